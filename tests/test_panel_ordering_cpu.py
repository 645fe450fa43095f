"""Memory ordering inside the panel's thread-block cluster, read from the source.

A CTA's tile is written by ordinary shared-memory stores. Another CTA of the
cluster may read it only behind a cluster barrier (release and acquire at
cluster scope): the arrival of a pivot record orders the record alone, and a
CTA barrier only that CTA. The waits for those records acquire at cluster
scope too, since other CTAs complete them."""

import pathlib
import re

SRC = (pathlib.Path(__file__).resolve().parent.parent / "algebra_linear_b200" / "csrc" / "dense_kernels.cuh").read_text()
CODE = re.sub(r"//[^\n]*", "", SRC)


def test_reads_of_another_ctas_tile_follow_a_cluster_barrier():
    body = CODE[CODE.index("panel_reg_kernel(PanelArgs<T> p)"):]
    body = body[:body.index("laswp_outside_kernel")]
    reads = [m.start() for m in re.finditer(r"\bld_cluster\(", body)]
    assert reads
    for at in reads:
        sync = list(re.finditer(r"cl\.sync\(\)|mbar_wait\(", body[:at]))[-1]
        assert sync.group() == "cl.sync()"


def test_record_waits_acquire_at_cluster_scope():
    waits = re.findall(r"mbarrier\.try_wait[\w.:]*", CODE)
    assert waits
    for w in waits:
        assert ".acquire.cluster" in w
