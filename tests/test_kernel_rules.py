"""Rules of the kernels' source that no run shows reliably: what a GPU does when one is broken depends on timing."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "metal-reax_b200" / "csrc"


def kernels():
    """(file, name, body without comments) of every __global__ definition."""
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\([^;{]*?\)\s*\{", text):
            depth, at = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
            yield path.name, m.group(1), text[m.end():at]


def test_cluster_meets_before_its_first_remote_access():
    """Another block's shared memory may be touched only once that block has started; the first cluster barrier is what
    says so."""
    remote = [(f, n, body) for f, n, body in kernels() if "map_shared_rank" in body]
    assert {n for _, n, _ in remote} >= {"k_cg_cluster", "k_cg_csr_static"}
    for f, n, body in remote:
        meet = body.find("cl.sync()")
        assert 0 <= meet < body.find("map_shared_rank"), "%s: %s reaches into another block before the cluster has met" % (f, n)


def test_warps_leave_after_a_list_overflow_together():
    """The overflow flags may be set while a kernel runs (by the other branch of the evaluation). A kernel whose lanes exchange
    values takes one decision a warp: a lane that left alone would be missed by the others."""
    seen = set()
    for f, n, body in kernels():
        if "lists_failed(d)" in body and re.search(r"_sync\(|warp_sum|lanes_sum", body.replace("__threadfence", "")):
            seen.add(n)
            assert not re.search(r"(?<!warp_)lists_failed\(d\)", body), "%s: %s leaves lane by lane" % (f, n)
    assert seen >= {"k_pairs", "k_nonbonded_half", "k_bonds", "k_bonded_atom", "k_hbond", "k_torsion"}
