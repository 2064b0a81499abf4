"""The charge solvers at the sizes where their work split changes: fewer rows than warps, ragged blocks of rows, empty and
long rows."""
import ctypes
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _random_csr(n, seed):
    """A symmetric positive definite (diag(eta) + H): rows of 0 to min(n - 1, 300) entries, |H| well below eta."""
    rng = np.random.default_rng(seed)
    H = np.zeros((n, n))
    for i in range(n):
        m = int(rng.integers(0, min(n, 150)))
        j = rng.choice(n, size=m, replace=False)
        H[i, j] = rng.uniform(0.0, 1.0, size=m)
    H = np.triu(H, 1)
    H += H.T
    eta = H.sum(1) + rng.uniform(1.0, 3.0, size=n)
    rows, cols = np.nonzero(H)
    rs = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    return H, rs, cols.astype(np.int32), H[rows, cols], eta, rng.uniform(-5.0, 5.0, size=n)


@pytest.mark.parametrize("n", [2, 3, 15, 16, 17, 31, 32, 33, 64, 65, 111, 112, 113, 127, 128, 129, 255, 256, 257, 1000, 1999])
def test_static_solve_sizes_match_dense(n):
    """Sizes on both sides of a row for every warp of a block (32), of the change from one block (112) to a cluster and of the
    cluster's halvings, against the dense FP64 solution. At tol 1e-12 the residual bounds the error: |x - x*| <= cond * tol *
    |x|; the matrices are diagonally dominant by a factor that keeps cond below 1e3, hence 1e-8 of the largest charge."""
    import torch
    import rxcuda
    H, rs, col, val, eta, chi = _random_csr(n, 100 + n)
    dev = torch.device("cuda", 0)
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    nnz = len(col)
    rs_d, col_d, val_d = up(rs), up(np.append(col, 0).astype(np.int32)), up(np.append(val, 0.0))
    eta_d, chi_d = up(eta), up(chi)
    s, t, q = (torch.zeros(n, dtype=torch.float64, device=dev) for _ in range(3))
    it, rel = torch.zeros(2, dtype=torch.int32, device=dev), torch.zeros(2, dtype=torch.float64, device=dev)
    lib = rxcuda.load()
    err = ctypes.create_string_buffer(256)
    rc = lib.rx_qeq_solve_static(n, rs_d.data_ptr(), col_d.data_ptr(), val_d.data_ptr(), eta_d.data_ptr(), chi_d.data_ptr(),
                                 s.data_ptr(), t.data_ptr(), q.data_ptr(), 1e-12, 500, it.data_ptr(), rel.data_ptr(),
                                 torch.cuda.current_stream(dev).cuda_stream, err, 256)
    assert rc == 0, err.value.decode()
    torch.cuda.synchronize(dev)
    A = np.diag(eta) + H
    s_ref, t_ref = np.linalg.solve(A, -chi), np.linalg.solve(A, -np.ones(n))
    q_ref = s_ref - s_ref.sum() / t_ref.sum() * t_ref
    assert nnz == rs[-1]
    assert rel.cpu().numpy().max() <= 1e-12 and it.cpu().numpy().max() < 500
    for got, ref in ((s, s_ref), (t, t_ref), (q, q_ref)):
        assert np.abs(got.cpu().numpy() - ref).max() <= 1e-8 * max(1.0, np.abs(ref).max())


def _jittered(n, seed, spacing=2.3):
    """n C/H/O atoms on random sites of a jittered cubic lattice (at least 20 A wide)."""
    rng = np.random.default_rng(seed)
    side = max(9, int(np.ceil(n ** (1.0 / 3.0))))
    sites = rng.permutation(side ** 3)[:n]
    x = np.stack([sites // side ** 2, sites // side % side, sites % side], axis=1) * spacing + rng.uniform(0.0, 0.7, size=(n, 3))
    return {"name": "jitter%d" % n, "origin": np.zeros(3), "box": np.eye(3) * side * spacing, "periodic": np.ones(3, dtype=np.int32),
            "x": x, "type": rng.integers(0, 3, size=n).astype(np.int32), "tag": np.arange(1, n + 1, dtype=np.int64)}


@pytest.fixture(scope="module")
def engine():
    import rxcuda
    from helpers import ffield_text
    e = rxcuda.Engine(0)
    e.set_forcefield(ffield_text())
    e.set_control()
    e.set_qeq(0.0, 10.0, 1e-12, 400)
    yield e
    e.close()


@pytest.fixture(scope="module")
def oracle():
    from helpers import ffield_text
    from oracle.oracle import COracle
    return COracle(ffield_text(), shell=15.0)


@pytest.mark.parametrize("n", [2, 7, 8, 9, 63, 128, 129, 1001, 4095, 4096, 4097, 6001])
def test_charge_solve_sizes_match_oracle(engine, oracle, n):
    """One system on both sides of a group of eight rows, of the blocks of a cluster (some own no row) and of the size where
    all SMs take the solve, against the oracle's charges: 1e-10 e at tol 1e-12, as for the other sizes."""
    s = _jittered(n, 7 + n)
    engine.set_systems([s])
    engine.qeq_reset()
    got = engine.qeq_solve()
    ref = oracle.qeq(s, tol=1e-12, imax=400)
    assert np.abs(got["q"] - ref["q"]).max() <= 1e-10
    # above 4096 atoms the solve restarts from an FP64 residual after every reduction by 1e6 (twice on the way to 1e-12),
    # and a restarted CG needs up to two more iterations to regain its directions
    assert np.abs(got["iters"][0] - ref["iters"]).max() <= (1 if n <= 4096 else 4)


def test_mixed_batch_solves_alone_and_together(engine, oracle):
    """Small systems beside larger ones: every small system's charges have the bits of its solve alone, whichever kernel and
    cluster size the batch takes; the large ones match the oracle."""
    ss = [_jittered(n, 90 + n) for n in (4500, 40, 700, 3, 4099, 2100)]
    engine.set_systems(ss)
    engine.qeq_reset()
    both = engine.qeq_solve()
    off = 0
    for k, s in enumerate(ss):
        n = len(s["type"])
        if n <= 4096:
            engine.set_systems([s])
            engine.qeq_reset()
            alone = engine.qeq_solve()
            assert np.array_equal(alone["q"], both["q"][off:off + n]), n
            assert np.array_equal(alone["iters"][0], both["iters"][k]), n
        ref = oracle.qeq(s, tol=1e-12, imax=400)
        assert np.abs(both["q"][off:off + n] - ref["q"]).max() <= 1e-10, n
        off += n


def test_more_systems_than_clusters(engine, oracle):
    """300 systems, more than the GPU holds clusters of even two blocks (148 SMs, one block each): every cluster takes several
    and uses its shared memory again for each. Each system's charges have the bits of its solve alone; every 25th matches the
    oracle to 1e-10 e at tol 1e-12, as for the other sizes."""
    sizes = np.random.default_rng(11).integers(5, 201, size=300)
    ss = [_jittered(int(n), 1000 + k) for k, n in enumerate(sizes)]
    engine.set_systems(ss)
    engine.qeq_reset()
    both = engine.qeq_solve()
    off = 0
    for k, s in enumerate(ss):
        n = len(s["type"])
        engine.set_systems([s])
        engine.qeq_reset()
        alone = engine.qeq_solve()
        assert np.array_equal(alone["q"], both["q"][off:off + n]), k
        assert np.array_equal(alone["iters"][0], both["iters"][k]), k
        if k % 25 == 0:
            ref = oracle.qeq(s, tol=1e-12, imax=400)
            assert np.abs(alone["q"] - ref["q"]).max() <= 1e-10, k
        off += n


# a stand-in for the runtime's occupancy query that refuses clusters of more than CLUSTERS_UP_TO blocks
FEW_CLUSTERS = r"""
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <stdlib.h>
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* f, const cudaLaunchConfig_t* c) {
  typedef cudaError_t (*Query)(int*, const void*, const cudaLaunchConfig_t*);
  for (unsigned k = 0; k < c->numAttrs; ++k)
    if (c->attrs[k].id == cudaLaunchAttributeClusterDimension && (int)c->attrs[k].val.clusterDim.x > atoi(getenv("CLUSTERS_UP_TO")))
      return cudaErrorInvalidClusterSize;
  return ((Query)dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), "cudaOccupancyMaxActiveClusters"))(n, f, c);
}
"""


def _with_few_clusters(tmp_path, limit, code):
    """Runs `code` (this module's names at hand) in a process whose runtime refuses clusters of more than `limit` blocks;
    returns the arrays that it puts into `out`."""
    src, lib, got = tmp_path / "few.c", tmp_path / "few.so", tmp_path / "out.npz"
    src.write_text("#define _GNU_SOURCE\n" + FEW_CLUSTERS)
    subprocess.run(["gcc", "-shared", "-fPIC", "-I/usr/local/cuda/include", str(src), "-o", str(lib), "-ldl"], check=True)
    here = Path(__file__).resolve().parent
    paths = [str(here), str(here.parent), str(here.parent / "metal-reax_b200")]
    code = "import sys; sys.path[:0] = %r\nfrom test_gpu_solvers import *\nfrom test_gpu_solvers import _jittered, _random_csr\n" \
           "out = {}\n%s\nnp.savez(%r, **out)\n" % (paths, code, str(got))
    run = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, LD_PRELOAD=str(lib), CLUSTERS_UP_TO=str(limit)),
                         capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]
    with np.load(got) as z:
        return {k: z[k] for k in z.files}


SOLVE_MIXED = """
import rxcuda
from helpers import ffield_text
e = rxcuda.Engine(0)
e.set_forcefield(ffield_text())
e.set_control()
e.set_qeq(0.0, 10.0, 1e-12, 400)
for name, sizes in (("batch", (4500, 40, 700, 3, 4096, 2100)), ("lone", (1001,))):
    e.set_systems([_jittered(n, 90 + n) for n in sizes])
    e.qeq_reset()
    got = e.qeq_solve()
    out[name + "_q"], out[name + "_iters"], out[name + "_rel"] = got["q"], got["iters"], got["rel"]
e.close()
"""


@pytest.mark.parametrize("limit", [0, 1, 8])
def test_charge_solve_where_clusters_are_refused(tmp_path, limit):
    """Where the GPU holds no cluster (or none of 16 blocks), the segmented solve takes the small systems too: the same
    charges, counts and residuals to the last bit."""
    few = _with_few_clusters(tmp_path, limit, SOLVE_MIXED)
    all_ = _with_few_clusters(tmp_path, 16, SOLVE_MIXED)
    for k in all_:
        assert np.array_equal(few[k], all_[k]), k


SOLVE_STATIC = """
import torch
import rxcuda
lib, err = rxcuda.load(), ctypes.create_string_buffer(256)
H, rs, col, val, eta, chi = _random_csr(300, 5)
up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
rs, col, val, eta, chi = up(rs), up(col), up(val), up(eta), up(chi)
s, t, q = (torch.zeros(300, dtype=torch.float64, device="cuda") for _ in range(3))
it, rel = torch.zeros(2, dtype=torch.int32, device="cuda"), torch.zeros(2, dtype=torch.float64, device="cuda")
rc = lib.rx_qeq_solve_static(300, *(a.data_ptr() for a in (rs, col, val, eta, chi, s, t, q)), 1e-12, 500, it.data_ptr(),
                             rel.data_ptr(), torch.cuda.current_stream().cuda_stream, err, 256)
assert rc == 0, err.value
torch.cuda.synchronize()
out["q"], out["rel"] = q.cpu().numpy(), rel.cpu().numpy()
"""


@pytest.mark.parametrize("limit", [0, 2, 8])
def test_static_solve_where_clusters_are_refused(tmp_path, limit):
    """Where the runtime refuses 16 blocks the solve takes the largest cluster that there is, down to one block. The blocks' sums
    are added in another order, hence the bound of the test above: 1e-8 of the largest charge at tol 1e-12."""
    few = _with_few_clusters(tmp_path, limit, SOLVE_STATIC)
    H, _, _, _, eta, chi = _random_csr(300, 5)
    A = np.diag(eta) + H
    s_ref, t_ref = np.linalg.solve(A, -chi), np.linalg.solve(A, -np.ones(300))
    q_ref = s_ref - s_ref.sum() / t_ref.sum() * t_ref
    assert few["rel"].max() <= 1e-12
    assert np.abs(few["q"] - q_ref).max() <= 1e-8 * max(1.0, np.abs(q_ref).max())


def test_static_solve_of_a_small_system_meets_in_one_block():
    """Up to 112 atoms the solve is one block's. Twenty iterations on 24 rows took 0.76 times as long as on 129 rows on a cluster
    while that block met as a cluster of one and divided twice. At most 0.7 times."""
    import torch
    import rxcuda
    lib, err = rxcuda.load(), ctypes.create_string_buffer(256)
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    took = []
    for n in (24, 129):
        rng = np.random.default_rng(n)   # a full matrix of condition 1e4: twenty iterations do not exhaust it
        Q = np.linalg.qr(rng.normal(size=(n, n)))[0]
        A = (Q * np.logspace(0.0, 4.0, n)) @ Q.T
        rs = np.arange(0, n * (n - 1) + 1, n - 1, dtype=np.int32)
        rows, col = np.nonzero(~np.eye(n, dtype=bool))
        col, val, eta, chi = col.astype(np.int32), A[rows, col], np.diag(A).copy(), rng.uniform(-5.0, 5.0, size=n)
        a = [up(x) for x in (rs, col, val, eta, chi)]
        guess = torch.zeros((3, 20, n), dtype=torch.float64, device="cuda")   # s, t and q of every solve
        it, rel = torch.zeros(2, dtype=torch.int32, device="cuda"), torch.zeros(2, dtype=torch.float64, device="cuda")
        best = float("inf")
        for _ in range(30):
            guess.zero_()
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            ev[0].record()
            for k in range(20):   # twenty iterations each
                rc = lib.rx_qeq_solve_static(n, *(x.data_ptr() for x in a), *(guess[c, k].data_ptr() for c in range(3)), 1e-300, 21,
                                             it.data_ptr(), rel.data_ptr(), torch.cuda.current_stream().cuda_stream, err, 256)
                assert rc == 0, err.value.decode()
            ev[1].record()
            torch.cuda.synchronize()
            best = min(best, ev[0].elapsed_time(ev[1]))
        assert it.tolist() == [21, 21]
        took.append(best)
    assert took[0] <= 0.7 * took[1], took


TIME_SOLVES = """
import time
import rxcuda
import systems
from helpers import ffield_text
e = rxcuda.Engine(0)
e.set_forcefield(ffield_text())
e.set_control()
e.set_qeq(0.0, 10.0, 1e-6, 200)
dense = systems.serving_request(0, seed=1, nmin=2000, nmax=2000)[0]
for name, ss in (("dense", [dense]), ("mixed", [systems.water_box(m) for m in (12, 3, 6, 5, 12, 9)])):
    e.set_systems(ss)
    e.qeq_solve()
    took = []
    for _ in range(9):
        e.qeq_reset()
        t = time.perf_counter()
        e.qeq_solve()
        took.append(time.perf_counter() - t)
    out[name] = min(took)
e.close()
"""


def test_charge_solve_takes_the_quicker_kernel(tmp_path):
    """A lone system of 2000 atoms in rows of 1000 entries, and small systems beside larger ones (water of 81 to 5184 atoms): the
    clusters take 1.3 times as long there as the segmented solve, so they are not taken. At most 1.2 times the solve
    without clusters, for the noise of the machine."""
    rule, without = (_with_few_clusters(tmp_path, limit, TIME_SOLVES) for limit in (16, 0))
    for k in rule:
        assert rule[k] <= 1.2 * without[k], (k, float(rule[k]), float(without[k]))


@pytest.mark.parametrize("n", [2, 33, 295, 296, 297, 600, 1999])
def test_single_system_solve_of_small_systems(engine, oracle, n):
    """The solve on all SMs below its usual sizes: blocks of one or two rows, some without rows, and both sides of 296 atoms
    (two rows a block). As for the other sizes: 1e-10 e at tol 1e-12."""
    s = _jittered(n, 300 + n)
    engine.set_tuning("lone_grid_min", 0)
    engine.set_systems([s])
    engine.qeq_reset()
    got = engine.qeq_solve()
    engine.set_tuning("lone_grid_min", 4096)
    ref = oracle.qeq(s, tol=1e-12, imax=400)
    assert np.abs(got["q"] - ref["q"]).max() <= 1e-10
    assert got["rel"].max() <= 1e-12


def test_charge_solve_with_vectors_in_global_memory(engine):
    """A system of more rows per block than shared memory holds (its vectors stay in global memory), against the segmented
    FP64 solve of the same system. Both stop at a relative residual of 1e-10; diag(eta) + H has a condition number of a few
    hundred, hence 1e-7 e."""
    s = _jittered(200000, 3)
    engine.set_qeq(0.0, 10.0, 1e-10, 400)
    engine.set_systems([s])
    engine.qeq_reset()
    whole = engine.qeq_solve()
    engine.set_tuning("lone_grid_min", 1 << 30)
    engine.qeq_reset()
    rows = engine.qeq_solve()
    engine.set_tuning("lone_grid_min", 4096)
    engine.set_qeq(0.0, 10.0, 1e-12, 400)
    assert whole["rel"].max() <= 1e-10 and rows["rel"].max() <= 1e-10
    assert np.abs(whole["q"] - rows["q"]).max() <= 1e-7


def test_bonded_time_grows_with_the_bonds(engine):
    """Carbon of 14 and of 18 bonds on its most bonded atom (two and three bonds to a lane) has 2.3 times the angles; the bonded
    terms take 1.5 times the time (they took 9 times when the lanes of a warp went through the exchange of the angles
    apart). At most 4 times, so that other users' work on the machine does not matter."""
    import systems
    took, most = [], []
    for density in (2.0, 3.0):
        engine.set_systems([systems.random_carbon(n=4000, density=density, seed=5)])
        engine.set_qeq(0.0, 10.0, 1e-6, 200)
        engine.compute(qeq=True)
        most.append(int(np.diff(engine.bonds()["start"]).max()))
        engine.set_timing(True)
        engine.compute(qeq=True)
        runs = []
        for _ in range(5):
            before = engine.phase_times()["bonded_terms"]
            engine.compute(qeq=True)
            runs.append(engine.phase_times()["bonded_terms"] - before)
        engine.set_timing(False)
        took.append(min(runs))
    engine.set_qeq(0.0, 10.0, 1e-12, 400)
    assert most[0] <= 16 < most[1]
    assert took[1] <= 4.0 * took[0], took


@pytest.mark.parametrize("n,density", [(2, 0.02), (30, 1.0), (61, 3.0), (200, 2.0)])
def test_bonded_terms_at_many_bonds_per_atom(engine, oracle, n, density):
    """Angles and torsions shared by the lanes of an atom or central bond: from no bond to more bonds than lanes (dense random
    carbon), against the oracle. FP64 terms, 1e-7 relative as in the parity tests; every decision identical."""
    import systems
    s = systems.random_carbon(n=n, density=density, seed=5 + n, dmin=0.95)
    ref = oracle.single_point(s, np.zeros(n))
    engine.set_systems([s])
    engine.set_charges(np.zeros(n))
    out = engine.compute(census=True)
    terms = [0, 1, 2, 3, 4, 5, 6, 8, 9]
    assert (np.abs(out["e"][0][terms] - ref["e"][terms]) / np.maximum(1.0, np.abs(ref["e"][terms]))).max() <= 1e-7
    assert np.array_equal(out["census"], ref["census"])
    scale = max(1.0, np.abs(ref["grad"]).max())
    assert np.abs(out["grad"] - ref["grad"]).max() <= 1e-6 * scale
    if density == 3.0:
        assert ref["census"][0].max() > 8
