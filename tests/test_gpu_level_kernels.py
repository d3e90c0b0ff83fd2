"""GPU tests of single level kernels at the sizes where their launch shapes
change, against the CPU oracle (the level parity over all degrees is in
test_gpu_parity.py)."""
import numpy as np
import pytest
import torch

import gputensorproductsmoother_b200 as tps

pytestmark = pytest.mark.gpu

# FP64: sums of at most 4 (2k+1) terms per stage, 6 stages deep; FP32 the same in
# 24 bits: the level parity's tolerances
TOL = {torch.float64: 1e-12, torch.float32: 2e-5}


def relerr(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


def sweep_matches(oracle, dim, k, n, dtype, seed=5, relaxation=1.0):
    npdt = np.float64 if dtype == torch.float64 else np.float32
    P = tps.PoissonProblem(dim, k, n, relaxation=relaxation)
    rng = np.random.default_rng(seed)
    x0, b = rng.uniform(-1, 1, P.n_dofs()).astype(npdt), rng.uniform(-1, 1, P.n_dofs()).astype(npdt)
    for zero, reverse in ((False, True), (True, False)):
        ref = oracle.smoother_step(dim, k, n, x0, b, omega=relaxation, zero_init=zero, reverse=reverse)
        x = torch.tensor(x0, device="cuda")
        S = tps.PatchSmoother(P)
        (S.vmult if zero else S.step)(x, torch.tensor(b, device="cuda"), reverse=reverse)
        torch.cuda.synchronize()
        assert relerr(x.cpu().numpy(), ref) < TOL[dtype], (zero, reverse)
    P.close()


# one warp per CTA, four warps per CTA, and more patches than the resident
# warps hold (Q1: 32 patches a warp); every colour lattice but the first is uneven
@pytest.mark.parametrize("k,n", [(1, 3), (1, 72), (1, 640), (1, 1536), (2, 5), (2, 160), (3, 224), (5, 3), (5, 96),
                                 (5, 288), (6, 72), (7, 5), (7, 128)])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_smoother_2d_launch_shapes(cuda, oracle, k, n, dtype):
    sweep_matches(oracle, 2, k, n, dtype, relaxation=0.9)


# A patch solve in FP32 rounds each of its stages and its result once, and its
# tables once: independent errors of at most 2^-24 each, of which the last ones
# count fully and the stages' average out.  Against the FP64 sweep they stay below
# three units in the 2-norm; one factor common to all entries (the rounding of a
# mode's length, left in) takes more than that by itself at degree 1.
@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 6, 7])
def test_smoother_2d_fp32_rounding(cuda, k):
    for n in (12, 48, 96):
        P = tps.PoissonProblem(2, k, n)
        S = tps.PatchSmoother(P)
        gen = torch.Generator(device="cuda").manual_seed(100 * k + n)
        x, b = (torch.rand(P.n_dofs(), device="cuda", generator=gen) * 2 - 1 for _ in range(2))
        x64 = x.double()
        S.step(x, b)
        S.step(x64, b.double())
        torch.cuda.synchronize()
        assert ((x.double() - x64).norm() / x64.norm()).item() < 3 * 2.0 ** -24
        P.close()


# the sweep on row-padded copies of the caller's vectors: one and several
# levels sharing the copies, the smallest level that takes them, rows that
# need 0..3 entries of padding
@pytest.mark.parametrize("k,n", [(3, 3), (3, 8), (4, 4), (5, 6), (6, 4), (7, 3), (2, 32), (1, 64)])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_smoother_3d_caller_vectors(cuda, oracle, k, n, dtype):
    if (n * k - 1) ** 3 > 4096 and n % 2:
        n += 1
    sweep_matches(oracle, 3, k, n, dtype, relaxation=0.9)


def test_smoother_3d_copies_serve_every_level_and_stream(cuda, oracle):
    """One handle: sweeps of two levels in turn on two streams, without a host
    wait between them, give each level's sweep; the memory-starved handle
    sweeps in place with the same result."""
    k, n = 4, 8
    P = tps.PoissonProblem(3, k, n)
    rng = np.random.default_rng(9)
    xs, bs, ref = {}, {}, {}
    for lv, nc in ((2, n), (1, n // 2)):
        x0, b = (rng.uniform(-1, 1, P.n_dofs(lv)) for _ in range(2))
        xs[lv], bs[lv] = torch.tensor(x0, device="cuda"), torch.tensor(b, device="cuda")
        ref[lv] = oracle.smoother_step(3, k, nc, oracle.smoother_step(3, k, nc, x0, b), b)
    start = {lv: x.clone() for lv, x in xs.items()}
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for _ in range(2):
        for lv, st in zip(xs, streams):
            with torch.cuda.stream(st):
                tps.PatchSmoother(P, lv).step(xs[lv], bs[lv])
    torch.cuda.synchronize()
    for lv in xs:
        assert relerr(xs[lv].cpu().numpy(), ref[lv]) < 1e-12
    from gputensorproductsmoother_b200 import _lib as L
    Q = tps.PoissonProblem(3, k, n)
    y = start[2].clone()
    tps.PatchSmoother(Q, 0).step(Q.new_vector(0), Q.new_vector(0))  # the error flag exists
    L.lib().tps_inject_alloc_failure(1)
    tps.PatchSmoother(Q, 2).step(y, bs[2])
    L.lib().tps_inject_alloc_failure(0)
    z = start[2].clone()
    tps.PatchSmoother(Q, 2).step(z, bs[2])
    torch.cuda.synchronize()
    assert torch.equal(y, z)
    P.close()
    Q.close()


def test_smoother_3d_copies_with_one_stream_handle(cuda):
    """Sweeps of two vector pairs on streams that share one handle: the
    per-thread default streams (handle 2) of two threads in turn, without a
    wait between them."""
    import threading
    from gputensorproductsmoother_b200 import _lib as L
    P = tps.PoissonProblem(3, 4, 16)
    gen = torch.Generator(device="cuda").manual_seed(4)
    x0, b = ([torch.rand(P.n_dofs(), device="cuda", dtype=torch.float64, generator=gen) for _ in range(2)]
             for _ in range(2))
    ref = [v.clone() for v in x0]
    for v, w in zip(ref, b):
        for _ in range(6):
            tps.PatchSmoother(P).step(v, w)
    x = [v.clone() for v in x0]
    torch.cuda.synchronize()

    def sweeps(i):
        for _ in range(3):
            L.check(L.lib().tps_smoother_step(P.handle, P.n_levels - 1, L.TPS_F64, x[i].data_ptr(), b[i].data_ptr(),
                                              0, 0, 2), P.handle)

    # the streams live on while their threads wait
    go, done = [threading.Event() for _ in range(5)], [threading.Event() for _ in range(4)]

    def worker(i):
        for r in (i, i + 2):
            go[r].wait()
            sweeps(i)
            done[r].set()
        go[4].wait()

    ts = [threading.Thread(target=worker, args=(i,)) for i in range(2)]
    for t in ts:
        t.start()
    for r in range(4):
        go[r].set()
        assert done[r].wait(60)
    torch.cuda.synchronize()
    go[4].set()
    for t in ts:
        t.join()
    for v, w in zip(x, ref):
        assert torch.equal(v, w)
    P.close()


def test_copies_are_given_back_where_memory_runs_out(cuda):
    """Sweeps on copies take no memory from the handle's other calls: an
    allocation that fails while the copies are held succeeds without them, and
    sweeps go on with new ones."""
    from gputensorproductsmoother_b200 import _lib as L
    P, Q = tps.PoissonProblem(3, 4, 8), tps.PoissonProblem(3, 4, 8)
    gen = torch.Generator(device="cuda").manual_seed(5)
    b = torch.rand(P.n_dofs(), device="cuda", dtype=torch.float64, generator=gen)
    x, y, z, w = torch.zeros_like(b), torch.zeros_like(b), torch.empty_like(b), torch.empty_like(b)
    tps.PatchSmoother(P).step(x, b)
    tps.PatchSmoother(Q).step(y, b)
    tps.MultigridSolvers(Q).vmult(w, b, precision="fp64")
    L.lib().tps_inject_alloc_failure(3)
    try:
        tps.MultigridSolvers(P).vmult(z, b, precision="fp64")
    finally:
        L.lib().tps_inject_alloc_failure(0)
    tps.PatchSmoother(P).step(x, b)
    tps.PatchSmoother(Q).step(y, b)
    torch.cuda.synchronize()
    assert torch.equal(z, w) and torch.equal(x, y)
    # nothing left to give back: the failure is reported
    R = tps.PoissonProblem(3, 4, 8)
    L.lib().tps_inject_alloc_failure(3)
    with pytest.raises(tps.TpsError):
        tps.MultigridSolvers(R).vmult(z, b, precision="fp64")
    L.lib().tps_inject_alloc_failure(0)
    for p in (P, Q, R):
        p.close()


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_captured_sweeps_share_nothing(cuda, dtype):
    """Sweeps captured after the handle has its copies: two branches of one
    graph, replayed while the handle sweeps other vectors on another stream."""
    P = tps.PoissonProblem(3, 4, 8)
    S = tps.PatchSmoother(P)
    gen = torch.Generator(device="cuda").manual_seed(3)
    x0, b = ([torch.rand(P.n_dofs(), device="cuda", dtype=dtype, generator=gen) for _ in range(3)] for _ in range(2))
    ref = [v.clone() for v in x0]
    for v, w in zip(ref, b):  # the copies exist from here on
        for _ in range(4):
            S.step(v, w)
    x = [v.clone() for v in x0]
    fork, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        fork.wait_stream(torch.cuda.current_stream())
        for _ in range(2):
            S.step(x[0], b[0])
            with torch.cuda.stream(fork):
                S.step(x[1], b[1])
        torch.cuda.current_stream().wait_stream(fork)
    for _ in range(2):
        g.replay()
        with torch.cuda.stream(other):
            S.step(x[2], b[2])
            S.step(x[2], b[2])
    torch.cuda.synchronize()
    for v, w in zip(x, ref):
        assert torch.equal(v, w)
    P.close()


def test_captured_solves_serve_any_vectors(cuda):
    """The captured CG iteration and the batch's graph are built once and read
    the caller's vectors from device memory: repeated solves with new right-hand
    sides, new and reused solution vectors (in place of b too) and on several
    streams match handles that never solved before."""
    def rhs(N1, seed):
        v = np.random.default_rng(seed).uniform(-1, 1, (N1,) * 3)
        v[[0, -1]] = v[:, [0, -1]] = v[:, :, [0, -1]] = 0.0
        return torch.tensor(v.ravel(), device="cuda")

    k, n = 3, 8
    N1 = n * k + 1
    P = tps.PoissonProblem(3, k, n)
    MG = tps.MultigridSolvers(P)
    systems = [(3, k, n), (3, 2, 6), (2, 3, 16)]
    B = tps.BatchSolver(systems)
    keep = []
    for i in range(4):
        st = torch.cuda.Stream() if i % 2 else torch.cuda.default_stream()
        with torch.cuda.stream(st):
            b = rhs(N1, 60 + i)
            x, rep = MG.solve_cg(b, rel_tol=1e-10)
            Q = tps.PoissonProblem(3, k, n)
            ref, rep_ref = tps.MultigridSolvers(Q).solve_cg(b.clone(), rel_tol=1e-10)
            assert torch.equal(x, ref) and rep.history == rep_ref.history
            keep.append((x, ref.clone()))
            bs = [b, rhs(13, 70 + i), torch.tensor(np.random.default_rng(80 + i).uniform(-1, 1, 49 ** 2), device="cuda")]
            xs = [torch.zeros_like(v) for v in bs]
            if i == 3:  # the first system's solution takes the place of its right-hand side
                xs[0] = bs[0]
            got, reps = B.solve(bs, x=xs)
            C = tps.BatchSolver(systems)
            if i < 3:
                want, wreps = C.solve(bs)
                for g, w, r, wr in zip(got, want, reps, wreps):
                    # autotuned tile depths may differ between two handles: rounding of p.q
                    assert r.iterations == wr.iterations
                    assert (g - w).abs().max().item() <= 1e-12 * w.abs().max().item()
            else:
                assert all(r.converged for r in reps)
            C.close()
            Q.close()
    for x, ref in keep:
        assert torch.equal(x, ref)
    P.close()
    B.close()


# one and several tiles per direction with remainders, one and several layer
# chunks; every entry of b is written (it starts as NaN), Dirichlet rows as zero
@pytest.mark.parametrize("dim,k,n", [(3, 1, 40), (3, 1, 72), (3, 2, 20), (3, 3, 12), (3, 4, 12), (3, 5, 8), (3, 6, 8),
                                     (3, 7, 8), (2, 1, 70), (2, 2, 2), (2, 3, 36), (2, 4, 20), (2, 6, 24)])
def test_assemble_tiles(cuda, oracle, dim, k, n):
    from gputensorproductsmoother_b200 import _lib as L
    P = tps.PoissonProblem(dim, k, n)
    fq = np.random.default_rng(31 * dim + k).uniform(-1, 1, (n ** dim, (k + 1) ** dim))
    b = torch.full((P.n_dofs(),), float("nan"), dtype=torch.float64, device="cuda")
    f = torch.tensor(fq, device="cuda")
    L.check(L.lib().tps_assemble_rhs(P.handle, P.n_levels - 1, f.data_ptr(), b.data_ptr(), None), P.handle)
    torch.cuda.synchronize()
    ref = oracle.assemble_rhs(dim, k, n, fq)
    got = b.cpu().numpy()
    assert np.isfinite(got).all()
    # sums of 2^dim (k+1)^dim products in another order
    assert relerr(got, ref) < 1e-13
    v = got.reshape((n * k + 1,) * dim)
    for ax in range(dim):
        assert not np.take(v, [0, -1], axis=ax).any()
    P.close()


# one level: the V-cycle is the dense inverse alone.  Sizes below, at and just
# past the inversion's 32-column blocks and 64-entry tiles, up to its largest
# ones, and the last on the host and the first on the device; cond(A) is at most 4 (2 n k)^2, so that a backward-stable inverse
# leaves a residual of a few cond * 2^-53
@pytest.mark.parametrize("dim,k,n", [(2, 1, 2), (2, 1, 3), (2, 2, 3), (2, 1, 7), (2, 1, 9), (2, 4, 2), (3, 1, 5),
                                     (2, 1, 33), (2, 1, 34), (3, 4, 3), (3, 1, 16), (2, 2, 32), (2, 1, 11), (2, 1, 12),
                                     (2, 3, 5), (3, 1, 7)])
@pytest.mark.parametrize("varying", [False, True])
def test_dense_coarse_inverse(cuda, dim, k, n, varying):
    kap = None
    if varying:
        kap = np.exp(np.random.default_rng(3).normal(0.0, 0.5, n ** dim))
    P = tps.PoissonProblem(dim, k, n, n_coarse=n, kappa=kap)
    b = np.random.default_rng(4).uniform(-1, 1, (n * k + 1,) * dim)
    for ax in range(dim):
        np.moveaxis(b, ax, 0)[[0, -1]] = 0.0
    b = torch.tensor(b.ravel(), device="cuda")
    for update in range(2 if varying else 1):
        if update:  # a new coefficient replaces the inverse
            P.set_kappa(kap[::-1].copy())
        for precision, tol in (("fp64", 1e-15), ("fp32", 4e-7)):
            z, r = P.new_vector(), P.new_vector()
            tps.MultigridSolvers(P).vmult(z, b, precision=precision)
            tps.LaplaceOperator(P).vmult(r, z)
            torch.cuda.synchronize()
            e = ((r - b).norm() / b.norm()).item()
            assert e < tol * 4 * (2 * n * k) ** 2, (update, precision, e)
    P.close()


def test_coefficients_at_the_limit_of_definiteness(cuda):
    """Coefficients over 1e30: where the device's elimination meets a pivot that
    rounding made negative, the host's factorisation decides, as it does for
    small coarse levels."""
    for seed in range(5):
        kap = np.exp(np.random.default_rng(seed).normal(0.0, 15.0, (2, 17 ** 2)))
        P = tps.PoissonProblem(2, 1, 17, n_coarse=17, kappa=kap[0])
        b = torch.rand(P.n_dofs(), dtype=torch.float64, device="cuda")
        z = P.new_vector()
        tps.MultigridSolvers(P).vmult(z, b, precision="fp64")
        P.set_kappa(np.ones(17 ** 2))  # a definite one afterwards is that of a new handle
        Q = tps.PoissonProblem(2, 1, 17, n_coarse=17, kappa=np.ones(17 ** 2))
        w = P.new_vector()
        tps.MultigridSolvers(P).vmult(z, b, precision="fp64")
        tps.MultigridSolvers(Q).vmult(w, b, precision="fp64")
        torch.cuda.synchronize()
        assert torch.equal(z, w)
        P.close()
        Q.close()


def test_kappa_update_needs_no_memory(cuda):
    """A new coefficient is taken up whole where device memory has run out, also
    with a large dense coarse level (2601 rows, 54 MB a matrix)."""
    from gputensorproductsmoother_b200 import _lib as L
    kap = np.exp(np.random.default_rng(3).normal(0.0, 0.5, (2, 26 ** 2)))
    P, Q = (tps.PoissonProblem(2, 2, 26, n_coarse=26, kappa=kap[i]) for i in range(2))
    b = torch.rand(P.n_dofs(), dtype=torch.float64, device="cuda")
    got, want = P.new_vector(), P.new_vector()
    tps.MultigridSolvers(P).vmult(got, b, precision="fp64")
    L.lib().tps_inject_alloc_failure(1)
    try:
        P.set_kappa(kap[1])
    finally:
        L.lib().tps_inject_alloc_failure(0)
    for f in (lambda p, v: tps.MultigridSolvers(p).vmult(v, b, precision="fp64"),
              lambda p, v: tps.LaplaceOperator(p).vmult(v, b)):
        f(P, got)
        f(Q, want)
        torch.cuda.synchronize()
        assert torch.equal(got, want)
    P.close()
    Q.close()


def test_constant_coarse_level_holds_no_workspace(cuda):
    """A constant coefficient's coarse operator is inverted once: the handle
    keeps its inverse (1331 rows, 14.2 MB), not what the inversion worked in."""
    make = lambda: tps.PoissonProblem(3, 4, 3, n_coarse=3)
    make().close()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    Ps = [make() for _ in range(8)]
    torch.cuda.synchronize()
    held = (free0 - torch.cuda.mem_get_info()[0]) / len(Ps)
    # one matrix, in pieces of at most 2 MB of a shared pool, and small buffers
    assert held < 1.5 * 8 * 1331 ** 2, held
    # FP32 V-cycles need the rounded inverse alone; a later FP64 one is that of
    # a handle that had no FP32 ones
    b = torch.rand(Ps[0].n_dofs(), dtype=torch.float64, device="cuda")
    for P in Ps:
        tps.MultigridSolvers(P).vmult(P.new_vector(), b, precision="fp32")
    torch.cuda.synchronize()
    held = (free0 - torch.cuda.mem_get_info()[0]) / len(Ps)
    assert held < 0.8 * 8 * 1331 ** 2, held
    Q = make()
    z = [P.new_vector() for P in (Q, Ps[0], Ps[0])]
    for P, v, precision in ((Q, z[0], "fp64"), (Ps[0], z[1], "fp64"), (Ps[0], z[2], "fp32")):
        tps.MultigridSolvers(P).vmult(v, b, precision=precision)
    tps.MultigridSolvers(Q).vmult(Q.new_vector(), b, precision="fp32")
    w = [Q.new_vector() for _ in range(2)]
    for v, precision in zip(w, ("fp64", "fp32")):
        tps.MultigridSolvers(Q).vmult(v, b, precision=precision)
    torch.cuda.synchronize()
    assert torch.equal(z[0], z[1]) and torch.equal(w[0], z[0]) and torch.equal(w[1], z[2])
    for P in Ps + [Q]:
        P.close()


# the varying-coefficient operator: tiles with remainders, several layer chunks,
# every degree (the smoother's are in test_gpu_kappa.py); padded rows are covered
# by the V-cycles elsewhere
@pytest.mark.parametrize("k,n", [(1, 9), (1, 40), (2, 3), (2, 24), (3, 5), (3, 12), (4, 2), (4, 12), (5, 3), (5, 8), (6, 2),
                                 (6, 8), (7, 2), (7, 4)])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_kappa_operator_tiles(cuda, oracle, k, n, dtype):
    if (tps.split_cells(n)[0] * k - 1) ** 3 > 4096:
        n = 4
    npdt = np.float64 if dtype == torch.float64 else np.float32
    rng = np.random.default_rng(17)
    kap = np.exp(rng.normal(0.0, 0.5, n ** 3))
    P = tps.PoissonProblem(3, k, n, kappa=kap)
    x = rng.uniform(-1, 1, P.n_dofs()).astype(npdt)
    y = torch.full((P.n_dofs(),), float("nan"), dtype=dtype, device="cuda")
    tps.LaplaceOperator(P).vmult(y, torch.tensor(x, device="cuda"))
    torch.cuda.synchronize()
    assert relerr(y.cpu().numpy(), oracle.laplace_vmult(3, k, n, x, kappa=kap)) < TOL[dtype]
    P.close()


@pytest.mark.parametrize("dim,k,n", [(2, 3, 16), (3, 3, 12), (3, 4, 8)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_vcycle_after_calls_that_leave_its_vectors_dirty(cuda, dim, k, n, precision):
    """A V-cycle starts from zero whatever ran before it on the handle's work
    vectors: timed sweeps, tensor-core sweeps on caller vectors with nonzero
    boundary entries, solves, FMG, other V-cycles."""
    P, Q = tps.PoissonProblem(dim, k, n), tps.PoissonProblem(dim, k, n)
    b = torch.tensor(np.random.default_rng(2).uniform(-1, 1, P.n_dofs()), device="cuda")
    ref, out = P.new_vector(), P.new_vector()
    tps.MultigridSolvers(Q).vmult(ref, b, precision=precision)
    MG = tps.MultigridSolvers(P)
    v = torch.rand(P.n_dofs(), device="cuda") + 1.0
    dirty = [lambda: [P.time_smoother(lv, precision, 2) for lv in range(P.n_levels)],
             lambda: MG.solve_cg(b, precision=precision),
             lambda: MG.solve_fmg([torch.ones_like(P.new_vector(lv)) for lv in range(P.n_levels)], precision=precision),
             lambda: MG.vmult(out, 2.0 * b, precision=precision, symmetric=True)]
    if dim == 3:
        dirty.append(lambda: tps.PatchSmoother(P, tensor_cores=True).step(v, v.clone()))
    for f in dirty:
        f()
        MG.vmult(out, b, precision=precision)
        torch.cuda.synchronize()
        assert torch.equal(out, ref)
    P.close()
    Q.close()


# levels whose sweep is one launch, and the first ones past its rule, at every
# degree: the oracle's sweep, and bit-identical to the per-colour kernels (an
# explicitly chosen variant in 3D)
@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_single_launch_sweeps(cuda, oracle, dim, k, dtype):
    for n in (3, 4, 5, 6, 8, 9, 10, 16):
        if (tps.split_cells(n)[0] * k - 1) ** dim > 1400 or (dim == 3 and n * k > 36):
            continue
        sweep_matches(oracle, dim, k, n, dtype, seed=n, relaxation=0.95)
        if dim == 3:
            P = tps.PoissonProblem(dim, k, n)
            S = tps.PatchSmoother(P)
            b = torch.rand(P.n_dofs(), device="cuda", dtype=dtype)
            x, y = torch.rand_like(b), None
            y = x.clone()
            S.step(x, b)
            prec = "fp64" if dtype == torch.float64 else "fp32"
            P.set_smoother_variant(0, prec)
            S.step(y, b)
            torch.cuda.synchronize()
            assert torch.equal(x, y)
            P.close()


# one iteration, restarts after a full basis (28 vectors), vectors shorter and
# longer than the reductions' grid; the coefficients come from the device.  The
# residual that the recurrence reports is |V(b - A x)| / |V b| in exact
# arithmetic; rounding separates the two by about 2^-53 |V b| times the
# operator's condition number (at most 1e6 here), so they are compared above
# 1e-9 and both have to be below it otherwise.
@pytest.mark.parametrize("dim,k,n,max_iter,reduce", [(2, 1, 4, 20, 1e-9), (2, 2, 256, 2, 1e-30), (2, 2, 256, 20, 1e-9),
                                                      (3, 2, 16, 40, 1e-30), (3, 3, 24, 1, 1e-30), (3, 3, 24, 3, 1e-30)])
def test_gmres_residual_is_the_reported_one(cuda, dim, k, n, max_iter, reduce):
    P = tps.PoissonProblem(dim, k, n)
    MG = tps.MultigridSolvers(P)
    b = np.random.default_rng(8).uniform(-1, 1, (n * k + 1,) * dim)
    for ax in range(dim):
        np.moveaxis(b, ax, 0)[[0, -1]] = 0.0
    b = torch.tensor(b.ravel(), device="cuda")
    x, rep = MG.solve_gmres(b, precision="fp64", max_iter=max_iter, reduce=reduce)
    r, z, z0 = P.new_vector(), P.new_vector(), P.new_vector()
    tps.LaplaceOperator(P).vmult(r, x)
    MG.vmult(z, b - r, precision="fp64")
    MG.vmult(z0, b, precision="fp64")
    torch.cuda.synchronize()
    true = (z.norm() / z0.norm()).item()
    # (an absolute tolerance of 1e-16 can end the long run early)
    assert 1 <= rep.iterations <= max_iter and (rep.converged or reduce < 1e-20)
    if rep.final_residual > 1e-9:
        assert abs(true - rep.final_residual) < 1e-3 * rep.final_residual, (true, rep.final_residual)
    else:
        assert true < 1e-9, (true, rep.final_residual)
    P.close()


# tiles with remainders in x and y at every degree; adds to what is there, on
# interior fine nodes only
@pytest.mark.parametrize("k,n", [(1, 6), (1, 40), (2, 20), (3, 12), (4, 12), (5, 8), (6, 8), (7, 8)])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_prolongation_tiles(cuda, oracle, k, n, dtype):
    P = tps.PoissonProblem(3, k, n)
    npdt = np.float64 if dtype == torch.float64 else np.float32
    rng = np.random.default_rng(23)
    L = P.n_levels - 1
    c, f = rng.uniform(-1, 1, P.n_dofs(L - 1)).astype(npdt), rng.uniform(-1, 1, P.n_dofs()).astype(npdt)
    ref = oracle.prolongate_add(3, k, n // 2, f, c)
    got = torch.tensor(f, device="cuda")
    tps.MGTransferCUDA(P).prolongate_and_add(L, got, torch.tensor(c, device="cuda"))
    torch.cuda.synchronize()
    assert relerr(got.cpu().numpy(), ref) < TOL[dtype]
    P.close()
