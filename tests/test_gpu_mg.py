"""Multigrid operators vs the CPU oracle (bit-exact per kernel: same order, no
contraction), the coarsest FP64 CG within FP32 output round-off, and the
solver's convergence to a 1e-8 relative FP64 residual."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _end(nb, n):
    """Domain extent giving cubic cells (h = 1 / max cells)."""
    g = max(nb[d] * n[d] for d in range(3))
    return tuple(nb[d] * n[d] / g for d in range(3))


def _setup(cn, nb, n, seed=1):
    e = _end(nb, n)
    k = cn.Grid.Cartesian(nb, n, end=e, dtype=np.float32)
    cn.workloads.poisson_coefficient(k, seed=seed)
    f = cn.Grid.Cartesian(nb, n, end=e, dtype=np.float32)
    cn.workloads.poisson_rhs(f, seed=seed + 1)
    return k, f


# blocks of 8^3 (one tile per block) and of 32^3, the C5 block size (the
# 32x8x4 tile path, several tiles per block)
BLOCKS = [((2, 3, 2), (8, 8, 8)), ((2, 2, 2), (32, 32, 32))]


@pytest.mark.parametrize("nb,n", BLOCKS)
def test_jacobi_and_restriction_match_oracle(cn, oracle_lib, nb, n):
    import torch
    k, f = _setup(cn, nb, n)
    m = cn.mg.Multigrid(k, omega=0.8)
    p = cn.Grid.Cartesian(nb, n, end=_end(nb, n), dtype=np.float32)
    rng = np.random.default_rng(2)
    ph = np.zeros(p.comp_stride, dtype=np.float32)
    p.blocks_view(ph)[:] = rng.standard_normal(p.blocks_view(ph).shape)
    p.upload(ph)
    out = cn.Grid.Cartesian(nb, n, end=_end(nb, n), dtype=np.float32)
    m.jacobi(p, f, out)
    torch.cuda.synchronize()
    kh, fh = k.download(), f.download()
    ih2 = np.float32(1.0 / p.getCellSize()[0] ** 2)
    want = oracle_lib.mg_jacobi(ph, kh, fh, nb, n, 0.8, ih2)
    assert np.array_equal(p.blocks_view(out.download()), p.blocks_view(want))
    fc = m.level(1, "f")
    m.restrict_residual(p, f, fc)
    torch.cuda.synchronize()
    want = oracle_lib.mg_resid_restrict(ph, kh, fh, nb, n, ih2)
    assert np.array_equal(fc.blocks_view(fc.download()), fc.blocks_view(want))
    # coarse coefficients
    kc = m.level(1, "k")
    want = oracle_lib.mg_restrict_mean(kh, nb, n)
    assert np.array_equal(kc.blocks_view(kc.download()), kc.blocks_view(want))
    # prolongation of a random coarse correction
    ec = m.level(1, "p")
    eh = np.zeros(ec.comp_stride, dtype=np.float32)
    ec.blocks_view(eh)[:] = rng.standard_normal(ec.blocks_view(eh).shape)
    ec.upload(eh)
    m.prolong(ec, p)
    torch.cuda.synchronize()
    want = oracle_lib.mg_prolong(ph, eh, nb, n)
    assert np.array_equal(p.blocks_view(p.download()), p.blocks_view(want))


@pytest.mark.parametrize("nb,n", [((2, 2, 2), (8, 8, 8)), ((2, 2, 2), (32, 32, 32))])
def test_fp64_residual_matches_oracle(cn, oracle_lib, nb, n):
    import torch
    k, f = _setup(cn, nb, n)
    m = cn.mg.Multigrid(k)
    p64 = cn.Grid.Cartesian(nb, n, dtype=np.float64)
    rng = np.random.default_rng(3)
    ph = np.zeros(p64.comp_stride)
    p64.blocks_view(ph)[:] = rng.standard_normal(p64.blocks_view(ph).shape) * 1e-3
    p64.upload(ph)
    r32 = cn.Grid.Cartesian(nb, n, dtype=np.float32)
    rr, ff = m.residual(p64, f, r32)
    torch.cuda.synchronize()
    wr, wrr, wff = oracle_lib.mg_resid64(ph, k.download(), f.download(), nb, n, 1.0 / p64.getCellSize()[0] ** 2)
    assert np.array_equal(r32.blocks_view(r32.download()), r32.blocks_view(wr))
    assert abs(rr - wrr) <= 1e-12 * wrr and abs(ff - wff) <= 1e-12 * wff


def test_vcycle_and_coarsest_solve(cn, oracle_lib):
    """A 2-level cycle (coarsest = CG) against the oracle composition; the
    coarse FP64 CG differs from the oracle's only by summation order."""
    import torch
    nb, n = (4, 4, 4), (2, 2, 2)
    k, f = _setup(cn, nb, n)
    m = cn.mg.Multigrid(k, nu1=1, nu2=1, omega=0.8, max_levels=2)
    assert m.nlevels == 2 and m.coarsest_cells == 64
    e = cn.Grid.Cartesian(nb, n, dtype=np.float32)
    m.vcycle(f, e)
    torch.cuda.synchronize()
    kh, fh = k.download(), f.download()
    ih2 = np.float32(1.0 / e.getCellSize()[0] ** 2)
    p1 = oracle_lib.mg_jacobi(None, kh, fh, nb, n, 0.8, ih2)
    fc = oracle_lib.mg_resid_restrict(p1, kh, fh, nb, n, ih2)
    kc = oracle_lib.mg_restrict_mean(kh, nb, n)
    ec, _ = oracle_lib.mg_coarse_cg(fc, kc, nb, (1, 1, 1), 1.0 / (2 * e.getCellSize()[0]) ** 2)
    p2 = oracle_lib.mg_prolong(p1, ec, nb, n)
    want = oracle_lib.mg_jacobi(p2, kh, fh, nb, n, 0.8, ih2)
    got = e.download()
    scale = np.max(np.abs(want))
    assert np.max(np.abs(got - want)) <= 1e-5 * scale


@pytest.mark.parametrize("nb,n", [((4, 4, 4), (16, 16, 16)), ((8, 8, 8), (32, 32, 32))])
def test_solver_reaches_1e8(cn, nb, n):
    """64^3 and the full 256^3 problem: FP64 relative residual <= 1e-8."""
    import torch
    k, f = _setup(cn, nb, n)
    m = cn.mg.Multigrid(k, nu1=2, nu2=2, omega=0.8)
    p64 = cn.Grid.Cartesian(nb, n, dtype=np.float64)
    cycles, rel = m.solve(f, p64, rtol=1e-8, max_cycles=60)
    print(f"{nb}x{n}: {m.nlevels} levels, {cycles} cycles, relres {rel:.3e}")
    assert rel <= 1e-8 and cycles < 60
    rr, ff = m.residual(p64, f)
    assert np.sqrt(rr / ff) <= 1e-8
    del m, p64, k, f
    torch.cuda.empty_cache()


def test_manufactured_solution_second_order(cn):
    """k = 1, f = L_exact(u) for u = sin(2 pi x) sin(2 pi y) sin(2 pi z): the
    discrete solution converges to u at second order."""
    import torch
    errs = []
    for N in (32, 64):
        nb, n = (4, 4, 4), (N // 4,) * 3
        k = cn.Grid.Cartesian(nb, n, dtype=np.float32)
        k.tensor(0).fill_(1.0)
        f = cn.Grid.Cartesian(nb, n, dtype=np.float32)
        x = ((torch.arange(N, device="cuda", dtype=torch.float64) + 0.5) / N)
        s = torch.sin(2 * np.pi * x)
        u = s[:, None, None] * s[None, :, None] * s[None, None, :]
        cn.workloads._global_to_blocks(f, -12 * np.pi ** 2 * u, torch)
        m = cn.mg.Multigrid(k)
        p64 = cn.Grid.Cartesian(nb, n, dtype=np.float64)
        m.solve(f, p64, rtol=1e-10, max_cycles=60)
        got = torch.from_numpy(p64.download()).cuda()
        cells = int(np.prod(n))
        gv = got.view(p64.size(), -1)[:, :cells].reshape(4, 4, 4, n[2], n[1], n[0]).permute(0, 3, 1, 4, 2, 5).reshape(N, N, N)
        errs.append(float((gv - u).abs().max()))
    assert errs[1] < errs[0] / 3.0, errs


@pytest.mark.parametrize("nb,n", [((2, 2, 2), (16, 16, 16)), ((12, 12, 12), (2, 2, 2))])
def test_solve_matches_oracle_solve(cn, oracle_lib, nb, n):
    """The whole solve (V(2,2) cycles in FP64 defect correction) against the
    oracle's composition of the same operators: the same cycle count (the
    device's coarsest solve is exact up to round-off like the oracle's CG:
    the dense inverse on an 8-cell coarsest level, the FP64 CG on a
    1728-cell one) and the same solution up to the periodic constant, within
    1e-5 of its range."""
    import torch
    k, f = _setup(cn, nb, n)
    m = cn.mg.Multigrid(k, nu1=2, nu2=2, omega=0.8)
    p64 = cn.Grid.Cartesian(nb, n, dtype=np.float64)
    cycles, rel = m.solve(f, p64, rtol=1e-8, max_cycles=60)
    torch.cuda.synchronize()
    want, wc, wrel = oracle_lib.mg_solve(k.download(), f.download(), nb, n, k.getCellSize()[0], rtol=1e-8,
                                         max_cycles=60)
    assert abs(cycles - wc) <= 1 and rel <= 1e-8 and wrel <= 1e-8
    got = p64.blocks_view(p64.download())
    ref = p64.blocks_view(want)
    got, ref = got - got.mean(), ref - ref.mean()
    assert np.max(np.abs(got - ref)) <= 1e-5 * np.ptp(ref)


@pytest.mark.parametrize("nb,n,nu", [((4, 4, 4), (16, 16, 16), (2, 2)), ((2, 2, 2), (12, 12, 12), (2, 1)),
                                     ((3, 2, 2), (8, 8, 8), (1, 2)), ((1, 1, 1), (32, 32, 32), (2, 0)),
                                     ((2, 1, 1), (8, 8, 8), (0, 2)), ((2, 2, 2), (2, 4, 8), (1, 1)),
                                     ((3, 3, 3), (5, 5, 5), (2, 2))])
def test_march_and_tail_match_tile_kernels(cn, nb, n, nu):
    """A Base BC (the periodic no-op) on every level's solution sends each
    operator through the tile kernels and its own launch; without BCs the
    marching kernels (rows of 4, 2 and 1 cells per thread) and the one-launch
    coarse part run.  Same operations in the same order: the same bits."""
    import torch
    k, f = _setup(cn, nb, n)
    out = []
    for plain in (True, False):
        m = cn.mg.Multigrid(k, nu1=nu[0], nu2=nu[1], omega=0.8)
        if not plain:
            for l in range(m.nlevels):
                g = m.level(l, "p")
                for b in range(g.size()):
                    g.field(b, 0).getBC().push_back(cn.BC.Base(0, 0))
                g.sync_bcs()
        e = cn.Grid.Cartesian(nb, n, end=_end(nb, n), dtype=np.float32)
        m.vcycle(f, e)
        p64 = cn.Grid.Cartesian(nb, n, end=_end(nb, n), dtype=np.float64)
        cycles, rel = m.solve(f, p64, rtol=1e-3, max_cycles=4)
        r32 = cn.Grid.Cartesian(nb, n, end=_end(nb, n), dtype=np.float32)
        if not plain:
            for b in range(p64.size()):
                p64.field(b, 0).getBC().push_back(cn.BC.Base(1, 0))
        rr, ff = m.residual(p64, f, r32)
        torch.cuda.synchronize()
        out.append((e.blocks_view(e.download()).copy(), p64.blocks_view(p64.download()).copy(),
                    r32.blocks_view(r32.download()).copy(), cycles, rr, ff))
    a, b = out
    assert a[3] == b[3]
    for x, y in zip(a[:3], b[:3]):
        assert np.array_equal(x, y)
    assert abs(a[4] - b[4]) <= 1e-12 * b[4] and abs(a[5] - b[5]) <= 1e-12 * b[5]


def test_more_multigrids_than_sum_places(cn):
    """Multigrids beyond the shared page of residual sums hold their own, and
    places come back: solves of the first and the last of 70, interleaved,
    and of one made after half of them are gone, give the same residuals."""
    nb, n = (2, 2, 2), (4, 4, 4)
    k, f = _setup(cn, nb, n)

    def rel(m):
        p64 = cn.Grid.Cartesian(nb, n, end=_end(nb, n), dtype=np.float64)
        return m.solve(f, p64, rtol=1e-30, max_cycles=2)[1]

    ms = [cn.mg.Multigrid(k) for _ in range(70)]
    want = rel(ms[0])
    assert [rel(m) for m in (ms[69], ms[1], ms[65], ms[0])] == [want] * 4
    del ms[10:45]
    assert rel(cn.mg.Multigrid(k)) == want and rel(ms[-1]) == want


@pytest.mark.parametrize("n64", [(16, 8, 8), (16, 16, 32), (16, 8, 32), (8, 16, 16)])
def test_solution_of_other_extents_is_refused(cn, n64):
    """The outer iteration takes p64 by the multigrid's block extents: fields
    of as many blocks whose extents differ along any dimension (along y and z
    only, with the storage of one component smaller, larger or the same), and
    residual fields too small for it, are refused before any of them is written."""
    nb, n = (2, 2, 2), (16, 16, 16)
    k, f = _setup(cn, nb, n)
    m = cn.mg.Multigrid(k)
    p64 = cn.Grid.Cartesian(nb, n64, dtype=np.float64)
    p64.tensor(0).fill_(7.0)
    for call in (lambda: m.solve(f, p64), lambda: m.residual(p64, f)):
        with pytest.raises(cn.CnError, match="unequal size"):
            call()
    assert float(p64.tensor(0).min()) == 7.0
    good = cn.Grid.Cartesian(nb, n, dtype=np.float64)
    small = cn.Grid.Cartesian(nb, (16, 8, 16), dtype=np.float32)
    with pytest.raises(cn.CnError, match="unequal size"):
        m.residual(good, f, small)
    with pytest.raises(cn.CnError, match="unequal size"):
        m.solve(f, f)  # an FP32 solution
    assert m.solve(f, good, rtol=1e-8)[1] <= 1e-8


def _base_bcs(cn, g):
    """A Base BC (the periodic no-op) on every block: the tile kernels run."""
    for b in range(g.size()):
        g.field(b, 0).getBC().push_back(cn.BC.Base(0, 0))
    g.sync_bcs()


@pytest.mark.parametrize("nb,n,nu", [((4, 4, 4), (16, 16, 16), (2, 2)), ((2, 2, 2), (12, 12, 12), (2, 1)),
                                     ((3, 2, 2), (8, 8, 8), (1, 2)), ((2, 2, 2), (2, 4, 8), (3, 2)),
                                     ((2, 1, 1), (24, 8, 16), (0, 1)), ((1, 1, 1), (32, 32, 32), (1, 0))])
def test_tile_kernels_from_the_face_means(cn, nb, n, nu):
    """Cycles with a BC on the solution of every level, on both of the fields
    that alternate as it where a sweep count is odd, against cycles without:
    the tile kernels and the marching ones read the same face means and give
    the same bits.  The first call of one multigrid is under stream capture,
    where nothing may be left to allocate or to fill."""
    import torch
    k, f = _setup(cn, nb, n)
    m, plain = (cn.mg.Multigrid(k, nu1=nu[0], nu2=nu[1], omega=0.8) for _ in range(2))
    e = [cn.Grid.Cartesian(nb, n, end=_end(nb, n), dtype=np.float32) for _ in range(3)]
    for l in range(m.nlevels):
        _base_bcs(cn, m.level(l, "p"))
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    g = cn.amr.Graph.capture(lambda: m.vcycle(f, e[0], stream=s), s)
    if sum(nu) % 2:  # now the other field of each level is its solution
        for l in range(m.nlevels - 1):
            _base_bcs(cn, m.level(l, "p"))
    g.launch(s)
    s.synchronize()
    m.vcycle(f, e[1])
    plain.vcycle(f, e[2])
    torch.cuda.synchronize()
    got = [x.blocks_view(x.download()) for x in e]
    assert np.array_equal(got[1], got[2])
    assert np.array_equal(got[0], got[2])


def test_tile_kernels_on_two_streams(cn):
    """The first sweeps of a new multigrid with BCs, on two streams that do not
    wait for one another."""
    import torch
    nb, n = (4, 4, 4), (32, 32, 32)
    k, f = _setup(cn, nb, n)
    m, plain = cn.mg.Multigrid(k), cn.mg.Multigrid(k)
    p, q, a, b, want = (cn.Grid.Cartesian(nb, n, dtype=np.float32) for _ in range(5))
    cn.workloads.poisson_rhs(p, seed=9)
    q.tensor(0).copy_(p.tensor(0))
    plain.jacobi(p, f, want)
    _base_bcs(cn, m.level(0, "p"))
    torch.cuda.synchronize()
    s, t = torch.cuda.Stream(), torch.cuda.Stream()
    m.jacobi(p, f, a, stream=s)
    m.jacobi(q, f, b, stream=t)
    torch.cuda.synchronize()
    assert torch.equal(a.tensor(0), want.tensor(0)) and torch.equal(b.tensor(0), want.tensor(0))


@pytest.mark.parametrize("nb,n", [((2, 3, 2), (5, 7, 3)), ((3, 1, 2), (1, 9, 1)), ((2, 2, 2), (6, 3, 3)), ((1, 2, 1), (12, 3, 6))])
@pytest.mark.parametrize("bcs", [False, True])
def test_jacobi_of_odd_blocks_matches_oracle(cn, oracle_lib, nb, n, bcs):
    """One sweep on blocks of odd extents, rows of one, two and four cells a
    thread: the marching and the tile kernel against the oracle."""
    import torch
    k, f = _setup(cn, nb, n)
    m = cn.mg.Multigrid(k)
    p, out = (cn.Grid.Cartesian(nb, n, end=_end(nb, n), dtype=np.float32) for _ in range(2))
    ph = np.zeros(p.comp_stride, dtype=np.float32)
    p.blocks_view(ph)[:] = np.random.default_rng(5).standard_normal(p.blocks_view(ph).shape)
    p.upload(ph)
    if bcs:
        _base_bcs(cn, m.level(0, "p"))
    m.jacobi(p, f, out)
    torch.cuda.synchronize()
    want = oracle_lib.mg_jacobi(ph, k.download(), f.download(), nb, n, 0.8, np.float32(1.0 / p.getCellSize()[0] ** 2))
    assert np.array_equal(p.blocks_view(out.download()), p.blocks_view(want))


@pytest.mark.parametrize("fine,coarse", [((5, 5, 5), (2, 2, 2)), ((8, 8, 7), (4, 4, 3)), ((8, 8, 8), (4, 4, 2)),
                                         ((8, 8, 8), (8, 8, 8)), ((8, 8, 8), (2, 2, 2))])
def test_prolongation_of_other_extents_is_refused(cn, fine, coarse):
    """The prolongation takes pairs of fine cells and indexes the coarse field
    by halves: anything but a field of half the extents is refused."""
    nb = (2, 2, 2)
    k, _ = _setup(cn, nb, (8, 8, 8))
    m = cn.mg.Multigrid(k)
    p, e = (cn.Grid.Cartesian(nb, n, dtype=np.float32) for n in (fine, coarse))
    with pytest.raises(cn.CnError, match="unequal size"):
        m.prolong(e, p)
