"""K1 fused lab + FD stencils vs the reference loops / oracle (bit-exact: no
FMA contraction on either side)."""
import ctypes as C

import numpy as np
import pytest

from devgrid import make_grid
from golden_io import c1_small

pytestmark = pytest.mark.gpu


def _run(cn, op, g, outs):
    import torch
    getattr(cn.ops, op)(g, *outs)
    torch.cuda.synchronize()


def test_c1_small_matches_reference_loops(cn):
    c = c1_small()
    g = make_grid(cn, c["comp"], c["nb"], c["n"], begin=(0, 0, 0), end=(1, 1, 1))
    lap = cn.Grid.Cartesian(c["nb"], c["n"])
    grad = cn.Grid.Cartesian(c["nb"], c["n"], ncomp=3)
    _run(cn, "lap_grad", g, (lap, grad))
    assert np.array_equal(lap.download(0), c["lap"])
    for d in range(3):
        assert np.array_equal(grad.download(d), c["grad"][d])
    # separate operators give the same bits
    lap2 = cn.Grid.Cartesian(c["nb"], c["n"])
    grad2 = cn.Grid.Cartesian(c["nb"], c["n"], ncomp=3)
    _run(cn, "laplacian", g, (lap2,))
    _run(cn, "gradient", g, (grad2,))
    assert np.array_equal(lap2.download(0), c["lap"])
    for d in range(3):
        assert np.array_equal(grad2.download(d), c["grad"][d])


def _c1_field(O, nb, n, seed=1234):
    """u = sin(2 pi x) sin(2 pi y) cos(2 pi z) + U(-1e-3, 1e-3) at cell centres."""
    stride = O.block_stride(n, np.float64)
    nbk = int(np.prod(nb))
    comp = np.zeros(nbk * stride)
    h = [1.0 / (nb[d] * n[d]) for d in range(3)]
    rng = np.random.default_rng(seed)
    cells = int(np.prod(n))
    for b in range(nbk):
        bi = (b % nb[0], (b // nb[0]) % nb[1], b // (nb[0] * nb[1]))
        z, y, x = np.meshgrid(*[(np.arange(n[d]) + n[d] * bi[d] + 0.5) * h[d] for d in (2, 1, 0)],
                              indexing="ij")
        comp[b * stride:b * stride + cells] = (np.sin(2 * np.pi * x) * np.sin(2 * np.pi * y) *
                                               np.cos(2 * np.pi * z)).ravel()
    comp += rng.uniform(-1e-3, 1e-3, size=comp.size)
    return comp, h


@pytest.mark.parametrize("with_bc", [False, True])
def test_c1_full_size_vs_oracle(cn, oracle_lib, with_bc):
    """128^3 cells as 8^3 blocks of 16^3 (the C1 geometry), FP64."""
    O = oracle_lib
    nb, n = (8, 8, 8), (16, 16, 16)
    comp, h = _c1_field(O, nb, n)
    bcl = {}
    if with_bc:
        for b in range(512):
            bi = (b % 8, (b // 8) % 8, b // 64)
            lst = []
            if bi[1] == 0: lst.append((1, 0, O.BC_ABSORBING, 0))
            if bi[1] == 7: lst.append((1, 1, O.BC_SYMMETRY, -1))
            if bi[2] == 0: lst.append((2, 0, O.BC_DIRICHLET, 0.5))
            if bi[2] == 7: lst.append((2, 1, O.BC_DIRICHLET, -0.25))
            if lst: bcl[b] = lst
    g = make_grid(cn, comp, nb, n, bcl)
    lap = cn.Grid.Cartesian(nb, n)
    grad = cn.Grid.Cartesian(nb, n, ncomp=3)
    _run(cn, "lap_grad", g, (lap, grad))
    hh = g.getCellSize()
    want_lap = O.laplacian_f64(comp, nb, n, bcl, [1.0 / (x * x) for x in hh])
    want_grad = O.gradient_f64(comp, nb, n, bcl, [1.0 / x for x in hh])
    assert np.array_equal(lap.download(0), want_lap)
    for d in range(3):
        assert np.array_equal(grad.download(d), want_grad[d])
    # accuracy vs the exact Laplacian -12 pi^2 u (noise-free part), a sanity bound
    if not with_bc:
        cells = lap.blocks_view(lap.download(0))
        assert np.isfinite(cells).all()


def test_divergence_periodic_vs_numpy(cn, oracle_lib):
    O = oracle_lib
    nb, n = (3, 2, 2), (8, 4, 6)
    stride = O.block_stride(n, np.float64)
    nbk = int(np.prod(nb))
    rng = np.random.default_rng(5)
    g = cn.Grid.Cartesian(nb, n, ncomp=3)
    comps = [rng.standard_normal(nbk * stride) for _ in range(3)]
    for c in range(3):
        g.upload(comps[c], c)
    out = cn.Grid.Cartesian(nb, n)
    cn.ops.divergence(g, out)
    got = out.blocks_view(out.download(0))
    # global periodic arrays (z, y, x)
    def glob(a):
        v = a.reshape(nbk, stride)[:, : int(np.prod(n))].reshape(nb[2], nb[1], nb[0], n[2], n[1], n[0])
        return v.transpose(0, 3, 1, 4, 2, 5).reshape(nb[2] * n[2], nb[1] * n[1], nb[0] * n[0])
    v0, v1, v2 = (glob(a) for a in comps)
    ih = [1.0 / x for x in g.getCellSize()]
    t0 = (np.roll(v0, -1, 2) - np.roll(v0, 1, 2)) * ih[0]
    t1 = (np.roll(v1, -1, 1) - np.roll(v1, 1, 1)) * ih[1]
    t2 = (np.roll(v2, -1, 0) - np.roll(v2, 1, 0)) * ih[2]
    want = 0.5 * ((t0 + t1) + t2)
    gotg = got.reshape(nb[2], nb[1], nb[0], n[2], n[1], n[0]).transpose(0, 3, 1, 4, 2, 5).reshape(want.shape)
    assert np.array_equal(gotg, want)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_ddx_kernel_abi(cn, oracle_lib, dtype):
    """ISPC benchmark kernel ABI on a pitched 32^3 lab (BaseBenchmark.cpp:55-95)."""
    import torch
    N, g = 32, 1
    L = N + 2 * g
    xps = L + 6  # padded pitch like an aligned FieldLab row
    rng = np.random.default_rng(9)
    lab = rng.standard_normal((L, L, xps)).astype(dtype)
    dst = np.zeros((N, N, N), dtype=dtype)
    factor = dtype(1.0 / N)
    off = g + xps * (g + L * g)
    fn = oracle_lib.lib().or_ddx_f64 if dtype == np.float64 else oracle_lib.lib().or_ddx_f32
    CT = C.c_double if dtype == np.float64 else C.c_float
    fn.argtypes = [C.c_int] * 3 + [C.c_void_p, C.c_int, C.c_int, C.c_void_p, C.c_int, C.c_int, CT]
    fn(N, N, N, C.c_void_p(lab.ctypes.data + off * lab.itemsize), xps, xps * L,
       dst.ctypes.data_as(C.c_void_p), N, N * N, CT(factor))
    tlab = torch.from_numpy(lab).cuda()
    tdst = torch.zeros((N, N, N), dtype=tlab.dtype, device="cuda")
    lib = cn._lib.lib()
    f = lib.cn_ddx_f64 if dtype == np.float64 else lib.cn_ddx_f32
    f(N, N, N, C.c_void_p(tlab.data_ptr() + off * lab.itemsize), xps, xps * L,
      C.c_void_p(tdst.data_ptr()), N, N * N, factor)
    torch.cuda.synchronize()
    assert np.array_equal(tdst.cpu().numpy(), dst)


def _glob(a, nb, n, stride):
    """Block-ordered component -> global periodic array (z, y, x)."""
    nbk = int(np.prod(nb))
    v = a.reshape(nbk, stride)[:, : int(np.prod(n))].reshape(nb[2], nb[1], nb[0], n[2], n[1], n[0])
    return v.transpose(0, 3, 1, 4, 2, 5).reshape(nb[2] * n[2], nb[1] * n[1], nb[0] * n[0])


@pytest.mark.parametrize("n", [(5, 3, 7), (7, 6, 4), (6, 5, 3), (2, 9, 2)])
def test_lap_grad_odd_extents_vs_oracle(cn, oracle_lib, n):
    """Block extents with odd x (one cell per thread) and odd y / z (two cells
    per thread), periodic and with a BC chain, bit-exact vs the oracle."""
    O = oracle_lib
    nb = (3, 2, 2)
    stride = O.block_stride(n, np.float64)
    rng = np.random.default_rng(sum(n))
    comp = rng.standard_normal(int(np.prod(nb)) * stride)
    for bcl in ({}, {b: [(0, 0, O.BC_DIRICHLET, 0.25), (1, 1, O.BC_ABSORBING, 0), (2, 0, O.BC_SYMMETRY, -1)]
                     for b in range(int(np.prod(nb)))}):
        g = make_grid(cn, comp, nb, n, bcl)
        lap = cn.Grid.Cartesian(nb, n)
        grad = cn.Grid.Cartesian(nb, n, ncomp=3)
        _run(cn, "lap_grad", g, (lap, grad))
        hh = g.getCellSize()
        want_lap = O.laplacian_f64(comp, nb, n, bcl, [1.0 / (x * x) for x in hh])
        want_grad = O.gradient_f64(comp, nb, n, bcl, [1.0 / x for x in hh])
        assert np.array_equal(lap.download(0), want_lap)
        for d in range(3):
            assert np.array_equal(grad.download(d), want_grad[d])


@pytest.mark.parametrize("n", [(8, 4, 6), (5, 3, 7)])
def test_fp32_lap_grad_div_periodic_vs_numpy(cn, oracle_lib, n):
    """FP32 grids: the same operation order in float32 numpy (every operation
    rounded on its own, no contraction) gives the same bits."""
    O = oracle_lib
    nb = (3, 2, 2)
    stride = O.block_stride(n, np.float32)
    rng = np.random.default_rng(7)
    f32 = np.float32
    comps = [rng.standard_normal(int(np.prod(nb)) * stride).astype(f32) for _ in range(3)]
    g = cn.Grid.Cartesian(nb, n, ncomp=3, dtype=f32)
    for c in range(3):
        g.upload(comps[c], c)
    lap = cn.Grid.Cartesian(nb, n, dtype=f32)
    grad = cn.Grid.Cartesian(nb, n, ncomp=3, dtype=f32)
    div = cn.Grid.Cartesian(nb, n, dtype=f32)
    _run(cn, "lap_grad", g, (lap, grad))
    cn.ops.divergence(g, div)
    import torch
    torch.cuda.synchronize()
    hh = g.getCellSize()
    ih = [f32(1.0 / x) for x in hh]
    ih2 = [f32(1.0 / (x * x)) for x in hh]
    u = _glob(comps[0], nb, n, stride)
    xp, xm = np.roll(u, -1, 2), np.roll(u, 1, 2)
    yp, ym = np.roll(u, -1, 1), np.roll(u, 1, 1)
    zp, zm = np.roll(u, -1, 0), np.roll(u, 1, 0)
    c2 = f32(2) * u
    want_lap = (ih2[0] * ((xp - c2) + xm) + ih2[1] * ((yp - c2) + ym)) + ih2[2] * ((zp - c2) + zm)
    want_g = [f32(0.5) * ((xp - xm) * ih[0]), f32(0.5) * ((yp - ym) * ih[1]), f32(0.5) * ((zp - zm) * ih[2])]
    v0, v1, v2 = (_glob(a, nb, n, stride) for a in comps)
    t0 = (np.roll(v0, -1, 2) - np.roll(v0, 1, 2)) * ih[0]
    t1 = (np.roll(v1, -1, 1) - np.roll(v1, 1, 1)) * ih[1]
    t2 = (np.roll(v2, -1, 0) - np.roll(v2, 1, 0)) * ih[2]
    want_div = f32(0.5) * ((t0 + t1) + t2)
    assert np.array_equal(_glob(lap.download(0), nb, n, stride), want_lap)
    for d in range(3):
        assert np.array_equal(_glob(grad.download(d), nb, n, stride), want_g[d])
    assert np.array_equal(_glob(div.download(0), nb, n, stride), want_div)


def _random_bcs(O, rng, nb):
    """BC lists of one component: on about half of the block faces one to
    three BCs (Base and repeats among them), faces inside the domain too."""
    out = {}
    for b in range(int(np.prod(nb))):
        lst = [(int(d), int(s), int(k), float(v)) for d in range(3) for s in range(2) if rng.random() < 0.5
               for k, v in zip(rng.integers(0, 4, size=rng.integers(1, 4)), (0.5, -1.0, 0.25))]
        if lst:
            out[b] = [lst[i] for i in rng.permutation(len(lst))]
    return out


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("nb,n", [((2, 1, 3), (8, 5, 3)), ((1, 3, 2), (6, 4, 9)), ((3, 2, 1), (7, 1, 2)),
                                  ((2, 2, 2), (12, 3, 33)), ((1, 1, 1), (4, 2, 1)), ((1, 2, 1), (1, 33, 40))])
def test_random_bc_vectors_vs_oracle_labs(cn, oracle_lib, dtype, nb, n):
    """Every component's own random BC vectors; rows of 4, 2 and 1 cells per
    thread, runs of one plane and longer, blocks of one cell along a
    direction.  The stencils, rounded operation by operation in numpy on the
    oracle's labs, give the same bits."""
    import torch
    O = oracle_lib
    rng = np.random.default_rng(sum(n))
    nbk, stride = int(np.prod(nb)), O.block_stride(n, dtype)
    comps = [rng.standard_normal(nbk * stride).astype(dtype) for _ in range(3)]
    bcl = [_random_bcs(O, rng, nb) for _ in range(3)]
    g = cn.Grid.Cartesian(nb, n, ncomp=3, dtype=dtype)
    kinds = {0: cn.BC.Base, 1: cn.BC.Dirichlet, 2: cn.BC.Absorbing, 3: cn.BC.Symmetry}
    for c in range(3):
        g.upload(comps[c], c)
        for b, lst in bcl[c].items():
            for d, s, k, v in lst:
                g.field(b, c).getBC().push_back(kinds[k](d, s, v) if k in (1, 3) else kinds[k](d, s))
    lap, div = (cn.Grid.Cartesian(nb, n, dtype=dtype) for _ in range(2))
    grad = cn.Grid.Cartesian(nb, n, ncomp=3, dtype=dtype)
    _run(cn, "lap_grad", g, (lap, grad))
    _run(cn, "divergence", g, (div,))
    T = dtype
    ih = [T(1.0 / x) for x in g.getCellSize()]
    ih2 = [T(1.0 / (x * x)) for x in g.getCellSize()]
    got = [a.blocks_view(a.download(k)) for a, k in ((lap, 0), (grad, 0), (grad, 1), (grad, 2), (div, 0))]
    m = slice(1, -1)
    for b in range(nbk):
        labs = []
        for c in range(3):
            lab, ok = O.lab_fill(comps[c], nb, n, (1, 1, 1), (1, 1, 1), False, bcl[c], b)
            labs.append(np.where(ok, lab, T(0)).astype(T))
        lo = [(m, m, slice(0, -2)), (m, slice(0, -2), m), (slice(0, -2), m, m)]
        hi = [(m, m, slice(2, None)), (m, slice(2, None), m), (slice(2, None), m, m)]
        u = labs[0]
        c2 = T(2) * u[m, m, m]
        dd = [ih2[d] * ((u[hi[d]] - c2) + u[lo[d]]) for d in range(3)]
        dv = [(labs[d][hi[d]] - labs[d][lo[d]]) * ih[d] for d in range(3)]
        want = [(dd[0] + dd[1]) + dd[2]] + [T(0.5) * ((u[hi[d]] - u[lo[d]]) * ih[d]) for d in range(3)]
        want.append(T(0.5) * ((dv[0] + dv[1]) + dv[2]))
        for what, (a, w) in enumerate(zip(got, want)):
            assert np.array_equal(a[b], w), f"output {what}, block {b}"


@pytest.mark.parametrize("nb,n,share", [((2, 2, 1), (12, 10, 40), 0.6), ((1, 1, 1), (36, 36, 60), 1.0),
                                        ((9, 8, 11), (4, 3, 5), 0.4), ((8, 8, 8), (2, 4, 3), 1.0),
                                        ((7, 5, 6), (8, 6, 2), 0.05), ((6, 6, 6), (32, 32, 32), 0.15)])
def test_faces_with_bcs_vs_oracle(cn, oracle_lib, nb, n, share):
    """BCs on a share of all block faces: large faces that several CTAs walk,
    many small ones to a CTA, CTAs without any, and outputs beyond L2, where x
    faces are taken by whole sectors.  Then without BCs again, and with BCs
    pushed between the capture of a call and its replay."""
    import torch
    O = oracle_lib
    rng = np.random.default_rng(nb[0] + n[0])
    nbk, stride = int(np.prod(nb)), O.block_stride(n, np.float64)
    comp = rng.standard_normal(nbk * stride)
    g = cn.Grid.Cartesian(nb, n)
    g.upload(comp)
    lap, grad = cn.Grid.Cartesian(nb, n), cn.Grid.Cartesian(nb, n, ncomp=3)
    h = g.getCellSize()

    def check(bcl):
        wl = O.laplacian_f64(comp, nb, n, bcl, [1 / (x * x) for x in h])
        wg = O.gradient_f64(comp, nb, n, bcl, [1 / x for x in h])
        assert np.array_equal(lap.blocks_view(lap.download(0)), lap.blocks_view(wl))
        for d in range(3):
            assert np.array_equal(grad.blocks_view(grad.download(d)), grad.blocks_view(wg[d]))

    kinds = {O.BC_DIRICHLET: cn.BC.Dirichlet, O.BC_ABSORBING: cn.BC.Absorbing, O.BC_SYMMETRY: cn.BC.Symmetry}
    faces = [(b, d, s) for b in range(nbk) for d in range(3) for s in range(2) if rng.random() < share]
    bcl = {}
    for b, d, s in faces:
        bcl.setdefault(b, []).append((d, s, int(rng.choice(list(kinds))), float(rng.choice([0.5, -1.0]))))

    def push():
        for b, lst in bcl.items():
            for d, s, k, v in lst:
                g.field(b).getBC().push_back(kinds[k](d, s) if k == O.BC_ABSORBING else kinds[k](d, s, v))
        g.sync_bcs()

    def clear():
        for b in bcl:
            g.field(b).getBC().clear()
        g.sync_bcs()

    push()
    cn.ops.lap_grad(g, lap, grad)
    torch.cuda.synchronize()
    check(bcl)
    clear()
    cn.ops.lap_grad(g, lap, grad)
    torch.cuda.synchronize()
    check({})
    s = torch.cuda.Stream()
    graph = cn.amr.Graph.capture(lambda: cn.ops.lap_grad(g, lap, grad, stream=s), s)
    push()
    graph.launch(s)
    s.synchronize()
    check(bcl)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("nb,n", [((1, 1, 1), (8, 8, 8)), ((1, 1, 1), (12, 10, 9)), ((2, 1, 3), (7, 6, 5))])
def test_outputs_on_top_of_inputs(cn, dtype, nb, n):
    """Operators written onto components they read give what they give into
    another grid."""
    import torch
    rng = np.random.default_rng(12)
    g, lap, grad = (cn.Grid.Cartesian(nb, n, ncomp=k, dtype=dtype) for k in (4, 1, 3))
    data = [rng.standard_normal(g.comp_stride).astype(dtype) for _ in range(4)]
    cells = lambda grid, c: grid.blocks_view(grid.download(c))

    def fresh():
        for c in range(4):
            g.upload(data[c], c)

    fresh()
    cn.ops.lap_grad(g, lap, grad, comp=1)
    torch.cuda.synchronize()
    want_l, want_g = cells(lap, 0), [cells(grad, d) for d in range(3)]
    cn.ops.laplacian(g, g, comp=1, out_comp=1)
    torch.cuda.synchronize()
    assert np.array_equal(cells(g, 1), want_l)
    fresh()
    cn.ops.gradient(g, g, comp=1, out_comp=0)
    torch.cuda.synchronize()
    assert all(np.array_equal(cells(g, d), want_g[d]) for d in range(3))
    fresh()
    cn.ops.divergence(g, lap, comp=1)
    torch.cuda.synchronize()
    want_d = cells(lap, 0)
    cn.ops.divergence(g, g, comp=1, out_comp=3)
    torch.cuda.synchronize()
    assert np.array_equal(cells(g, 3), want_d)
