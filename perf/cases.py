"""Performance cases: the work that programs built on this framework have it do.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare(case, seed)`` makes what a program holds before the call (grids with
their boundary conditions, solvers, labs and file buffers, filled from the
seed), ``run(state)`` is one pass through the public entry points,
``work(case)`` the bytes and operations that pass cannot do without and
``exact(case, seed)`` the same outputs from plain torch in 64 bits.

Eight kinds of work:

* ``lab``      ghost-cell labs of a block range (Cartesian.loadLab for user stencils)
* ``fd``       fused Laplacian / gradient / divergence on a scalar or vector grid
* ``euler``    one SSP-RK3 step of the compressible Euler equations
* ``loop``     one iteration of an Euler time loop: CFL time step, RK3 step, conservation sums
* ``amr``      one SSP-RK3 step on blocks of uneven sizes on two refinement levels
* ``poisson``  one multigrid solve of div(k grad p) = f to a 1e-8 relative residual
* ``io``       a checkpoint: grid into the FP32 file buffer, and a file buffer back into a grid
* ``learned``  loss and gradients of one training batch of the learned smoother

Global arrays are (z, y, x); grids store blocks x fastest, each block's cells
x fastest.  Boundary conditions: "periodic", or "walls" (x periodic, y
absorbing on both sides, z Dirichlet).
"""
import math

import numpy as np
import torch

import cubismnova_b200 as cn

DEV = "cuda"
F64 = torch.float64
GAMMA = 1.4
DT = {"f64": np.float64, "f32": np.float32}
TDT = {"f64": torch.float64, "f32": torch.float32}


# ------------------------------------------------------------------- cases
def listed():
    return [
        # a user stencil's loop over blocks loads one lab at a time: launch latency
        dict(name="lab_one_block", kind="lab", nb0=4, nb1=4, nb2=4, n0=16, n1=16, n2=16, dtype="f64", bc="periodic",
             lo=-1, hi=2, tensorial=True, first=21, count=1),
        # all labs of a production grid (512^3 as 16^3 blocks of 32^3), the WENO5 stencil, with walls
        dict(name="lab_all_512", kind="lab", nb0=16, nb1=16, nb2=16, n0=32, n1=32, n2=32, dtype="f64", bc="walls",
             lo=-3, hi=4, tensorial=False, first=0, count=4096),
        # the reference's Laplacian benchmark size
        dict(name="lap_grad_128", kind="fd", op="lap_grad", nb0=4, nb1=4, nb2=4, n0=32, n1=32, n2=32, dtype="f64",
             bc="periodic"),
        # a large vector field in single precision on blocks of uneven extents, with walls
        dict(name="div_ragged_f32", kind="fd", op="div", nb0=12, nb1=10, nb2=8, n0=30, n1=33, n2=27, dtype="f32",
             bc="walls"),
        # a small simulation's time loop: latency, host round trips
        dict(name="euler_loop_64", kind="loop", nb0=2, nb1=2, nb2=2, n0=32, n1=32, n2=32, dtype="f64", bc="walls"),
        # the production size in double precision
        dict(name="euler_f64_512", kind="euler", nb0=16, nb1=16, nb2=16, n0=32, n1=32, n2=32, dtype="f64",
             bc="walls"),
        # a single-precision run
        dict(name="euler_f32_384", kind="euler", nb0=12, nb1=12, nb2=12, n0=32, n1=32, n2=32, dtype="f32",
             bc="walls"),
        # adaptive blocks: a refined ball in a coarse box, about 4200 blocks of 8^3, 16^3 and 32^3 cells
        dict(name="amr_f64", kind="amr", r0=7, r1=6, r2=6, radius=0.25, dtype="f64"),
        # a small pressure solve inside a time loop: launch latency of the coarse levels
        dict(name="poisson_64", kind="poisson", nb=4, n=16),
        # a large solve
        dict(name="poisson_256", kind="poisson", nb=8, n=32),
        # velocity checkpoint: three FP64 components to and from the FP32 file order
        dict(name="io_384", kind="io", nb0=12, nb1=12, nb2=12, n0=32, n1=32, n2=32, dtype="f64", file="f32",
             ncomp=3),
        # one training batch of the learned smoother (32 patches of 32^3 cells)
        dict(name="learned_batch", kind="learned", batch=32, patch=32),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lab", "fd", "euler", "loop", "amr", "poisson", "io", "learned"])

    def blocks(cells_lo, cells_hi, extents):
        """Block extents from `extents` and block counts for about a drawn number of cells."""
        n = [rng.choice(extents) for _ in range(3)]
        target = math.exp(rng.uniform(math.log(cells_lo), math.log(cells_hi))) / (n[0] * n[1] * n[2])
        side = max(1.0, target ** (1.0 / 3.0))
        nb = [max(1, int(side * rng.uniform(0.8, 1.25))) for _ in range(3)]
        return dict(nb0=nb[0], nb1=nb[1], nb2=nb[2], n0=n[0], n1=n[1], n2=n[2])

    if kind == "lab":
        c = dict(kind=kind, **blocks(1 << 16, 1 << 26, [8, 13, 16, 20, 24, 27, 32, 33]))
        c.update(dtype=rng.choice(["f64", "f32"]), tensorial=rng.random() < 0.4)
        c["bc"] = "periodic" if c["tensorial"] else rng.choice(["periodic", "walls"])
        c["lo"], c["hi"] = rng.choice([(-1, 2), (-2, 3), (-3, 4), (0, 2)])
        total = c["nb0"] * c["nb1"] * c["nb2"]
        c["count"] = rng.choice([1, total, max(1, total // 3)])
        c["first"] = rng.randrange(0, total - c["count"] + 1)
        return c
    if kind == "fd":
        c = dict(kind=kind, op=rng.choice(["lap", "grad", "lap_grad", "div"]),
                 **blocks(1 << 16, 1 << 26, [8, 16, 17, 21, 24, 30, 32, 33]))
        c.update(dtype=rng.choice(["f64", "f32"]), bc=rng.choice(["periodic", "walls"]))
        return c
    if kind in ("euler", "loop"):
        c = dict(kind=kind, **blocks(1 << 15, 1 << 25, [8, 16, 24, 32]))
        c.update(dtype=rng.choice(["f64", "f32"]), bc=rng.choice(["periodic", "walls"]))
        return c
    if kind == "amr":
        return dict(kind=kind, r0=rng.randint(2, 7), r1=rng.randint(2, 6), r2=rng.randint(2, 6),
                    radius=round(rng.uniform(0.2, 0.42), 3), dtype=rng.choice(["f64", "f64", "f32"]))
    if kind == "poisson":
        nb, n = rng.choice([(2, 16), (2, 32), (3, 16), (3, 24), (3, 32), (4, 24), (4, 32), (5, 16), (5, 24), (6, 16),
                            (6, 32), (7, 32), (8, 16)])
        return dict(kind=kind, nb=nb, n=n)
    if kind == "io":
        c = dict(kind=kind, **blocks(1 << 16, 1 << 25, [8, 15, 16, 20, 27, 32]))
        c.update(dtype=rng.choice(["f64", "f32"]), ncomp=rng.choice([1, 3, 5]))
        c["file"] = rng.choice(["f64", "f32"])
        return c
    return dict(kind="learned", batch=_log_int(rng, 2, 32), patch=rng.choice([8, 12, 16, 24, 32]))


# --------------------------------------------------------- shared geometry
def _nb(c):
    return (c["nb0"], c["nb1"], c["nb2"])


def _n(c):
    return (c["n0"], c["n1"], c["n2"])


def _global(c):
    return tuple(a * b for a, b in zip(_nb(c), _n(c)))


def _end(c):
    """Cubic cells: the box's extents in units of its longest side."""
    g = _global(c)
    return tuple(v / max(g) for v in g)


def _h(c):
    return 1.0 / max(_global(c))


def _to_blocks(a, nb, n):
    """(nz, ny, nx) -> (blocks, cells of a block)."""
    v = a.reshape(nb[2], n[2], nb[1], n[1], nb[0], n[0]).permute(0, 2, 4, 1, 3, 5)
    return v.reshape(nb[0] * nb[1] * nb[2], n[0] * n[1] * n[2])


def _grid(c, ncomp=1, dtype=None):
    return cn.Grid.Cartesian(_nb(c), _n(c), end=_end(c), ncomp=ncomp, dtype=DT[dtype or c["dtype"]])


def _fill(grid, arrays):
    nb, n = grid.getSize(), grid.getBlockCells()
    cells = n[0] * n[1] * n[2]
    for comp, a in enumerate(arrays):
        t = grid.tensor(comp)
        t.zero_()
        t[:, :cells].copy_(_to_blocks(a, nb, n))


def _held(tensor, owner):
    """A view of library memory that keeps the object owning that memory alive."""
    tensor.owner = owner
    return tensor


def _values(grid):
    n = grid.getBlockCells()
    cells = n[0] * n[1] * n[2]
    return [_held(grid.tensor(comp)[:, :cells], grid) for comp in range(grid.ncomp)]


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _axes(c):
    h = _h(c)
    x, y, z = ((torch.arange(m, device=DEV, dtype=F64) + 0.5) * h for m in _global(c))
    return x[None, None, :], y[None, :, None], z[:, None, None]


def _noise(shape, gen, amp):
    return torch.rand(shape, generator=gen, device=DEV, dtype=F64).mul_(2 * amp).sub_(amp)


def _phases(seed, k):
    return np.random.default_rng([int(seed), 5]).random(k)


def _wave(c, seed, ncomp):
    """Smooth waves with a little noise, stored in the case's type."""
    x, y, z = _axes(c)
    gx, gy, gz = _global(c)
    gen, ph = _gen(seed), _phases(seed, 3 * ncomp)
    out = []
    for k in range(ncomp):
        p = 2 * math.pi * ph[3 * k:3 * k + 3]
        u = torch.sin(2 * math.pi * x + p[0]) * torch.sin(2 * math.pi * y + p[1]) * torch.cos(2 * math.pi * z + p[2])
        u += _noise((gz, gy, gx), gen, 1e-3)
        out.append(u.to(TDT[c["dtype"]]))
    return out


WALL = 0.25  # Dirichlet value of the scalar cases' z walls


def _scalar_bcs(c, grid):
    if c["bc"] == "walls":
        for comp in range(grid.ncomp):
            for s in (0, 1):
                grid.push_boundary_bc(lambda d, s: cn.BC.Absorbing(d, s), 1, s, comp=comp)
                grid.push_boundary_bc(lambda d, s: cn.BC.Dirichlet(d, s, WALL), 2, s, comp=comp)
        grid.sync_bcs()


def _pad(a, lo, hi, bc, wall):
    """a (nz, ny, nx) with lo ghost cells below and hi above per direction
    (edges of walls in the order x, y, z: only faces are used there)."""
    def ext(v, dim, mode):
        m = v.shape[dim]
        if mode == "wrap":
            i = torch.arange(-lo, m + hi, device=v.device) % m
            return v.index_select(dim, i)
        if mode == "edge":
            i = torch.arange(-lo, m + hi, device=v.device).clamp(0, m - 1)
            return v.index_select(dim, i)
        s = list(v.shape)
        s[dim] = m + lo + hi
        w = torch.full(s, wall, dtype=v.dtype, device=v.device)
        w.narrow(dim, lo, m).copy_(v)
        return w
    a = ext(a, 2, "wrap")
    a = ext(a, 1, "wrap" if bc == "periodic" else "edge")
    return ext(a, 0, "wrap" if bc == "periodic" else "const")


# ----------------------------------------------------------------- Euler
def _far():
    return (1.0, 0.0, 0.0, 0.0, 1.0 / (GAMMA - 1.0))


def _pulse(r2, gen, seed, dtype):
    """Conservative state of a density pulse with velocity noise, p = 1."""
    ph = _phases(seed, 5)
    rho = torch.exp(r2 / (-2 * 0.1 ** 2)).mul_(0.4 + 0.2 * ph[3]).add_(1.0)
    vel = [_noise(rho.shape, gen, 1e-2) for _ in range(3)]
    ke = (vel[0] ** 2 + vel[1] ** 2 + vel[2] ** 2).mul_(rho).mul_(0.5)
    state = [rho.to(dtype)] + [(rho * v).to(dtype) for v in vel]
    state.append(ke.add_(1.0 / (GAMMA - 1.0)).to(dtype))
    return state


def _euler_state(c, seed):
    x, y, z = _axes(c)
    end, ph = _end(c), _phases(seed, 5)
    r2 = sum((a - e * (0.4 + 0.2 * q)) ** 2 for a, e, q in zip((x, y, z), end, ph))
    return _pulse(r2, _gen(seed), seed, TDT[c["dtype"]])


def _euler_dt(h):
    # CFL 0.3 of the pulse's fastest signals (sound speed at rho = 1 plus the noise)
    return 0.3 * h / (3 * (math.sqrt(GAMMA) + 1e-2))


def _euler_bcs(c, U):
    if c["bc"] == "walls":
        for comp, v in enumerate(_far()):
            for s in (0, 1):
                U.push_boundary_bc(lambda d, s: cn.BC.Absorbing(d, s), 1, s, comp=comp)
                U.push_boundary_bc(lambda d, s, v=v: cn.BC.Dirichlet(d, s, v), 2, s, comp=comp)
        U.sync_bcs()


def _primitive(U):
    rho, m0, m1, m2, E = U
    u, v, w = m0 / rho, m1 / rho, m2 / rho
    return rho, u, v, w, (GAMMA - 1) * (E - 0.5 * (m0 * u + m1 * v + m2 * w))


def _weno(a, b, c, d, e):
    """WENO5-JS value at the upper face of cell c from cells a .. e."""
    q0 = (2 * a - 7 * b + 11 * c) / 6
    q1 = (-b + 5 * c + 2 * d) / 6
    q2 = (2 * c + 5 * d - e) / 6
    s0 = 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2
    s1 = 13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2
    s2 = 13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2
    w0, w1, w2 = 0.1 / (1e-6 + s0) ** 2, 0.6 / (1e-6 + s1) ** 2, 0.3 / (1e-6 + s2) ** 2
    return (w0 * q0 + w1 * q1 + w2 * q2) / (w0 + w1 + w2)


def _flux(W, d):
    rho, p, un = W[0], W[4], W[1 + d]
    E = p / (GAMMA - 1) + 0.5 * rho * (W[1] ** 2 + W[2] ** 2 + W[3] ** 2)
    U = [rho, rho * W[1], rho * W[2], rho * W[3], E]
    F = [u * un for u in U]
    F[1 + d] = F[1 + d] + p
    F[4] = F[4] + p * un
    return U, F, un.abs() + torch.sqrt(GAMMA * p / rho)


def _rhs(lab, h):
    """-div F on the inner cells of a lab (5 x ... x z x y x x) with 3 ghosts a side."""
    W = _primitive(lab)
    out = None
    for d in range(3):
        ax = -1 - d

        def inner(v):
            for o in (-1, -2, -3):
                if o != ax:
                    v = v.narrow(o, 3, v.shape[o] - 6)
            return v
        V = [inner(v) for v in W]
        m = V[0].shape[ax] - 6  # inner cells along d
        left, right = [], []
        for v in V:
            s = [v.narrow(ax, k, m + 1) for k in range(6)]  # cells f-3 .. f+2 of face f
            left.append(_weno(*s[:5]))
            right.append(_weno(*s[:0:-1]))
        UL, FL, aL = _flux(left, d)
        UR, FR, aR = _flux(right, d)
        a = torch.maximum(aL, aR)
        div = []
        for ul, ur, fl, fr in zip(UL, UR, FL, FR):
            F = 0.5 * (fl + fr) - 0.5 * a * (ur - ul)
            div.append((F.narrow(ax, 1, m) - F.narrow(ax, 0, m)) / h)
        out = div if out is None else [o + v for o, v in zip(out, div)]
    return [-o for o in out]


def _rk3(U, dt, rhs):
    """SSP-RK3 (Shu & Osher); rhs(U) gives the list of right-hand sides."""
    U1 = [u + dt * r for u, r in zip(U, rhs(U))]
    U2 = [0.75 * u + 0.25 * (v + dt * r) for u, v, r in zip(U, U1, rhs(U1))]
    del U1
    return [u / 3 + 2 / 3 * (v + dt * r) for u, v, r in zip(U, U2, rhs(U2))]


def _euler_rhs_global(c):
    far = _far()

    def rhs(U):
        out = [torch.empty_like(u) for u in U]
        nz = U[0].shape[0]
        pad = [_pad(u, 3, 3, c["bc"], far[k]) for k, u in enumerate(U)]
        step = max(1, (1 << 23) // (U[0].shape[1] * U[0].shape[2]))
        for z in range(0, nz, step):
            m = min(step, nz - z)
            for o, r in zip(out, _rhs([p[z:z + m + 6] for p in pad], _h(c))):
                o[z:z + m] = r
        return out
    return rhs


# ------------------------------------------------------------------- AMR
def _amr_layout(c):
    """Blocks on two levels: root cubes of 64 level-1 cells; inside a ball the
    layout is refined to level 1, and cubes are split near its surface and,
    now and then, elsewhere.  Returns levels, cells, origins, box extents."""
    L = tuple(64 * c["r%d" % d] for d in range(3))
    rng = np.random.default_rng(11)
    centre = (0.4 + 0.2 * rng.random(3)) * np.array(L)
    R = c["radius"] * min(L)
    levels, cells, origins = [], [], []

    def side(o, e):
        """1: the cube lies inside the ball, -1: outside, 0: across its surface."""
        o = np.array(o)
        near = np.clip(centre, o, o + e)
        far = np.where(centre - o > e / 2, o, o + e)
        if np.sum((far - centre) ** 2) <= R * R:
            return 1
        return -1 if np.sum((near - centre) ** 2) >= R * R else 0

    def place(level, e, o):
        levels.append(level)
        cells.append(e if level else e // 2)
        origins.append(o)

    def visit(o, e):
        s = side(o, e)
        keep = rng.random()
        if e == 8:
            return place(1, 8, o)
        if e == 16 and s < 0:
            return place(0, 16, o)
        if e == 16 and keep < 0.8 or e == 32 and s > 0 and keep < 0.8:
            return place(1, e, o)
        if s < 0 and keep < 0.8:
            return place(0, e, o)
        half = e // 2
        for q in range(8):
            visit((o[0] + (q & 1) * half, o[1] + ((q >> 1) & 1) * half, o[2] + (q >> 2) * half), half)

    for k in range(c["r2"]):
        for j in range(c["r1"]):
            for i in range(c["r0"]):
                visit((64 * i, 64 * j, 64 * k), 64)
    return np.array(levels), np.array(cells), np.array(origins), L


def _amr_groups(layout):
    """Blocks of one level and size, as (level, n, block numbers)."""
    levels, cells, _, _ = layout
    for lev in (0, 1):
        for n in (8, 16, 32):
            ids = np.flatnonzero((levels == lev) & (cells == n))
            if len(ids):
                yield lev, n, ids


def _amr_state(c, seed, layout):
    """The pulse state in block order, each block's cells x fastest."""
    levels, cells, origins, L = layout
    off = np.concatenate([[0], np.cumsum(cells.astype(np.int64) ** 3)])
    r2 = torch.empty(int(off[-1]), device=DEV, dtype=F64)
    box = [v / L[0] for v in L]
    mid = [b * (0.4 + 0.2 * q) for b, q in zip(box, _phases(seed, 5))]
    for lev, n, ids in _amr_groups(layout):
        cs = 2 - lev
        i = (torch.arange(n, device=DEV, dtype=F64) + 0.5) * cs
        o = torch.tensor(origins[ids], device=DEV, dtype=F64)
        t = []
        for d in range(3):
            a = (o[:, d, None] + i[None, :]) / L[0] - mid[d]
            t.append((a - box[d] * torch.round(a / box[d])) ** 2)
        v = t[2][:, :, None, None] + t[1][:, None, :, None] + t[0][:, None, None, :]
        at = torch.tensor(off[ids], device=DEV)[:, None] + torch.arange(n ** 3, device=DEV)[None, :]
        r2[at] = v.reshape(len(ids), -1)
    return _pulse(r2, _gen(seed), seed, TDT[c["dtype"]])


def _amr_rhs(layout):
    """Right-hand side on a layout in plain torch: ghosts by copy, trilinear
    prolongation (3/4, 1/4 per direction, clamped to the source block) or the
    mean of 8 children."""
    levels, cells, origins, L = layout
    t = lambda a: torch.tensor(np.asarray(a), device=DEV, dtype=torch.int64)  # noqa: E731
    off = t(np.concatenate([[0], np.cumsum(cells.astype(np.int64) ** 3)]))
    lev_t, n_t, org = t(levels), t(cells), t(origins)
    look = np.zeros((L[2] // 8, L[1] // 8, L[0] // 8), dtype=np.int64)
    for b, (lv, n, o) in enumerate(zip(levels, cells, origins)):
        e = int(n) * (2 - int(lv)) // 8
        x, y, z = (int(v) // 8 for v in o)
        look[z:z + e, y:y + e, x:x + e] = b
    look = t(look)

    def plan(lev, n, ids):
        cs = 2 - lev
        q = torch.arange(-3, n + 3, device=DEV) * cs
        b = t(ids)
        X = [((org[b, d][:, None] + q[None, :]) % L[d]) for d in range(3)]
        E = n + 6
        shape = (len(ids), E, E, E)
        x = X[0][:, None, None, :].expand(shape).reshape(-1)
        y = X[1][:, None, :, None].expand(shape).reshape(-1)
        z = X[2][:, :, None, None].expand(shape).reshape(-1)
        s = look[z // 8, y // 8, x // 8]
        f = [x - org[s, 0], y - org[s, 1], z - org[s, 2]]
        same = lev_t[s] == lev
        css = 2 - lev_t[s]

        def at(s, p):
            return off[s] + p[0] + n_t[s] * (p[1] + n_t[s] * p[2])
        base = at(s, [v // css for v in f])
        other = torch.nonzero(~same).reshape(-1)
        so, fo = s[other], [v[other] for v in f]
        idx, wgt = [], []
        for k in range(8):
            if lev == 1:  # coarse source
                p = [v // 2 for v in fo]
                w = 1.0
                for d in range(3):
                    if (k >> d) & 1:
                        p[d] = torch.minimum((p[d] + 2 * (fo[d] % 2) - 1).clamp(min=0), n_t[so] - 1)
                        w *= 0.25
                    else:
                        w *= 0.75
            else:
                p, w = [fo[d] + ((k >> d) & 1) for d in range(3)], 0.125
            idx.append(at(so, p))
            wgt.append(w)
        return shape, base, other, idx, wgt

    def rhs(U):
        out = [torch.empty_like(u) for u in U]
        for lev, n, all_ids in _amr_groups(layout):
            for ids in np.array_split(all_ids, max(1, len(all_ids) * (n + 6) ** 3 // (1 << 23))):
                shape, base, other, idx, wgt = plan(lev, n, ids)
                labs = []
                for u in U:
                    v = u[base.clamp(max=u.numel() - 1)]
                    if other.numel():
                        v[other] = sum(w * u[i] for w, i in zip(wgt, idx))
                    labs.append(v.reshape(shape))
                at = off[t(ids)][:, None] + torch.arange(n ** 3, device=DEV)[None, :]
                for o, r in zip(out, _rhs(labs, (2 - lev) / L[0])):
                    o[at] = r.reshape(len(ids), -1)
        return out
    return rhs


# --------------------------------------------------------------- Poisson
def _poisson_inputs(c, seed):
    """k: smoothed log-normal (sigma 0.5), f: 32 Gaussians, mean removed (FP32)."""
    N = c["nb"] * c["n"]
    gen = _gen(seed)
    a = torch.exp(torch.randn((N, N, N), generator=gen, device=DEV, dtype=F64) * 0.5)
    for dim in range(3):
        a = (torch.roll(a, 1, dim) + a + torch.roll(a, -1, dim)) / 3.0
    rng = np.random.default_rng([int(seed), 7])
    g = (torch.arange(N, device=DEV, dtype=F64) + 0.5) / N
    f = torch.zeros((N, N, N), device=DEV, dtype=F64)
    for _ in range(32):
        m, w, s = rng.random(3), 0.02 + 0.06 * rng.random(), 2 * rng.random() - 1
        e = []
        for d in range(3):
            t = g - m[d]
            t = t - torch.round(t)
            e.append(torch.exp(t * t / (-2 * w * w)))
        f += s * e[2][:, None, None] * e[1][None, :, None] * e[0][None, None, :]
    f -= f.mean()
    return a.to(torch.float32), f.to(torch.float32)


def _poisson_exact(k, f, N):
    """Conjugate gradients in FP64, preconditioned by the constant-coefficient
    operator (FFT); the solution of zero mean."""
    k, f = k.to(F64), f.to(F64)
    ih2 = float(N) ** 2
    kf = []
    for dim in (2, 1, 0):
        kn = torch.roll(k, -1, dim)
        kf.append(2 * k * kn / (k + kn))

    def A(p):  # -L p
        out = torch.zeros_like(p)
        for dim, kk in zip((2, 1, 0), kf):
            g = kk * (torch.roll(p, -1, dim) - p)
            out += torch.roll(g, 1, dim) - g
        return out * ih2
    w = 2 - 2 * torch.cos(2 * math.pi * torch.arange(N, device=DEV, dtype=F64) / N)
    lam = (w[:, None, None] + w[None, :, None] + w[None, None, :N // 2 + 1]) * ih2 * float(k.mean())
    lam[0, 0, 0] = 1.0

    def M(r):
        z = torch.fft.rfftn(r) / lam
        z[0, 0, 0] = 0
        return torch.fft.irfftn(z, s=r.shape)
    b = -(f - f.mean())
    x = torch.zeros_like(b)
    r = b.clone()
    z = M(r)
    p = z.clone()
    rz = (r * z).sum()
    stop = 1e-12 * b.norm()
    for _ in range(200):
        q = A(p)
        a = rz / (p * q).sum()
        x += a * p
        r -= a * q
        if r.norm() <= stop:
            break
        z = M(r)
        rz, old = (r * z).sum(), rz
        p = z + (rz / old) * p
    return x - x.mean()


# --------------------------------------------------------------- learned
def _learned_inputs(c, seed):
    """Patches as the smoother's training sees them: residuals, their Jacobi
    correction x0 = -r / D, x1 = x0 ln k and the coefficient (FP32)."""
    B, P = c["batch"], c["patch"]
    gen = _gen(seed)
    S = P + 8

    def smooth(a):
        for dim in (1, 2, 3):
            a = (torch.roll(a, 1, dim) + a + torch.roll(a, -1, dim)) / 3.0
        return a
    k = smooth(torch.exp(torch.randn((B, S, S, S), generator=gen, device=DEV, dtype=F64) * 0.5))
    r = smooth(torch.randn((B, S, S, S), generator=gen, device=DEV, dtype=F64))
    ih2 = float(8 * P) ** 2
    x0 = -r / (6 * ih2 * k)
    x0 = x0 * ih2  # patches are scaled with the operator: ih2 = 1 in the loss
    x = torch.stack([x0, x0 * torch.log(k)], 1)
    f = lambda a: a.to(torch.float32).reshape(B, -1).contiguous()  # noqa: E731
    kk, rr = k[:, 3:-3, 3:-3, 3:-3], r[:, 4:-4, 4:-4, 4:-4]
    return x.to(torch.float32).reshape(B, 2, -1).contiguous(), f(kk), f(rr)


def _learned_weights():
    rng = np.random.default_rng(3)
    return [(rng.standard_normal(s) * a).astype(np.float32)
            for s, a in (((27, 2, 16), 0.2), ((27, 16, 16), 0.07), ((27, 16, 1), 0.01))]


OMEGA = 0.8


def _conv(x, W):
    """x (Ci, S, S, S) with W (27, Ci, Co), valid."""
    S = x.shape[1] - 2
    out = None
    for t in range(27):
        dx, dy, dz = t % 3, (t // 3) % 3, t // 9
        v = x[:, dz:dz + S, dy:dy + S, dx:dx + S].reshape(x.shape[0], -1)
        o = W[t].t() @ v
        out = o if out is None else out + o
    return out.reshape(W.shape[2], S, S, S)


def _learned_exact(c, seed):
    B, P = c["batch"], c["patch"]
    x, k, r = (a.to(F64) for a in _learned_inputs(c, seed))
    x, k, r = x.reshape(B, 2, P + 8, P + 8, P + 8), k.reshape(B, P + 2, P + 2, P + 2), r.reshape(B, P, P, P)
    Ws = [torch.tensor(w, device=DEV, dtype=F64, requires_grad=True) for w in _learned_weights()]
    total = 0.0
    for b in range(B):
        y = _conv(torch.relu(_conv(torch.relu(_conv(x[b], Ws[0])), Ws[1])), Ws[2])[0]
        cc = OMEGA * x[b, 0, 3:-3, 3:-3, 3:-3] + y
        kb, m = k[b], slice(1, -1)
        res = r[b]
        for ax in range(3):
            up, dn = [m, m, m], [m, m, m]
            up[ax], dn[ax] = slice(2, None), slice(0, -2)
            up, dn = tuple(up), tuple(dn)
            mid = (m, m, m)
            kp = 2 * kb[mid] * kb[up] / (kb[mid] + kb[up])
            km = 2 * kb[mid] * kb[dn] / (kb[mid] + kb[dn])
            res = res - (kp * (cc[up] - cc[mid]) - km * (cc[mid] - cc[dn]))
        loss = (res ** 2).sum() / (r[b] ** 2).sum() / B
        loss.backward()
        total += float(loss.detach())
    return {"loss": total, "grads": [w.grad for w in Ws]}


# --------------------------------------------------------------- prepare
class _State:
    def __init__(self, case, **kw):
        self.case = case
        self.__dict__.update(kw)
        # the program's own views of its result grids
        self.out = kw["out"] if "out" in kw else [v for g in kw.get("results", ()) for v in _values(g)]


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "lab":
        g = _grid(c)
        _fill(g, _wave(c, seed, 1))
        _scalar_bcs(c, g)
        st = cn.Core.Stencil(c["lo"], c["hi"], c["tensorial"])
        E = [v - c["lo"] + c["hi"] - 1 for v in _n(c)]
        out = torch.zeros((c["count"], E[2], E[1], E[0]), dtype=TDT[c["dtype"]], device=DEV)
        return _State(c, grid=g, stencil=st, out=out)
    if kind == "fd":
        g = _grid(c, 3 if c["op"] == "div" else 1)
        _fill(g, _wave(c, seed, g.ncomp))
        _scalar_bcs(c, g)
        scalar = _grid(c) if c["op"] != "grad" else None
        vector = _grid(c, 3) if c["op"] in ("grad", "lap_grad") else None
        return _State(c, grid=g, scalar=scalar, vector=vector, results=[v for v in (scalar, vector) if v])
    if kind in ("euler", "loop"):
        U = _grid(c, 5)
        _fill(U, _euler_state(c, seed))
        _euler_bcs(c, U)
        return _State(c, U=U, w1=cn.euler.like(U), w2=cn.euler.like(U), dt=_euler_dt(_h(c)), results=[U])
    if kind == "amr":
        layout = _amr_layout(c)
        U = cn.amr.AmrGrid(*layout, ncomp=5, dtype=DT[c["dtype"]])
        for k, a in enumerate(_amr_state(c, seed, layout)):
            U.tensor(k).copy_(a)
        return _State(c, U=U, w1=U.like(), w2=U.like(), dt=_euler_dt(1.0 / layout[3][0]),
                      out=[_held(U.tensor(k), U) for k in range(5)])
    if kind == "poisson":
        nb, n = (c["nb"],) * 3, (c["n"],) * 3
        k = cn.Grid.Cartesian(nb, n, dtype=np.float32)
        f = cn.Grid.Cartesian(nb, n, dtype=np.float32)
        p = cn.Grid.Cartesian(nb, n, dtype=np.float64)
        ka, fa = _poisson_inputs(c, seed)
        _fill(k, [ka])
        _fill(f, [fa])
        torch.cuda.synchronize()
        return _State(c, f=f, p=p, results=[p], mg=cn.mg.Multigrid(k, nu1=2, nu2=2, omega=6.0 / 7.0))
    if kind == "io":
        g = _grid(c, c["ncomp"])
        _fill(g, _wave(c, seed, c["ncomp"]))
        gx, gy, gz = _global(c)
        shape = (gz, gy, gx, c["ncomp"])
        saved = torch.rand(shape, generator=_gen(seed + 1), device=DEV, dtype=TDT[c["file"]])
        back = _grid(c, c["ncomp"])
        return _State(c, grid=g, back=back, results=[back], saved=saved,
                      buf=torch.zeros(shape, dtype=TDT[c["file"]], device=DEV))
    x, k, r = _learned_inputs(c, seed)
    nn = cn.learned.LearnedSmoother(seed=1, omega=OMEGA)
    nn.set_weights(*_learned_weights())
    return _State(c, nn=nn, x=x, k=k, r=r)


def run(state):
    s, c = state, state.case
    kind = c["kind"]
    if kind == "lab":
        return cn.ops.load_labs(s.grid, s.stencil, s.out, 0, c["first"], c["count"])
    if kind == "fd":
        if c["op"] == "lap":
            cn.ops.laplacian(s.grid, s.scalar)
        elif c["op"] == "grad":
            cn.ops.gradient(s.grid, s.vector)
        elif c["op"] == "div":
            cn.ops.divergence(s.grid, s.scalar)
        else:
            cn.ops.lap_grad(s.grid, s.scalar, s.vector)
        return s.out
    if kind == "euler":
        cn.euler.rk3_step(s.U, s.w1, s.w2, s.dt)
        return s.out
    if kind == "loop":
        dt = cn.euler.cfl_dt(s.U, 0.3)
        sums = cn.euler.rk3_step(s.U, s.w1, s.w2, dt, want_sums=True)
        return {"state": s.out, "sums": sums, "dt": dt}
    if kind == "amr":
        cn.amr.rk3_step(s.U, s.w1, s.w2, s.dt)
        return s.out
    if kind == "poisson":
        s.mg.solve(s.f, s.p, rtol=1e-8, max_cycles=60)
        return s.out
    if kind == "io":
        cn.IO.Field2AOS(s.grid, file_dtype=DT[c["file"]], out=s.buf)
        cn.IO.AOS2Field(s.saved, s.back)
        return {"file": s.buf, "grid": s.out}
    loss, grads = s.nn.loss_grad(s.x, s.k, s.r, c["patch"], 1.0)
    return {"loss": loss, "grads": grads}


# ------------------------------------------------------------------ work
def work(case):
    c, kind = case, case["kind"]
    if kind == "learned":
        # three layers forward, three weight gradients, two data gradients
        B, P = c["batch"], c["patch"]
        c1, c2, c3 = (P + 6) ** 3, (P + 4) ** 3, (P + 2) ** 3
        macs = 27 * (2 * 32 * c1 + 3 * 256 * c2 + 3 * 16 * c3)
        return {"bytes": 4.0 * B * (2 * (P + 8) ** 3 + (P + 2) ** 3 + P ** 3), "flops": 2.0 * B * macs}
    if kind == "amr":
        layout = _amr_layout(c)
        cells = float(np.sum(layout[1].astype(np.int64) ** 3))
        return {"bytes": cells * 10 * np.dtype(DT[c["dtype"]]).itemsize, "flops": cells * 3 * 1000.0}
    if kind == "poisson":
        cells = float(c["nb"] * c["n"]) ** 3
        # f and k read, p written; about 15 V(2,2) cycles, each cell visited
        # 4 x 8/7 times by 15 operations of the smoother, twice by the residuals
        return {"bytes": 16 * cells, "flops": 15 * cells * 100.0}
    es = np.dtype(DT[c["dtype"]]).itemsize
    cells = float(np.prod(_global(c)))
    if kind == "lab":
        n, w = _n(c), c["hi"] - c["lo"] - 1
        lab = (n[0] + w) * (n[1] + w) * (n[2] + w) if c["tensorial"] else (
            n[0] * n[1] * n[2] + w * (n[0] * n[1] + n[1] * n[2] + n[0] * n[2]))
        return {"bytes": float(c["count"]) * es * (n[0] * n[1] * n[2] + lab), "flops": 0.0}
    if kind == "fd":
        io, ops = {"lap": (2, 13), "grad": (4, 9), "lap_grad": (5, 22), "div": (4, 9)}[c["op"]]
        return {"bytes": cells * es * io, "flops": cells * ops}
    if kind == "io":
        return {"bytes": 2 * cells * c["ncomp"] * (es + np.dtype(DT[c["file"]]).itemsize), "flops": 0.0}
    # one RK3 step: the state read and written once; about 1000 operations per cell and stage
    return {"bytes": cells * 10 * es, "flops": cells * 3 * 1000.0}


# ----------------------------------------------------------------- exact
def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "learned":
        return _learned_exact(c, seed)
    if kind == "amr":
        layout = _amr_layout(c)
        U = [u.to(F64) for u in _amr_state(c, seed, layout)]
        return _rk3(U, _euler_dt(1.0 / layout[3][0]), _amr_rhs(layout))
    if kind == "poisson":
        N = c["nb"] * c["n"]
        k, f = _poisson_inputs(c, seed)
        return [_to_blocks(_poisson_exact(k, f, N), (c["nb"],) * 3, (c["n"],) * 3)]
    nb, n = _nb(c), _n(c)
    if kind in ("euler", "loop"):
        U = [u.to(F64) for u in _euler_state(c, seed)]
        dt = _euler_dt(_h(c))
        if kind == "loop":
            W = _primitive(U)
            cs = torch.sqrt(GAMMA * W[4] / W[0])
            dt = 0.3 / sum(float((W[1 + d].abs() + cs).max()) / _h(c) for d in range(3))
        V = _rk3(U, dt, _euler_rhs_global(c))
        state = [_to_blocks(v, nb, n) for v in V]
        if kind == "euler":
            return state
        return {"state": state, "sums": [float(v.sum()) * _h(c) ** 3 for v in V], "dt": dt}
    u = [a.to(F64) for a in _wave(c, seed, {"fd": 3 if c.get("op") == "div" else 1, "lab": 1}.get(kind, c.get("ncomp")))]
    if kind == "io":
        gx, gy, gz = _global(c)
        saved = torch.rand((gz, gy, gx, c["ncomp"]), generator=_gen(seed + 1), device=DEV, dtype=TDT[c["file"]])
        back = saved.to(TDT[c["dtype"]]).to(F64)
        return {"file": torch.stack(u, -1), "grid": [_to_blocks(back[..., k], nb, n) for k in range(c["ncomp"])]}
    if kind == "lab":
        lo, hi = -c["lo"], c["hi"] - 1
        p = _pad(u[0], lo, hi, c["bc"], WALL)
        E = [v + lo + hi for v in n]
        out = torch.zeros((c["count"], E[2], E[1], E[0]), dtype=F64, device=DEV)
        for i in range(c["count"]):
            b = c["first"] + i
            x, y, z = b % nb[0] * n[0], b // nb[0] % nb[1] * n[1], b // (nb[0] * nb[1]) * n[2]
            out[i] = p[z:z + E[2], y:y + E[1], x:x + E[0]]
        if not c["tensorial"]:  # edges and corners are not part of the lab
            ghost = [(torch.arange(E[d], device=DEV) < lo) | (torch.arange(E[d], device=DEV) >= lo + n[d])
                     for d in range(3)]
            edge = (ghost[2][:, None, None].int() + ghost[1][None, :, None].int() + ghost[0][None, None, :].int()) > 1
            out.masked_fill_(edge[None], 0.0)
        return out
    ih = 1.0 / _h(c)
    p = [_pad(a, 1, 1, c["bc"], WALL) for a in u]
    m = slice(1, -1)

    def at(a, d, s):
        q = [m, m, m]
        q[2 - d] = slice(2, None) if s > 0 else slice(0, -2)
        return a[tuple(q)]

    def lap(a):
        return sum((at(a, d, 1) - 2 * a[m, m, m] + at(a, d, -1)) * ih * ih for d in range(3))

    def der(a, d):
        return 0.5 * ih * (at(a, d, 1) - at(a, d, -1))
    if c["op"] == "div":
        out = [sum(der(p[d], d) for d in range(3))]
    else:
        out = [] if c["op"] == "grad" else [lap(p[0])]
        if c["op"] != "lap":
            out += [der(p[0], d) for d in range(3)]
    return [_to_blocks(v, nb, n) for v in out]
