"""Learned smoother: device loss/gradients vs the numpy oracle (itself checked
by finite differences), training reduces the loss, and multigrid with the
trained smoother converges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# Tolerances of the tensor-core training path (BF16 hidden-layer weights,
# activations and activation gradients; FP32 accumulation) against the
# float64 oracle that rounds to BF16 at the same points: what is left is
# FP32 summation order and BF16 ties decided differently by a last-bit FP32
# difference.  Measured: loss 1.4e-6, gradients <= 1.1e-3 (3 x 4^3 patches)
# and <= 5.4e-5 (2 x 16^3); against the unrounded float64 oracle the same
# gradients differ by up to 4e-2 (the BF16 storage itself).
TOL_TC_LOSS = 1e-4
TOL_TC_GRAD = 5e-3


def _batch(B, P, seed):
    rng = np.random.default_rng(seed)
    S, R = P + 8, P + 2
    x = rng.standard_normal((B, 2, S, S, S))
    k = 0.5 + rng.random((B, R, R, R))
    r = rng.standard_normal((B, P, P, P))
    return x, k, r


def _device_loss_grad(nn, x, k, r, P, ih2):
    import torch
    B = x.shape[0]
    tx = torch.tensor(x, dtype=torch.float32, device="cuda").reshape(B, 2, -1).contiguous()
    tk = torch.tensor(k, dtype=torch.float32, device="cuda").reshape(B, -1).contiguous()
    tr = torch.tensor(r, dtype=torch.float32, device="cuda").reshape(B, -1).contiguous()
    return nn.loss_grad(tx, tk, tr, P, ih2)


def _rel(got, want):
    return float(np.max(np.abs(got - want)) / np.max(np.abs(want)))


def test_loss_and_gradient_match_oracle(cn):
    """FP32 CUDA-core training path against the float64 oracle."""
    from oracle import nn_oracle as N
    B, P = 3, 4
    x, k, r = _batch(B, P, 0)
    nn = cn.learned.LearnedSmoother(seed=3, omega=0.8, init_scale=0.05)
    nn.set_training("fp32")
    W1, W2, W3 = [w.astype(np.float64) for w in nn.weights()]
    ih2 = 16.0
    loss, (g1, g2, g3) = _device_loss_grad(nn, x, k, r, P, ih2)
    x32, k32, r32 = (a.astype(np.float32).astype(np.float64) for a in (x, k, r))
    wl, w1, w2, w3 = N.loss_and_grad(x32, k32, r32, W1, W2, W3, 0.8, ih2)
    assert abs(loss - wl) <= 1e-4 * abs(wl)
    for got, want in ((g1, w1), (g2, w2), (g3, w3)):
        err = _rel(got, want)
        assert err < 1e-3, err
    assert N.fd_check(x32, k32, r32, W1, W2, W3, 0.8, ih2, n=4) < 1e-5


@pytest.mark.parametrize("B,P", [(3, 4), (2, 5), (2, 16)])
def test_tensor_core_training_matches_bf16_oracle(cn, B, P):
    """Tensor-core training path (tcgen05 forward, data gradient and weight
    gradient of the hidden layer) against the float64 oracle rounded to BF16
    where the device stores BF16; 3 x 4^3 patches end in partial 128-cell
    chunks (1536 and 3000 rows), 2 x 5^3 patches have odd cube sides (ragged
    bricks), 2 x 16^3 patches span many chunks."""
    from oracle import nn_oracle as N
    x, k, r = _batch(B, P, 7 + P)
    nn = cn.learned.LearnedSmoother(seed=5, omega=0.8, init_scale=0.05)
    nn.set_training("tensor")
    W1, W2, W3 = [w.astype(np.float64) for w in nn.weights()]
    ih2 = 16.0
    loss, grads = _device_loss_grad(nn, x, k, r, P, ih2)
    x32, k32, r32 = (a.astype(np.float32).astype(np.float64) for a in (x, k, r))
    bl, *bw = N.loss_and_grad(x32, k32, r32, W1, W2, W3, 0.8, ih2, bf16_path=True)
    pl, *pw = N.loss_and_grad(x32, k32, r32, W1, W2, W3, 0.8, ih2)
    errs = [_rel(g, w) for g, w in zip(grads, bw)]
    plain = [_rel(g, w) for g, w in zip(grads, pw)]
    print(f"B={B} P={P}: loss {loss:.6f} bf16-oracle {bl:.6f} fp64-oracle {pl:.6f}; "
          f"grad rel vs bf16 oracle {['%.2e' % e for e in errs]}, vs fp64 oracle {['%.2e' % e for e in plain]}")
    assert abs(loss - bl) <= TOL_TC_LOSS * abs(bl)
    for e in errs:
        assert e < TOL_TC_GRAD, errs


@pytest.mark.parametrize("B,P,offset", [(1, 1, 0), (5, 3, 0), (3, 7, 0), (2, 8, 1)])
def test_tensor_core_training_edges(cn, B, P, offset):
    """The first and last layers where their tiles end: cubes shorter than a
    run of cells along x or z, column groups with idle lanes, and inputs whose
    rows are not on 16-byte boundaries.  The tolerances of the other sizes."""
    import torch
    from oracle import nn_oracle as N
    x, k, r = _batch(B, P, 31 + P)
    nn = cn.learned.LearnedSmoother(seed=5, omega=0.8, init_scale=0.05)
    nn.set_training("tensor")
    W1, W2, W3 = [w.astype(np.float64) for w in nn.weights()]
    tx, tk, tr = (torch.tensor(a, dtype=torch.float32, device="cuda") for a in (x, k, r))
    buf = torch.zeros(offset + tx.numel(), dtype=torch.float32, device="cuda")
    buf[offset:] = tx.reshape(-1)
    loss, grads = nn.loss_grad(buf[offset:].view(B, 2, -1), tk.reshape(B, -1), tr.reshape(B, -1), P, 16.0)
    x32, k32, r32 = (a.astype(np.float32).astype(np.float64) for a in (x, k, r))
    want, *bw = N.loss_and_grad(x32, k32, r32, W1, W2, W3, 0.8, 16.0, bf16_path=True)
    assert abs(loss - want) <= TOL_TC_LOSS * abs(want)
    for g, w in zip(grads, bw):
        assert _rel(g, w) < TOL_TC_GRAD


def _fma32(a, b, c):
    """float32 fused multiply-add: the product is exact in float64, the sum is
    rounded to odd there, so that the rounding to float32 is the only one."""
    p, c = a.astype(np.float64) * b.astype(np.float64), c.astype(np.float64)
    s = p + c
    v = s - p
    err = (p - (s - v)) + (c - v)
    even = (s.view(np.int64) & 1) == 0
    s = np.where((err != 0) & even, np.nextafter(s, np.where(err > 0, np.inf, -np.inf)), s)
    return s.astype(np.float32)


def _bf16(v):
    u = np.ascontiguousarray(v, dtype=np.float32).view(np.uint32).astype(np.uint64)
    return (((u + 0x7FFF + ((u >> 16) & 1)) >> 16) << 16).astype(np.uint32).view(np.float32)


@pytest.mark.parametrize("B,P,seed", [(1, 1, 0), (1, 2, 1), (2, 5, 2), (3, 8, 3), (1, 8, 4), (2, 13, 5), (1, 30, 6),
                                      (1, 63, 7)])
def test_last_layer_sums_in_tap_order(cn, B, P, seed):
    """The last layer's forward and data gradient, bit for bit in the order of
    one cell at a time: taps x fastest, then y, then z, the channels of a tap in
    turn, one chain of fused multiply-adds per result.  Both come before BF16
    roundings, so another order shows in the gradients.

    One cell of h1 is 1 and all others are 0, so h2 is W2 (in BF16) in the 27
    cells around it, and the gradient of W2 is gh2 there, single exact products.
    With k = 1, ih2 = 1, omega = 0 and r = +-1 near that cell, the loss kernels'
    float32 operations have one order and no rounding that a contraction changes;
    the loss (sums in float64) then shows any last bit of y."""
    import torch
    rng = np.random.default_rng(100 + seed)
    S, S1, R = P + 8, P + 6, P + 2
    active = B - 1
    ends = (2, S1 - 3)  # 27 cells of h2 around the h1 cell: [2, S1 - 3]
    c = np.array([ends[seed % 2], int(rng.integers(2, S1 - 2)), ends[(seed // 2) % 2]])  # x, y, z
    W1 = np.zeros((27, 2, 16), np.float32)
    W1[13, 0, 0] = 1.0
    W2 = np.zeros((27, 16, 16), np.float32)
    W2[:, 0, :] = _bf16(rng.uniform(0.5, 1.5, (27, 16)).astype(np.float32))
    W3 = rng.standard_normal((27, 16, 1)).astype(np.float32)
    nn = cn.learned.LearnedSmoother(seed=1, omega=0.0, init_scale=0.05)
    nn.set_training("tensor")
    nn.set_weights(W1, W2, W3)
    x = np.zeros((B, 2, S, S, S), np.float32)
    x[active, 0, c[2] + 1, c[1] + 1, c[0] + 1] = 1.0
    r = np.zeros((B, P, P, P), np.float32)
    lo, hi = np.maximum(c - 6, 0), np.minimum(c + 2, P)
    win = tuple(slice(lo[d], hi[d]) for d in (2, 1, 0))
    r[active][win] = rng.choice(np.array([-1.0, 1.0], np.float32), size=r[active][win].shape)
    t = lambda a: torch.tensor(a, device="cuda").reshape(B, -1).contiguous()
    loss, grads = nn.loss_grad(t(x), t(np.ones((B, R, R, R), np.float32)), t(r), P, 1.0)

    # the same in float32, [z][y][x] windows of the whole cubes padded by zeros
    h2 = np.zeros((P + 4,) * 3 + (16,), np.float32)
    taps = [(q % 3, (q // 3) % 3, q // 9) for q in range(27)]
    for q, d in enumerate(taps):
        h2[c[2] - d[2], c[1] - d[1], c[0] - d[0]] = W2[q, 0]
    y = np.zeros((R, R, R), np.float32)
    a, b = np.maximum(c - 4, 0), np.minimum(c + 1, R)
    acc = np.zeros(tuple((b - a)[::-1]), np.float32)
    for q, d in enumerate(taps):
        v = h2[a[2] + d[2]:b[2] + d[2], a[1] + d[1]:b[1] + d[1], a[0] + d[0]:b[0] + d[0]]
        for i in range(16):
            acc = _fma32(v[..., i], W3[q, i], acc)
    y[a[2]:b[2], a[1]:b[1], a[0]:b[0]] = acc
    m = y[1:-1, 1:-1, 1:-1]
    f = [(y[1:-1, 1:-1, 2:] - m) - (m - y[1:-1, 1:-1, :-2]), (y[1:-1, 2:, 1:-1] - m) - (m - y[1:-1, :-2, 1:-1]),
         (y[2:, 1:-1, 1:-1] - m) - (m - y[:-2, 1:-1, 1:-1])]
    e = r[active] - ((f[0] + f[1]) + f[2])
    rr = float(np.sum(r[active].astype(np.float64) ** 2))
    want = float(np.sum(e.astype(np.float64) ** 2)) / rr / B
    ep = np.pad(e, 2)  # e at (z, y, x) of the cube of side R is ep[z + 1, y + 1, x + 1]
    g = ep[1:-1, 1:-1, 1:-1] * np.float32(-6.0)
    for o in ((0, 0, 1), (0, 0, -1), (0, 1, 0), (0, -1, 0), (1, 0, 0), (-1, 0, 0)):
        g = g + ep[1 + o[0]:R + 1 + o[0], 1 + o[1]:R + 1 + o[1], 1 + o[2]:R + 1 + o[2]]
    g = np.float32(-2.0 / (rr * B)) * g
    gp = np.pad(g, 2)  # gc at c - 2 + e of h2's cell c is gp[c + e]
    for q, d in enumerate(taps):
        cell = c - np.array(d)
        acc = np.zeros(16, np.float32)
        for e_, s in enumerate(taps):
            v = gp[cell[2] + s[2], cell[1] + s[1], cell[0] + s[0]]
            acc = _fma32(np.full(16, v, np.float32), W3[26 - e_, :, 0], acc)
        assert np.array_equal(grads[1][q, 0], _bf16(acc)), (q, grads[1][q, 0], _bf16(acc))
    # the float64 sums' own rounding: at most 9^3 terms
    assert abs(loss - want) <= 1e-12 * want, (loss, want)


def test_tensor_core_training_step_matches_fp32(cn):
    """One Adam step from the same weights with either training path moves
    the weights the same way (BF16 gradients point where the FP32 ones do)."""
    B, P = 4, 8
    x, k, r = _batch(B, P, 11)
    a = cn.learned.LearnedSmoother(seed=2, omega=0.8, init_scale=0.05)
    b = cn.learned.LearnedSmoother(seed=2, omega=0.8, init_scale=0.05)
    a.set_training("fp32")
    b.set_training("tensor")
    _, ga = _device_loss_grad(a, x, k, r, P, 4.0)
    _, gb = _device_loss_grad(b, x, k, r, P, 4.0)
    for u, v in zip(ga, gb):
        cos = float(np.dot(u.ravel(), v.ravel()) / (np.linalg.norm(u) * np.linalg.norm(v)))
        assert cos > 0.99, cos


def _poisson(cn, nb, n, seed=1):
    k = cn.Grid.Cartesian(nb, n, dtype=np.float32)
    cn.workloads.poisson_coefficient(k, seed=seed)
    f = cn.Grid.Cartesian(nb, n, dtype=np.float32)
    cn.workloads.poisson_rhs(f, seed=seed + 1)
    return k, f


def test_training_and_learned_multigrid(cn):
    import torch
    nb, n = (4, 4, 4), (16, 16, 16)
    k, f = _poisson(cn, nb, n)
    m = cn.mg.Multigrid(k, nu1=2, nu2=2, omega=0.8)
    x, kk, r, P = cn.learned.collect_patches(m, f, cycles=6, per_snapshot=16, max_patches=192, seed=5)
    assert x.shape[0] == 192
    nn = cn.learned.LearnedSmoother(seed=1, omega=0.8, init_scale=1e-3)
    ih2 = 1.0 / k.getCellSize()[0] ** 2
    l0, _ = nn.loss_grad(x[:32], kk[:32], r[:32], P, ih2)
    last = nn.train(x, kk, r, P, ih2, epochs=8, batch=16, lr=2e-3, seed=2)
    l1, _ = nn.loss_grad(x[:32], kk[:32], r[:32], P, ih2)
    print(f"loss before {l0:.4f} after {l1:.4f} (last epoch {last:.4f})")
    assert l1 < l0
    p64 = cn.Grid.Cartesian(nb, n, dtype=np.float64)
    cyc_plain, rel_plain = m.solve(f, p64, rtol=1e-8, max_cycles=60)
    # what training gains: the same network untrained (near-zero weights,
    # i.e. damped Jacobi) against the trained one, both replacing Jacobi on
    # the finest level, where the training residuals came from
    untrained = cn.learned.LearnedSmoother(seed=1, omega=0.8, init_scale=1e-3)
    cn.learned.use_in(m, untrained, level_mask=0x1)
    cyc_u, rel_u = m.solve(f, p64, rtol=1e-8, max_cycles=60)
    cn.learned.use_in(m, nn, level_mask=0x1)
    cyc_nn, rel_nn = m.solve(f, p64, rtol=1e-8, max_cycles=60)
    print(f"plain: {cyc_plain} cycles ({rel_plain:.2e}); untrained: {cyc_u} ({rel_u:.2e}); "
          f"trained: {cyc_nn} cycles ({rel_nn:.2e})")
    assert rel_nn <= 1e-8 and rel_u <= 1e-8 and rel_plain <= 1e-8
    rr, ff = m.residual(p64, f)
    assert np.sqrt(rr / ff) <= 1e-8
    # measured here: plain 15, untrained 15, trained 11 cycles
    assert cyc_nn <= cyc_plain - 2 and cyc_nn <= cyc_u - 2
