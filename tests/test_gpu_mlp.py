"""BF16 MLP kernels against the CPU oracle (oracle/mlp_oracle.py): forward,
loss gradient and every parameter gradient; a training smoke test; the IDW
kernel against eval/core.py's formula."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _setup(rows=512, seed=0):
    import torch
    from eulersr_b200.warmstart.mlp import MLP, K_IN
    m = MLP(seed=seed)
    g = torch.Generator().manual_seed(seed + 1)
    # non-zero head so gradients reach every layer
    m.view("W4").copy_((torch.randn(4, 256, generator=g) * 0.05).cuda())
    m.view("b4").copy_((torch.randn(4, generator=g) * 0.1).cuda())
    m.pb.copy_(m.p.to(torch.bfloat16))
    X = torch.zeros(rows, K_IN)
    X[:, :13] = torch.randn(rows, 13, generator=g)
    X = X.to(torch.bfloat16).cuda()
    base = (torch.randn(rows, 4, generator=g) * 0.5).cuda()
    tgt = (torch.randn(rows, 4, generator=g) * 0.5).cuda()
    w = (1 + torch.rand(rows, generator=g) * 4).cuda()
    inv_den = torch.tensor([1.3, 0.7, 2.0, 1.1]).cuda()
    return m, X, base, tgt, w, inv_den


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


def test_forward_backward_match_oracle():
    import torch
    from oracle import mlp_oracle as MO
    m, X, base, tgt, w, inv_den = _setup()
    y, acts = m.forward(X, base, keep=True)
    L, dpred = m.loss(y, tgt, w, inv_den)
    m.backward(acts, dpred)
    torch.cuda.synchronize()
    P = m.params_numpy()
    Xn = X.float().cpu().numpy()
    yo, ao = MO.forward(P, Xn, base.cpu().numpy())
    assert _rel(y.cpu().numpy(), yo) < 1e-3
    Lo, dyo = MO.loss_and_grad(yo, tgt.cpu().numpy(), w.cpu().numpy(), inv_den.cpu().numpy())
    assert abs(float(L.item()) - Lo) <= 1e-3 * Lo
    go = MO.backward(P, ao, dpred.cpu().numpy().astype(np.float64))
    gg = m.grads_numpy()
    for k in ("W4", "b4", "W3", "b3", "W2", "b2", "W1", "b1", "W0", "b0"):
        assert _rel(gg[k], go[k]) < 2e-2, (k, _rel(gg[k], go[k]))
    # the BF16 gradients also track exact float64 backpropagation
    y64, a64 = MO.forward(P, Xn, base.cpu().numpy(), bf16=False)
    _, dy64 = MO.loss_and_grad(y64, tgt.cpu().numpy(), w.cpu().numpy(), inv_den.cpu().numpy())
    g64 = MO.backward(P, a64, dy64, bf16=False)
    for k in ("W3", "W1", "W0"):
        assert _rel(gg[k], g64[k]) < 6e-2, (k, _rel(gg[k], g64[k]))


def test_training_reduces_loss():
    import torch
    m, X, base, tgt, w, inv_den = _setup(rows=2048, seed=3)
    # a learnable target: a smooth function of the inputs
    Xf = X.float()
    tgt = torch.stack([torch.tanh(Xf[:, 0] + 0.5 * Xf[:, 1]), Xf[:, 2] * 0.3, torch.sin(Xf[:, 3]),
                       0.2 * Xf[:, 4] ** 2], 1).contiguous()
    base = torch.zeros_like(tgt)
    losses = []
    for it in range(300):
        y, acts = m.forward(X, base, keep=True)
        L, dpred = m.loss(y, tgt, w, inv_den)
        m.backward(acts, dpred)
        m.adamw(lr=2e-3)
        losses.append(float(L.item()))
    assert losses[-1] < 0.2 * losses[0], (losses[0], losses[-1])


def test_idw_kernel_matches_formula():
    import torch
    from eulersr_b200 import _ffi as F
    from oracle import euler_oracle as O
    rng = np.random.default_rng(0)
    src = rng.standard_normal((300, 4)).astype(np.float32)
    idx = rng.integers(0, 300, (1000, 6)).astype(np.int32)
    dist = rng.uniform(1e-3, 0.5, (1000, 6)).astype(np.float32)
    ds, di, dd = (torch.from_numpy(a).cuda() for a in (src, idx, dist))
    out = torch.empty((1000, 4), dtype=torch.float32, device="cuda")
    F.check(F.lib().esr_idw_apply(C.c_void_p(ds.data_ptr()), 300, 4, C.c_void_p(di.data_ptr()),
                                  C.c_void_p(dd.data_ptr()), 1000, 6, C.c_void_p(out.data_ptr()), None))
    torch.cuda.synchronize()
    ref = O.idw_predict(src, idx, dist)
    assert np.max(np.abs(out.cpu().numpy() - ref)) <= 2e-6 * max(1.0, np.abs(ref).max())
    bad = C.c_int32(7)
    F.check(F.lib().esr_idw_status(C.byref(bad)))
    assert bad.value == 0


def test_idw_kernel_refuses_out_of_range_indices():
    """A neighbour index outside [0, n_src) is never dereferenced: its row
    comes out NaN, the other rows are unchanged, and the status flag reports
    it once (reading it clears it)."""
    import torch
    from eulersr_b200 import _ffi as F
    from oracle import euler_oracle as O
    rng = np.random.default_rng(1)
    src = rng.standard_normal((50, 4)).astype(np.float32)
    idx = rng.integers(0, 50, (64, 6)).astype(np.int32)
    idx[5, 2] = 50          # one past the end
    idx[9, 0] = -1          # negative
    dist = rng.uniform(1e-3, 0.5, (64, 6)).astype(np.float32)
    ds, di, dd = (torch.from_numpy(a).cuda() for a in (src, idx, dist))
    out = torch.empty((64, 4), dtype=torch.float32, device="cuda")
    F.check(F.lib().esr_idw_apply(C.c_void_p(ds.data_ptr()), 50, 4, C.c_void_p(di.data_ptr()),
                                  C.c_void_p(dd.data_ptr()), 64, 6, C.c_void_p(out.data_ptr()), None))
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    assert np.isnan(got[[5, 9]]).all()
    good = np.setdiff1d(np.arange(64), [5, 9])
    ref = O.idw_predict(src, idx[good], dist[good])
    assert np.max(np.abs(got[good] - ref)) <= 2e-6 * max(1.0, np.abs(ref).max())
    bad = C.c_int32(0)
    F.check(F.lib().esr_idw_status(C.byref(bad)))
    assert bad.value == 1
    F.check(F.lib().esr_idw_status(C.byref(bad)))
    assert bad.value == 0


def test_feature_and_decode_kernels_match_formula():
    """esr_mlp_features builds the 13 inputs of preprocessing/dataset.py:140-176
    (geometry statics, IDW primitives normalised by mu/sig, asinh of the IDW
    pressure gradient over sig_p, normalised Mach and alpha; zero padding) in
    BF16 plus the float32 IDW base; esr_mlp_decode turns normalised primitives
    back into conserved rows with the density/pressure floors."""
    import torch
    from eulersr_b200 import _ffi as F
    rng = np.random.default_rng(5)
    rows, ld = 777, 128
    stat5 = rng.standard_normal((rows, 5)).astype(np.float32)
    prim = (rng.standard_normal((rows, 4)) * [0.3, 0.5, 0.2, 0.4] + [1.0, 2.0, 0.1, 1.0]).astype(np.float32)
    gradp = (rng.standard_normal((rows, 2)) * 5.0).astype(np.float32)
    mu = np.array([1.1, 1.9, 0.05, 0.9], np.float32)
    sig = np.array([0.25, 0.6, 0.3, 0.5], np.float32)
    mach_n, aoa_n = np.float32(0.37), np.float32(-0.6)
    d = {k: torch.from_numpy(v).cuda() for k, v in dict(stat5=stat5, prim=prim, gradp=gradp, mu=mu, sig=sig).items()}
    X = torch.full((rows, ld), 7.0, dtype=torch.bfloat16, device="cuda")
    base = torch.empty((rows, 4), dtype=torch.float32, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())   # noqa: E731
    F.check(F.lib().esr_mlp_features(p(d["stat5"]), p(d["prim"]), p(d["gradp"]), rows, float(mach_n), float(aoa_n),
                                     p(d["mu"]), p(d["sig"]), ld, p(X), p(base), None))
    torch.cuda.synchronize()
    q = (prim - mu) / sig                                  # float32, correctly rounded on both sides
    assert np.array_equal(base.cpu().numpy(), q)
    want = np.zeros((rows, ld), np.float32)
    want[:, :5] = stat5
    want[:, 5:9] = q
    want[:, 9:11] = np.arcsinh(gradp / (sig[3] + np.float32(1e-8)))
    want[:, 11], want[:, 12] = mach_n, aoa_n
    got = X.float().cpu().numpy()
    bf = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(torch.bfloat16).float().numpy()   # noqa: E731
    assert np.array_equal(got[:, :9], bf(want[:, :9]))
    assert np.array_equal(got[:, 11:], bf(want[:, 11:]))
    # asinh may differ from numpy's in the last float32 bit: one BF16 step at most
    assert np.all(np.abs(got[:, 9:11] - bf(want[:, 9:11])) <= np.abs(bf(want[:, 9:11])) * 2.0 ** -7 + 1e-30)
    # decode: rho = max(q0 sig0 + mu0, floor), u, v, p = max(q3 sig3 + mu3, floor) -> conserved float64
    pred = rng.standard_normal((rows, 4)).astype(np.float32)
    pred[:5, 0] = -10.0                                    # density below the floor
    pred[5:10, 3] = -10.0                                  # pressure below the floor
    W = torch.empty((rows, 4), dtype=torch.float64, device="cuda")
    dp = torch.from_numpy(pred).cuda()
    F.check(F.lib().esr_mlp_decode(p(dp), rows, p(d["mu"]), p(d["sig"]), 1.4, 0.05, 0.05, p(W), None))
    torch.cuda.synchronize()
    r = np.maximum(pred[:, 0].astype(np.float64) * sig[0] + mu[0], 0.05)
    u = pred[:, 1].astype(np.float64) * sig[1] + mu[1]
    v = pred[:, 2].astype(np.float64) * sig[2] + mu[2]
    pr = np.maximum(pred[:, 3].astype(np.float64) * sig[3] + mu[3], 0.05)
    ref = np.stack([r, r * u, r * v, pr / 0.4 + 0.5 * r * (u * u + v * v)], 1)
    assert np.allclose(W.cpu().numpy(), ref, rtol=2e-6, atol=1e-6)
    assert np.all(W.cpu().numpy()[:5, 0] == np.float32(0.05))


@pytest.mark.parametrize("ta,tb,epi,M,N,K,splits", [
    (0, 0, 1, 256, 256, 256, 1),     # forward: z = X W^T + b, h = res + relu(z)
    (0, 0, 1, 128, 256, 128, 1),     # input layer (K = 128)
    (0, 1, 2, 256, 128, 256, 1),     # backward dX with the relu mask
    (1, 1, 0, 256, 128, 512, 2),     # weight gradient, split-K partials
    (1, 1, 0, 128, 256, 2048, 4),    # long K: the stage barriers wrap several times
    (0, 0, 0, 256, 256, 192, 1),     # K-blocks = stages
    (0, 1, 0, 128, 256, 64, 1),      # a single K-block
    (0, 0, 2, 128, 128, 320, 1),
])
def test_tcgen05_gemm_matches_mma_sync(ta, tb, epi, M, N, K, splits):
    """The tcgen05 GEMM (operands in swizzled shared memory, accumulators in
    tensor memory) against the mma.sync kernel and a float64 product of the
    same BF16 operands, for every layout/epilogue the MLP uses."""
    import torch
    from eulersr_b200 import _ffi as F
    L = F.lib()
    g = torch.Generator().manual_seed(M + N + K + 7 * epi)
    A = torch.randn((K, M) if ta else (M, K), generator=g).to(torch.bfloat16).cuda()
    B = torch.randn((K, N) if tb else (N, K), generator=g).to(torch.bfloat16).cuda()
    bias = torch.randn(N, generator=g).cuda()
    res = torch.randn(M, N, generator=g).to(torch.bfloat16).cuda()
    aux = torch.randn(M, N, generator=g).to(torch.bfloat16).cuda()
    lda = M if ta else K
    ldb = N if tb else K
    p = lambda t: C.c_void_p(t.data_ptr()) if t is not None else None

    def run(fn):
        if epi == 0:
            o0, o1 = torch.zeros(splits, M, N, device="cuda"), None
        else:
            o0, o1 = torch.zeros(M, N, dtype=torch.bfloat16, device="cuda"), torch.zeros(M, N, dtype=torch.bfloat16, device="cuda")
        F.check(fn(ta, tb, M, N, K, p(A), lda, p(B), ldb, epi, p(bias) if epi == 1 else None,
                   p(res) if epi else None, p(aux) if epi == 2 else None, p(o0), p(o1), N, splits, None))
        torch.cuda.synchronize()
        return o0, o1

    t0, t1 = run(L.esr_gemm_bf16)
    r0, r1 = run(L.esr_gemm_bf16_mma_sync)
    flag = C.c_int32(-1)
    F.check(L.esr_gemm_tc_status(C.byref(flag)))
    assert flag.value == 0
    Ad = A.double().cpu()
    Bd = B.double().cpu()
    ref = (Ad.T if ta else Ad) @ (Bd if tb else Bd.T)
    if epi == 0:
        got = t0.double().sum(0).cpu()
        assert _rel(got.numpy(), ref.numpy()) < 1e-5
        assert _rel(got.numpy(), r0.double().sum(0).cpu().numpy()) < 1e-5
    else:
        # BF16 outputs: both paths agree to BF16 rounding
        for a, b in ((t0, r0), (t1, r1)):
            assert _rel(a.float().cpu().numpy(), b.float().cpu().numpy()) < 4e-3
        if epi == 1:
            z = ref + bias.double().cpu()
            assert _rel(t1.double().cpu().numpy(), z.numpy()) < 4e-3


@pytest.mark.parametrize("rows,cols", [(1, 256), (7, 256), (129, 256), (1000, 256), (300, 40), (65, 7), (33, 264)])
@pytest.mark.parametrize("shift", [0, 1])
def test_column_sums_and_split_reduction_edges(rows, cols, shift):
    """esr_colsum_bf16 and esr_reduce_splits at the edges of their row lanes,
    column groups and split groups, on buffers aligned to 16 bytes and shifted
    by one element. Tolerance: float32 sums of at most 1,000 BF16 values of
    magnitude ~1 in 8 x 128 partial chains, 1e-5 of the sum of magnitudes."""
    import torch
    from eulersr_b200 import _ffi as F
    g = torch.Generator().manual_seed(rows)
    X = torch.randn(rows * cols + shift, generator=g).to(torch.bfloat16).cuda()[shift:]
    rpb = 100
    nb = (rows + rpb - 1) // rpb
    part = torch.full((nb, cols), float("nan"), device="cuda")
    out = torch.full((cols,), float("nan"), device="cuda")
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = lambda t: C.c_void_p(t.data_ptr())
    F.check(F.lib().esr_colsum_bf16(p(X), rows, cols, rpb, p(part), st))
    F.check(F.lib().esr_reduce_splits(p(part), nb, cols, cols, p(out), st))
    x = X.view(rows, cols).double()
    ref, mag = x.sum(0), x.abs().sum(0)
    assert torch.all((out.double() - ref).abs() <= 1e-5 * mag + 1e-12)
    for splits in (1, 7, 8, 9, 33):
        q = torch.randn(splits, cols + 3, generator=g).cuda()
        F.check(F.lib().esr_reduce_splits(p(q), splits, cols + 3, cols, p(out), st))
        r = q[:, :cols].double()
        assert torch.all((out.double() - r.sum(0)).abs() <= 1e-6 * r.abs().sum(0) + 1e-12)


@pytest.mark.parametrize("rows", [1, 15, 128, 1001])
@pytest.mark.parametrize("shift", [0, 1])
def test_head_kernels_edges(rows, shift):
    """The head's forward and backward at row counts around its blocks and
    warps, with aligned and shifted BF16 buffers, against float64. Tolerances:
    float32 sums of 256 (forward) or `rows` (weight gradient) products, 1e-5
    of the sum of magnitudes; dH and dZ are BF16 roundings, 2^-8 relative."""
    import torch
    from eulersr_b200 import _ffi as F
    K, rpb = 256, 128
    g = torch.Generator().manual_seed(rows + shift)
    bf = lambda: torch.randn(rows * K + shift, generator=g).to(torch.bfloat16).cuda()[shift:].view(rows, K)
    H, Z = bf(), bf()
    dH = torch.zeros(rows * K + shift, dtype=torch.bfloat16, device="cuda")[shift:].view(rows, K)
    dZ = torch.zeros_like(H) if not shift else torch.zeros(rows * K + 1, dtype=torch.bfloat16, device="cuda")[1:].view(rows, K)
    W, b = torch.randn(4, K, generator=g).cuda(), torch.randn(4, generator=g).cuda()
    dY, base = torch.randn(rows, 4, generator=g).cuda(), torch.randn(rows, 4, generator=g).cuda()
    y = torch.empty(rows, 4, device="cuda")
    nb = (rows + rpb - 1) // rpb
    part = torch.full((nb, 4 * K + 4), float("nan"), device="cuda")
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = lambda t: C.c_void_p(t.data_ptr())
    F.check(F.lib().esr_mlp_head_fwd(p(H), rows, K, p(W), p(b), p(base), p(y), st))
    h, w = H.double(), W.double()
    assert torch.all((y.double() - (h @ w.T + b + base)).abs() <= 1e-5 * (h.abs() @ w.abs().T + 1))
    F.check(F.lib().esr_mlp_head_bwd(p(dY), p(H), p(Z), rows, K, p(W), p(dH), p(dZ), p(part), rpb, st))
    dh = dY.double() @ w
    tol = 2.0 ** -8 * dh.abs() + 1e-5 * (dY.double().abs() @ w.abs())
    assert torch.all((dH.double() - dh).abs() <= tol)
    assert torch.all((dZ.double() - dh * (Z > 0)).abs() <= tol)
    tot = part.double().sum(0)
    gw, mag = dY.double().T @ h, dY.double().abs().T @ h.abs()
    assert torch.all((tot[:4 * K].view(4, K) - gw).abs() <= 1e-5 * mag + 1e-12)
    assert torch.all((tot[4 * K:] - dY.double().sum(0)).abs() <= 1e-5 * dY.double().abs().sum(0) + 1e-12)


def test_gemm_epilogue_aligned_and_shifted_buffers_agree():
    """The 16-byte epilogue and the element-pair one (outputs 4 bytes off the
    16-byte grid) write the same bits, forward and backward."""
    import torch
    from eulersr_b200 import _ffi as F
    M, N, K = 384, 256, 128
    g = torch.Generator().manual_seed(2)
    rnd = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16).cuda()
    A, B, res, aux = rnd(M, K), rnd(N, K), rnd(M, N), rnd(M, N)
    bias = torch.randn(N, generator=g).cuda()
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = lambda t: C.c_void_p(t.data_ptr())
    for epi in (1, 2):
        got = []
        for off in (0, 2):
            o0 = torch.zeros(M * N + off, dtype=torch.bfloat16, device="cuda")[off:]
            o1 = torch.zeros(M * N + off, dtype=torch.bfloat16, device="cuda")[off:]
            F.check(F.lib().esr_gemm_bf16(0, 0, M, N, K, p(A), K, p(B), K, epi, p(bias), p(res), p(aux), p(o0), p(o1),
                                          N, 1, st))
            got.append((o0.clone(), o1.clone()))
        assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
        assert got[0][1].abs().sum() > 0


@pytest.mark.parametrize("rows", [128, 384, 148 * 128, 149 * 128])
@pytest.mark.parametrize("with_base", [True, False])
def test_fused_forward_equals_layer_calls(rows, with_base):
    """esr_mlp_forward (one tile, a few, one per SM, and an odd number in pairs) gives the bits
    of the layer-by-layer GEMM and head calls: y, and h and z when kept."""
    import torch
    from eulersr_b200 import _ffi as F
    m, X, base, *_ = _setup(rows=rows, seed=5)
    base = base if with_base else None
    got = []
    for fused in (True, False):
        m.fused = fused
        y, acts = m.forward(X, base, keep=True)
        y2 = m.forward(X, base)
        assert torch.equal(y, y2)
        got.append([y.clone()] + [t.clone() for t in acts["h"] + acts["z"]])
    assert all(torch.equal(a, b) for a, b in zip(*got))
    bad = C.c_int32(-1)
    F.check(F.lib().esr_gemm_tc_status(C.byref(bad)))
    assert bad.value == 0


@pytest.mark.parametrize("rows,rows_out", [(1, 128), (127, 128), (128, 128), (300, 384)])
def test_warm_inputs_equal_separate_calls(rows, rows_out):
    """esr_warm_inputs gives the bits of two esr_idw_apply calls and
    esr_mlp_features, zero rows after the last, and the same NaN row and error
    flag for an out-of-range neighbour."""
    import torch
    from eulersr_b200 import _ffi as F
    L, n_src, ld = F.lib(), 50, 128
    g = torch.Generator().manual_seed(rows)
    f = lambda *s: torch.randn(*s, generator=g).cuda()
    prim, gradp, stat = f(n_src, 4), f(n_src, 2), f(rows, 5)
    idx = torch.randint(0, n_src, (rows, 6), generator=g, dtype=torch.int32).cuda()
    dist = torch.rand(rows, 6, generator=g).cuda()
    mu, sig = f(4), torch.rand(4, generator=g).cuda() + 0.5
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = lambda t: C.c_void_p(t.data_ptr())
    bad = C.c_int32(0)
    for wrong in (False, True):
        if wrong:
            idx[rows // 2, 3] = n_src
        ip, ig = torch.empty(rows, 4, device="cuda"), torch.empty(rows, 2, device="cuda")
        X0 = torch.zeros(rows_out, ld, dtype=torch.bfloat16, device="cuda")
        b0 = torch.zeros(rows_out, 4, device="cuda")
        F.check(L.esr_idw_apply(p(prim), n_src, 4, p(idx), p(dist), rows, 6, p(ip), st))
        F.check(L.esr_idw_apply(p(gradp), n_src, 2, p(idx), p(dist), rows, 6, p(ig), st))
        F.check(L.esr_mlp_features(p(stat), p(ip), p(ig), rows, 0.3, -0.2, p(mu), p(sig), ld, p(X0), p(b0), st))
        F.check(L.esr_idw_status(C.byref(bad)))
        assert bad.value == int(wrong)
        X1 = torch.full((rows_out, ld), 7.0, dtype=torch.bfloat16, device="cuda")
        b1 = torch.full((rows_out, 4), 7.0, device="cuda")
        F.check(L.esr_warm_inputs(p(prim), p(gradp), n_src, p(idx), p(dist), p(stat), rows, rows_out, 0.3, -0.2, p(mu),
                                  p(sig), ld, p(X1), p(b1), st))
        F.check(L.esr_idw_status(C.byref(bad)))
        assert bad.value == int(wrong)
        assert torch.equal(X0.view(torch.int16), X1.view(torch.int16))
        assert torch.equal(torch.nan_to_num(b0, 99.0), torch.nan_to_num(b1, 99.0))


@pytest.mark.parametrize("rows,splits", [(128, 1), (384, 1), (640, 2), (1024, 4), (1152, 9), (2816, 11), (5632, 22), (2688, 42)])
def test_batched_weight_gradients_equal_layer_calls(rows, splits):
    """esr_mlp_wgrad at one K-block per range, one to four ranges per block, a
    block with fewer, more ranges than fit one wave, and rings that wrap: the
    bits of the split-K GEMM and of the column sums of each layer."""
    import torch
    from eulersr_b200 import _ffi as F
    g = torch.Generator().manual_seed(rows + splits)
    rnd = lambda *s: (torch.randn(*s, generator=g) + 0.25).to(torch.bfloat16).cuda()
    dz = [rnd(rows, 256) for _ in range(4)]
    src = [rnd(rows, 128)] + [rnd(rows, 256) for _ in range(3)]
    nblk = (rows + 255) // 256
    sums = splits == 1 or rows // splits % 256 == 0
    new = lambda: ([torch.full((splits, 256, s.shape[1]), float("nan"), device="cuda") for s in src],
                   torch.full((4, nblk, 256), float("nan"), device="cuda"))
    dw, db = new()
    want, wantb = new()
    arr = lambda ts: (C.c_void_p * 4)(*[t.data_ptr() for t in ts])
    p = lambda t: C.c_void_p(t.data_ptr())
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    L = F.lib()
    F.check(L.esr_mlp_wgrad(arr(dz), arr(src), rows, splits, arr(dw), p(db) if sums else None, st))
    for l in range(4):
        kin = src[l].shape[1]
        F.check(L.esr_gemm_bf16(1, 1, 256, kin, rows, p(dz[l]), 256, p(src[l]), kin, 0, None, None, None, p(want[l]), None,
                                kin, splits, st))
        F.check(L.esr_colsum_bf16(p(dz[l]), rows, 256, 256, p(wantb[l]), st))
        assert torch.equal(dw[l], want[l])
    assert torch.equal(db, wantb) if sums else True
    bad = C.c_int32(-1)
    F.check(L.esr_gemm_tc_status(C.byref(bad)))
    assert bad.value == 0
    for r, s in ((rows + 64, 1), (rows, 0), (rows, rows // 64 + 1)):
        assert L.esr_mlp_wgrad(arr(dz), arr(src), r, s, arr(dw), None, st) != 0


@pytest.mark.parametrize("rows", [128, 384, 2048, 2688, 4352])
def test_backward_in_one_call_equals_layer_calls(rows):
    """esr_mlp_backward (in-place dh, one weight-gradient launch, with the
    column sums in it or, where a range is no whole number of 256-row blocks,
    beside it) gives the bits of the layer-by-layer calls."""
    import torch
    m, X, base, tgt, w, inv_den = _setup(rows=rows, seed=9)
    y, acts = m.forward(X, base, keep=True)
    _, dpred = m.loss(y, tgt, w, inv_den)
    splits = 1
    while rows % (128 * splits) == 0 and rows // (splits * 2) >= 1024:
        splits *= 2
    m.backward(acts, dpred, splits=splits)
    want = m.g.clone()
    m.g.fill_(float("nan"))
    m.backward(acts, dpred)
    assert torch.equal(m.g, want)
    assert m.L.esr_mlp_backward_workspace(rows + 64) == -1


@pytest.mark.parametrize("rows", [128, 2688])
def test_views_of_larger_buffers_run(rows):
    """Flat parameters and kept activations that are views into a larger
    buffer, at 4-byte addresses, give the bits of buffers of their own: the
    layer calls take them where the one-call kernels' 16-byte accesses cannot."""
    import torch
    m, X, base, tgt, w, inv_den = _setup(rows=rows, seed=11)

    def passes(acts_of=lambda acts: acts):
        y, acts = m.forward(X, base, keep=True)
        _, dpred = m.loss(y, tgt, w, inv_den)
        m.backward(acts_of(acts), dpred)
        return y.clone(), m.g.clone()

    def shifted(acts):
        z = []
        for t in acts["z"]:
            big = torch.zeros(t.numel() + 2, dtype=t.dtype, device=t.device)
            big[2:].copy_(t.reshape(-1))
            z.append(big[2:].view(t.shape))
        return dict(acts, z=z)

    want = passes()
    assert all(torch.equal(a, b) for a, b in zip(passes(shifted), want))
    big = torch.zeros(m.n_params + 1, device=m.p.device)
    big[1:].copy_(m.p)
    m.p = big[1:]
    assert m.p.data_ptr() % 16 == 4
    assert all(torch.equal(a, b) for a, b in zip(passes(), want))
    assert torch.equal(m.forward(X, base), want[0])
