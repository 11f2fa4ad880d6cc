"""Fused tap kernels (telephone attention, adaptive local convolution) against the unfused PyTorch restatement."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp(min=1e-12)).item()


@pytest.mark.parametrize("B,L,H,D,K,half", [(2, 300, 4, 64, 64, 8), (1, 1000, 2, 16, 16, 21), (2, 130, 3, 128, 8, 3), (1, 257, 8, 8, 33, 5)])
def test_telephone_fused(B, L, H, D, K, half):
    from ml_experiments_b200.ops import fused_taps as T

    g = torch.Generator().manual_seed(B * L + K)
    dev = "cuda"
    x = torch.randn(B, L, H * D, generator=g).bfloat16().float().to(dev)
    freq = (torch.rand(B, L, H, generator=g) * 15 + 1).to(dev)
    phase = ((torch.rand(B, L, H, generator=g) * 2 - 1) * 16).to(dev)
    kern = torch.randn(B, L, H, K, generator=g).to(dev)
    expo = (torch.rand(B, L, 1, generator=g) * 3.5 + 0.5).to(dev)
    leaves = [t.clone().requires_grad_(True) for t in (x, freq, phase, kern, expo)]
    ref_leaves = [t.clone().requires_grad_(True) for t in (x, freq, phase, kern, expo)]
    max_rec = half * 16.0
    out = T.telephone_gather(*leaves, H, half, max_rec)
    ref = T.telephone_gather_ref(*ref_leaves, H, half, max_rec)
    assert _rel(out, ref) < 1e-2
    dout = torch.randn(B, L, H * D, generator=g).bfloat16().float().to(dev)
    out.backward(dout)
    ref.backward(dout)
    for name, a, b in zip(("dx", "dfreq", "dphase", "dkern", "dexpo"), leaves, ref_leaves):
        assert _rel(a.grad, b.grad) < 2e-2, (name, _rel(a.grad, b.grad))


def _band_inputs(B, L, H, D, K, seed, freq):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(B, L, H * D, generator=g).bfloat16().float()
    u = torch.rand(B, L, H, generator=g)
    f = {"wide": u * 15 + 1, "narrow": u * 1.5, "signed": (u - 0.5) * 20, "zero": torch.where(u < 0.3, 0.0, u * 4)}[freq]
    phase = (torch.rand(B, L, H, generator=g) * 2 - 1) * 16
    kern = torch.randn(B, L, H, K, generator=g)
    expo = torch.rand(B, L, 1, generator=g) * 3.5 + 0.5
    return [t.to("cuda") for t in (x, f, phase, kern, expo)], torch.randn(B, L, H * D, generator=g).bfloat16().float().to("cuda")


def _by_band(B, L, H, D, K, half, max_rec=None):
    """Whether the band products take a call, forward and backward."""
    from ml_experiments_b200.ops.runtime import ops

    x = torch.empty(B, L, H * D, device="cuda", dtype=torch.bfloat16)
    return tuple(ops().tele_band_takes(x, x, H, K, half, half * 16.0 if max_rec is None else max_rec, back) for back in (False, True))


@pytest.mark.parametrize("B,L,H,D,K,half,fwd,bwd", [
    (8, 16384, 4, 64, 16, 117, True, True), (8, 16384, 4, 64, 64, 117, True, True),                     # 3570, 1120 us and 10350, 3400; 10130, 4300
    (8, 16384, 4, 16, 16, 117, True, True),                                                             # 1290, 1104 and 3770, 3350
    (1, 1200, 1, 128, 33, 52, False, False), (1, 2000, 1, 64, 64, 70, True, False),                      # backward 62, 105 us and 85, 130
    (1, 6000, 4, 16, 33, 66, True, False), (8, 16384, 4, 16, 64, 119, False, False),                    # 142, 208; forward 1300, 1617
    (8, 700, 8, 16, 64, 19, False, False), (2, 3001, 8, 32, 16, 45, True, True)])                        # forward 33, 43; both 96, 74 and 239, 200
def test_telephone_goes_the_faster_way(B, L, H, D, K, half, fwd, bwd):
    """Calls for which both were timed (gather, band products), large tables and few blocks among them."""
    assert _by_band(B, L, H, D, K, half) == (fwd, bwd)


@pytest.mark.parametrize("B,L,H,D,K,half,freq", [
    (12, 128, 1, 64, 16, 50, "wide"), (2, 129, 2, 32, 16, 57, "wide"), (1, 191, 4, 16, 64, 59, "signed"), (8, 193, 1, 128, 33, 61, "narrow"),
    (2, 1000, 3, 64, 16, 54, "zero"), (1, 2051, 2, 128, 64, 51, "signed"), (1, 3001, 2, 32, 16, 55, "wide"), (1, 2500, 1, 64, 2, 117, "narrow"),
    (1, 2500, 1, 128, 6, 118, "wide"), (2, 1201, 4, 64, 16, 37, "wide"), (1, 300, 2, 64, 16, 4, "wide"),
    (6, 2051, 2, 128, 64, 51, "signed"), (5, 3001, 2, 32, 16, 55, "wide"), (6, 2500, 1, 64, 2, 117, "narrow"), (4, 2500, 1, 128, 6, 118, "wide"),
    (8, 601, 4, 64, 64, 20, "wide"), (8, 577, 2, 128, 47, 60, "zero"), (16, 193, 2, 128, 33, 61, "narrow"), (4, 1000, 3, 64, 16, 54, "zero")])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_telephone_band(B, L, H, D, K, half, freq, dtype):
    """Edges of the tiles of 128 rows and 64 keys, tables that are no multiple of four, strides below one (several taps on a row), negative
    and zero ones, results in both precisions. Those in `gathered` are too little work for the products, forward or backward."""
    from ml_experiments_b200.ops import fused_taps as T

    gathered = {(1, 2051, 2, 128, 64, 51): (1, 1), (1, 3001, 2, 32, 16, 55): (0, 1), (1, 2500, 1, 64, 2, 117): (0, 1), (1, 2500, 1, 128, 6, 118): (1, 1),
                (1, 300, 2, 64, 16, 4): (1, 1)}
    assert _by_band(B, L, H, D, K, half) == tuple(not g for g in gathered.get((B, L, H, D, K, half), (0, 0)))
    ins, dout = _band_inputs(B, L, H, D, K, L + D, freq)
    leaves = [t.clone().to(dtype if i == 0 else t.dtype).requires_grad_(True) for i, t in enumerate(ins)]
    ref = [t.clone().requires_grad_(True) for t in ins]
    y = T.telephone_gather(*leaves, H, half, half * 16.0)
    yr = T.telephone_gather_ref(*ref, H, half, half * 16.0)      # positions in fp32 as here: the same rows are read
    assert y.dtype == dtype and _rel(y, yr) < 5e-3         # bf16 results
    y.backward(dout.to(dtype))
    yr.backward(dout)
    for i, (name, a, b) in enumerate(zip(("dx", "dfreq", "dphase", "dkern", "dexpo"), leaves, ref)):
        tol = 5e-3 if i == 0 and dtype == torch.bfloat16 else 2e-4         # results rounded to 2^-9; sums of up to 30000 fp32 products
        assert _rel(a.grad, b.grad) < tol, (name, _rel(a.grad, b.grad), tol)


@pytest.mark.parametrize("D,H", [(16, 4), (64, 4), (128, 4)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_telephone_band_weights_have_24_bits(D, H, dtype):
    """Two rows of opposite sign and nothing else: a result is the difference of the weights of two neighbouring taps, 6.8e-5 of them. It is
    off by their rounding to fp32 (three of 2^-24 each, 0.3 % of it) and by its own to bf16 (0.2 %); by 16 bits it would be off by 10 %."""
    from ml_experiments_b200.ops import fused_taps as T

    L, K, half, j = 1000, 16, 54, 500
    B = 4
    assert _by_band(B, L, H, D, K, half) == (True, True)
    pair = torch.zeros(B, L, H * D, device="cuda", dtype=dtype)
    pair[:, j], pair[:, j + 1] = 1, -1
    x = pair.clone().requires_grad_()
    one, zero = torch.ones(B, L, H, device="cuda"), torch.zeros(B, L, H, device="cuda")
    kern = (1 + torch.arange(K, device="cuda") / 256).expand(B, L, H, K).contiguous()
    y = T.telephone_gather(x, one, zero, kern, torch.zeros(B, L, 1, device="cuda"), H, half, half * 16.0)
    y.backward(pair)
    tap = (torch.arange(L, device="cuda") - j).abs().double()
    step = (K - 1) / (half * 16.0) / 256
    want = step * torch.where(torch.arange(L, device="cuda") <= j, -1.0, 1.0).double()
    both = (tap <= half) & ((torch.arange(L, device="cuda") - j - 1).abs() <= half)
    for got in (y, x.grad):                     # (the gradient is the same sum over the queries that sample a row)
        assert ((got[0, both].double() - want[both, None]).abs() / step).max().item() < 1e-2


@pytest.mark.parametrize("B", [1, 4])
def test_telephone_band_keeps_what_is_not_finite_where_it_is_sampled(B):
    """A row of x (of the gradient) that is not finite reaches the queries that sample it (the rows that it samples) and no others,
    although products with weights of zero are formed."""
    from ml_experiments_b200.ops import fused_taps as T

    L, H, D, half = 700, 2, 64, 54
    assert _by_band(B, L, H, D, 16, half) == (True, True)
    ins, dout = _band_inputs(B, L, H, D, 16, 5, "wide")
    ins[0][0, 350, 3] = float("nan")
    ins[0][0, 200, 70] = float("inf")
    dout[0, 333, 5] = float("nan")
    leaves, ref = [t.clone().requires_grad_(True) for t in ins], [t.clone().requires_grad_(True) for t in ins]
    y = T.telephone_gather(*leaves, H, half, half * 16.0)
    yr = T.telephone_gather_ref(*ref, H, half, half * 16.0)
    bad = yr.isfinite().logical_not()
    assert bad.any() and torch.equal(y.isfinite().logical_not(), bad)
    assert _rel(y[~bad], yr[~bad]) < 5e-3
    y.backward(dout)
    yr.backward(dout)
    inner = slice(2, L - 2)                                # taps outside are moved to the ends in the restatement, with weight zero
    bad = ref[0].grad[:, inner].isfinite().logical_not()
    dx, dxr = leaves[0].grad[:, inner], ref[0].grad[:, inner]
    assert bad.any() and torch.equal(dx.isfinite().logical_not(), bad)
    assert _rel(dx[~bad], dxr[~bad]) < 2e-4


@pytest.mark.parametrize("B,L,H,D,K", [(1, 4001, 4, 64, 16), (2, 1000, 4, 16, 16), (2, 3000, 2, 128, 64)])
def test_telephone_band_takes_about_as_long_where_nothing_is_finite(B, L, H, D, K):
    """A step that has diverged: results are formed tap by tap there, until they are no numbers (an element at a time and to the end, it
    took 30 times as long and more)."""
    from ml_experiments_b200.ops import fused_taps as T

    half = 54
    assert _by_band(B, L, H, D, K, half) == (True, True)
    ins, dout = _band_inputs(B, L, H, D, K, 7, "wide")
    ins[0] = ins[0].bfloat16()

    def pair(x, g):
        leaves = [t.clone().requires_grad_(True) for t in (x, *ins[1:])]
        best = [1e9, 1e9]
        for _ in range(4):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(3)]
            torch.cuda._sleep(2000000)                   # the calls are issued meanwhile
            e[0].record()
            y = T.telephone_gather(*leaves, H, half, half * 16.0)
            e[1].record()
            grads = torch.autograd.grad(y, leaves, g)
            e[2].record()
            torch.cuda.synchronize()
            best = [min(b, e[i].elapsed_time(e[i + 1])) for i, b in enumerate(best)]
        return best, y, grads[0]

    nan = torch.full_like(dout, float("nan")).bfloat16()
    (fwd, bwd), *_ = pair(ins[0], dout.bfloat16())
    (fwd_nan, _), y, _ = pair(nan, dout.bfloat16())
    (_, bwd_nan), _, dx = pair(ins[0], nan)
    assert y.isnan().all() and dx[:, 300:-300].isnan().all()
    assert fwd_nan < 4 * fwd and bwd_nan < 4 * bwd, (fwd, fwd_nan, bwd, bwd_nan)      # (measured: 1.4 and 2.1 at most)


@pytest.mark.parametrize("D", [32, 128])
@pytest.mark.parametrize("stride", [float("nan"), float("inf"), float("-inf"), 1e38, -1e38])
def test_telephone_band_strides_that_leave_the_sequence(D, stride):
    """A stride that is no number or infinite has no tap in the sequence (0 * stride is no number either): nothing comes out of it, and its
    gradients are zero. A very large one has tap 0 alone, as 1e6 has."""
    from ml_experiments_b200.ops import fused_taps as T

    B, L, H, half, at = 4, 700, 4, 54, (0, slice(100, 700, 150), 0)
    assert _by_band(B, L, H, D, 16, half) == (True, True)
    ins, dout = _band_inputs(B, L, H, D, 16, 6, "wide")
    ins[4][0, ::100] *= -1                       # weights that grow with the distance
    grads, ys = [], []
    for f in (stride, 1e6):
        ins[1][at] = f
        leaves = [t.clone().requires_grad_(True) for t in ins]
        ys.append(T.telephone_gather(*leaves, H, half, half * 16.0))
        ys[-1].backward(dout)
        grads.append([t.grad for t in leaves])
        assert all(t.isfinite().all() for t in [ys[-1], *grads[-1]])
    if abs(stride) < float("inf"):
        assert torch.equal(*ys) and all(torch.equal(a, b) for a, b in zip(*grads))
        assert all(g[at].abs().sum() > 0 for g in grads[0][2:4])
    else:
        assert not ys[0].view(B, L, H, D)[at].any() and not any(g[at].any() for g in grads[0][1:4])


@pytest.mark.parametrize("B,L,H,D,K,half", [(2, 300, 4, 64, 64, 29), (1, 1000, 2, 16, 16, 9), (2, 130, 3, 128, 8, 3), (1, 257, 8, 8, 64, 12)])
def test_adaptive_local_fused(B, L, H, D, K, half):
    from ml_experiments_b200.ops import fused_taps as T

    g = torch.Generator().manual_seed(B * L + K + 1)
    dev = "cuda"
    x = torch.randn(B, L, H * D, generator=g).bfloat16().float().to(dev)
    half_w = (torch.rand(B, L, H, generator=g) * half + 0.5).to(dev)
    half_w[:, ::7] = 0.5                      # narrow windows: the tap sum stays below the normalisation threshold
    center = ((torch.rand(B, L, H, generator=g) * 2 - 1) * 12).to(dev)
    kern = torch.randn(B, L, H, K, generator=g).to(dev)
    leaves = [t.clone().requires_grad_(True) for t in (x, half_w, center, kern)]
    ref_leaves = [t.clone().requires_grad_(True) for t in (x, half_w, center, kern)]
    out = T.adaptive_local_gather(*leaves, H, half)
    ref = T.alc_gather_ref(*ref_leaves, H, half)
    assert _rel(out, ref) < 1e-2
    dout = torch.randn(B, L, H * D, generator=g).bfloat16().float().to(dev)
    out.backward(dout)
    ref.backward(dout)
    for name, a, b in zip(("dx", "dhalf_w", "dcenter", "dkern"), leaves, ref_leaves):
        assert _rel(a.grad, b.grad) < 2e-2, (name, _rel(a.grad, b.grad))


@pytest.mark.parametrize("C", [1, 4, 8, 64, 256, 300, 512, 768, 1024])
@pytest.mark.parametrize("act", ["none", "silu", "sigmoid", "tanh"])
@pytest.mark.parametrize("dtypes", [(torch.bfloat16, torch.float32), (torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16)])
def test_rms_norm_act(C, act, dtypes):
    from ml_experiments_b200.ops.norm_act import rms_norm_act, rms_norm_act_ref

    din, dout = dtypes
    g = torch.Generator().manual_seed(C)
    x = torch.randn(3, 37, C, generator=g).to("cuda", din)
    w = (torch.rand(C, generator=g) + 0.5).to("cuda")
    xa, wa = x.clone().requires_grad_(True), w.clone().requires_grad_(True)
    xb, wb = x.float().clone().requires_grad_(True), w.clone().requires_grad_(True)
    ya = rms_norm_act(xa, wa, 1e-6, act, dout)
    yb = rms_norm_act_ref(xb, wb, 1e-6, act, torch.float32)
    assert ya.dtype == dout and _rel(ya, yb) < (1e-2 if dout == torch.bfloat16 else 1e-5)
    gy = torch.randn(3, 37, C, generator=g).to("cuda")
    ya.backward(gy.to(dout))
    yb.backward(gy.to(dout).float())
    tol = 2e-2 if torch.bfloat16 in dtypes else 1e-4
    assert _rel(xa.grad, xb.grad) < tol and _rel(wa.grad, wb.grad) < tol


@pytest.mark.parametrize("C", [256, 300, 512, 768, 1024, 1280])
@pytest.mark.parametrize("rows,off", [(1, 0), (37, 0), (6001, 0), (37, 1)])
def test_rms_norm_act_with_bf16_weights_is_the_same_as_with_their_fp32_values(C, rows, off):
    """Weights are read in either type; rows on and off the 16-byte boundary (the latter take the general path)."""
    from ml_experiments_b200.ops.norm_act import rms_norm_act, rms_norm_act_ref

    g = torch.Generator().manual_seed(C + rows)
    x = torch.randn(rows * C + 8, generator=g).bfloat16().cuda()[off:off + rows * C].view(rows, C)
    w = (torch.rand(C, generator=g) + 0.5).bfloat16().cuda()
    xa, wa, xb, wb = x.clone().requires_grad_(), w.clone().requires_grad_(), x.clone().requires_grad_(), w.float().requires_grad_()
    if off:
        xa, xb = x.detach().requires_grad_(), x.detach().requires_grad_()
    ya, yb = rms_norm_act(xa, wa, 1e-6, "silu"), rms_norm_act(xb, wb, 1e-6, "silu")
    assert torch.equal(ya, yb) and _rel(ya, rms_norm_act_ref(x.float(), w.float(), 1e-6, "silu")) < 4e-3
    gy = torch.randn(rows, C, generator=g).bfloat16().cuda()
    ya.backward(gy)
    yb.backward(gy)
    assert torch.equal(xa.grad, xb.grad) and wa.grad.dtype == torch.bfloat16 and _rel(wa.grad, wb.grad) < 4e-3


def test_rms_norm_act_bf16_weights_may_change_before_the_backward():
    """An optimizer may step between a forward and its backward: the gradients are those of the weights that the forward had."""
    from ml_experiments_b200.ops.norm_act import rms_norm_act, rms_norm_act_skip

    g = torch.Generator().manual_seed(3)
    for C in (512, 300):
        x = torch.randn(50, C, generator=g).bfloat16().cuda()
        w = (torch.rand(C, generator=g) + 0.5).bfloat16().cuda()
        gy = torch.randn(50, C, generator=g).bfloat16().cuda()
        for norm in (lambda a, b: rms_norm_act(a, b, 1e-6, "silu"), lambda a, b: rms_norm_act_skip(a, b, 1e-6, "silu")[0]):
            grads = []
            for change in (False, True):
                xa, wa = x.clone().requires_grad_(), w.clone().requires_grad_()
                y = norm(xa, wa)
                if change:
                    with torch.no_grad():
                        wa.mul_(3)
                y.backward(gy)
                grads.append((xa.grad, wa.grad))
            assert torch.equal(grads[0][0], grads[1][0]) and _rel(grads[1][1], grads[0][1]) < 4e-3     # (dw: sums in any order)


@pytest.mark.parametrize("C,dtype,lead", [(768, torch.bfloat16, 12), (1024, torch.bfloat16, 0), (512, torch.bfloat16, 9), (300, torch.bfloat16, 12),
                                          (256, torch.float32, 5)])
def test_rms_norm_act_skip_adds_the_skip_gradient_in_the_backward_kernel(C, dtype, lead):
    """``h, skip[, first] = rms_norm_act_skip(x, w)``; ``out = skip + f(h) + g(first)``: dx = norm backward of (dh with
    d first added into its leading columns) + the skip's gradient, from one kernel (16-byte path for bf16 rows of 256 k
    columns, several rows per warp; the general path otherwise)."""
    from ml_experiments_b200.ops.norm_act import rms_norm_act_ref, rms_norm_act_skip

    g = torch.Generator().manual_seed(C)
    x = torch.randn(6000, C, generator=g).to("cuda", dtype)
    w = (torch.rand(C, generator=g) + 0.5).to("cuda")
    xa, wa = x.clone().requires_grad_(True), w.clone().requires_grad_(True)
    xb, wb = x.float().clone().requires_grad_(True), w.clone().requires_grad_(True)
    outs = rms_norm_act_skip(xa, wa, 1e-6, "silu", lead_cols=lead)
    h, skip = outs[0], outs[1]
    loss = (skip.float() * 0.5 + torch.sin(h.float())).sum()
    if lead:
        assert outs[2].shape == (6000, lead) and torch.equal(outs[2], h[:, :lead])
        loss = loss + (outs[2].float() * 3.0).pow(2).sum()
    loss.backward()
    hb = rms_norm_act_ref(xb, wb, 1e-6, "silu", torch.float32)
    hq = hb.detach().to(dtype).float() + (hb - hb.detach())          # the slice's consumer sees the rounded output
    loss_b = (xb * 0.5 + torch.sin(hb)).sum() + ((hq[:, :lead] * 3.0).pow(2).sum() if lead else 0.0)
    loss_b.backward()
    tol = 2e-2 if dtype == torch.bfloat16 else 1e-4
    assert _rel(h, hb) < (1e-2 if dtype == torch.bfloat16 else 1e-5)
    assert _rel(xa.grad, xb.grad) < tol and _rel(wa.grad, wb.grad) < tol
