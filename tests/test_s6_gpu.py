"""S6 selective-scan kernels against the sequential fp32 oracle, and the S6 LM end to end."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def default_scan_shape():
    yield
    from ml_experiments_b200.ops.selective_scan import set_states_per_thread
    set_states_per_thread()


@pytest.mark.parametrize("qs", [(4, 4), (2, 4), (4, 2), (2, 2)])
@pytest.mark.parametrize("bsz,L,din", [(2, 200, 128), (1, 64, 72), (3, 333, 192), (2, 50, 100), (1, 33, 7)])
def test_scan_forward_backward(bsz, L, din, qs, default_scan_shape):
    from ml_experiments_b200.ops.selective_scan import selective_scan, selective_scan_ref, set_states_per_thread

    set_states_per_thread(*qs)
    torch.manual_seed(0)
    n = 16
    dev = "cuda"
    u = torch.randn(bsz, L, din, device=dev).bfloat16().float().requires_grad_(True)
    delta = (torch.rand(bsz, L, din, device=dev) * 0.2 + 0.01).requires_grad_(True)
    A = (-torch.rand(din, n, device=dev) * 4 - 0.2).requires_grad_(True)
    B = torch.randn(bsz, L, n, device=dev).requires_grad_(True)
    C = torch.randn(bsz, L, n, device=dev).requires_grad_(True)
    D = torch.randn(din, device=dev).requires_grad_(True)
    z = torch.randn(bsz, L, din, device=dev).bfloat16().float().requires_grad_(True)
    g = torch.randn(bsz, L, din, device=dev)
    ref = selective_scan_ref(u, delta, A, B, C, D, z)
    ref.backward(g)
    want = [t.grad.clone() for t in (u, delta, A, B, C, D, z)]
    for t in (u, delta, A, B, C, D, z):
        t.grad = None
    out = selective_scan(u, delta, A, B, C, D, z)
    assert ((out - ref).abs().max() / ref.abs().max()).item() < 2e-2
    out.backward(g)
    for name, t, w in zip("u delta A B C D z".split(), (u, delta, A, B, C, D, z), want):
        rel = ((t.grad - w).norm() / (w.norm() + 1e-9)).item()
        assert rel < 3e-2, (name, rel)


@pytest.mark.parametrize("delta_dtype", [torch.float32, torch.bfloat16])
def test_scan_fused_softplus_bias_gate(delta_dtype):
    """Raw step + bias + softplus and the silu(z) gate run inside the kernels; gradients reach the raw step and the bias."""
    from ml_experiments_b200.ops.selective_scan import selective_scan, selective_scan_ref

    torch.manual_seed(1)
    bsz, L, din, n, dev = 2, 150, 100, 16, "cuda"
    u = torch.randn(bsz, L, din, device=dev).bfloat16().float().requires_grad_(True)
    raw = (torch.randn(bsz, L, din, device=dev) - 3).to(delta_dtype).float().requires_grad_(True)
    bias = torch.randn(din, device=dev).requires_grad_(True)
    A = (-torch.rand(din, n, device=dev) * 4 - 0.2).requires_grad_(True)
    B = torch.randn(bsz, L, n, device=dev).requires_grad_(True)
    C = torch.randn(bsz, L, n, device=dev).requires_grad_(True)
    z = torch.randn(bsz, L, din, device=dev).bfloat16().float().requires_grad_(True)
    g = torch.randn(bsz, L, din, device=dev)
    leaves = (u, raw, bias, A, B, C, z)
    ref = selective_scan_ref(u, raw, A, B, C, None, z, delta_bias=bias, delta_softplus=True)
    ref.backward(g)
    want = [t.grad.clone() for t in leaves]
    for t in leaves:
        t.grad = None
    raw_in = raw.to(delta_dtype)
    raw_in.retain_grad()
    out = selective_scan(u, raw_in, A, B, C, None, z, delta_bias=bias, delta_softplus=True)
    assert ((out - ref).abs().max() / ref.abs().max()).item() < 2e-2
    out.backward(g)
    tol = 3e-2 if delta_dtype == torch.float32 else 5e-2
    for name, t, w in zip("u raw bias A B C z".split(), leaves, want):
        rel = ((t.grad.float() - w).norm() / (w.norm() + 1e-9)).item()
        assert rel < tol, (name, rel)


def test_s6_lm_trains():
    from ml_experiments_b200.models.s6 import S6Config, S6LM

    torch.manual_seed(0)
    m = S6LM(S6Config(d_model=128, n_layers=2, vocab_size=256)).cuda().bfloat16()
    ids = torch.randint(0, 256, (2, 256), device="cuda")
    ids[:, 1::2] = ids[:, 0::2]  # every second byte repeats the previous one: learnable
    opt = torch.optim.AdamW(m.parameters(), lr=3e-3)
    first = None
    for _ in range(30):
        loss = m(ids[:, :-1], ids[:, 1:])
        opt.zero_grad()
        loss.backward()
        opt.step()
        first = first if first is not None else loss.item()
    assert loss.item() < 0.8 * first


def test_causal_conv1d_silu():
    from ml_experiments_b200.ops.causal_conv import causal_conv1d_silu, causal_conv1d_silu_ref

    torch.manual_seed(1)
    B, L, C = 2, 150, 264
    wide = torch.randn(B, L, 2 * C, device="cuda").bfloat16()
    x = wide[..., :C].detach().requires_grad_(True)           # channel slice of a wider tensor
    w = (torch.randn(C, 1, 4, device="cuda") * 0.5).requires_grad_(True)
    b = torch.randn(C, device="cuda").requires_grad_(True)
    g = torch.randn(B, L, C, device="cuda").bfloat16()
    xr = x.detach().float().requires_grad_(True)
    wr, br = w.detach().clone().requires_grad_(True), b.detach().clone().requires_grad_(True)
    ref = causal_conv1d_silu_ref(xr, wr, br)
    ref.backward(g.float())
    y = causal_conv1d_silu(x, w, b)
    assert ((y.float() - ref).abs().max() / ref.abs().max()).item() < 2e-2
    y.backward(g)
    for name, got, want in (("dx", x.grad, xr.grad), ("dw", w.grad, wr.grad), ("db", b.grad, br.grad)):
        rel = ((got.float() - want).norm() / want.norm()).item()
        assert rel < 2e-2, (name, rel)


@pytest.mark.parametrize("bsz,L,din,off", [(1, 1, 8, 0), (2, 15, 24, 0), (2, 17, 40, 0), (1, 33, 7, 0), (2, 40, 48, 4),
                                           (10, 37, 1024, 0), (1, 4097, 16, 0)])
@pytest.mark.parametrize("delta_dtype", [torch.float32, torch.bfloat16])
def test_scan_tile_edges(bsz, L, din, off, delta_dtype):
    """Sequences and channel counts around the tiles (16 steps; 8, 16 and 32 channels), enough channels for the
    four-states-a-thread forward, rows that are not 16-byte aligned (odd channel counts, a tensor that starts inside an
    allocation)."""
    from ml_experiments_b200.ops.selective_scan import selective_scan, selective_scan_ref

    g = torch.Generator(device="cuda").manual_seed(L)

    def make(*shape, dtype=torch.bfloat16):
        n = 1
        for s in shape:
            n *= s
        flat = torch.randn(n + off, generator=g, device="cuda").to(dtype)
        return flat[off:].view(*shape)

    u, z = make(bsz, L, din), make(bsz, L, din)
    raw = (make(bsz, L, din) - 2).to(delta_dtype)
    B, C = make(bsz, L, 16, dtype=torch.float32), make(bsz, L, 16, dtype=torch.float32)
    A = -torch.rand(din, 16, generator=g, device="cuda") * 4 - 0.2
    D, bias = make(din, dtype=torch.float32), make(din, dtype=torch.float32) * 0.5
    dy = make(bsz, L, din)
    ins = [t.detach().requires_grad_() for t in (u, raw, A, B, C, D, z, bias)]
    out = selective_scan(*ins[:7], delta_bias=ins[7], delta_softplus=True)
    got = torch.autograd.grad(out, ins, dy)
    ref_in = [t.detach().float().requires_grad_() for t in ins]
    ref = selective_scan_ref(*ref_in[:7], delta_bias=ref_in[7], delta_softplus=True)
    want = torch.autograd.grad(ref, ref_in, dy.float())
    # outputs are rounded to bf16 (2^-9), the gate's backward reads the bf16 value in front of the gate (2^-9 more)
    assert ((out.float() - ref).norm() / ref.norm()).item() < 4e-3
    for name, a, w in zip("u raw A B C D z bias".split(), got, want):
        assert ((a.float() - w).norm() / (w.norm() + 1e-12)).item() < 1e-2, name


@pytest.mark.parametrize("bsz,L,C", [(1, 1, 8), (2, 3, 24), (1, 4, 264), (2, 7, 40), (3, 33, 128), (1, 66, 520), (2, 257, 48),
                                     (64, 200, 1024)])
@pytest.mark.parametrize("sliced", [False, True])
def test_causal_conv1d_tile_edges(bsz, L, C, sliced):
    """Sequences around the four-step groups and the tiles, channel counts that end inside a warp, a channel slice as input,
    and (the last one) enough work for the longest tiles."""
    from ml_experiments_b200.ops.causal_conv import causal_conv1d_silu, causal_conv1d_silu_ref

    g = torch.Generator(device="cuda").manual_seed(L)
    wide = torch.randn(bsz, L, 2 * C if sliced else C, generator=g, device="cuda").bfloat16()
    x = wide[..., :C].detach().requires_grad_()
    w = torch.randn(C, 1, 4, generator=g, device="cuda").requires_grad_()
    b = torch.randn(C, generator=g, device="cuda").requires_grad_()
    dy = torch.randn(bsz, L, C, generator=g, device="cuda").bfloat16()
    y = causal_conv1d_silu(x, w, b)
    got = torch.autograd.grad(y, (x, w, b), dy)
    ref_in = [t.detach().double().contiguous().requires_grad_() for t in (x, w, b)]   # 64 bits: no TF32 in the oracle
    ref = causal_conv1d_silu_ref(*ref_in)
    want = torch.autograd.grad(ref, ref_in, dy.double())
    assert ((y.double() - ref).norm() / ref.norm()).item() < 3e-3              # bf16 output: 2^-9
    assert ((got[0].double() - want[0]).norm() / want[0].norm()).item() < 3e-3
    for a, e in zip(got[1:], want[1:]):
        assert ((a.double() - e).norm() / e.norm()).item() < 1e-4              # fp32 sums of fp32 products


def test_causal_conv1d_off_the_16_byte_boundary():
    """A channel slice that starts 8 bytes into a 16-byte piece takes the general path, a gradient that does so is copied, and
    the operators refuse both."""
    from ml_experiments_b200.ops.causal_conv import causal_conv1d_silu, causal_conv1d_silu_ref
    from ml_experiments_b200.ops.runtime import ops

    bsz, L, C = 2, 37, 40
    wide = torch.randn(bsz, L, C + 8, device="cuda").bfloat16()
    w, b = torch.randn(C, 1, 4, device="cuda").requires_grad_(), torch.randn(C, device="cuda").requires_grad_()
    dy = torch.randn(bsz * L * C + 4, device="cuda").bfloat16()[4:].view(bsz, L, C)
    w32, y = w.detach().reshape(C, 4).contiguous(), torch.empty(bsz, L, C, device="cuda", dtype=torch.bfloat16)
    for first in (0, 4):
        x = wide[..., first:first + C].detach().requires_grad_()
        out = causal_conv1d_silu(x, w, b)
        got = torch.autograd.grad(out, (x, w, b), dy)
        ref_in = [t.detach().double().contiguous().requires_grad_() for t in (x, w, b)]
        ref = causal_conv1d_silu_ref(*ref_in)
        want = torch.autograd.grad(ref, ref_in, dy.double())
        # bf16 outputs, and in the general path bf16 weights, pre-activations and gradients: 2^-9 each
        for a, e in zip((out, *got), (ref, *want)):
            assert ((a.double() - e).norm() / e.norm()).item() < 1e-2
    with pytest.raises(RuntimeError, match="16-byte"):
        ops().causal_conv1d_silu_fwd(wide[..., 4:4 + C], w32, None, y)
    with pytest.raises(RuntimeError, match="16-byte"):
        ops().causal_conv1d_silu_bwd(wide[..., :C], w32, None, dy, y, torch.zeros_like(w32), None)


@pytest.mark.parametrize("bsz,auto", [(1, 2), (10, 4)])
def test_states_per_thread_of_the_forward_can_be_chosen(bsz, auto, default_scan_shape):
    """Two and four states a thread add a channel's sixteen products in another order, so a choice shows in the last bits; left
    alone, few channels in flight take two and many take four."""
    from ml_experiments_b200.ops.selective_scan import selective_scan, set_states_per_thread

    g = torch.Generator(device="cuda").manual_seed(bsz)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    L, din = 64, 1024
    ins = (rand(bsz, L, din).bfloat16(), rand(bsz, L, din) * 0.1 + 0.2, -rand(din, 16).abs() - 0.2, rand(bsz, L, 16),
           rand(bsz, L, 16))
    outs = {}
    for qs in (2, 4, None):
        set_states_per_thread(qs)
        outs[qs] = selective_scan(*ins)
    assert not torch.equal(outs[2], outs[4])
    assert ((outs[2].float() - outs[4].float()).norm() / outs[4].float().norm()).item() < 4e-3    # bf16 outputs: 2^-9
    assert torch.equal(outs[None], outs[auto])
    with pytest.raises(RuntimeError, match="2 or 4"):
        set_states_per_thread(3)


@pytest.mark.parametrize("bsz,L,c,rank,dtype", [(1, 1, 64, 8, torch.bfloat16), (2, 33, 72, 8, torch.float32), (3, 130, 128, 16, torch.bfloat16),
                                               (1, 257, 1024, 64, torch.bfloat16)])
def test_s6_inner_is_convolution_projections_and_scan(bsz, L, c, rank, dtype):
    """The node of an S6 mixer (small parameters packed, B and C split off and their gradients joined by kernels of its own) against the
    separate operators, values and every gradient; parameters in both types."""
    from ml_experiments_b200.ops.causal_conv import causal_conv1d_silu
    from ml_experiments_b200.ops.linear import linear, linear_tee
    from ml_experiments_b200.ops.selective_scan import s6_inner, selective_scan

    g = torch.Generator().manual_seed(L + c)
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()  # noqa: E731
    x = [rnd(bsz, L, c).bfloat16(), rnd(bsz, L, c).bfloat16()]
    p = [rnd(c, 1, 4) * 0.4, rnd(c) * 0.1, rnd(rank + 32, c) * c ** -0.5, rnd(c, rank) * rank ** -0.5, rnd(c) - 3,
         torch.log(torch.arange(1.0, 17.0).cuda()).repeat(c, 1) + 0.1 * rnd(c, 16), rnd(c)]
    a = [t.clone().requires_grad_() for t in x] + [t.to(dtype).requires_grad_() for t in p]
    b = [t.detach().clone().requires_grad_() for t in a]
    y = s6_inner(*a)
    xi, z, cw, cb, xw, dw, db, al, d = b
    dbc, u = linear_tee(causal_conv1d_silu(xi, cw, cb), xw)
    dt, B, C = torch.split(dbc, [rank, 16, 16], dim=-1)
    yr = selective_scan(u.contiguous(), linear(dt, dw), -torch.exp(al.float()), B, C, d, z, delta_bias=db, delta_softplus=True)
    # exp(A_log) is rounded once here and within an ulp there: a few results fall on the other side of a bf16 rounding
    assert ((y.float() - yr.float()).norm() / yr.float().norm()).item() < 5e-4
    dy = rnd(bsz, L, c).bfloat16()
    y.backward(dy)
    yr.backward(dy)
    for name, s, t in zip(("xi", "z", "conv_w", "conv_b", "x_w", "dt_w", "dt_b", "A_log", "D"), a, b):
        assert s.grad.dtype == t.grad.dtype and s.grad.shape == t.grad.shape
        # the same sums in another order (atomics, partial sums): bf16 results differ by a rounding here and there
        err = ((s.grad.float() - t.grad.float()).norm() / t.grad.float().norm().clamp(min=1e-20)).item()
        assert err < 3e-3, (name, err)
    with torch.no_grad():
        assert torch.equal(s6_inner(*a), y)


def _mixer_backward(frozen=(), change=(), dtype=torch.bfloat16):
    """Gradients of a mixer's input and parameters and the launches of its backward; ``change``: parameters that are tripled before it."""
    from ml_experiments_b200.models.s6 import S6Config, S6Mixer
    from ml_experiments_b200.ops.runtime import launch_count

    torch.manual_seed(5)
    m = S6Mixer(S6Config(d_model=128, n_layers=1)).cuda().to(dtype)
    x = torch.randn(2, 100, 128, device="cuda").bfloat16().requires_grad_()
    params = dict(m.named_parameters())
    for n in frozen:
        params[n].requires_grad_(False)
    y = m(x)
    with torch.no_grad():
        for n in change:
            params[n].mul_(3)
    before = launch_count()
    (y.float() * torch.randn(y.shape, device="cuda")).sum().backward()
    return {"x": x.grad, **{n: p.grad for n, p in params.items()}}, launch_count() - before


def test_s6_inner_forms_no_gradients_of_frozen_projections():
    want, full = _mixer_backward()
    for frozen in (["x_proj.weight"], ["dt_proj.weight"], ["x_proj.weight", "dt_proj.weight"]):
        got, launches = _mixer_backward(frozen)
        assert launches == full - len(frozen)
        assert all(got[n] is None if n in frozen else torch.allclose(got[n].float(), g.float(), rtol=2e-2, atol=1e-3 * g.abs().max().item()) for n, g in want.items())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_s6_inner_small_parameters_may_change_before_the_backward(dtype):
    """An optimizer may step between a forward and its backward: the gradients are those of the parameters that the forward had."""
    change = ["conv1d.weight", "conv1d.bias", "A_log", "D", "dt_proj.bias"]
    want, _ = _mixer_backward(dtype=dtype)
    got, _ = _mixer_backward(change=change, dtype=dtype)
    for n, g in want.items():
        assert torch.allclose(got[n].float(), g.float(), rtol=2e-2, atol=1e-3 * g.abs().max().item()), n      # (bf16; sums in any order)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("din", [16, 1000, 37])          # the pipelined kernels, their last block half full, the general ones
def test_softplus_of_delta(dtype, din):
    """dt read off a state checkpoint (no decay, one input) and its derivative off ddelta, against 64 bits, over the range of delta.

    Bound: t = exp(-|x|) has the hardware's 2^-22 and the rounding of its argument, |x| log2(e) 2^-24 ln 2 in t; then 6 roundings."""
    from ml_experiments_b200.ops.runtime import ops

    x = torch.cat([torch.linspace(-40, 40, din - 9), torch.tensor([0.0, -0.0, 19.99, 20.01, 88.0, -80.0, 100.0, -3e-5, 4e-6])]).to(dtype)
    length = 20
    delta = torch.zeros(1, length, din, dtype=dtype)
    delta[0, 0] = x
    one = torch.zeros(1, length, 16)
    one[0, :, 0] = 1.0
    u = torch.zeros(1, length, din, dtype=torch.bfloat16)
    u[0, 0] = 1.0
    delta, u, B, C = (a.cuda() for a in (delta, u, one, one))
    A = torch.zeros(din, 16, device="cuda")
    e = lambda *s, t: torch.zeros(*s, device="cuda", dtype=t)
    y, out = e(1, length, din, t=torch.bfloat16), e(1, length, din, t=torch.bfloat16)
    state = e(1, 2, 4, din, 4, t=torch.float32)
    ops().s6_scan_fwd(u, delta, None, True, A, B, C, None, None, y, out, state)
    dout = torch.zeros_like(u)
    dout[0, 0] = 1.0
    ddelta, du, dA = torch.zeros_like(delta), torch.zeros_like(u), torch.zeros_like(A)
    parts = [e(1, (din + 31) // 32, length, 16, t=torch.float32) for _ in range(2)]
    ops().s6_scan_bwd(u, delta, None, True, A, B, C, None, None, None, dout, state, du, ddelta, dA, *parts, None, None, None)
    xd = x.double()
    dt = torch.where(xd < 0, torch.log1p(torch.exp(xd)), xd + torch.log1p(torch.exp(-xd)))
    tol = 2.0 ** -22 + 2.0 ** -24 * (xd.abs() * 1.5 + 6)
    got = state[0, 1, 0, :, 0].double().cpu()
    assert ((got - dt).abs() <= tol * dt).all()
    tol = tol + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0)       # (stored as delta's type)
    sp = 1 / (1 + torch.exp(-xd))
    assert ((ddelta[0, 0].double().cpu() - sp).abs() <= tol * sp).all()
