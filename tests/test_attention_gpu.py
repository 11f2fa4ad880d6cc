"""tcgen05 flash attention (forward and backward) against a dense fp32 oracle."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _setup(t, h, d, doc_len, seed=0):
    torch.manual_seed(seed)
    qkv = torch.randn(t, 3, h, d, device="cuda", dtype=torch.bfloat16)
    q, k, v = qkv[:, 0], qkv[:, 1], qkv[:, 2]  # strided views, heads contiguous
    from ml_experiments_b200.ops.attention import doc_bounds_from_starts

    is_start = torch.zeros(t, dtype=torch.bool, device="cuda")
    is_start[::doc_len] = True
    ds, de = doc_bounds_from_starts(is_start)
    return q, k, v, ds, de


@pytest.mark.parametrize("t,doc_len,window", [(256, 256, 0), (1024, 1024, 0), (1024, 384, 0), (2048, 1000, 3), (1536, 1536, 2)])
@pytest.mark.parametrize("d", [128, 64])
def test_attention_forward(t, doc_len, window, d):
    from ml_experiments_b200.ops import attention as A

    q, k, v, ds, de = _setup(t, 3, d, doc_len)
    o, lse = A.flash_attention_forward(q, k, v, ds, de, 0.12, window)
    ref = A.attention_reference(q, k, v, ds, 0.12, window)
    err = (o.float() - ref).abs().max().item()
    assert err < 2e-2, err


@pytest.mark.parametrize("t,doc_len,window", [(256, 256, 0), (1024, 1024, 0), (1024, 384, 0), (2048, 1000, 3)])
@pytest.mark.parametrize("d", [128, 64])
def test_attention_backward(t, doc_len, window, d):
    from ml_experiments_b200.ops import attention as A

    q, k, v, ds, de = _setup(t, 2, d, doc_len, seed=1)
    d_o = torch.randn(t, 2, d, device="cuda", dtype=torch.bfloat16)
    qf, kf, vf = (x.float().detach().requires_grad_(True) for x in (q, k, v))
    ref = A.attention_reference(qf, kf, vf, ds, 0.12, window)
    ref.backward(d_o.float())
    o, lse = A.flash_attention_forward(q, k, v, ds, de, 0.12, window)
    dq, dk, dv = A.flash_attention_backward(q, k, v, o, d_o, lse, ds, de, 0.12, window)
    for name, got, want in (("dq", dq, qf.grad), ("dk", dk, kf.grad), ("dv", dv, vf.grad)):
        rel = ((got.float() - want).norm() / want.norm()).item()
        assert rel < 2e-2, (name, rel)


def test_doc_bounds():
    from ml_experiments_b200.ops.attention import doc_bounds_from_starts

    s = torch.tensor([1, 0, 0, 1, 0, 1, 0, 0], dtype=torch.bool)
    ds, de = doc_bounds_from_starts(s)
    assert ds.tolist() == [0, 0, 0, 3, 3, 5, 5, 5]
    assert de.tolist() == [3, 3, 3, 5, 5, 8, 8, 8]


def test_doc_bounds_kernel_matches_the_scan_formulation():
    from ml_experiments_b200.ops.attention import doc_bounds_from_starts, doc_bounds_from_tokens

    g = torch.Generator(device="cuda").manual_seed(3)
    for t, p in ((1, 0.5), (77, 0.1), (1024, 0.01), (49152, 0.001), (5000, 0.0)):
        tok = torch.randint(0, 50, (t,), device="cuda", generator=g)
        tok = torch.where(torch.rand(t, device="cuda", generator=g) < p, torch.full_like(tok, 99), tok)
        s0, e0 = doc_bounds_from_starts(tok == 99)
        s1, e1 = doc_bounds_from_tokens(tok, 99)
        assert torch.equal(s0, s1) and torch.equal(e0, e1), t


@pytest.mark.parametrize("d,dv", [(32, 64), (16, 32), (64, 128)])
def test_differential_flash_attention_matches_two_sdpa_calls(d, dv):
    import torch.nn.functional as F

    from ml_experiments_b200.ops.attention import differential_flash_attention

    torch.manual_seed(d)
    B, L, H = 2, 200, 3
    mk = lambda w: torch.randn(B, L, H, w, device="cuda").bfloat16().float().requires_grad_(True)
    q1, k1, q2, k2, v = mk(d), mk(d), mk(d), mk(d), mk(dv)
    o1, o2 = differential_flash_attention(q1, k1, q2, k2, v)
    t = lambda x: x.transpose(1, 2)
    r1 = t(F.scaled_dot_product_attention(t(q1), t(k1), t(v), is_causal=True))
    r2 = t(F.scaled_dot_product_attention(t(q2), t(k2), t(v), is_causal=True))
    assert o1.shape == r1.shape and (o1.float() - r1).abs().max() < 3e-2 and (o2.float() - r2).abs().max() < 3e-2
    w1, w2 = torch.randn_like(r1), torch.randn_like(r2)
    (o1.float() * w1).sum().add((o2.float() * w2).sum()).backward()
    got = [x.grad.clone() for x in (q1, k1, q2, k2, v)]
    for x in (q1, k1, q2, k2, v):
        x.grad = None
    ((r1 * w1).sum() + (r2 * w2).sum()).backward()
    for name, g, x in zip("q1 k1 q2 k2 v".split(), got, (q1, k1, q2, k2, v)):
        rel = ((g - x.grad).norm() / x.grad.norm()).item()
        assert rel < 3e-2, (name, rel)


def test_causal_self_attention_module_uses_the_flash_path_in_eval():
    from ml_experiments_b200.models.ripple_ops import CausalSelfAttention

    torch.manual_seed(0)
    m = CausalSelfAttention(256, num_heads=4, differential=True).cuda().eval()
    x = torch.randn(2, 160, 256, device="cuda")
    y, _ = m(x)
    ref, _ = m.cpu()(x.cpu())
    assert (y.cpu() - ref).abs().max() < 5e-2 * ref.abs().max() + 1e-2



@pytest.mark.parametrize("t,starts,window,scale", [
    (1, [0], 0, 0.12), (127, [0], 0, 0.12), (129, [0, 5], 0, 0.12), (256, [0, 128], 1, 0.12), (257, [0, 250], 0, 0.12),
    (385, [0, 128, 256, 384], 0, 0.12), (1001, [0, 3, 130, 383, 640], 2, 0.12), (2300, [0, 700, 701, 2200], 0, -0.12),
    (640, [0], 0, 0.0), (20000, [0, 9000], 5, 0.5)])
@pytest.mark.parametrize("d", [128, 64])
def test_attention_forward_tile_edges(t, starts, window, scale, d):
    """Sequence ends, document starts and windows on and beside the 128 / 256 boundaries of the query pairs; scales of
    every sign; more work items than multiprocessors; the saved log-sum-exp."""
    from ml_experiments_b200.ops import attention as A

    h = 5 if t < 5000 else 2
    q, k, v, _, _ = _setup(t, h, d, t)
    is_start = torch.zeros(t, dtype=torch.bool, device="cuda")
    is_start[starts] = True
    ds, de = A.doc_bounds_from_starts(is_start)
    o, lse = A.flash_attention_forward(q, k, v, ds, de, scale, window)
    for lo in range(0, t, 5000):                                # rows in parts: a dense oracle of 20000 x 20000 is large
        sl = slice(lo, min(t, lo + 5000))
        m = A.attention_mask(ds, window)[sl]
        s = ((q[sl].float().transpose(0, 1) @ k.float().permute(1, 2, 0)) * scale).masked_fill(~m[None], float("-inf"))
        want = (torch.softmax(s, -1) @ v.float().transpose(0, 1)).transpose(0, 1)
        # bf16 probabilities and outputs: 2^-9 relative each, values up to ~4.5
        assert (o[sl].float() - want).abs().max().item() < 2e-2
        assert (lse[:, sl] * 0.6931471805599453 - torch.logsumexp(s, -1)).abs().max().item() < 1e-3


@pytest.mark.parametrize("t,starts,window", [(1, [0], 0), (129, [0, 5], 0), (256, [0, 128], 1), (385, [0, 127, 128, 129, 384], 0),
                                             (1001, [0, 3, 63, 64, 130, 383, 640], 2), (1100, [0, 700, 701], 0)])
@pytest.mark.parametrize("d", [128, 64])
def test_attention_backward_tile_edges(t, starts, window, d):
    """Document starts on and beside the 64-query and 128-key boundaries and several inside one tile."""
    from ml_experiments_b200.ops import attention as A

    q, k, v, _, _ = _setup(t, 3, d, t, seed=t)
    is_start = torch.zeros(t, dtype=torch.bool, device="cuda")
    is_start[starts] = True
    ds, de = A.doc_bounds_from_starts(is_start)
    d_o = torch.randn(t, 3, d, device="cuda", dtype=torch.bfloat16)
    ins = [x.float().detach().requires_grad_(True) for x in (q, k, v)]
    want = torch.autograd.grad(A.attention_reference(*ins, ds, 0.12, window), ins, d_o.float())
    o, lse = A.flash_attention_forward(q, k, v, ds, de, 0.12, window)
    got = A.flash_attention_backward(q, k, v, o, d_o, lse, ds, de, 0.12, window)
    for name, a, w in zip("qkv", got, want):     # bf16 P, dS and outputs: 2^-9 each (dq and dk vanish at one token)
        assert (a.float() - w).norm().item() <= 1e-2 * w.norm().item() + 1e-2, name


def _blocked_oracle(q, k, v, ds, scale, window):
    """The forward's rounding restated: keys in blocks of 64, the offset of a row's exponents raised where a block's maximum
    exceeds it by more than 8 (log2), probabilities rounded to bf16; sums and products in 64 bits."""
    from ml_experiments_b200.ops import attention as A

    t = q.shape[0]
    sl2 = torch.tensor(scale, dtype=torch.float32) * torch.tensor(1.4426950408889634, dtype=torch.float32)
    s = (q.double().transpose(0, 1) @ k.double().permute(1, 2, 0)).float() * sl2.item()
    s = s.masked_fill(~A.attention_mask(ds, window)[None], float("-inf"))
    m = s.new_full(s.shape[:2], float("-inf"))
    l, o = torch.zeros_like(m, dtype=torch.float64), torch.zeros_like(q, dtype=torch.float64).transpose(0, 1)
    for lo in range(0, t, 64):
        x = s[:, :, lo:lo + 64]
        top = x.amax(-1)
        new = torch.where(top > m + 8, top, m)
        alpha = torch.where(new == m, torch.ones_like(m), torch.exp2(m - new)).double()
        m = new
        p = torch.exp2(x - torch.where(m == float("-inf"), torch.zeros_like(m), m)[..., None])
        l = l * alpha + p.double().sum(-1)
        o = o * alpha[..., None] + p.bfloat16().double() @ v.double().transpose(0, 1)[:, lo:lo + 64]
    return (o / l[..., None]).transpose(0, 1)


@pytest.mark.parametrize("t", [64, 65, 128, 192, 250, 320, 384, 449, 830])
@pytest.mark.parametrize("d", [128, 64])
def test_attention_backward_tiles_in_turn(t, d):
    """One to thirteen query tiles a key tile: first and last turns of the buffers (two groups of warps, three sets of scores, three or six
    of queries), and how the report at the end finds each of them."""
    from ml_experiments_b200.ops import attention as A

    q, k, v, ds, de = _setup(t, 2, d, t, seed=t)
    dy = torch.randn(t, 2, d, device="cuda").bfloat16()
    grads = []
    for fn, dt in ((lambda *x: A.flash_attention(*x, ds, de, 0.12, 0), torch.bfloat16), (lambda *x: A.attention_reference(*x, ds, 0.12), torch.float32)):
        ins = [u.detach().to(dt).requires_grad_() for u in (q, k, v)]
        grads.append(torch.autograd.grad(fn(*ins), ins, dy.to(dt)))
    for got, want in zip(*grads):
        assert ((got.float() - want).norm() / want.norm()).item() < 1.5e-2     # bf16 probabilities and results


@pytest.mark.parametrize("t,starts,window", [(64, [0], 0), (200, [0], 0), (513, [0, 70, 190, 333], 0), (1500, [0, 900], 0),
                                             (1500, [0], 3)])
@pytest.mark.parametrize("rising", [False, True])
@pytest.mark.parametrize("d", [128, 64])
def test_attention_forward_rounds_per_64_keys(t, starts, window, rising, d):
    from ml_experiments_b200.ops import attention as A

    q, k, v, _, _ = _setup(t, 3, d, t, seed=t + d)
    if rising:       # later keys score higher, so that offsets are raised, inside of 128-key tiles too
        k = (k.float() * torch.linspace(0.05, 4, t, device="cuda")[:, None, None]).bfloat16()
    is_start = torch.zeros(t, dtype=torch.bool, device="cuda")
    is_start[starts] = True
    ds, de = A.doc_bounds_from_starts(is_start)
    o, _ = A.flash_attention_forward(q, k, v, ds, de, 0.12, window)
    want = _blocked_oracle(q, k, v, ds, 0.12, window).bfloat16()
    # with the same offsets only the last bits of the fp32 scores, exponentials (2^-22) and sums differ; that moves one
    # output in some hundred over a bf16 boundary. Another offset rounds the probabilities anew (2^-9) and moves one in three.
    assert (o != want).float().mean().item() < 0.03


@pytest.mark.parametrize("pairs", [37, 74, 75, 150, 223, 400])
@pytest.mark.parametrize("t", [128, 300, 640])
@pytest.mark.parametrize("d", [128, 64])
def test_attention_forward_items_of_one_and_two_tiles(pairs, t, d):
    """Heads such that the pairs of query tiles are around half of the multiprocessors and just above one and two rounds of
    them: all single tiles, all pairs, pairs and a last round of singles; one, three and five tiles a head."""
    from ml_experiments_b200.ops import attention as A

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    h = max(1, pairs * sms // 148 // ((t + 255) // 256))
    q, k, v, _, _ = _setup(t, h, d, t, seed=pairs + t)
    is_start = torch.zeros(t, dtype=torch.bool, device="cuda")
    is_start[::130] = True
    ds, de = A.doc_bounds_from_starts(is_start)
    for starts in (ds, torch.zeros_like(ds)):
        o, lse = A.flash_attention_forward(q, k, v, starts, torch.full_like(de, t) if starts is not ds else de, 0.12)
        want = A.attention_reference(q, k, v, starts, 0.12)
        assert (o.float() - want).abs().max().item() < 2e-2      # bf16 probabilities and outputs, values up to ~4.5
        assert bool(lse.isfinite().all())


@pytest.mark.parametrize("d", [128, 64])
def test_attention_forward_captured_after_a_call_of_another_size(d):
    """A call of few tiles readies the build that a call of many takes: the latter may come first in a capture."""
    from ml_experiments_b200.ops import attention as A
    from ml_experiments_b200.ops.runtime import ops, status

    def args(t, h):
        q, k, v, _, _ = _setup(t, h, d, t, seed=t)
        ds, de = A.doc_bounds_from_starts(torch.zeros(t, dtype=torch.bool, device="cuda"))
        return q, k, v, torch.empty_like(q), torch.empty(h, t, device="cuda"), ds, de, 0.12, 0, status(q.device)

    small, large = args(200, 1), args(1024, 60)
    ops().attn_fwd(*small)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops().attn_fwd(*large)
    graph.replay()
    got = large[3].clone()
    ops().attn_fwd(*large)
    assert torch.equal(got, large[3]) and bool(got.isfinite().all())
