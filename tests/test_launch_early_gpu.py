"""Kernels that start under the end of the one before (programmatic dependent launch): chains in which each reads what the last wrote,
and overwrites what it read, give the bits of the same chains with a synchronisation after every launch; so do their CUDA graphs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _chain(x, w, qkv, lam, cos, sin, bounds, h, d, pause):
    from ml_experiments_b200.ops import attention as A, fused as Fz, gemm as G
    from ml_experiments_b200.ops.runtime import ops

    t, c = x.shape
    y = torch.empty(t, 3 * c, device=x.device, dtype=torch.bfloat16)
    z = torch.empty(t, c, device=x.device, dtype=torch.bfloat16)
    dlam = torch.zeros(2, device=x.device)
    packed, dqkv = torch.empty(t, 3, h, d, device=x.device, dtype=torch.bfloat16), torch.empty_like(qkv)
    keep = []
    for _ in range(3):
        x = Fz.rmsnorm(x); pause()
        G.gemm(x, w, out=y); pause()                                              # [t, 3 c], overwritten on each pass
        ops().qkv_post_fwd(y.view(t, 3, h, d), None, lam, cos, sin, packed, h, d, 1e-6); pause()
        q, k, v = packed.unbind(1)
        o, lse = A.flash_attention_forward(q, k, v, *bounds, 0.1); pause()
        dq, dk, dv = A.flash_attention_backward(q, k, v, o, o, lse, *bounds, 0.1); pause()
        ops().qkv_post_bwd(torch.zeros_like(dq), dk, dv, y.view(t, 3, h, d), None, lam, cos, sin, dqkv, None, dlam, h, d, 1e-6); pause()
        G.gemm(dqkv.view(t, 3 * c), w, b_mn=True, out=z); pause()
        x = Fz.norm_bwd_add(z, x, o.view(t, c)); pause()
        keep += [o.clone(), dk, dv, z.clone(), x.clone()]
    return keep


@pytest.mark.parametrize("t,h,d", [(72, 1, 128), (1000, 6, 128), (4096, 3, 64), (20000, 6, 64)])
def test_a_chain_is_the_chain_with_waits(t, h, d):
    from ml_experiments_b200.ops.attention import doc_bounds_from_starts
    from ml_experiments_b200.ops.fused import rotary_tables

    torch.manual_seed(0)
    c = h * d
    x = torch.randn(t, c, device="cuda").bfloat16()
    w = (torch.randn(3 * c, c, device="cuda") / c ** 0.5).bfloat16()
    qkv = torch.empty(t, 3, h, d, device="cuda", dtype=torch.bfloat16)
    lam = torch.tensor([0.8, 0.2], device="cuda")
    cos, sin = rotary_tables(d, t, "cuda")
    starts = torch.zeros(t, dtype=torch.bool, device="cuda")
    starts[::t // 3] = True
    args = (x, w, qkv, lam, cos, sin, doc_bounds_from_starts(starts), h, d)
    want = _chain(*args, torch.cuda.synchronize)
    got = _chain(*args, lambda: None)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = _chain(*args, lambda: None)
    for g in got:
        g.zero_()
    graph.replay()
    graph.replay()
    assert all(torch.equal(a, b) for a, b in zip(got, want))


def _block_chain(x, x0, lam, fc, pj, h, buf, d, acc, dw, dlam, pause):
    """An MLP forward and backward around a mix: aux operands written by the launch in front, a weight gradient into a cleared buffer."""
    from ml_experiments_b200.ops import fused as Fz, gemm as G
    from ml_experiments_b200.ops.runtime import ops

    keep = []
    for _ in range(2):
        mix, xn = Fz.mix_norm(x, x0, lam); pause()
        G.gemm(xn, fc, out=h, epilogue=G.EPI_RELU2); pause()
        G.gemm(h, pj, out=buf, epilogue=G.EPI_AXPBY, aux=mix, beta=1.0); pause()                # aux from two launches before
        G.gemm(buf, pj, b_mn=True, out=d, epilogue=G.EPI_RELU2_BWD, aux=h); pause()             # `buf` from the launch in front
        G.gemm(d, xn, a_mn=True, b_mn=True, out=dw, split_k=2); pause()
        G.gemm(d, fc, b_mn=True, out=buf); pause()
        G.gemm(xn, fc, out=h, epilogue=G.EPI_AXPBY, aux=d, beta=0.5); pause()                   # aux from three, `h` overwritten
        G.gemm(h, pj, out=xn, epilogue=G.EPI_AXPBY, aux=buf, beta=1.0); pause()
        dx = Fz.norm_bwd_add(xn, mix, buf); pause()
        x, _ = ops().gpt_mix_bwd(dx, mix, x0, None, lam, None, acc, dlam, None, xn); pause()
        keep += [mix, h.clone(), buf.clone(), d.clone(), dw.clone(), dx, x, acc.clone()]
    return keep


@pytest.mark.parametrize("t,c", [(1000, 256), (20000, 768)])
def test_a_block_is_the_block_with_waits(t, c):
    from ml_experiments_b200.ops.runtime import ops

    torch.manual_seed(1)
    bf = lambda *s: torch.randn(*s, device="cuda").bfloat16()  # noqa: E731
    x, x0, fc, pj = bf(t, c), bf(t, c), bf(4 * c, c) * c ** -0.5, bf(c, 4 * c) * c ** -0.5
    assert ops().gemm_by_pairs(t, 4 * c, c, 1, False, 2, 1) == ops().gemm_by_pairs(t, c, 4 * c, 1, False, 2, 1) == (t == 20000)
    lam, dlam = torch.tensor([0.8, 0.2], device="cuda"), torch.zeros(2, device="cuda")          # (dlam: added up in any order)
    h, buf, d, acc, dw = bf(t, 4 * c), bf(t, c), bf(t, 4 * c), torch.zeros(t, c, device="cuda"), torch.empty(4 * c, c, device="cuda")
    args = (x, x0, lam, fc, pj, h, buf, d, acc, dw, dlam)
    want = _block_chain(*args, torch.cuda.synchronize)
    acc.zero_()
    got = _block_chain(*args, lambda: None)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        acc.zero_()
        got = _block_chain(*args, lambda: None)
    for g in got:
        g.zero_()
    graph.replay()
    graph.replay()
    assert all(torch.equal(a, b) for a, b in zip(got, want))


def _dq_chain(qkv, packed, lam, cos, sin, bounds, dq, dqkv, dlam, h, d, eps, pause):
    from ml_experiments_b200.ops import attention as A
    from ml_experiments_b200.ops.runtime import ops

    keep = []
    for _ in range(3):
        ops().qkv_post_fwd(qkv, None, lam, cos, sin, packed, h, d, eps); pause()
        q, k, v = packed.unbind(1)
        o, lse = A.flash_attention_forward(q, k, v, *bounds, 0.1); pause()
        dq.zero_(); pause()
        _, dk, dv = A.flash_attention_backward(q, k, v, o, o, lse, *bounds, 0.1, 0, dq); pause()
        ops().qkv_post_bwd(dq, dk, dv, qkv, None, lam, cos, sin, dqkv, None, dlam, h, d, eps); pause()    # right behind the TMA additions to dq
        ops().qkv_post_fwd(dqkv, None, lam, cos, sin, packed, h, d, eps); pause()
        qkv = packed.clone()
        keep += [o, dq.clone(), dqkv.clone(), qkv]
    return keep


@pytest.mark.parametrize("t,h,d", [(128, 1, 128), (1000, 6, 128), (1000, 4, 64), (20000, 6, 128), (20000, 6, 64)])
def test_dq_is_read_as_a_whole(t, h, d):
    """Documents of 128 tokens: a row of dQ is one addition to zero, so that its bits are the same in any order."""
    from ml_experiments_b200.ops.attention import doc_bounds_from_starts
    from ml_experiments_b200.ops.fused import rotary_tables

    torch.manual_seed(2)
    bf = lambda *s: torch.randn(*s, device="cuda").bfloat16()  # noqa: E731
    qkv, packed, dqkv = bf(t, 3, h, d), bf(t, 3, h, d), bf(t, 3, h, d)
    lam, dlam = torch.tensor([0.8, 0.2], device="cuda"), torch.zeros(2, device="cuda")
    starts = torch.zeros(t, dtype=torch.bool, device="cuda")
    starts[::128] = True
    args = (qkv, packed, lam, *rotary_tables(d, t, "cuda"), doc_bounds_from_starts(starts), torch.empty(t, h, d, device="cuda"), dqkv, dlam, h, d, 1e-6)
    want = _dq_chain(*args, torch.cuda.synchronize)
    for _ in range(3):
        assert all(torch.equal(a, b) for a, b in zip(_dq_chain(*args, lambda: None), want))
