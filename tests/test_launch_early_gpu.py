"""Kernels that start under the end of the one before (programmatic dependent launch): a chain in which each reads what the last wrote,
and overwrites what it read, gives the bits of the same chain with a synchronisation after every launch; so does its CUDA graph."""
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
