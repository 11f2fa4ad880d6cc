"""tcgen05 GEMM against fp32 torch matmul: every operand majorness, ragged shapes, batches, epilogues, fp8."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(a, b, a_mn, b_mn):
    A = a.float().transpose(-1, -2) if a_mn else a.float()
    B = b.float().transpose(-1, -2) if b_mn else b.float()
    return A @ B.transpose(-1, -2)


def _rel_err(x, y):
    return ((x.float() - y).norm() / (y.norm() + 1e-12)).item()


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("m,n,k", [(128, 128, 64), (256, 512, 256), (384, 768, 1024), (200, 136, 72), (1024, 2304, 768)])
def test_gemm_bf16_majors(a_mn, b_mn, m, n, k):
    from ml_experiments_b200.ops.gemm import gemm

    torch.manual_seed(0)
    a = torch.randn((k, m) if a_mn else (m, k), device="cuda", dtype=torch.bfloat16)
    b = torch.randn((k, n) if b_mn else (n, k), device="cuda", dtype=torch.bfloat16)
    ref = _ref(a, b, a_mn, b_mn)
    out = gemm(a, b, a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32)
    assert _rel_err(out, ref) < 2e-3
    out16 = gemm(a, b, a_mn=a_mn, b_mn=b_mn)
    assert out16.dtype == torch.bfloat16
    assert _rel_err(out16, ref) < 6e-3


def test_gemm_batched_and_epilogues():
    from ml_experiments_b200.ops import gemm as G

    torch.manual_seed(1)
    a = torch.randn(3, 256, 320, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(3, 384, 320, device="cuda", dtype=torch.bfloat16)
    ref = _ref(a, b, False, False)
    assert _rel_err(G.gemm(a, b, out_dtype=torch.float32), ref) < 2e-3
    # relu^2
    out = G.gemm(a, b, epilogue=G.EPI_RELU2, alpha=0.05)
    assert _rel_err(out, torch.relu(ref * 0.05) ** 2) < 1e-2
    # alpha * acc + beta * aux
    aux = torch.randn(3, 256, 384, device="cuda", dtype=torch.bfloat16)
    out = G.gemm(a, b, epilogue=G.EPI_AXPBY, aux=aux, alpha=0.5, beta=-2.0, out_dtype=torch.float32)
    assert _rel_err(out, 0.5 * ref - 2.0 * aux.float()) < 2e-3
    # relu^2 backward: acc * 2 * sqrt(h)
    h = (torch.relu(torch.randn(3, 256, 384, device="cuda")) ** 2).bfloat16()
    out = G.gemm(a, b, epilogue=G.EPI_RELU2_BWD, aux=h, out_dtype=torch.float32)
    assert _rel_err(out, ref * 2 * h.float().sqrt()) < 2e-3


def test_gemm_split_k_and_accumulate():
    from ml_experiments_b200.ops import gemm as G

    torch.manual_seed(2)
    # weight-gradient shape: both operands MN-major, long K
    dy = torch.randn(8192, 768, device="cuda", dtype=torch.bfloat16)
    x = torch.randn(8192, 768, device="cuda", dtype=torch.bfloat16)
    ref = dy.float().T @ x.float()
    out = G.gemm(dy, x, a_mn=True, b_mn=True, split_k=8)
    assert out.dtype == torch.float32
    assert _rel_err(out, ref) < 2e-3
    out2 = G.gemm(dy, x, a_mn=True, b_mn=True, split_k=4, out=out.clone(), accumulate=True)
    assert _rel_err(out2, 2 * ref) < 2e-3


def test_gemm_strided_views():
    from ml_experiments_b200.ops import gemm as G

    torch.manual_seed(3)
    big = torch.randn(512, 3 * 256, device="cuda", dtype=torch.bfloat16)
    a = big[:, 256:512]  # row pitch 768, K = 256
    w = torch.randn(384, 256, device="cuda", dtype=torch.bfloat16)
    outbuf = torch.zeros(512, 1024, device="cuda", dtype=torch.bfloat16)
    G.gemm(a, w, out=outbuf[:, 128:512])
    assert _rel_err(outbuf[:, 128:512], a.float() @ w.float().T) < 6e-3
    assert outbuf[:, :128].abs().max().item() == 0 and outbuf[:, 512:].abs().max().item() == 0


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_gemm_fp8(a_mn, b_mn):
    from ml_experiments_b200.ops.gemm import gemm

    torch.manual_seed(4)
    m, n, k = 512, 640, 768
    a = torch.randn((k, m) if a_mn else (m, k), device="cuda").to(torch.float8_e4m3fn)
    b = torch.randn((k, n) if b_mn else (n, k), device="cuda").to(torch.float8_e5m2 if b_mn else torch.float8_e4m3fn)
    ref = _ref(a, b, a_mn, b_mn)
    out = gemm(a, b, a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32, alpha=0.25)
    assert _rel_err(out, 0.25 * ref) < 2e-3


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False)])
@pytest.mark.parametrize("m,n,k,batch", [(8193, 2312, 1096, None), (16384 + 128, 776, 1608, None), (640, 1032, 1032, 33), (776, 760, 3080, 16)])
def test_gemm_by_pairs(a_mn, b_mn, m, n, k, batch):
    """Products large enough for pairs of CTAs on tiles of 256 x 256: a last tile of one row, of one CTA only, of a few columns; a K that
    is no multiple of a stage; batches (33 of them leave too many tiles for the last round: by single CTAs); every epilogue."""
    from ml_experiments_b200.ops import gemm as G
    from ml_experiments_b200.ops.runtime import ops

    m = (m + 7) // 8 * 8 if a_mn else m          # (rows of 16-byte multiples)
    assert 2 * m * n * k * (batch or 1) >= 4e10
    assert ops().gemm_by_pairs(m, n, k, batch or 1, False, 2, 1) == (batch != 33)
    torch.manual_seed(7)
    pre = () if batch is None else (batch,)
    a = torch.randn(*pre, *((k, m) if a_mn else (m, k)), device="cuda", dtype=torch.bfloat16)
    b = torch.randn(*pre, *((k, n) if b_mn else (n, k)), device="cuda", dtype=torch.bfloat16)
    aux = torch.randn(*pre, m, n, device="cuda", dtype=torch.bfloat16).square()
    ref = _ref(a, b, a_mn, b_mn)
    kw = dict(a_mn=a_mn, b_mn=b_mn)
    assert _rel_err(G.gemm(a, b, **kw), ref) < 6e-3
    assert _rel_err(G.gemm(a, b, out_dtype=torch.float32, **kw), ref) < 2e-3
    assert _rel_err(G.gemm(a, b, epilogue=G.EPI_RELU2, alpha=0.05, **kw), torch.relu(ref * 0.05) ** 2) < 1e-2
    assert _rel_err(G.gemm(a, b, epilogue=G.EPI_AXPBY, aux=aux, alpha=0.5, beta=-2.0, **kw), 0.5 * ref - 2.0 * aux.float()) < 6e-3
    assert _rel_err(G.gemm(a, b, epilogue=G.EPI_RELU2_BWD, aux=aux, **kw), ref * 2 * aux.float().sqrt()) < 1e-2


@pytest.mark.parametrize("m,n,k,element_bytes,pairs", [
    (49152, 3072, 768, 2, True), (49152, 768, 3072, 2, True), (16384, 4096, 1536, 1, True),                       # 162, 174 us; 165, 173; 128, 140
    (49152, 3072, 256, 2, False), (49152, 5120, 384, 2, False), (49152, 1536, 512, 2, False),                     # 119, 90; 190, 169; 76, 72
    (49152, 50304, 768, 1, False), (16384, 50304, 768, 1, False), (49152, 768, 1024, 1, False)])                  # 2552, 1906; 726, 636; 46, 42
def test_pairs_only_where_they_are_faster(m, n, k, element_bytes, pairs):
    """Sizes at which both were timed (pairs, single CTAs): tiles of a few stages of K are not for pairs."""
    from ml_experiments_b200.ops.runtime import ops

    assert ops().gemm_by_pairs(m, n, k, 1, False, element_bytes, 1) == pairs


def test_gemm_fp8_by_pairs():
    from ml_experiments_b200.ops.gemm import gemm
    from ml_experiments_b200.ops.runtime import ops

    assert ops().gemm_by_pairs(3000, 5008, 1424, 1, False, 1, 1)

    torch.manual_seed(8)
    m, n, k = 3000, 5008, 1424
    a = torch.randn(m, k, device="cuda").to(torch.float8_e4m3fn)
    for b_mn in (False, True):
        b = torch.randn((k, n) if b_mn else (n, k), device="cuda").to(torch.float8_e5m2 if b_mn else torch.float8_e4m3fn)
        assert _rel_err(gemm(a, b, b_mn=b_mn, out_dtype=torch.float32, alpha=0.25), 0.25 * _ref(a, b, False, b_mn)) < 2e-3


_BACKWARD_FIRST = """
import torch
from ml_experiments_b200.ops.linear import linear
x, w = (torch.randn(128, 128, device="cuda", dtype=torch.bfloat16, requires_grad=True) for _ in range(2))
y = linear(x, w)
y.backward(torch.ones_like(y))
assert ((x.grad.float() - w.detach().float().sum(0)).abs() < 0.2).all()
"""


def test_a_product_as_the_first_operator_of_a_backward():
    """The thread of autograd has not touched the device then. (A process of its own: here it has.)"""
    import os
    import subprocess
    import sys

    r = subprocess.run([sys.executable, "-c", _BACKWARD_FIRST], capture_output=True, text=True, timeout=300,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0, r.stderr[-500:]


def test_output_aliasing_an_operand_is_refused():
    """In-place products are a timing-dependent race between CTAs (one stores a tile of the operand another still
    reads); the front end rejects them instead of returning numbers that are right most of the time."""
    from ml_experiments_b200.ops import gemm as G

    x = torch.randn(4, 256, 256, device="cuda").bfloat16()
    w = torch.randn(4, 256, 256, device="cuda").bfloat16()
    with pytest.raises(ValueError, match="alias"):
        G.gemm(w, x, b_mn=True, out=x)
    with pytest.raises(ValueError, match="alias"):
        G.gemm(x, w, out=x[:, :, :])
    out = torch.empty_like(x)
    G.gemm(w, x, b_mn=True, out=out, epilogue=G.EPI_AXPBY, aux=x, alpha=1.0, beta=0.5)      # aux may be an operand
