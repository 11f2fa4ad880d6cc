"""Ways out of a kernel that would wait for ever: the device status word (after a wait has expired, kernels leave before they
touch anything, and a CTA leaves as a whole), and the check of register splits."""
import re
from pathlib import Path

import pytest
import torch


def test_no_thread_returns_by_its_own_read_of_the_status_word():
    """Warps of a CTA that read the word at different times must not part: named barriers, register allocation and
    tensor-memory set-up of the rest would wait for ever. (Shown on the source: the race cannot be provoked safely.)"""
    csrc = Path(__file__).resolve().parent.parent / "ml_experiments_b200" / "csrc"
    for path in sorted(csrc.rglob("*.cu")):
        found = re.findall(r"status_poisoned\([^;{]*\)\)\s*\{?\s*return", path.read_text())
        assert not found, (path.name, found)


@pytest.mark.gpu
@pytest.mark.parametrize("op", ["attn_fwd", "attn_bwd", "gemm", "gemm_pair", "ssd_fwd"])
def test_kernels_leave_at_once_while_the_word_is_set(op):
    from ml_experiments_b200.ops import attention as A
    from ml_experiments_b200.ops.runtime import check_status, ops, status

    t, h, d = 300, 2, 128
    bf = lambda *s: torch.randn(*s, device="cuda").bfloat16()  # noqa: E731
    mark = lambda *s, dt=torch.bfloat16: torch.full(s, 7.0, device="cuda", dtype=dt)  # noqa: E731
    st = status()
    if op.startswith("attn"):
        q, k, v, d_o = (bf(t, h, d) for _ in range(4))
        ds, de = A.doc_bounds_from_starts(torch.zeros(t, dtype=torch.bool, device="cuda"))
        o, lse = A.flash_attention_forward(q, k, v, ds, de, 0.12)
        if op == "attn_fwd":
            outs = [mark(t, h, d), mark(h, t, dt=torch.float32)]
            call = lambda: ops().attn_fwd(q, k, v, *outs, ds, de, 0.12, 0, st)  # noqa: E731
        else:
            outs = [mark(t, h, d, dt=torch.float32), mark(t, h, d), mark(t, h, d)]
            delta = torch.empty(h, t, device="cuda")
            call = lambda: ops().attn_bwd(q, k, v, o, d_o, lse, delta, *outs, ds, de, 0.12, 0, st)  # noqa: E731
    elif op.startswith("gemm"):
        m, k = (256, 128) if op == "gemm" else (40960, 2048)         # by pairs of CTAs, whose both must leave
        a, b, outs = bf(m, k), bf(384, k), [mark(m, 384)]
        call = lambda: ops().gemm(a, b, outs[0], None, False, False, 0, 1.0, 0.0, 1, False, st)  # noqa: E731
    else:
        x, B, C = bf(1, 256, 2, 64), bf(1, 256, 2, 64), bf(1, 256, 2, 64)
        la, g, outs = -torch.rand(1, 256, 2, device="cuda"), torch.rand(1, 256, 2, device="cuda"), [mark(1, 256, 2, 64)]
        call = lambda: ops().ssd_fwd(x, B, C, la, g, g, outs[0], None, None, st)  # noqa: E731
    st.fill_(6)
    call()
    with pytest.raises(RuntimeError):
        check_status()                       # clears the word
    assert all(bool((u == 7.0).all()) for u in outs)
    call()
    check_status()
    assert all(bool((u != 7.0).any()) for u in outs)


def test_register_splits_are_checked_against_what_the_block_was_launched_with():
    """What the attention forward asks before its first launch: a build with fewer registers a thread must be refused, as its
    setmaxnreg would wait for ever."""
    from ml_experiments_b200.ops.runtime import ops

    need = 256 * 208 + 128 * 88
    fits = ops().register_split_fits
    assert fits(168, 384, need) and fits(161, 384, need)          # registers are handed out 8 a thread
    assert not fits(160, 384, need) and not fits(128, 384, need)
    source = (Path(__file__).resolve().parent.parent / "ml_experiments_b200" / "csrc" / "attn" / "attn_sm100.cu").read_text()
    assert source.index("register_split_fits(attr.numRegs") < source.index("launch_early(kern, grid, FWD_THREADS")
