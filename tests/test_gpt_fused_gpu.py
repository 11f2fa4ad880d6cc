"""Fused GPT step (loss and every parameter gradient) against the plain PyTorch path of the same module."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(fp8):
    from ml_experiments_b200.models.gpt import GPT, GPTConfig

    torch.manual_seed(0)
    cfg = GPTConfig(vocab_size=50257, num_layers=4, num_heads=2, model_dim=256, head_dim=128, max_seq_len=2048,
                    skip_attn_layers=(2,), num_value_embeds=1, use_fp8_head=fp8)
    m = GPT(config=cfg).cuda().cast_embeddings_bf16()
    # non-trivial values for the zero-initialised / identity parameters so every gradient path is exercised
    with torch.no_grad():
        for blk in m.blocks:
            blk.lambdas.copy_(torch.tensor([0.9, 0.2]))
            blk.mlp.c_proj.weight.normal_(0, 0.02)
            if blk.attn is not None:
                blk.attn.c_proj.weight.normal_(0, 0.02)
                blk.attn.lambdas.copy_(torch.tensor([0.6, 0.4]))
        m.lm_head.weight.normal_(0, 0.02)
        m.skip_weights.copy_(torch.tensor([0.8, 1.1]))
    return m


@pytest.mark.parametrize("fp8", [False, True])
def test_fused_matches_reference(fp8):
    m = _model(fp8)
    t = 2048
    x = torch.randint(0, 50257, (t,), device="cuda")
    x[::512] = 50256
    y = torch.randint(0, 50257, (t,), device="cuda")
    import copy

    oracle = copy.deepcopy(m).float()  # fp32 everywhere, plain autograd
    oracle.fused = False
    loss_ref = oracle(x, y, 2)
    loss_ref.backward()
    ref = {n: p.grad.float().clone() for n, p in oracle.named_parameters()}
    m.fused = True
    loss = m(x, y, 2)
    loss.backward()
    assert abs(loss.item() - loss_ref.item()) < 2e-2 * abs(loss_ref.item())
    tol = 0.12 if fp8 else 0.06
    for n, p in m.named_parameters():
        assert p.grad is not None, n
        assert p.grad.dtype == p.dtype and p.grad.shape == p.shape, n
        g, r = p.grad.float(), ref[n]
        rel = ((g - r).norm() / (r.norm() + 1e-12)).item()
        # scalar parameters have tiny gradients that are sums of bf16-rounded products: looser bound
        if p.ndim < 2:
            assert (g - r).norm().item() <= max(3 * tol * r.norm().item(), 3e-4), (n, rel, r.norm().item())
        else:
            assert rel < tol, (n, rel, r.norm().item())


def test_muon_fused_matches_torch():
    from ml_experiments_b200.optim import Muon

    torch.manual_seed(1)
    shapes = [(3, 256, 256), (256, 256), (1024, 256), (256, 1024)]
    ps = [torch.randn(s, device="cuda").requires_grad_(True) for s in shapes]
    qs = [p.detach().cpu().clone().requires_grad_(True) for p in ps]
    oa, ob = Muon(ps, lr=0.05, momentum=0.95), Muon(qs, lr=0.05, momentum=0.95)
    for _ in range(2):
        for p, q in zip(ps, qs):
            g = torch.randn_like(p)
            p.grad, q.grad = g, g.cpu()
        oa.step(); ob.step()
    for p, q in zip(ps, qs):
        delta = (p.detach().cpu() - q.detach()).norm() / (q.detach() - q.detach().round()).norm().clamp_min(1e-3)
        upd_err = (p.detach().cpu() - q.detach()).abs().max().item()
        assert upd_err < 2e-2, upd_err


def test_loss_and_grad_equals_backward_of_the_loss():
    """The trainer's direct path fills p.grad with what autograd would have produced, and accumulates on a second call."""
    m = _model(True)
    t = 1024
    x = torch.randint(0, 50257, (t,), device="cuda")
    y = torch.randint(0, 50257, (t,), device="cuda")
    loss = m(x, y, 2)
    loss.backward()
    want = {n: p.grad.clone() for n, p in m.named_parameters() if p.grad is not None}
    m.zero_grad(set_to_none=True)
    loss2 = m.loss_and_grad(x, y, 2)
    assert not loss2.requires_grad and torch.allclose(loss2, loss.detach())
    got = {n: p.grad for n, p in m.named_parameters() if p.grad is not None}
    assert set(got) == set(want)
    for n in want:
        assert got[n].dtype == want[n].dtype and got[n].shape == want[n].shape, n
        # weight-gradient GEMMs use split-K atomics: equal up to summation order
        assert (got[n].float() - want[n].float()).norm() <= 2e-3 * want[n].float().norm() + 1e-8, n
    m.loss_and_grad(x, y, 2)
    for n in want:
        assert (m.get_parameter(n).grad.float() - 2 * want[n].float()).norm() <= 1e-2 * (2 * want[n].float()).norm() + 1e-8, n


def test_gradient_hooks_are_called_before_the_rest_of_the_block_is_issued():
    """A hook hands a finished gradient over (to a collective, say): that of an output projection comes before its half of the block goes on:
    that of the MLP 3 kernels earlier, of the attention 6."""
    from ml_experiments_b200.ops.runtime import launch_count

    m = _model(False)
    t = 1024
    x, y = torch.randint(0, 50257, (t,), device="cuda"), torch.randint(0, 50257, (t,), device="cuda")
    m.loss_and_grad(x, y, 2)
    before = launch_count()
    m.loss_and_grad(x, y, 2)
    all_launches = launch_count() - before
    want = {n: p.grad.clone() / 2 for n, p in m.named_parameters()}
    called = {}
    m._grad_hooks = {id(p): lambda p, g, n=n: called.update({n: (launch_count(), g)}) for n, p in m.named_parameters() if p.dim() > 1}
    m.zero_grad(set_to_none=True)
    before = launch_count()
    m.loss_and_grad(x, y, 2)
    assert launch_count() - before == all_launches
    for i, blk in enumerate(m.blocks):
        at = {n[9:]: c[0] for n, c in called.items() if n.startswith(f"blocks.{i}.")}
        assert at["mlp.c_fc.weight"] - at["mlp.c_proj.weight"] == 3
        if blk.attn is not None:
            assert at["attn.qkv_w"] - at["attn.c_proj.weight"] >= 6        # and the scatter of a value embedding
    for n, p in m.named_parameters():
        if p.dim() > 1:
            assert called[n][1].shape == p.shape and torch.allclose(called[n][1].float(), want[n].float(), rtol=5e-2, atol=2e-3 * want[n].abs().max().item()), n


def test_muon_momentum_survives_a_state_dict_round_trip():
    """A momentum buffer restored from a checkpoint is moved into the optimizer's stacked buffer before the next step."""
    from ml_experiments_b200.optim import Muon

    torch.manual_seed(2)
    shapes = [(2, 256, 256), (256, 256), (512, 256)]
    grads = [[torch.randn(s, device="cuda") for s in shapes] for _ in range(3)]

    def run(resume_after):
        torch.manual_seed(3)
        ps = [torch.randn(s, device="cuda").requires_grad_(True) for s in shapes]
        opt = Muon(ps, lr=0.05, momentum=0.9)
        for step, gs in enumerate(grads):
            if step == resume_after:
                import copy
                sd = copy.deepcopy(opt.state_dict())
                opt = Muon(ps, lr=0.05, momentum=0.9)
                opt.load_state_dict(sd)
            for p, g in zip(ps, gs):
                p.grad = g.clone()
            opt.step()
        return [p.detach().clone() for p in ps]

    a, b = run(resume_after=-1), run(resume_after=2)
    for x, y in zip(a, b):
        assert torch.allclose(x, y, rtol=0, atol=1e-3)     # a lost momentum buffer would move the weights by ~5e-2
