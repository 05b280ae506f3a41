"""Training calls where operators are looked at or tensors have no memory: fake tensors, tracing, vmap, batched gradients, dispatch modes.
Outside of these the calls bypass the dispatcher (ops._Train, projected._Projected); inside they must not."""
import pytest
import torch

from flashdeberta_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"
KW = dict(max_seqlen=96, position_buckets=32, max_relative_positions=64)


def _leaves(device, batch=2):
    g = torch.Generator().manual_seed(3)
    make = lambda *s: torch.randn(*s, generator=g).bfloat16().to(device).requires_grad_(True)
    return [make(batch, 96, 2, 64) for _ in range(3)] + [make(2, 64, 64) for _ in range(2)]


def test_forward_and_backward_on_fake_tensors():
    """Shapes of a training step without its memory, as a memory planner or an ahead-of-time tracer asks for them."""
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode():
        leaves = [torch.empty(*s, dtype=torch.bfloat16, device="cuda", requires_grad=True) for s in [(2, 96, 2, 64)] * 3 + [(2, 64, 64)] * 2]
        out = ops.disentangled_attention(*leaves, **KW)
        grads = torch.autograd.grad(out, leaves, torch.empty_like(out))
    assert out.shape == (2, 96, 2, 64) and out.dtype == torch.bfloat16
    assert [g.shape for g in grads] == [t.shape for t in leaves]


def _module():
    from flashdeberta_b200.attention import FlashDisentangledSelfAttention
    from tests.test_configs_gpu import _small_config
    torch.manual_seed(5)
    return FlashDisentangledSelfAttention(_small_config("b200")).bfloat16().train()


def test_module_on_fake_tensors():
    from torch._subclasses.fake_tensor import FakeTensorMode
    module = _module()
    with FakeTensorMode(allow_non_fake_inputs=True):
        module = module.to("cuda")
        x = torch.empty(2, 96, 256, dtype=torch.bfloat16, device="cuda", requires_grad=True)
        rel = torch.empty(512, 256, dtype=torch.bfloat16, device="cuda")
        out, _ = module(x, torch.ones(2, 96, device="cuda"), rel_embeddings=rel)
        grad, = torch.autograd.grad(out, x, torch.empty_like(out))
    assert out.shape == grad.shape == x.shape


def test_vmap_over_a_training_call():
    leaves = _leaves(DEV, batch=3)
    call = lambda q, k, v: ops.disentangled_attention(q, k, v, *leaves[3:], **KW)
    out = torch.vmap(call)(*(t.unsqueeze(1) for t in leaves[:3]))
    want = torch.cat([call(*(t[i:i + 1] for t in leaves[:3])) for i in range(3)])
    assert torch.equal(out[:, 0], want)


def _spread(run, leaves, out_shape):
    """Gradients of two output gradients: one after the other, and as one batch."""
    g = torch.Generator().manual_seed(4)
    douts = torch.randn(2, *out_shape, generator=g).bfloat16().to(DEV)
    single = [torch.autograd.grad(run(), leaves, d) for d in douts]
    batched = torch.autograd.grad(run(), leaves, douts, is_grads_batched=True)
    for i, b in enumerate(batched):
        want = torch.stack([s[i] for s in single])
        err = (b.float() - want.float()).norm() / want.float().norm().clamp_min(1e-30)
        assert b.shape == want.shape and err < 1e-2, (i, err.item())


def test_batched_gradients_of_the_operator():
    leaves = _leaves(DEV)
    _spread(lambda: ops.disentangled_attention(*leaves, **KW), leaves, (2, 96, 2, 64))


def test_batched_gradients_of_the_module():
    module = _module().to(DEV)
    x = torch.randn(2, 96, 256, device=DEV).bfloat16().requires_grad_(True)
    rel = torch.randn(515, 256, device=DEV).bfloat16().requires_grad_(True)
    mask = (torch.arange(96, device=DEV)[None] < torch.tensor([96, 50], device=DEV)[:, None]).long()
    leaves = [x, rel, *(p for n, p in module.named_parameters() if n != "key_proj.bias")]  # (that gradient cancels to rounding)
    _spread(lambda: module(x, mask, rel_embeddings=rel)[0], leaves, (2, 96, 256))


def test_dispatch_modes_see_the_attention():
    from torch.utils._python_dispatch import TorchDispatchMode

    class Seen(TorchDispatchMode):
        def __init__(self):
            super().__init__()
            self.names = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.names.append(func.name())
            return func(*args, **(kwargs or {}))

    from flashdeberta_b200 import FlashDebertaV2Model
    from tests.test_configs_gpu import _small_config
    model = FlashDebertaV2Model(_small_config("b200")).eval().to(DEV).bfloat16()
    with torch.no_grad(), Seen() as seen:  # inference: the linear layers
        model(input_ids=torch.ones(1, 40, dtype=torch.int64, device=DEV))
    assert sum("addmm" in n or "linear" in n for n in seen.names) >= 3 * 5
    leaves, module = _leaves(DEV), _module().to(DEV)
    x = torch.randn(2, 96, 256, device=DEV).bfloat16().requires_grad_(True)
    rel = torch.randn(512, 256, device=DEV).bfloat16()
    for run in (lambda: ops.disentangled_attention(*leaves, **KW), lambda: module(x, None, rel_embeddings=rel)[0]):
        with Seen() as seen:
            run().sum().backward()
        assert "flashdeberta_b200::attn_fwd_train" in seen.names and "flashdeberta_b200::attn_bwd" in seen.names


@pytest.mark.parametrize("mode", ["real", "fake"])
def test_make_fx_records_the_attention(mode):
    from torch.fx.experimental.proxy_tensor import make_fx
    leaves = _leaves(DEV)

    def step(q, k, v, pk, pq):
        out = ops.disentangled_attention(q, k, v, pk, pq, **KW)
        return torch.autograd.grad(out, (q, k, v, pk, pq), torch.ones_like(out))

    traced = make_fx(step, tracing_mode=mode)(*leaves)
    assert "attn_fwd_train" in traced.code and "attn_bwd" in traced.code
    other = [(2 * t).detach().requires_grad_(True) for t in leaves]
    for a, b in zip(traced(*other), step(*other)):
        assert (a.float() - b.float()).norm() <= 1e-2 * b.float().norm()


def test_saved_tensors_may_be_stored_elsewhere():
    """Hooks that keep what the backward needs on the host: the addresses are those of what comes back."""
    leaves, module = _leaves(DEV), _module().to(DEV)
    x = torch.randn(2, 96, 256, device=DEV).bfloat16().requires_grad_(True)
    rel = torch.randn(512, 256, device=DEV).bfloat16().requires_grad_(True)
    for run, wrt in ((lambda: ops.disentangled_attention(*leaves, **KW), leaves),
                     (lambda: module(x, None, rel_embeddings=rel)[0], [x, rel, *module.parameters()])):
        want = torch.autograd.grad(run().sum(), wrt)
        with torch.autograd.graph.save_on_cpu():
            out = run()
        junk = [torch.full((1 << 20,), float("nan"), device=DEV) for _ in range(8)]
        for a, b in zip(torch.autograd.grad(out.sum(), wrt), want):
            assert torch.equal(a, b)
        del junk
