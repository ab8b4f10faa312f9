"""The operators with gradients disabled take a shorter way to the same kernels: same bits, shapes and types as with them
enabled, and nothing that requires a gradient."""
import pytest
import torch

from tinyinfinitrain_b200 import ops

pytestmark = pytest.mark.gpu
BF, F32 = torch.bfloat16, torch.float32


def _rnd(dtype, *shape, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, device="cuda", generator=g).to(dtype).requires_grad_()


def _x(dtype, seed=1):
    return _rnd(dtype, 2, 65, 128, seed=seed)


CASES = {
    "linear": lambda d: (ops.linear, _x(d), _rnd(d, 96, 128)),
    "linear bias": lambda d: (ops.linear, _x(d), _rnd(d, 96, 128), _rnd(d, 96)),
    "linear bias residual": lambda d: (ops.linear, _x(d), _rnd(d, 128, 128), _rnd(d, 128), _x(d, 2)),
    "linear strided": lambda d: (ops.linear, _rnd(d, 65, 2, 128).transpose(0, 1), _rnd(d, 96, 128)),
    "mlp": lambda d: (ops.mlp_gelu, _x(d), _rnd(d, 512, 128), _rnd(d, 512), _rnd(d, 128, 512), _rnd(d, 128)),
    "mlp residual": lambda d: (ops.mlp_gelu, _x(d), _rnd(d, 512, 128), _rnd(d, 512), _rnd(d, 128, 512), _rnd(d, 128), _x(d, 2)),
    "layernorm": lambda d: (ops.layernorm, _x(d), _rnd(d, 128), _rnd(d, 128)),
    "layernorm fork": lambda d: (ops.layernorm_fork, _x(d), _rnd(d, 128), _rnd(d, 128)),
    "rmsnorm": lambda d: (ops.rmsnorm, _x(d), _rnd(d, 128)),
    "rmsnorm fork": lambda d: (ops.rmsnorm_fork, _x(d), _rnd(d, 128)),
    "gelu": lambda d: (ops.gelu, _x(d)),
    "swiglu": lambda d: (ops.swiglu, _x(d)),
    "embedding": lambda d: (ops.embedding, torch.arange(130, device="cuda").view(2, 65) % 50, _rnd(d, 50, 128), _rnd(d, 65, 128)),
    "attention qkv": lambda d: (ops.causal_attention_qkv, _rnd(d, 2, 65, 4 * 64), 2, 1),
    "attention": lambda d: (ops.causal_attention, _rnd(d, 2, 65, 2, 64), _rnd(d, 2, 65, 1, 64), _rnd(d, 2, 65, 1, 64)),
}


@pytest.mark.parametrize("dtype", [BF, F32], ids=["bf16", "fp32"])
@pytest.mark.parametrize("name", CASES)
def test_operator_without_gradients(name, dtype):
    f, *args = CASES[name](dtype)
    with_grad = f(*args)
    with torch.no_grad():
        without = f(*args)
    with torch.inference_mode():
        inference = f(*args)
    tup = lambda r: r if isinstance(r, tuple) else (r,)
    for a, b, c in zip(tup(with_grad), tup(without), tup(inference)):
        assert a.requires_grad and not b.requires_grad and not c.requires_grad
        assert a.shape == b.shape == c.shape and a.dtype == b.dtype == c.dtype and a.stride() == b.stride()
        assert torch.equal(a, b) and torch.equal(a, c)
    # what came back without gradients can be written to without touching the graph of the first result
    grads = torch.autograd.grad(sum(r.float().sum() for r in tup(with_grad)), [a for a in args if torch.is_tensor(a) and a.requires_grad])
    assert all(torch.isfinite(g).all() for g in grads)
