"""The count of kernel launches against the kernels that the profiler sees on the GPU."""
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from multimesh_jax_b200.ops import _lib, attention
from multimesh_jax_b200.ops import kernels as K
from multimesh_jax_b200.ops.moe import moe_ffn

pytestmark = pytest.mark.gpu


def _rand(*shape):
    return torch.randn(*shape, device="cuda").bfloat16()


def _norm_gradient(rows, D):
    x, w, dy, rstd = _rand(rows, D), _rand(D), _rand(rows, D), torch.rand(rows, device="cuda") + 0.5
    return lambda: K.rmsnorm_bwd(x, w, dy, rstd)


def _attention_gradient(S):
    qkv, dout = _rand(2, S, 3, 128), _rand(2, S, 1, 128)
    out, lse = attention.attention_fwd_packed(qkv, 1)
    return lambda: attention.attention_bwd_packed(dout, qkv, out, lse, 1)


def _linear_gradient(T, N, Kd):
    dy, w, x, dx, dw = _rand(T, N), _rand(N, Kd), _rand(T, Kd), _rand(T, Kd), torch.empty(N, Kd, device="cuda")
    return lambda: _lib.load().mm_linear_bwd_bf16(*[t.data_ptr() for t in (dy, w, x, dx, dw)], 1, T, N, Kd, K.PAIR_MIN_M, K._stream())


def _updates(n):
    ts = [[torch.zeros(n, device="cuda", dtype=torch.bfloat16 if k == 1 else torch.float32) for k in range(5)] for _ in range(3)]
    step = torch.tensor([1], device="cuda")
    args = [a for t in ts for a in (*[x.data_ptr() for x in t], n)]
    return lambda: _lib.load().mm_adamw_group(*args, 1e-3, 0.9, 0.95, 1e-8, 0.1, 1.0, step.data_ptr(), K._stream())


def _experts():
    x, wr, wgu, wdown = _rand(64, 128), _rand(4, 128), _rand(4, 2, 256, 128), _rand(4, 128, 256)
    ins = [t.requires_grad_(True) for t in (x, wr, wgu, wdown)]
    return lambda: torch.autograd.grad(moe_ffn(*ins, 2).sum(), ins)


@pytest.mark.parametrize("make,expected", [
    (lambda: _norm_gradient(100, 256), 1), (lambda: _norm_gradient(100, 2048), 2),
    (lambda: _attention_gradient(128), 1), (lambda: _attention_gradient(129), 3),
    (lambda: _linear_gradient(256, 256, 256), 1), (lambda: _linear_gradient(4096, 4096, 256), 2),
    (lambda: _updates(1 << 10), 1), (lambda: _updates(1 << 24), 3), (_experts, 19)],
    ids=["norm-one", "norm-two", "attention-one", "attention-three", "linear-one", "linear-two", "adamw-one", "adamw-three", "experts"])
def test_every_kernel_launch_is_counted_once(make, expected):
    step = make()
    step()
    torch.cuda.synchronize()
    before = K.launch_count
    with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as prof:
        step()
        torch.cuda.synchronize()
    seen = sum("mm::" in e.name for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA)
    assert K.launch_count - before == seen == expected
