"""Fused element-wise kernels against the separate ones they replace."""
import pytest
import torch

from multimesh_jax_b200.ops import _lib
from multimesh_jax_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


def _rand(*shape):
    return torch.randn(*shape, device="cuda").bfloat16()


# one vector per row, the edges of every block size, rows that no step of two divides
@pytest.mark.parametrize("D", [8, 1024, 1032, 2056, 4104, 16384])
@pytest.mark.parametrize("rows", [1, 2, 3, 1301])
def test_add_rmsnorm_and_its_weight_gradient(D, rows):
    torch.manual_seed(D + rows)
    x, delta, w, dy = _rand(rows, D), _rand(rows, D), _rand(D), _rand(rows, D)
    xn, y, rstd = K.add_rmsnorm_fwd(x, delta, w, 1e-5)
    assert torch.equal(xn, K.add(x, delta))
    y2, rstd2 = K.rmsnorm_fwd(xn, w, 1e-5)
    assert torch.equal(y, y2) and torch.equal(rstd, rstd2)
    dx, dw = K.rmsnorm_bwd(xn, w, dy, rstd)
    lib = _lib.load()
    part = torch.empty(lib.mm_rmsnorm_bwd_parts(rows), D, device="cuda")
    dx2, dw2 = torch.empty_like(xn), torch.empty(D, device="cuda", dtype=torch.bfloat16)
    rc = lib.mm_rmsnorm_bwd_bf16(xn.data_ptr(), w.data_ptr(), dy.data_ptr(), rstd.data_ptr(), dx2.data_ptr(), dw2.data_ptr(),
                                 part.data_ptr(), rows, D, 0, torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and torch.equal(dx, dx2) and torch.equal(dw.bfloat16(), dw2)
    acc = torch.randn(D, device="cuda")
    for accumulate, want in ((0, dw2.float()), (1, acc + dw2.float())):
        rc = lib.mm_rmsnorm_bwd_acc(xn.data_ptr(), w.data_ptr(), dy.data_ptr(), rstd.data_ptr(), dx2.data_ptr(),
                                    (out := acc.clone()).data_ptr(), part.data_ptr(), rows, D, accumulate, 0,
                                    torch.cuda.current_stream().cuda_stream)
        assert rc == 0 and torch.equal(out, want)


# a table shorter and longer than the token count; one head; groups with heads that are only copied
@pytest.mark.parametrize("T,S,H,rot,group", [(1, 1, 1, 1, 1), (300, 300, 6, 2, 3), (256, 64, 12, 5, 6), (77, 1000, 3, 2, 3),
                                             (33, 33, 16, 3, 4), (31, 7, 17, 1, 1), (9, 9, 48, 5, 6)])
def test_rotated_copy(T, S, H, rot, group):
    x = _rand(T, H, 128)
    cos, sin = K.rope_tables(S, 128, 1e4, "cuda")
    out, want = K.rope(x, cos, sin, rot, group), K.rope_(x.clone(), cos, sin, rot_per_group=rot, group_size=group)
    # the two kernels may contract products and sums differently: 2^-24 of the summands, then one bf16 rounding
    torch.testing.assert_close(out, want, rtol=2.0 ** -7, atol=1e-5)
    keep = torch.tensor([h % group >= rot for h in range(H)], device="cuda")
    assert torch.equal(out[:, keep], x[:, keep])


@pytest.mark.parametrize("F", [8, 512, 520, 1032, 11008])
def test_swiglu_widths(F):
    gu, dh = _rand(37, 2 * F), _rand(37, F)
    g, u, d = gu[:, :F].double(), gu[:, F:].double(), dh.double()
    s = torch.sigmoid(g)
    # one bf16 rounding (2^-8 of the value at most) of a few 32-bit operations
    torch.testing.assert_close(K.swiglu_fwd(gu).double(), g * s * u, rtol=2.0 ** -8 + 1e-5, atol=1e-6)
    want = torch.cat([d * u * s * (1 + g * (1 - s)), d * g * s], 1)
    torch.testing.assert_close(K.swiglu_bwd(gu, dh).double(), want, rtol=2.0 ** -8 + 1e-4, atol=1e-5)


# narrow rows, of which a block takes many, up to the width from which it takes one; counts that fill no block
@pytest.mark.parametrize("F", [8, 24, 1016, 1024])
@pytest.mark.parametrize("T,live", [(1, None), (301, None), (301, 0), (301, 7), (301, 400)])
def test_swiglu_rows(F, T, live):
    gu, dh = _rand(T, 2 * F), _rand(T, F)
    g, u, d = gu[:, :F].double(), gu[:, F:].double(), dh.double()
    s = torch.sigmoid(g)
    rows = None if live is None else torch.tensor([live], device="cuda", dtype=torch.int32)
    n = T if live is None else min(live, T)
    lib, stream = _lib.load(), torch.cuda.current_stream().cuda_stream
    count = rows.data_ptr() if rows is not None else None
    h, dgu = torch.full((T, F), 7.0, device="cuda").bfloat16(), torch.full((T, 2 * F), 7.0, device="cuda").bfloat16()
    assert lib.mm_swiglu_fwd_rows(gu.data_ptr(), h.data_ptr(), T, F, count, stream) == 0
    assert lib.mm_swiglu_bwd_rows(gu.data_ptr(), dh.data_ptr(), dgu.data_ptr(), T, F, count, stream) == 0
    # one bf16 rounding (2^-8 of the value at most) of a few 32-bit operations
    torch.testing.assert_close(h[:n].double(), (g * s * u)[:n], rtol=2.0 ** -8 + 1e-5, atol=1e-6)
    want = torch.cat([d * u * s * (1 + g * (1 - s)), d * g * s], 1)
    torch.testing.assert_close(dgu[:n].double(), want[:n], rtol=2.0 ** -8 + 1e-4, atol=1e-5)
    assert (h[n:] == 7.0).all() and (dgu[n:] == 7.0).all()


@pytest.mark.parametrize("n", [4, 1024, 1028, 4 * 256 * 6 * 200 + 12])     # one vector; one block; a last block of a few vectors
def test_adamw_up_to_the_last_vector(n):
    torch.manual_seed(n)
    cpu = [torch.randn(n), torch.empty(n, dtype=torch.bfloat16), torch.randn(n), torch.rand(n), torch.randn(n)]
    gpu = [t.cuda() for t in cpu]
    kw = dict(lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1)
    K.adamw_step_(*cpu, step=3, **kw)
    K.adamw_step_(*gpu, step=torch.tensor([3], device="cuda"), **kw)
    for a, b in zip(gpu, cpu):
        torch.testing.assert_close(a.cpu().float(), b.float(), rtol=2.0 ** -7 if b.dtype == torch.bfloat16 else 1e-5, atol=1e-6)


def test_scaling_in_place_by_one_and_by_another_factor():
    x = _rand(1003)[:1000].clone()
    for f in (1.0, -0.5):
        want, s = (x.float() * f).bfloat16(), torch.tensor([f], device="cuda").bfloat16()
        y = x.clone()
        for out in (y, torch.empty_like(x)):
            rc = _lib.load().mm_scale_bf16((y if out is y else x).data_ptr(), s.data_ptr(), out.data_ptr(), x.numel(),
                                           torch.cuda.current_stream().cuda_stream)
            assert rc == 0 and torch.equal(out, want)


@pytest.mark.parametrize("rows,V", [(1, 8), (512, 1000), (8192, 32000), (1024, 128256)])
def test_loss_does_not_depend_on_the_gradient_that_is_written_over_the_logits(rows, V):
    logits, targets = _rand(rows, V), torch.randint(0, V, (rows,), device="cuda")
    want = K.cross_entropy_fwd_bwd(logits, targets, 1.0, write_grad=False)
    exact = torch.nn.functional.cross_entropy(logits[:512].double(), targets[:512], reduction="none")
    torch.testing.assert_close(want[:512].double(), exact, rtol=1e-5, atol=1e-5)     # fp32 sums of V exponentials
    for _ in range(4):
        assert torch.equal(K.cross_entropy_fwd_bwd(logits.clone(), targets, 1.0, write_grad=True), want)


# one element per thread of a block and one more; a tensor that is missing or empty; sizes far apart
@pytest.mark.parametrize("sizes", [(4, 1024, 1028), (1 << 16, 4, 2052), (8, 0, 1024), (2048, 1020, 0), (0, 0, 12),
                                   (1 << 24, 1 << 24, 4)])      # above the size that shares a launch
def test_grouped_adamw_equals_single_updates(sizes):
    from multimesh_jax_b200.ops import _lib
    torch.manual_seed(sum(sizes))
    make = lambda n: [torch.randn(n, device="cuda"), torch.zeros(n, device="cuda", dtype=torch.bfloat16), torch.randn(n, device="cuda"),
                      torch.rand(n, device="cuda"), torch.randn(n, device="cuda")]
    one = [make(n) for n in sizes]
    group = [[t.clone() for t in ts] for ts in one]
    step = torch.tensor([3], device="cuda")
    hyper = (1e-2, 0.9, 0.95, 1e-8, 0.1)
    stream = torch.cuda.current_stream().cuda_stream
    for ts, n in zip(one, sizes):
        assert _lib.load().mm_adamw(*[t.data_ptr() for t in ts], n, *hyper, 1, 0.5, step.data_ptr(), stream) == 0
    args = [a for ts, n in zip(group, sizes) for a in (*[t.data_ptr() if n else None for t in ts], n)]
    assert _lib.load().mm_adamw_group(*args, *hyper, 0.5, step.data_ptr(), stream) == 0
    for a, b in zip(one, group):
        assert all(torch.equal(x, y) for x, y in zip(a, b))


# one cluster: a row, fewer rows than warps, a second pair of rows for some warps only, widths that end inside a warp's
# vectors; two launches: few partial sums, many
@pytest.mark.parametrize("rows,D", [(1, 8), (7, 256), (129, 248), (300, 264), (257, 504), (512, 256), (513, 256), (100, 2048), (1500, 1024)])
@pytest.mark.parametrize("accumulate,add", [(0, 0), (1, 1)])
def test_norm_gradient_of_small_and_large_rows(rows, D, accumulate, add):
    x, dy, w = _rand(rows, D), _rand(rows, D), _rand(D)
    rstd = torch.rand(rows, device="cuda") + 0.5
    dx, dw = _rand(rows, D), torch.randn(D, device="cuda")
    xf, gf, r = x.double(), dy.double(), rstd.double()[:, None]
    gw = gf * w.double()
    want = (dx.double() if add else 0) + gw * r - xf * r ** 3 * (gw * xf).sum(1, keepdim=True) / D
    dw_want = (dw.double() if accumulate else 0) + (gf * xf * r).sum(0)
    lib = _lib.load()
    scratch = torch.empty(lib.mm_rmsnorm_bwd_parts(rows) * D, device="cuda")
    rc = lib.mm_rmsnorm_bwd(x.data_ptr(), w.data_ptr(), dy.data_ptr(), rstd.data_ptr(), dx.data_ptr(), dw.data_ptr(), scratch.data_ptr(),
                            rows, D, accumulate, add, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    # one bf16 rounding (2^-9 of the norm) of 32-bit sums; sums of `rows` terms in 32 bits
    assert ((dx.double() - want).norm() <= 2.0 ** -8 * want.norm())
    assert ((dw.double() - dw_want).norm() <= 4 * rows ** 0.5 * 2.0 ** -24 * dw_want.norm().clamp_min(1.0))


# the same sums rounded to the weight's type, and rounded before they are added: one cluster of each width, two launches
@pytest.mark.parametrize("rows,D", [(3, 248), (257, 256), (129, 264), (257, 504), (256, 512), (257, 512), (600, 1032)])
def test_norm_gradient_is_rounded_as_the_weight_is(rows, D):
    x, dy, w, rstd = _rand(rows, D), _rand(rows, D), _rand(D), torch.rand(rows, device="cuda") + 0.5
    lib, stream = _lib.load(), torch.cuda.current_stream().cuda_stream
    scratch, dx = torch.empty(lib.mm_rmsnorm_bwd_parts(rows) * D, device="cuda"), torch.empty_like(x)
    ins = [t.data_ptr() for t in (x, w, dy, rstd, dx)]
    full, half, acc = torch.empty(D, device="cuda"), torch.empty(D, device="cuda").bfloat16(), torch.randn(D, device="cuda")
    want = acc.clone()
    assert lib.mm_rmsnorm_bwd(*ins, full.data_ptr(), scratch.data_ptr(), rows, D, 0, 0, stream) == 0
    assert lib.mm_rmsnorm_bwd_bf16(*ins, half.data_ptr(), scratch.data_ptr(), rows, D, 0, stream) == 0
    assert lib.mm_rmsnorm_bwd_acc(*ins, acc.data_ptr(), scratch.data_ptr(), rows, D, 1, 0, stream) == 0
    assert torch.equal(half, full.bfloat16()) and torch.equal(acc, want + half.float())


@pytest.mark.parametrize("rows,V", [(1, 8), (300, 2056), (70, 32000)])
def test_loss_gradient_into_another_buffer(rows, V):
    logits, targets = _rand(rows, V), torch.randint(0, V, (rows,), device="cuda")
    targets[::7] = -1
    before = logits.clone()
    loss, grad = K.cross_entropy_to(logits, targets, 0.5)
    assert torch.equal(logits, before)
    want = before.clone()
    assert torch.equal(K.cross_entropy_fwd_bwd(want, targets, 0.5), loss) and torch.equal(want, grad)


@pytest.mark.parametrize("offset", [1, 4, 8])
def test_loss_gradient_of_logits_that_start_off_16_bytes(offset):
    rows, V = 70, 2056
    flat, targets = _rand(rows * V + 8), torch.randint(0, V, (rows,), device="cuda")
    logits = flat[offset:offset + rows * V].view(rows, V)
    assert logits.is_contiguous() and logits.data_ptr() % 16 == offset * 2 % 16
    loss, grad = torch.ops.mm_ops.cross_entropy(logits, targets, 0.5)
    want = logits.clone()
    assert torch.equal(K.cross_entropy_fwd_bwd(want, targets, 0.5).sum() * 0.5, loss) and torch.equal(want, grad)
