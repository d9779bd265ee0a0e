"""Operators that may write a result over an operand do so only when nothing needs its memory any more.
Native programs are built without a GPU, their recorded calls replayed on CPU tensors and compared with
the eager function; the interpreted programs run the same steps."""
import pytest
import torch

import multimesh_jax_b200 as mm
from multimesh_jax_b200.compiler import lower, native
from multimesh_jax_b200.compiler.capture import DTYPE_FROM_NAME
from multimesh_jax_b200.ops import kernels as K
from multimesh_jax_b200.ops import mm_ops  # noqa: F401  (registers the operators)

ops = torch.ops.mm_ops


def _mem(slots, s):
    return slots[s.slot][s.off:s.off + s.nbytes].view(s.dtype).view(s.shape)


def _gemm(m, a, a_mn, lda, b, b_mn, ldb, out, mode, *_):
    c = K.gemm(m(a), m(b), a_mn=bool(a_mn), b_mn=bool(b_mn), out_dtype=m(out).dtype)
    m(out).copy_(c.float() + m(out).float() if mode in (2, 3) else c)


def _cross_entropy(m, buf, targets, loss, _, __, rows, V, ___, ____, scale, grad, *_rest):
    m(loss).copy_(K.cross_entropy_fwd_bwd(m(buf).view(rows, V), m(targets).reshape(-1), scale, bool(grad)))


def _norm_bwd(m, x, w, dy, rstd, dx, dw, accumulate, add):
    assert not add
    got, d = K.rmsnorm_bwd(m(x), m(w), m(dy), m(rstd))
    m(dx).copy_(got)
    m(dw).copy_((m(dw) if accumulate else 0) + d.bfloat16().float())


REPLAY = {
    "mm_gemm_auto_bf16": _gemm,
    "mm_cross_entropy": _cross_entropy,
    "mm_scale_bf16": lambda m, x, s, out, *_: m(out).copy_(m(x) * m(s).reshape(())),
    "mm_memcpy_d2d": lambda m, dst, src, *_: m(dst).copy_(m(src).view(m(dst).shape)),
    "mm_swiglu_fwd": lambda m, gu, h, T, F, *_: m(h).copy_(K.swiglu_fwd(m(gu).view(T, 2 * F)).view(h.shape)),
    "mm_add_bf16": lambda m, x, y, out, *_: m(out).copy_(m(x) + m(y)),
    "mm_bf16_to_f32": lambda m, x, out, n, acc, *_: m(out).copy_(m(x).float().view(out.shape) + (m(out) if acc else 0)),
    "mm_embedding_fwd": lambda m, table, tok, out, *_: m(out).copy_(m(table)[m(tok)]),
    "mm_accumulate_f32": lambda m, acc, x, *_: m(acc).add_(m(x).view(acc.shape)),
    "mm_rmsnorm_fwd": lambda m, x, w, y, rstd, rows, D, eps, *_: [m(o).copy_(r.view(o.shape)) for o, r in zip(
        (y, rstd), K.rmsnorm_fwd(m(x), m(w), eps))],
    "mm_rmsnorm_bwd_bf16": lambda m, *a: _norm_bwd(m, *a[:6], 0, 0),
    "mm_rmsnorm_bwd_acc": lambda m, *a: _norm_bwd(m, *a[:6], a[9], a[10]),
    "mm_sum_scale_f32": lambda m, x, n, scale, out, *_: m(out).copy_(m(x).sum() * scale),
}


def _compile(fn, args, donate=()):
    with mm.enable_fast_path(False):
        return mm.compile_function(fn, args, num_devices=1, backend="cpu", donate_argnums=donate)


def _replay(exe, args, monkeypatch):
    """Runs every task of the plan by replaying its native program. A tile is a byte buffer per store; returns
    the step's results and the final contents of the arguments' tiles."""
    calls = []
    emit = native._Builder.call
    monkeypatch.setattr(native._Builder, "call", lambda self, name, *a: (calls.append((name, a)), emit(self, name, *a))[1])
    plan, tiles = exe.plan, {}
    for i, sid in enumerate(plan["param_stores"]):
        if sid >= 0:
            tiles[sid] = args[i].clone()
    for op in plan["ops"]:
        if op["kind"] != "task":
            continue
        t = plan["templates"][op["template"]]
        prog = exe.programs[t["id"]]
        calls.clear()
        have = any(m == 2 for m in op["accumulate"])
        np_ = native.build_native(exe.cap, plan, t, prog, tuple(int(m > 0) for m in op["accumulate"]), have)
        ins = [tiles[s].contiguous().view(-1).view(torch.uint8) for s in op["inputs"]]
        accs = [tiles[op["outputs"][k]].view(-1).view(torch.uint8) for k in np_.acc_positions]
        blocks = [torch.zeros(max(n, 1), dtype=torch.uint8) for n in np_.out_chunks] or [torch.zeros(1, dtype=torch.uint8)]
        slots = ins + [blocks[0], torch.zeros(max(np_.scratch_bytes, 1), dtype=torch.uint8)] + accs + blocks[1:]
        for name, a in calls:
            # microbatch slices: the slot's address moves by the launch's scalar times the bytes of a row
            a = [native.Sym(x[1].slot, x[1].off + op["scalars"][x[2]] * x[3], x[1].shape, x[1].dtype) if isinstance(x, tuple) else x
                 for x in a]
            REPLAY[name](lambda s: _mem(slots, s), *a)
        for spec, s in zip(np_.outputs, op["outputs"]):
            if spec[0] == "block":
                n = spec[4].itemsize * torch.Size(spec[3]).numel()
                tiles[s] = blocks[spec[1]][spec[2]:spec[2] + n].view(spec[4]).view(spec[3])
            elif spec[0] == "input":
                tiles[s] = ins[spec[1]].view(DTYPE_FROM_NAME[plan["stores"][s]["shape"]["dtype"]]).view(spec[2])
            elif spec[0] == "slice":
                tiles[s] = tiles[op["inputs"][spec[1]]].narrow(0, op["scalars"][0], spec[2][0]).view(spec[2])
    return [tiles[s] for s in plan["root_stores"]], {s: tiles[s] for s in plan["param_stores"] if s >= 0}


def _b(*shape):
    return (torch.randn(*shape) / shape[-1] ** 0.5).bfloat16()


def _view_read_later(x, w, w2, s):
    y = ops.linear(x, w)
    z = ops.linear(y.view(4, 2, 64) * s, w2)
    return z, ops.linear(y, w2)


def _detached_read_later(x, w, w2, s):
    y = ops.linear(x, w)
    return y.detach() * s, ops.linear(y, w2)


def _view_of_argument_scaled(x, w, w2, s):
    return ops.linear((x.view(4, 2, 64) * s).view(8, 64), w), ops.linear(x, w2)


def _view_is_a_result(x, w, w2, s):
    y = ops.linear(x, w)
    return y.view(4, 2, 64) * s, y


def _two_fused_halves(x, w, w2, s):
    y = ops.linear(x, w)
    z = y.view(8, 1, 64) * s
    return z, ops.swiglu(y.view(8, 2, 32))


def _scaled_weight(x, w, w2, s):
    return (ops.linear(x, w * s),)


def _nothing_left(x, w, w2, s):
    return (ops.linear(x, w).view(4, 2, 64) * s,)


FORMS = [_view_read_later, _detached_read_later, _view_of_argument_scaled, _view_is_a_result, _two_fused_halves, _scaled_weight,
         _nothing_left]


@pytest.mark.parametrize("form", FORMS, ids=lambda f: f.__name__.strip("_"))
def test_product_with_a_device_scalar(form, monkeypatch):
    torch.manual_seed(0)
    args = (_b(8, 64), _b(64, 64), _b(64, 64), torch.tensor([0.5]).bfloat16())
    want = form(*args)
    exe = _compile(form, args)
    got, kept = _replay(exe, args, monkeypatch)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    for sid, a in zip(exe.plan["param_stores"], args):
        assert sid < 0 or torch.equal(kept[sid], a)
    for a, b in zip(exe(*args), want):
        assert torch.equal(a.full_tensor(), b)
    exe.shutdown()


def test_product_over_a_dead_intermediate_still_takes_its_memory():
    args = (_b(8, 64), _b(64, 64), _b(64, 64), torch.tensor([0.5]).bfloat16())
    exe = _compile(_nothing_left, args)
    taken = {exe.cap.graph.node(p.instrs[idx].node_id)["op"] for p in exe.programs.values() for idx, _ in p.takes_over}
    assert taken == {"aten.mul.Tensor"}
    exe.shutdown()


def test_loop_invariant_argument_is_scaled_once_per_microbatch(monkeypatch):
    torch.manual_seed(1)
    w, s = _b(64, 64), torch.tensor([0.5]).bfloat16()
    x, t = torch.randint(0, 64, (8,)), torch.randint(0, 64, (8,))

    def step(w, s, x, t):
        def loss(w, batch):
            h = ops.embedding(w, batch[0])
            return ops.cross_entropy(ops.linear(h, w * s), batch[1], 1.0 / 8)[0]
        return mm.microbatch(lambda w, batch: loss(w, batch), size=2, argnum=1, accumulate_dtype=torch.float32)(w, (x, t))

    with mm.ignore_transforms():
        want = step(w, s, x, t)
    exe = _compile(step, (w, s, x, t))
    assert len([op for op in exe.plan["ops"] if op["kind"] == "task"]) >= 4
    (got,), kept = _replay(exe, (w, s, x, t), monkeypatch)
    torch.testing.assert_close(got, want.float(), rtol=1e-5, atol=1e-5)     # fp32 sums of four losses
    assert all(torch.equal(kept[sid], a) for sid, a in zip(exe.plan["param_stores"], (w, s)))
    torch.testing.assert_close(exe(w, s, x, t).full_tensor(), want.float(), rtol=1e-5, atol=1e-5)
    exe.shutdown()


@pytest.mark.parametrize("form", ["plain", "scaled", "other shape"])
def test_norm_weight_gradient_on_its_way_into_the_accumulator(form, monkeypatch):
    torch.manual_seed(5)
    table, w, s, tokens = _b(32, 64), torch.rand(64).bfloat16(), torch.tensor([0.5]).bfloat16(), torch.randint(0, 32, (8,))

    def step(table, w, s, tokens):
        def gradient(w, batch):
            x = ops.embedding(table, batch)
            y, rstd = ops.rmsnorm(x, w, 1e-5)
            dw = ops.rmsnorm_bwd(x, w, y, rstd)[1]
            return dw * s if form == "scaled" else dw.view(8, 8) if form == "other shape" else dw
        return mm.microbatch(gradient, size=2, argnum=1, accumulate_dtype=torch.float32)(w, tokens)

    args = (table, w, s, tokens)
    want = sum(step_part.float() for step_part in (
        (lambda x: ops.rmsnorm_bwd(x, w, *ops.rmsnorm(x, w, 1e-5))[1] * (s if form == "scaled" else 1))(ops.embedding(table, tokens[i:i + 2]))
        for i in range(0, 8, 2))).view((8, 8) if form == "other shape" else (64,))
    exe = _compile(step, args)
    (got,), _ = _replay(exe, args, monkeypatch)
    assert torch.equal(got, want)
    assert torch.equal(exe(*args).full_tensor(), want)
    exe.shutdown()


def test_results_that_are_views_of_an_operand_survive_its_operator(monkeypatch):
    """The interpreted variants that work in place follow the same rule."""
    torch.manual_seed(2)
    x, w, t = _b(8, 64), _b(64, 64), torch.randint(0, 64, (8,))

    def logits_in_another_shape(x, w, t):
        y = ops.linear(x, w)
        z = y.view(4, 2, 64)
        return ops.cross_entropy(y, t, 0.125)[0], z

    exe = _compile(logits_in_another_shape, (x, w, t))
    want = logits_in_another_shape(x, w, t)
    got, _ = _replay(exe, (x, w, t), monkeypatch)
    for a, b, c in zip(got, exe(x, w, t), want):
        torch.testing.assert_close(a, c, rtol=1e-6, atol=0)
        torch.testing.assert_close(b.full_tensor(), c, rtol=1e-6, atol=0)
    exe.shutdown()

    qkv, (cos, sin) = _b(1, 4, 3, 16), K.rope_tables(4, 16, 1e4, "cpu")

    def projection_in_another_shape(q, cos, sin):
        p = q + q
        z = p.view(4, 48)
        return ops.attention(p, cos, sin, 1)[0], z

    exe = _compile(projection_in_another_shape, (qkv, cos, sin))
    for a, b in zip(exe(qkv, cos, sin), projection_in_another_shape(qkv, cos, sin)):
        assert torch.equal(a.full_tensor(), b)
    exe.shutdown()


def test_update_keeps_operands_that_are_read_again():
    torch.manual_seed(3)
    p, master, m, v, g = _b(64), torch.randn(64), torch.randn(64), torch.rand(64), torch.randn(64)
    t = torch.tensor([3])

    def step(p, master, m, v, g, t):
        p2, master2, m2, v2 = ops.adamw(p, master, m, v, g, t, 1e-2, 0.9, 0.95, 1e-8, 0.1, 1.0)
        return p2, master2, m2, v2, master2 - master, m.view(8, 8)

    args = (p, master, m, v, g, t)
    want = step(*args)
    exe = _compile(step, args, donate=(0, 1, 2, 3))
    for a, b in zip(exe(*(x.clone() for x in args)), want):
        assert torch.equal(a.full_tensor(), b)
    exe.shutdown()
    # not donated: neither plain tensors nor tiles of an earlier step's results change
    first = _compile(lambda *a: tuple(x + 0 for x in a), args[:4])
    tiles = first(*args[:4])
    exe = _compile(lambda *a: ops.adamw(*a, 1e-2, 0.9, 0.95, 1e-8, 0.1, 1.0), args)
    exe(*tiles, g, t)
    assert all(torch.equal(a.full_tensor(), b) for a, b in zip(tiles, args))
    exe(*args)
    assert torch.equal(args[1], master) and all(torch.equal(a.full_tensor(), b) for a, b in zip(tiles, args))
    exe.shutdown()
    first.shutdown()


def test_which_operators_return_views():
    assert all(lower.returns_view(op) for op in ("aten.view.default", "aten._unsafe_view.default", "aten.expand.default", "aten.t.default",
                                           "aten.split.Tensor", "aten.select.int", "no.such.operator"))
    assert not any(lower.returns_view(op) for op in ("aten.mul.Tensor", "aten.clone.default", "mm_ops.linear.default"))


@pytest.mark.gpu
@pytest.mark.parametrize("form", FORMS, ids=lambda f: f.__name__.strip("_"))
def test_product_on_the_device(form):
    torch.manual_seed(4)
    args = tuple(a.cuda() for a in (_b(8, 64), _b(64, 64), _b(64, 64), torch.tensor([0.5]).bfloat16()))
    want = form(*args)
    with mm.enable_fast_path(False):
        exe = mm.compile_function(form, args, num_devices=1, backend="cuda")
    for _ in range(2):
        got = exe(*args)
        for a, b in zip(got, want):
            assert torch.equal(a.full_tensor(), b)
    assert any(v.startswith("native") for v in exe.native_report().values())
    exe.shutdown()


def test_results_of_one_task_that_share_memory_are_left_to_each_other(monkeypatch):
    """A task hands on a value twice, once as a view; the task that reads the first scales it, the next reads the second."""
    torch.manual_seed(6)
    args = (_b(8, 64), _b(64, 64), torch.tensor([0.5]).bfloat16())
    mesh = mm.TaskMesh((1,), ("x",), [0])
    first = mm.task(lambda x, w: (lambda y: (y, y.view(4, 2, 64)))(ops.linear(x, w)), name="first", mesh=mesh)
    second = mm.task(lambda y, s, w: ops.linear(y * s, w), name="second", mesh=mesh)
    third = mm.task(lambda v, w: ops.linear(v.view(8, 64), w), name="third", mesh=mesh)

    def step(x, w, s):
        y, v = first(x, w)
        return second(y, s, w), third(v, w)

    with mm.ignore_transforms():
        want = step(*args)
    mm.init(cpus=1)
    exe = _compile(step, args)
    assert len([op for op in exe.plan["ops"] if op["kind"] == "task"]) >= 3
    assert not any(p.takes_over for p in exe.programs.values())
    got, _ = _replay(exe, args, monkeypatch)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert all(torch.equal(a.full_tensor(), b) for a, b in zip(exe(*args), want))
    exe.shutdown()
