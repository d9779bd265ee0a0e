"""Kernel programs of the native task launcher, built (not launched) on a machine without a GPU."""
import torch

import multimesh_jax_b200 as mm
from multimesh_jax_b200.compiler.native import build_native
from multimesh_jax_b200.models import llama


def _pp2_plan():
    cfg = llama.LlamaConfig.tiny(n_layers=4, n_heads=1, n_kv_heads=1, d_model=128, d_ff=256, vocab=256)
    cfg.dtype = torch.bfloat16
    B, S, MB = 8, 128, 2
    params = llama.init_params(cfg)
    opt_state = llama.init_opt_state(params)
    tokens = torch.randint(0, cfg.vocab, (B, S))
    cos, sin = llama.rope_tables(cfg, S, "cpu")
    step = llama.make_train_step(cfg, llama.AdamWConfig(lr=1e-2), seq_len=S, global_batch=B, microbatch_size=MB,
                                 schedule="1f1b")
    mesh = mm.MultiMesh((2, 1), ("stage", "model"))
    llama.register_pipeline_tasks(cfg, mesh, num_stages=2)
    with mesh:
        return mm.compile_function(step, (params, opt_state, tokens, tokens, cos, sin), mesh=mesh, backend="cpu",
                                   donate_argnums=(0, 1))


def test_outputs_read_by_a_reshard_are_written_into_an_external_tile_without_a_copy():
    exe = _pp2_plan()
    plan = exe.plan
    sources = {op["src_store"] for op in plan["ops"] if op["kind"] == "reshard"}
    assert sources
    seen_ext = 0
    for t in plan["templates"]:
        if not t["name"].endswith("_loop"):
            continue
        ops = [op for op in plan["ops"] if op["kind"] == "task" and op["template"] == t["id"]]
        ext = None
        for op in ops:
            here = {k for k, (sid, m) in enumerate(zip(op["outputs"], op["accumulate"])) if m == 0 and sid in sources}
            ext = here if ext is None else ext & here
        protect = sorted({i for op in ops for i, sid in enumerate(op["inputs"]) if sid in sources})
        modes = tuple(1 if m else 0 for m in ops[0]["accumulate"])
        prog = exe.programs[t["id"]]
        plain = build_native(exe.cap, plan, t, prog, modes, False)
        direct = build_native(exe.cap, plan, t, prog, modes, False, sorted(ext), protect)
        assert direct.external == sorted(ext)
        # the producer writes into the tile: no kernel call is added, the output block shrinks
        # by exactly the bytes that moved out of it
        assert direct.num_calls == plain.num_calls
        moved = 0
        for k in ext:
            spec = direct.outputs[k]
            assert spec[0] == "ext"
            n = spec[3].itemsize
            for e in spec[2]:
                n *= e
            moved += (n + 255) // 256 * 256
            seen_ext += 1
        assert plain.out_block_bytes - direct.out_block_bytes == moved
        assert [o[0] for i, o in enumerate(direct.outputs) if i not in ext] == \
               [o[0] for i, o in enumerate(plain.outputs) if i not in ext]
    assert seen_ext >= 3          # x and h forward, their cotangents backward
    exe.shutdown()


def test_fresh_outputs_are_carved_from_bounded_chunks(monkeypatch):
    from multimesh_jax_b200.compiler import native
    exe = _pp2_plan()
    plan = exe.plan
    t = next(t for t in plan["templates"] if t["name"].endswith("stage0_loop"))
    ops = [op for op in plan["ops"] if op["kind"] == "task" and op["template"] == t["id"]]
    modes = tuple(1 if m else 0 for m in ops[0]["accumulate"])
    whole = build_native(exe.cap, plan, t, exe.programs[t["id"]], modes, False)
    assert len(whole.out_chunks) == 1 and whole.out_chunks[0] == whole.out_block_bytes
    monkeypatch.setattr(native._Builder, "OUT_CHUNK", 256 << 10)
    split = build_native(exe.cap, plan, t, exe.programs[t["id"]], modes, False)
    assert len(split.out_chunks) > 1 and sum(split.out_chunks) == split.out_block_bytes
    # every chunk respects the bound unless it holds a single larger output
    sizes = {}
    for spec in split.outputs:
        if spec[0] != "block":
            continue
        _, chunk, off, shape, dtype = spec
        n = dtype.itemsize
        for e in shape:
            n *= e
        assert 0 <= chunk < len(split.out_chunks) and off + n <= split.out_chunks[chunk]
        sizes.setdefault(chunk, []).append(n)
    for chunk, total in enumerate(split.out_chunks):
        assert total <= (256 << 10) or len(sizes.get(chunk, ())) <= 1
    assert split.num_calls == whole.num_calls
    exe.shutdown()


def test_tasks_are_interpreted_when_the_scratch_tile_cannot_be_reserved():
    from types import SimpleNamespace
    from multimesh_jax_b200.runtime.executable import Executable
    for answers, native in (([64], True), ([0, 64], True), ([0, 0], False)):
        exe = SimpleNamespace(topology=SimpleNamespace(local_devices=[0]), _native={(3, False): "a", (3, True): "b"}, _native_why={},
                              _scratch_base={}, context=SimpleNamespace(reserve_scratch=lambda d, n: answers.pop(0)))
        Executable._reserve_scratch(exe, 5 << 20)
        assert answers == [] and bool(exe._native) == native and exe._scratch_base == ({0: 64} if native else {})
        assert native or exe._native_why == {3: "5 MiB of task scratch could not be reserved on device 0"}


def _sym(slot, off, *shape, dtype=torch.bfloat16):
    from multimesh_jax_b200.compiler.native import Sym
    return Sym(slot, off, shape, dtype)


def _products(dx, dw, dy=None, x=None):
    """The calls of a linear layer's gradient: 64 rows, 32 columns of dY, 16 of X."""
    from multimesh_jax_b200.compiler.native import STREAM
    dy, w, x = dy or _sym(0, 0, 64, 32), _sym(1, 0, 32, 16), x or _sym(2, 0, 64, 16)
    return [("mm_gemm_auto_bf16", (dy, 0, 32, w, 1, 16, dx, 0, 16, 64, 16, 32, 256, STREAM)),
            ("mm_gemm_auto_bf16", (dy, 1, 32, x, 1, 16, dw, 2, 16, 32, 16, 64, 256, STREAM))]


def test_products_of_a_linear_gradient_share_a_launch_only_when_neither_needs_the_other():
    from multimesh_jax_b200.compiler.native import merge_calls
    dx, dw = _sym(3, 0, 64, 16), _sym(4, 0, 32, 16, dtype=torch.float32)
    a, b = _products(dx, dw)
    for pair in ([a, b], [b, a]):
        (name, args), = merge_calls(pair)
        assert name == "mm_linear_bwd_bf16" and args[5:9] == (2, 64, 32, 16) and args[3] is dx and args[4] is dw
    assert len(merge_calls([a, ("mm_zero", (dx, 8, None)), b])) == 3
    # dX over X or over dY (their last reader is the other product), results that overlap, another dY, bf16 accumulation
    assert len(merge_calls(_products(_sym(2, 512, 64, 16), dw))) == 2
    assert len(merge_calls(_products(_sym(0, 2048, 64, 16), dw))) == 2
    assert len(merge_calls(_products(_sym(4, 1024, 64, 16), dw))) == 2
    assert len(merge_calls([a, _products(dx, dw, dy=_sym(0, 4096, 64, 32))[1]])) == 2
    assert len(merge_calls([a, (b[0], b[1][:7] + (3,) + b[1][8:])])) == 2


def test_updates_share_a_launch_three_at_a_time():
    from multimesh_jax_b200.compiler.native import STREAM, merge_calls
    step = _sym(9, 0, 1, dtype=torch.int64)

    def update(k, lr=0.1, slots=None, at=step):
        s = slots or [5 * k + 10 + j for j in range(5)]
        f = [_sym(i, 0, 8, dtype=torch.bfloat16 if j == 1 else torch.float32) for j, i in enumerate(s)]
        return "mm_adamw", (*f, 8, lr, 0.9, 0.99, 1e-8, 0.0, 1, 1.0, at, STREAM)

    merged = merge_calls([update(k) for k in range(7)])
    assert [n for n, _ in merged] == ["mm_adamw_group", "mm_adamw_group", "mm_adamw"]
    assert all(len(a) == 26 for n, a in merged[:2])
    (name, args), = merge_calls([update(0), update(1)])
    assert name == "mm_adamw_group" and args[12:18] == (None,) * 5 + (0,)
    assert [n for n, _ in merge_calls([update(0), update(1, lr=0.2)])] == ["mm_adamw"] * 2
    assert [n for n, _ in merge_calls([update(0), update(1, at=_sym(8, 0, 1, dtype=torch.int64))])] == ["mm_adamw"] * 2
    # the second update reads what the first one wrote; both read one gradient (a tied weight's) and write apart
    assert [n for n, _ in merge_calls([update(0), update(1, slots=[10, 20, 21, 22, 23])])] == ["mm_adamw"] * 2
    assert [n for n, _ in merge_calls([update(0), update(1, slots=[20, 21, 22, 23, 14])])] == ["mm_adamw_group"]


def test_a_copy_of_the_logits_for_their_gradient_is_one_pass():
    from multimesh_jax_b200.compiler.native import STREAM, merge_calls
    logits, grad, tok, loss = _sym(0, 0, 4, 16), _sym(1, 0, 4, 16), _sym(2, 0, 4, dtype=torch.int64), _sym(1, 512, 4, dtype=torch.float32)
    copy = ("mm_memcpy_d2d", (grad, logits, 128, STREAM))
    ce = ("mm_cross_entropy", (grad, tok, loss, None, None, 4, 16, 16, 0, 0.5, 1, STREAM))
    (name, args), = merge_calls([copy, ce])
    assert name == "mm_cross_entropy_to" and args[:7] == (logits, grad, tok, loss, 4, 16, 0.5)
    other = _sym(1, 256, 4, 16)
    assert len(merge_calls([("mm_memcpy_d2d", (other, logits, 128, STREAM)), ce])) == 2
    assert len(merge_calls([("mm_memcpy_d2d", (grad, logits, 64, STREAM)), ce])) == 2        # part of the rows
    assert len(merge_calls([copy, (ce[0], ce[1][:10] + (0, STREAM))])) == 2                  # no gradient


def test_the_losses_do_not_go_over_logits_that_the_same_pass_reads(monkeypatch):
    """Logits that are copied by the program itself die with the copy, so the losses of the rows take their memory:
    fine behind the copy, not in one pass that reads them."""
    from multimesh_jax_b200.compiler import native
    logits, grad, tok = _sym(0, 0, 4, 16), _sym(1, 0, 4, 16), _sym(2, 0, 4, dtype=torch.int64)
    for at, calls in ((0, 2), (112, 2), (128, 1)):
        loss = _sym(0, at, 4, dtype=torch.float32)
        copy = ("mm_memcpy_d2d", (grad, logits, 128, native.STREAM))
        ce = ("mm_cross_entropy", (grad, tok, loss, None, None, 4, 16, 16, 0, 0.5, 1, native.STREAM))
        assert len(native.merge_calls([copy, ce])) == calls

    seen = []
    add = native._Builder._add_call
    monkeypatch.setattr(native._Builder, "_add_call", lambda self, name, a: (seen.append((name, a)), add(self, name, a))[1])
    ops = torch.ops.mm_ops
    x, w, t = torch.randn(64, 64).bfloat16(), torch.randn(512, 64).bfloat16(), torch.randint(0, 512, (64,))

    def step(x, w, t):
        z = ops.linear(x, w).to(torch.bfloat16, copy=True)
        return tuple(ops.cross_entropy(z, t, 0.125))

    with mm.enable_fast_path(False):
        exe = mm.compile_function(step, (x, w, t), num_devices=1, backend="cpu")
    for op in exe.plan["ops"]:
        if op["kind"] == "task":
            tm = exe.plan["templates"][op["template"]]
            build_native(exe.cap, exe.plan, tm, exe.programs[tm["id"]], tuple(int(m > 0) for m in op["accumulate"]), False)
    exe.shutdown()
    (copied,) = [a for n, a in seen if n == "mm_memcpy_d2d"]
    (ce,) = [a for n, a in seen if n == "mm_cross_entropy"]
    assert not native._disjoint([ce[2]], [copied[1]])       # the case in question: losses over the copied logits
    for name, a in seen:
        if name == "mm_cross_entropy_to":
            assert native._disjoint([a[1], a[3]], [a[0]])


def test_the_gradient_of_a_loss_is_not_written_when_nothing_reads_it(monkeypatch):
    from multimesh_jax_b200.compiler import native
    seen = []
    emit = native._Builder.call
    monkeypatch.setattr(native._Builder, "call", lambda self, name, *a: (seen.append((name, a)), emit(self, name, *a))[1])
    ops = torch.ops.mm_ops
    x, w, t = torch.randn(8, 64).bfloat16(), torch.randn(32, 64).bfloat16(), torch.randint(0, 32, (8,))

    def logits_and_loss(x, w, t):
        y = ops.linear(x, w)
        return ops.cross_entropy(y, t, 0.125)[0], y

    def gradient_too(x, w, t):
        y = ops.linear(x, w)
        return (*ops.cross_entropy(y, t, 0.125), y)

    for fn, write in ((logits_and_loss, 0), (gradient_too, 1)):
        seen.clear()
        with mm.enable_fast_path(False):
            exe = mm.compile_function(fn, (x, w, t), num_devices=1, backend="cpu")
        for op in exe.plan["ops"]:
            if op["kind"] == "task":
                tm = exe.plan["templates"][op["template"]]
                build_native(exe.cap, exe.plan, tm, exe.programs[tm["id"]], tuple(int(m > 0) for m in op["accumulate"]), False)
        (ce,) = [a for n, a in seen if n == "mm_cross_entropy"]
        assert ce[10] == write and ("mm_memcpy_d2d" in [n for n, _ in seen]) == bool(write)
        exe.shutdown()
