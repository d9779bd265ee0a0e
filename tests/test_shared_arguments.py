"""Arguments that a compiled step works on in the caller's memory, without a private copy."""
import pytest
import torch
from torch.utils import _pytree as pytree

import multimesh_jax_b200 as mm
from multimesh_jax_b200.compiler.lower import Instr, TemplateProgram
from multimesh_jax_b200.compiler.native import inputs_left_alone
from multimesh_jax_b200.models import llama


def _loss_step(device, train):
    cfg = llama.LlamaConfig.tiny(n_layers=2, n_heads=1, n_kv_heads=1, d_model=128, d_ff=256, vocab=256)
    cfg.dtype = torch.bfloat16
    B, S = 2, 128
    params = llama.init_params(cfg, device=device)
    tokens = torch.randint(0, cfg.vocab, (B, S), device=device)
    cos, sin = llama.rope_tables(cfg, S, device)
    mesh = mm.MultiMesh((1, 1), ("stage", "model"))
    llama.register_pipeline_tasks(cfg, mesh, num_stages=1)
    if train:
        step = llama.make_train_step(cfg, llama.AdamWConfig(lr=1e-2), seq_len=S, global_batch=B, microbatch_size=1)
        args = (params, llama.init_opt_state(params), tokens, tokens, cos, sin)
    else:
        def step(p, tokens, labels, cos, sin):
            return llama.loss_fn(cfg, p, tokens, labels, cos, sin, 1.0 / (B * S)), p["final_norm"]
        args = (params, tokens, tokens, cos, sin)
    with mesh:
        return mm.compile_function(step, args, mesh=mesh, backend=device), args


def test_only_inputs_that_no_operator_writes_are_left_alone():
    exe, args = _loss_step("cpu", train=True)
    names = [jp for jp, _ in pytree.tree_flatten_with_path(args)[0]]
    written = set()
    for op in exe.plan["ops"]:
        if op["kind"] != "task":
            continue
        prog = exe.programs[op["template"]]
        alone = inputs_left_alone(exe.cap, prog)
        written |= {s for s, v in zip(op["inputs"], prog.inputs) if v not in alone}
    clean = [pytree.keystr(names[i]) for i, sid in enumerate(exe.plan["param_stores"]) if sid >= 0 and sid not in written]
    # AdamW may write over weights and moments, token ids are handed on to the backward tasks; the step
    # counter, the labels and the rotary tables are only read
    assert clean == ["[1]['step']", "[3]", "[4]", "[5]"]
    exe.shutdown()


@pytest.mark.gpu
def test_shared_arguments_keep_their_values_and_follow_updates():
    exe, args = _loss_step("cuda", train=False)
    assert exe._shared_params
    before = [t.clone() for t in pytree.tree_leaves(args)]
    loss, norm = exe(*args)
    first = loss.full_tensor().item()
    for a, b in zip(pytree.tree_leaves(args), before):
        assert torch.equal(a, b)
    # a result that is an argument is a copy of it: neither changes with the other
    out = norm.full_tensor()
    kept = out.clone()
    args[0]["final_norm"].mul_(3.0)
    assert torch.equal(out, kept)
    args[0]["embed"].mul_(2.0)
    assert exe(*args)[0].full_tensor().item() != first
    exe.shutdown()


def _offset_view(t):
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    flat[1:] = t.reshape(-1)
    return flat[1:].view(t.shape)


@pytest.mark.parametrize("donate", [False, True])
def test_tiles_of_arguments_start_on_vector_boundaries(donate):
    exe, args = _loss_step("cpu", train=donate)
    exe._shared_params = set(range(len(exe.plan["param_stores"])))      # as on a device: nothing is copied for privacy
    exe.donated = set(exe._shared_params) if donate else set()
    exe._plan_binding()
    want = exe(*pytree.tree_map(torch.clone, args))[0].full_tensor()
    odd = pytree.tree_map(_offset_view, args)
    even = pytree.tree_map(torch.clone, args)
    assert any(t.data_ptr() % 16 for t in pytree.tree_leaves(odd))
    for call in (odd, even):
        bound = {}
        bind = exe._submit_task

        def first_task(k, op, d, *rest):
            bound.update({sid: exe.tiles[sid][0] for sid in exe.plan["param_stores"] if sid >= 0 and not bound.get(sid) is not None
                          and 0 in exe.tiles[sid]})
            return bind(k, op, d, *rest)

        exe._submit_task = first_task
        loss = exe(*call)[0].full_tensor()
        exe._submit_task = bind
        assert torch.equal(loss, want)
        leaves = pytree.tree_leaves(call)
        for i, sid in enumerate(exe.plan["param_stores"]):
            if sid >= 0:
                assert bound[sid].data_ptr() % 16 == 0
                assert (bound[sid].data_ptr() == leaves[i].data_ptr()) == (leaves[i].data_ptr() % 16 == 0)
    exe.shutdown()


def test_microbatch_slices_start_on_vector_boundaries():
    prog = TemplateProgram({"name": "t", "mesh_dims": [1], "device_start": 0}, [Instr(3, None, 0, None, [1], None, 0, (0, 1, 1))],
                           [0], [1], {})
    for x in (torch.randn(6, 12).bfloat16(), torch.randn(6, 8).bfloat16(), torch.arange(6).view(6, 1)):
        for row in range(6):
            (piece,) = prog.run(None, [row], [x])
            assert torch.equal(piece, x[row:row + 1])
            assert piece.data_ptr() % 16 == 0 or not piece.is_floating_point()
            # rows that start well, and token ids wherever they start, stay in the argument's memory
            assert (piece.data_ptr() == x[row].data_ptr()) == (x[row].data_ptr() % 16 == 0 or not x.is_floating_point())


@pytest.mark.gpu
def test_arguments_at_odd_offsets_on_the_device():
    exe, args = _loss_step("cuda", train=False)
    want = exe(*args)[0].full_tensor()
    assert torch.equal(exe(*pytree.tree_map(_offset_view, args))[0].full_tensor(), want)
    exe.shutdown()


def test_one_tensor_passed_as_a_written_and_as_a_read_argument():
    """AdamW writes over donated state; another argument in the same memory keeps what it was passed with."""
    ops = torch.ops.mm_ops
    torch.manual_seed(0)
    p, g, t = torch.randn(64).bfloat16(), torch.randn(64), torch.tensor([3])
    flat = torch.randn(192).abs()

    def step(p, master, m, v, g, t, ref):
        new = ops.adamw(p, master, m, v, g, t, 1e-2, 0.9, 0.95, 1e-8, 0.1, 1.0)
        return (*new, new[1] - ref)

    with mm.enable_fast_path(False):
        exe = mm.compile_function(step, (p, *[flat[:64]] * 3, g, t, flat[:64]), num_devices=1, backend="cpu",
                                  donate_argnums=(0, 1, 2, 3))
    exe._shared_params = {4, 5, 6}      # as on a device
    exe._plan_binding()
    # (master, m, v, ref): apart; ref is the master; ref lies across two of them; both moments and ref are one tensor
    for spans in ((0, 64, 128, None), (0, 64, 128, 0), (0, 64, 128, 32), (0, 64, 64, 64), (0, 0, 0, 0)):
        memory = flat.clone()
        parts = [memory[s:s + 64] if s is not None else flat[3:67].clone() for s in spans]
        want = step(p, *(x.clone() for x in parts[:3]), g, t, parts[3].clone())
        got = exe(p.clone(), *parts[:3], g, t, parts[3])
        for a, b in zip(got, want):
            assert torch.equal(a.full_tensor(), b), spans
    exe.shutdown()
