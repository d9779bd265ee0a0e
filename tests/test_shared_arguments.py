"""Arguments that a compiled step works on in the caller's memory, without a private copy."""
import pytest
import torch
from torch.utils import _pytree as pytree

import multimesh_jax_b200 as mm
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
