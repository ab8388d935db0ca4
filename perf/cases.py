"""Timed cases of the LoRA fine-tuning framework: what a program built on it runs, through its public entry points.

    train   one turn of the training loop on a LoraStepEngine: the optimizer step on the gradients of the batch before,
            then forward + loss + backward of this batch (the same work as train_step, cut between backward and
            optimizer so that gradients and updated adapters are both there to be compared)
    ppl     corpus perplexity (LoraStepEngine.perplexity): forward and loss only
    score   multiple-choice evaluation (LoraStepEngine.score_tokens): one call per question, prompts of unequal length
    attn    the attention operator by itself, forward and backward (ops.attention_fwd / attention_bwd)
    mlp_f32 a gated MLP of the eager f32 operators (the C++ operator API's default type), forward and backward
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mobilefinetuner_b200 import _lib as L
from mobilefinetuner_b200 import configs as Cf
from mobilefinetuner_b200 import ops as O
from mobilefinetuner_b200 import synth
from mobilefinetuner_b200.engine import LoraStepEngine

MODELS = {"gpt2_small": Cf.GPT2_SMALL, "qwen25_05b": Cf.QWEN25_05B, "gemma3_270m": Cf.GEMMA3_270M, "gemma3_1b": Cf.GEMMA3_1B}
LR, CLIP = 2e-4, 1.0
CANDIDATES = 4                        # answer letters of a multiple-choice question
MIN_TOKENS, MAX_TOKENS, MAX_SEQ = 512, 16384, 2048     # smallest and largest batch, largest sequence of the configurations


def listed():
    return [
        # the four benchmark configurations of configs.CONFIGS at their own sizes: small and launch-bound, two ordinary
        # ones, and the largest step the framework is run at
        dict(name="train_gpt2_small_4x128", kind="train", model="gpt2_small", batch=4, seq=128, pad=0.0),
        dict(name="train_qwen25_05b_8x512", kind="train", model="qwen25_05b", batch=8, seq=512, pad=0.0),
        dict(name="train_gemma3_270m_16x1024", kind="train", model="gemma3_270m", batch=16, seq=1024, pad=0.0),
        dict(name="train_gemma3_1b_8x2048", kind="train", model="gemma3_1b", batch=8, seq=2048, pad=0.0),
        # short sequences on the largest model, as many tokens as the smallest configuration
        dict(name="train_gemma3_1b_4x128", kind="train", model="gemma3_1b", batch=4, seq=128, pad=0.0),
        # batches cut to the longest example: lengths that are no multiple of anything, shorter examples padded with
        # ignored labels
        dict(name="train_qwen25_05b_5x397", kind="train", model="qwen25_05b", batch=5, seq=397, pad=0.25),
        dict(name="train_gemma3_270m_3x1001", kind="train", model="gemma3_270m", batch=3, seq=1001, pad=0.25),
        # evaluation: perplexity over full-context windows, and letter scoring over four prompts
        dict(name="ppl_gpt2_small_4x1024", kind="ppl", model="gpt2_small", batch=4, seq=1024, pad=0.0),
        dict(name="score_gemma3_270m_437", kind="score", model="gemma3_270m", seq=437, questions=4),
        # the operator: the long end of the grouped-query sweep, and Gemma's head size with its window on a ragged length
        dict(name="attn_14x2x64_8x4096", kind="attn", batch=8, heads=14, kv_heads=2, head_dim=64, seq=4096, window=0),
        dict(name="attn_4x1x256_4x1000_w512", kind="attn", batch=4, heads=4, kv_heads=1, head_dim=256, seq=1000, window=512),
        # eager f32 operators at the widths of the 0.5 B model, a batch of 4 x 128 tokens
        dict(name="mlp_f32_512x896x4864", kind="mlp_f32", tokens=512, hidden=896, inter=4864),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "ppl", "score", "attn", "attn", "mlp_f32"])
    if kind in ("train", "ppl"):
        model = rng.choice(sorted(MODELS))
        seq = _log_int(rng, 64, MODELS[model].n_positions or MAX_SEQ)
        if rng.random() < 0.4:
            seq = max(64, seq // 64 * 64)
        batch = _log_int(rng, -(-MIN_TOKENS // seq), min(16, MAX_TOKENS // seq))
        return dict(kind=kind, model=model, batch=batch, seq=seq, pad=rng.choice([0.0, 0.0, 0.25]))
    if kind == "score":
        model = rng.choice(sorted(MODELS))
        return dict(kind=kind, model=model, seq=_log_int(rng, 96, 1000), questions=rng.choice([1, 2, 4]))
    if kind == "attn":
        heads, kv_heads, head_dim = rng.choice([(14, 2, 64), (12, 12, 64), (4, 1, 256)])
        seq = _log_int(rng, 64, 4096)
        if rng.random() < 0.4:
            seq = max(64, seq // 64 * 64)
        batch = _log_int(rng, 1, max(1, min(8, 32768 // seq)))
        window = rng.choice([0, 512]) if head_dim == 256 else 0
        return dict(kind=kind, batch=batch, heads=heads, kv_heads=kv_heads, head_dim=head_dim, seq=seq, window=window)
    hidden, inter = rng.choice([(640, 2048), (896, 4864), (1152, 6912)])
    return dict(kind=kind, tokens=_log_int(rng, 64, 2048), hidden=hidden, inter=inter)


# ------------------------------------------------------------------ inputs
def _frozen(spec, gen):
    """Random weights in parameters() order, generated on the device: N(0, 0.02) matrices and biases, neutral norms
    with some jitter.  None: derived by the engine from another tensor."""
    for kind, shape in spec.param_shapes():
        if kind == "lm_head":
            yield None
        elif kind in ("wte", "wpe", "embed", "linear", "bias"):
            yield torch.randn(shape, device="cuda", generator=gen) * 0.02
        else:
            base = 1.0 if kind == "ln" or (kind == "norm" and spec.family != Cf.GEMMA) else 0.0
            yield base + 0.05 * torch.randn(shape, device="cuda", generator=gen)


def _engine(spec, batch, seq, seed):
    eng = LoraStepEngine(spec, batch, seq)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    for i, a in enumerate(_frozen(spec, gen)):
        if a is not None:
            L.call("mft_model_set_param_dev", eng._h, i, a.data_ptr())
    torch.cuda.synchronize()
    eng.set_lora(synth.make_lora(spec, seed))
    return eng


def _batch(spec, case, seed):
    ids, labels = synth.make_batch(spec, case["batch"], case["seq"], seed)
    if case["pad"] > 0:
        # row b keeps a prefix: the first row is full, the others end up to `pad` earlier
        s = case["seq"]
        for b in range(1, case["batch"]):
            labels[b, s - int(s * case["pad"] * b / case["batch"]):] = -100
    return ids, labels


_last = {}


def prepare(case, seed):
    kind = case["kind"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if {k: v for k, v in case.items() if k != "name"} != _last.get("case"):
        _last["case"] = {k: v for k, v in case.items() if k != "name"}
        L.init(torch.cuda.current_device())
        L.call("mft_empty_cache")          # another model: the memory of the last one goes back to the driver
    if kind == "train":
        spec = MODELS[case["model"]]
        eng = _engine(spec, case["batch"], case["seq"], seed)
        ids, labels = _batch(spec, case, seed + 1)
        eng.forward_backward(*_batch(spec, case, seed + 2))      # gradients of the batch before
        grads, params = eng.grad_bucket(), eng.param_bucket()
        grads.engine = params.engine = eng                       # the views live in the engine's memory
        return dict(kind=kind, eng=eng, ids=ids, labels=labels, grads=grads, params=params)
    if kind == "ppl":
        spec = MODELS[case["model"]]
        return dict(kind=kind, eng=_engine(spec, case["batch"], case["seq"], seed), batches=[_batch(spec, case, seed + 1)])
    if kind == "score":
        spec = MODELS[case["model"]]
        n = case["questions"]
        g = synth.rng(seed + 1)
        prompts = [synth.zipf_ids(g, (case["seq"] - 19 * i,), spec.vocab) for i in range(n)]
        letters = [np.asarray(g.choice(spec.vocab, CANDIDATES, replace=False), np.int32) for _ in range(n)]
        return dict(kind=kind, eng=_engine(spec, 1, case["seq"], seed), prompts=prompts, letters=letters)
    if kind == "attn":
        def heads(n):
            return torch.randn(case["batch"], case["seq"], n, case["head_dim"], device="cuda", generator=gen).bfloat16().permute(0, 2, 1, 3)
        q, k, v, d_o = heads(case["heads"]), heads(case["kv_heads"]), heads(case["kv_heads"]), heads(case["heads"])
        return dict(kind=kind, q=q, k=k, v=v, d_o=d_o, scale=case["head_dim"] ** -0.5, window=case["window"])
    t, h, i = case["tokens"], case["hidden"], case["inter"]

    def rnd(*shape, scale=1.0):
        return torch.randn(shape, device="cuda", generator=gen) * scale
    s = dict(kind=kind, x=rnd(t, h), dy=rnd(t, h), wg=rnd(h, i, scale=h ** -0.5), wu=rnd(h, i, scale=h ** -0.5), wd=rnd(i, h, scale=i ** -0.5))
    for name, cols in (("g", i), ("u", i), ("a", i), ("y", h), ("da", i), ("dg", i), ("du", i), ("dx", h), ("dx_up", h)):
        s[name] = torch.empty(t, cols, device="cuda")
    return s


# ------------------------------------------------------------------ one pass
def _matmul(a, b, out, trans_b):
    m, k = a.shape
    L.call("mft_matmul_f32", a.data_ptr(), b.data_ptr(), out.data_ptr(), 1, m, out.shape[1], k, 0, 0, 0, trans_b,
           torch.cuda.current_stream().cuda_stream)


def run(state):
    kind = state["kind"]
    if kind == "train":
        eng = state["eng"]
        eng.optimizer_step(LR, max_grad_norm=CLIP)
        loss, scored = eng.forward_backward(state["ids"], state["labels"])
        return {"loss": loss, "scored": scored, "grads": state["grads"], "params": state["params"]}
    if kind == "ppl":
        nll, ppl, tokens = state["eng"].perplexity(state["batches"])
        return {"nll": nll, "ppl": ppl, "tokens": tokens}
    if kind == "score":
        return [state["eng"].score_tokens(p, c) for p, c in zip(state["prompts"], state["letters"])]
    if kind == "attn":
        q, k, v = state["q"], state["k"], state["v"]
        o, lse = O.attention_fwd(q, k, v, state["scale"], state["window"])
        dq, dk, dv = O.attention_bwd(q, k, v, o, state["d_o"], lse, state["scale"], state["window"])
        return {"o": o, "lse": lse, "dq": dq, "dk": dk, "dv": dv}
    st = torch.cuda.current_stream().cuda_stream
    s = state
    _matmul(s["x"], s["wg"], s["g"], 0)
    _matmul(s["x"], s["wu"], s["u"], 0)
    L.call("mft_swiglu_f32", s["g"].data_ptr(), s["u"].data_ptr(), None, s["a"].data_ptr(), None, s["a"].numel(), st)
    _matmul(s["a"], s["wd"], s["y"], 0)
    _matmul(s["dy"], s["wd"], s["da"], 1)
    L.call("mft_swiglu_f32", s["g"].data_ptr(), s["u"].data_ptr(), s["da"].data_ptr(), s["dg"].data_ptr(), s["du"].data_ptr(), s["a"].numel(), st)
    _matmul(s["dg"], s["wg"], s["dx"], 1)
    _matmul(s["du"], s["wu"], s["dx_up"], 1)
    L.call("mft_add_f32", s["dx"].data_ptr(), s["dx_up"].data_ptr(), s["dx"].data_ptr(), s["dx"].numel(), st)
    return {"y": s["y"], "dx": s["dx"]}


# ------------------------------------------------------------------ what a pass cannot do without
def _pairs(seq, window):
    return sum(min(j + 1, window) for j in range(seq)) if window > 0 else seq * (seq + 1) // 2


def _forward_flops(spec, batch, seq, lm_rows):
    """Forward share of ModelSpec.step_flops, with the lm head on `lm_rows` positions."""
    t, h, qd, kd = batch * seq, spec.hidden, spec.n_heads * spec.head_dim, spec.n_kv_heads * spec.head_dim
    up = 1 if spec.family == Cf.GPT2 else 2
    per_token = h * (qd + 2 * kd) + qd * h + (up + 1) * h * spec.inter
    lora = sum(math.prod(shape) for _, shape in spec.lora_shapes())
    f = 2.0 * t * (spec.layers * per_token + lora) + 2.0 * lm_rows * h * spec.vocab
    for i in range(spec.layers):
        f += 4.0 * spec.head_dim * spec.n_heads * batch * _pairs(seq, spec.sliding_window if spec.layer_is_sliding(i) else 0)
    return f


def work(case):
    kind = case["kind"]
    if kind in ("train", "ppl", "score"):
        spec = MODELS[case["model"]]
        # frozen weights once, in bf16 (Gemma's lm_head is the tied table)
        frozen = 2.0 * sum(math.prod(shape) for k, shape in spec.param_shapes() if k != "lm_head")
        adapters = 4.0 * sum(math.prod(shape) for _, shape in spec.lora_shapes())
        if kind == "train":
            # adapters, gradients and the two Adam moments are each read and written; ids and labels are int32
            t, h = case["batch"] * case["seq"], spec.hidden
            flops = spec.step_flops(case["batch"], case["seq"])
            if spec.family == Cf.GPT2 and spec.gpt2_detach_attn:
                # nothing flows back through attention and its two projections there
                flops -= spec.layers * (8.0 * t * h * h + 8.0 * h * case["batch"] * _pairs(case["seq"], 0))
            return {"bytes": frozen + 8 * adapters + 8.0 * t, "flops": flops}
        if kind == "ppl":
            t = case["batch"] * case["seq"]
            return {"bytes": frozen + adapters + 8.0 * t, "flops": _forward_flops(spec, case["batch"], case["seq"], t)}
        lengths = [case["seq"] - 19 * i for i in range(case["questions"])]
        return {"bytes": len(lengths) * (frozen + adapters) + 4.0 * sum(lengths), "flops": sum(_forward_flops(spec, 1, s, 1) for s in lengths)}
    if kind == "attn":
        rows = case["batch"] * case["seq"]
        q, kv = 2.0 * rows * case["heads"] * case["head_dim"], 2.0 * rows * case["kv_heads"] * case["head_dim"]
        # in: q, k, v, dO; out: O, dQ, dK, dV and the f32 row log-sum-exp
        pairs = case["batch"] * case["heads"] * _pairs(case["seq"], case["window"])
        return {"bytes": 4 * q + 4 * kv + 4.0 * rows * case["heads"], "flops": 12.0 * case["head_dim"] * pairs}
    t, h, i = case["tokens"], case["hidden"], case["inter"]
    return {"bytes": 4.0 * (4 * t * h + 3 * h * i), "flops": 12.0 * t * h * i}


def tolerance(case):
    if case["kind"] == "mlp_f32":
        return {"rel": 1e-5}                  # f32 sums of up to 6912 terms, two products deep
    if case["kind"] == "attn":
        return {"rel": 1e-2}                  # bf16 operands and probabilities, f32 accumulation
    if case["kind"] == "train":
        return {"rel": 2e-2}                  # gradients through up to 26 layers of bf16 activations
    return {"rel": 2e-3}                      # losses and log-probabilities, formed in f32 from bf16 activations
