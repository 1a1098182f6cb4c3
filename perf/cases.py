"""The workloads this library is measured on, through the calls a user's program makes: the isolated quantised product
(`fc_qmatmul_dev` on device buffers), generation with a resident model (`prefill`, `decode_greedy`, `topk`,
`feed_greedy`, `feed_batch`) and scoring (`score_batch`, `score_ragged`).

Models are the repository's benchmark configurations (`hostmodel.config_c1/c3/c4/c5`) with seeded N(0, 0.02) weights,
packed as the blocks of a quantised file. Every case is a dict of plain values; `draw` gives more of the same ranges:
products of 1..4096 rows, K 256..4096 in whole blocks of 32, any N in 256..32000; models of 2 layers up to the
configuration's own depth, 1..64 streams, prompts up to 1536 tokens; 1..256 sequences of 17..1024 ids. Packed weights
are Q8_0 or Q4_0.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from ferrum_gpu_b200 import CudaGpt2, CudaLlama, Device, Mode, QKind, upload_qweight
from ferrum_gpu_b200 import _ffi, hostmodel
from ferrum_gpu_b200.engine import Rng, SampleParams, sample_candidates

CONFIGS = {"c1": hostmodel.config_c1, "c3": hostmodel.config_c3, "c4": hostmodel.config_c4, "c5": hostmodel.config_c5}
TIED = {"c1": False, "c3": False, "c4": True, "c5": True}
STD = 0.02
_device = None


def listed():
    return [
        # -- the product alone --
        # the smallest projection of a small model at batch 1: a call is launch and latency
        {"name": "product_1x768x768_q8", "path": "product", "m": 1, "k": 768, "n": 768, "weights": "Q8_0", "mode": "exact"},
        # the vocabulary head of a 4096-wide model at batch 1: the weight stream from HBM
        {"name": "product_1x4096x32000_q4", "path": "product", "m": 1, "k": 4096, "n": 32000, "weights": "Q4_0", "mode": "exact"},
        # a feed-forward product of batched decode, a batch that fills no tile
        {"name": "product_40x2048x11008_q4", "path": "product", "m": 40, "k": 2048, "n": 11008, "weights": "Q4_0", "mode": "exact"},
        # the head over one prompt of odd length on the tensor cores
        {"name": "product_500x2048x32000_q4", "path": "product", "m": 500, "k": 2048, "n": 32000, "weights": "Q4_0", "mode": "tensor"},
        # a feed-forward product of batched scoring, the largest of the product grid but the head
        {"name": "product_4096x4096x11008_q8", "path": "product", "m": 4096, "k": 4096, "n": 11008, "weights": "Q8_0", "mode": "tensor"},
        # -- generation --
        # one user of the small GPT-2-style model: 16 prompt tokens, 128 more, greedy
        {"name": "generate_c1_b1", "path": "generate", "model": "c1", "layers": 6, "weights": "Q8_0", "streams": 1,
         "prompt": 16, "steps": 128, "top_k": 0},
        # one user of the Llama-style model, sampled: candidates selected on the device, one draw per token on the host
        {"name": "sample_c3_b1", "path": "generate", "model": "c3", "layers": 12, "weights": "Q4_0", "streams": 1,
         "prompt": 128, "steps": 64, "top_k": 40},
        # a handful of users at once: prompts of different lengths in the default arithmetic, then decoded together
        {"name": "serve_c3_b6", "path": "generate", "model": "c3", "layers": 12, "weights": "Q4_0", "streams": 6,
         "prompt": 600, "steps": 64, "top_k": 0},
        # a full server: 64 streams of the Qwen2-style model decoding together
        {"name": "decode_c4_b64", "path": "generate", "model": "c4", "layers": 24, "weights": "Q8_0", "streams": 64,
         "prompt": 0, "steps": 128, "top_k": 0},
        # a long prompt and a short answer, in the default arithmetic: time to first token and decode over a long cache
        {"name": "long_prompt_c4_b1", "path": "generate", "model": "c4", "layers": 24, "weights": "Q8_0", "streams": 1,
         "prompt": 1536, "steps": 64, "top_k": 0},
        # -- scoring --
        # the batched scoring run: 256 sequences of 1024 ids
        {"name": "score_c3_256x1024", "path": "score", "model": "c3", "layers": 12, "weights": "Q4_0", "seqs": 256,
         "length": 1024, "ragged": False, "mode": "tensor"},
        # a server's concurrent scoring requests: texts of all lengths against a large tied vocabulary
        {"name": "score_c5_ragged", "path": "score", "model": "c5", "layers": 12, "weights": "Q4_0", "seqs": 23,
         "length": 1000, "ragged": True, "mode": "tensor"},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    weights = rng.choice(["Q8_0", "Q4_0"])
    path = rng.choice(["product", "product", "generate", "score"])
    if path == "product":
        m = _log_int(rng, 1, 4096)
        # beyond the decode widths most callers ask for the tensor cores, some for the default
        mode = "exact" if m <= 64 or (m <= 512 and rng.random() < 0.25) else "tensor"
        # (the tensor-core product takes K in steps of 64)
        k = 32 * _log_int(rng, 8, 128) if mode == "exact" else 64 * _log_int(rng, 4, 64)
        return {"path": path, "m": m, "k": k, "n": _log_int(rng, 256, 32000), "weights": weights, "mode": mode}
    model = rng.choice(sorted(CONFIGS))
    cfg = CONFIGS[model]()
    layers = rng.randint(2, cfg.layers)
    if path == "generate":
        streams = _log_int(rng, 1, 64)
        steps = rng.randint(8, 96)
        most = min(cfg.ctx - steps - 1, 4096 // streams)
        prompt = 0 if rng.random() < 0.25 else _log_int(rng, 2, min(1536, most))
        top_k = rng.choice([0, 0, 20, 100]) if streams == 1 and prompt else 0
        return {"path": path, "model": model, "layers": layers, "weights": weights, "streams": streams, "prompt": prompt,
                "steps": steps, "top_k": top_k}
    length = _log_int(rng, 17, min(1024, cfg.ctx))
    mode = "exact" if rng.random() < 0.25 else "tensor"
    most = (2048 if mode == "exact" else 32768) // length
    return {"path": path, "model": model, "layers": layers, "weights": weights, "seqs": _log_int(rng, 1, min(256, max(2, most))),
            "length": length, "ragged": rng.random() < 0.5, "mode": mode}


# ---- inputs ------------------------------------------------------------------------------------------------------

def _dev() -> Device:
    global _device
    if _device is None:
        _device = Device.open(0)
    return _device


def _blocks(w: torch.Tensor, kind: str) -> np.ndarray:
    """An `[n, k]` f32 matrix as the bytes of a quantised file: n rows of k / 32 blocks."""
    b = w.reshape(-1, 32)
    peak = b.gather(1, b.abs().argmax(dim=1, keepdim=True))
    scale = (peak.abs() / 127 if kind == "Q8_0" else peak / -8).to(torch.float16)
    q = torch.where(scale == 0, torch.zeros_like(b), b / scale.float())
    if kind == "Q8_0":
        codes = q.round().clamp(-127, 127).to(torch.int8).view(torch.uint8)
    else:
        q = (q.round() + 8).clamp(0, 15).to(torch.uint8)
        codes = q[:, :16] | (q[:, 16:] << 4)
    return torch.cat([scale.view(torch.uint8), codes], dim=1).reshape(-1).cpu().numpy()


def _lengths(case):
    """Prompt or sequence lengths, spread over the upper three quarters of the largest one where they differ."""
    n, top = (case["seqs"], case["length"]) if case["path"] == "score" else (case["streams"], case["prompt"])
    if n == 1 or (case["path"] == "score" and not case["ragged"]):
        return [top] * n
    low = max(2 if case["path"] == "score" else 1, top // 4)
    return [top - (i * 617) % max(1, top - low + 1) for i in range(n)]


def _config(case):
    cfg = CONFIGS[case["model"]]()
    cfg.layers = case["layers"]
    return cfg


def _model(case, gen):
    """The model as a quantised file holds it (packed blocks, f32 norms and biases), resident on the device."""
    cfg = _config(case)
    kind = case["weights"]
    none = np.zeros(0, dtype=np.float32)

    def mat(k, n):
        return _blocks(torch.randn(n, k, device="cuda", generator=gen) * STD, kind)

    def vec(n, std):
        return (torch.randn(n, device="cuda", generator=gen) * std).cpu().numpy()

    packed = {"tok": mat(cfg.dim, cfg.vocab)}
    packed["head"] = packed["tok"] if TIED[case["model"]] else mat(cfg.dim, cfg.vocab)
    ones = np.ones(cfg.dim, dtype=np.float32)
    zeros = np.zeros(max(cfg.dim, cfg.hidden), dtype=np.float32)
    blocks = []
    if isinstance(cfg, hostmodel.LlamaConfig):
        biased = case["model"] == "c4"
        for _ in range(cfg.layers):
            blocks.append(hostmodel.LlamaBlock(
                attn_norm=ones, wq=none, wk=none, wv=none, wo=none, ffn_norm=ones, gate=none, up=none, down=none,
                bq=vec(cfg.q_dim, STD) if biased else None, bk=vec(cfg.kv_dim, STD) if biased else None,
                bv=vec(cfg.kv_dim, STD) if biased else None))
        model = hostmodel.Llama(cfg, none, blocks, ones, none, TIED[case["model"]])
        names, cls = _ffi.LLAMA_MATS, CudaLlama
    else:
        d, h = cfg.dim, cfg.hidden
        for _ in range(cfg.layers):
            blocks.append(hostmodel.Gpt2Block(
                ln1_g=ones, ln1_b=zeros[:d], wq=none, bq=zeros[:d], wk=none, bk=zeros[:d], wv=none, bv=zeros[:d],
                wo=none, bo=zeros[:d], ln2_g=ones, ln2_b=zeros[:d], w1=none, b1=zeros[:h], w2=none, b2=zeros[:d]))
        model = hostmodel.Gpt2(cfg, none, vec(cfg.ctx * d, STD), blocks, ones, zeros[:d], none)
        names, cls = _ffi.GPT2_MATS, CudaGpt2
    for i in range(cfg.layers):
        for name in names:
            packed[(i, name)] = mat(*model.mat_shape(name))
    return cls(_dev(), model, QKind[kind], max_streams=case.get("streams", 1), packed=packed)


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    dev = _dev()
    if case["path"] == "product":
        m, k, n = case["m"], case["k"], case["n"]
        w = upload_qweight(dev, QKind[case["weights"]], _blocks(torch.randn(n, k, device="cuda", generator=gen) * STD, case["weights"]), k, n)
        x = torch.randn(m, k, device="cuda", generator=gen)
        y = torch.empty(m, n, device="cuda")
        torch.cuda.synchronize()
        return {"case": case, "w": w, "x": x, "y": y}
    cfg = _config(case)
    state = {"case": case, "model": _model(case, gen)}
    ids = np.random.default_rng(seed)
    seqs = [ids.integers(0, cfg.vocab, size=n, dtype=np.int32) for n in _lengths(case)]
    if case["path"] == "score":
        state["ids"] = seqs if case["ragged"] else np.stack(seqs)
    else:
        state["prompts"] = seqs
        state["first"] = ids.integers(0, cfg.vocab, size=case["streams"], dtype=np.int32)
        state["seed"] = seed
    return state


# ---- one pass ----------------------------------------------------------------------------------------------------

def _mode(case):
    return Mode.EXACT_F32 if case["mode"] == "exact" else Mode.TENSOR_F16


def _sampled(m, prompt, case, seed):
    """`generate` with a top-k draw: the prompt in one pass, then one draw per token over the device's candidates."""
    params = SampleParams(temperature=0.8, top_k=case["top_k"], top_p=0.95, repetition_penalty=1.1)
    rng = Rng(seed)
    logits = m.prefill(prompt)
    history, values = prompt.tolist(), []
    for step in range(case["steps"]):
        if step:
            m.feed_greedy(history[-1])
        idx, val = m.topk(params.top_k, 0, params.repetition_penalty, history[-64:])
        values.append(val)
        history.append(sample_candidates(idx, val, params, rng))
    return {"first": logits, "tokens": np.array(history[prompt.size:], dtype=np.int32), "values": np.stack(values),
            "last": m.feed(history[-1])}


def run(state):
    case = state["case"]
    if case["path"] == "product":
        w = state["w"]
        w.dev.check(_ffi.load().fc_qmatmul_dev(w.handle, state["x"].data_ptr(), case["m"], state["y"].data_ptr(), int(_mode(case))))
        return state["y"]
    m = state["model"]
    if case["path"] == "score":
        logprob, greedy, nll = (m.score_ragged if case["ragged"] else m.score_batch)(state["ids"], _mode(case))
        if case["ragged"]:
            logprob, greedy = np.concatenate(logprob), np.concatenate(greedy)
        return {"logprob": logprob, "greedy": greedy, "nll": nll}
    for s in range(case["streams"]):
        m.reset(s)
    if case["top_k"]:
        return _sampled(m, state["prompts"][0], case, state["seed"])
    out = {}
    if case["prompt"]:
        out["first"] = np.stack([m.prefill(p, stream=s) for s, p in enumerate(state["prompts"])])
    else:
        _, out["first"] = m.feed_batch(state["first"], want_logits=True)
    out["tokens"] = m.decode_greedy(out["first"].argmax(axis=1), case["steps"])
    if case["streams"] <= 8:
        # (among thousands of picks one that rounding decides is likely, and it sends its stream another way:
        # with many streams only the logits before the chain are comparable)
        _, out["last"] = m.feed_batch(out["tokens"][-1], want_logits=True)
    return out


# ---- what a pass cannot do without --------------------------------------------------------------------------------

def _weight_bytes(case, params):
    return params * (34 if case["weights"] == "Q8_0" else 18) / 32


def work(case):
    if case["path"] == "product":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": _weight_bytes(case, k * n) + 4.0 * m * (k + n), "flops": 2.0 * m * n * k}
    cfg = _config(case)
    llama = isinstance(cfg, hostmodel.LlamaConfig)
    q_dim, kv_dim = (cfg.q_dim, cfg.kv_dim) if llama else (cfg.dim, cfg.dim)
    trunk = cfg.layers * (cfg.dim * (2 * q_dim + 2 * kv_dim) + (3 if llama else 2) * cfg.dim * cfg.hidden)
    head = cfg.dim * cfg.vocab
    kv = cfg.layers * 2 * kv_dim * 4.0  # bytes of one position's k and v
    bytes_ = flops = 0.0
    if case["path"] == "score":
        for n in _lengths(case):
            t = n - 1
            flops += 2.0 * (trunk + head) * t + 2.0 * q_dim * t * (t + 1) * cfg.layers
            bytes_ += 4.0 * n + 5.0 * t + 8
        return {"bytes": bytes_ + _weight_bytes(case, trunk + head), "flops": flops}
    for p in _lengths(case):
        if p:  # the prompt: weights once per prompt, its k and v written, one row of logits
            flops += 2.0 * trunk * p + 2.0 * head + 2.0 * q_dim * p * (p + 1) * cfg.layers
            bytes_ += _weight_bytes(case, trunk + head) + kv * p + 4.0 * cfg.vocab
        for i in range(case["steps"] + 1):
            flops += 2.0 * (trunk + head) + 4.0 * q_dim * (p + i + 1) * cfg.layers
            bytes_ += kv * (p + i + 2)
    # every step reads the weights once for all streams; beside the chained steps one whose logits come back
    bytes_ += (case["steps"] + 1) * _weight_bytes(case, trunk + head) + 4.0 * case["streams"] * cfg.vocab
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # about four times what was measured: a product against the same in f64 7e-7 (exact) and 2.9e-4 (fp16 operands),
    # a prompt in one pass against the same token by token 2.2e-6, fp16-operand log-probabilities against exact 5.6e-5
    if case["path"] == "generate":
        return {"rel": 1e-5, "max": 5e-5, "differ": 0.01}
    if case["mode"] == "exact":
        return {"rel": 5e-6, "max": 2e-5, "differ": 0.001}
    if case["path"] == "product":
        return {"rel": 1e-3, "max": 8e-3}
    return {"rel": 2.5e-4, "max": 1e-3, "differ": 0.001}
