"""The work a user of this library has it do, as cases that can be timed and compared.

Three kinds of caller are covered, each through the public Python mirror of the C ABI:

* an engine that calls the operator surface with HOST pointers, one call per projection or expert batch
  (``op`` = matvec, chain, fp4_batch);
* a decode loop over a device-resident stack of MoE layers, activations in HBM (``op`` = decode), the same with the
  activations in host memory (``op`` = decode_host), or with the whole feed-forward block of a layer (``op`` = block);
* prefill through the two-phase layer calls on the tensor cores (``op`` = prefill).

Sizes are those of the repository's benchmark configurations (affine-Q4: hidden 2816, 128 experts of 704, top-8;
NVFP4: hidden 5120, 64 experts of 1536, top-4; single projection 4096 x 4096) and one generic smaller MoE geometry
(hidden 2048, 64 experts of 768, top-8).  The weights of a geometry are laid out once per process, as a serving
program does; every state holds its own tokens.
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

synth = importlib.import_module("salt-core_b200.synth")
backend = importlib.import_module("salt-core_b200.backend")
stack_mod = importlib.import_module("salt-core_b200.stack")

Q4_GEOMETRIES = ((2816, 704, 128, 8), (2048, 768, 64, 8))
FP4_GEOMETRY = (5120, 1536, 64, 4)
Q4_LAYERS, FP4_LAYERS = 6, 2
Q4_TOKENS, FP4_TOKENS = 2048, 256
DENSE_INTER = 2112


def listed():
    q4 = dict(zip(("hidden", "inter", "experts", "topk"), Q4_GEOMETRIES[0]), format="q4")
    fp4 = dict(zip(("hidden", "inter", "experts", "topk"), FP4_GEOMETRY), format="nvfp4")
    return [
        # one dense projection of one token: the smallest call of an engine that keeps its activations on the host
        {"name": "abi-q4-matvec", "op": "matvec", "rows": 4096, "cols": 4096},
        # the eight selected experts of one token, gate | up | GeGLU | down, from the host
        dict(q4, name="abi-q4-chain", op="chain", count=8, group=1),
        # a few draft tokens through one NVFP4 projection, from the host
        {"name": "abi-nvfp4-batch", "op": "fp4_batch", "rows": 1536, "cols": 5120, "batch": 7},
        # single-stream decode: the latency a chat user sees
        dict(q4, name="q4-decode-b1", op="decode", batch=1, layers=6),
        # a few streams whose activations come from and go to the host
        dict(q4, name="q4-decode-host-b3", op="decode_host", batch=3, layers=6),
        # small and full decode batches of a server
        dict(q4, name="q4-decode-b16", op="decode", batch=16, layers=6),
        dict(q4, name="q4-decode-b64", op="decode", batch=64, layers=6),
        # whole feed-forward block of one layer (dense branch beside the experts) for two streams
        dict(q4, name="q4-block-b2", op="block", batch=2, layers=1),
        # prompts: the accurate form on a chunk of 512 tokens, the fast form on a long ragged prompt
        dict(q4, name="q4-prefill-split-512", op="prefill", batch=512, precision="split", layers=1),
        dict(q4, name="q4-prefill-single-1999", op="prefill", batch=1999, precision="single", layers=1),
        # NVFP4 experts: single-stream decode with the exact kernels, a prompt chunk on block-scaled tensor cores
        dict(fp4, name="nvfp4-decode-b1", op="decode", batch=1, layers=2),
        dict(fp4, name="nvfp4-prefill-256", op="prefill", batch=256, precision="split", layers=1),
    ]


def _log(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    op = rng.choice(("matvec", "chain", "fp4_batch", "decode", "decode", "decode", "decode_host", "block", "prefill",
                     "prefill", "fp4_decode", "fp4_prefill"))
    if op == "matvec":
        return {"op": op, "rows": _log(rng, 64, 8192), "cols": 64 * _log(rng, 4, 128)}
    if op == "fp4_batch":
        return {"op": op, "rows": _log(rng, 64, 6144), "cols": 256 * _log(rng, 1, 20), "batch": _log(rng, 1, 32)}
    if op in ("fp4_decode", "fp4_prefill"):
        c = dict(zip(("hidden", "inter", "experts", "topk"), FP4_GEOMETRY), format="nvfp4")
        if op == "fp4_decode":
            return dict(c, op="decode", batch=_log(rng, 1, 16), layers=rng.randint(1, FP4_LAYERS))
        return dict(c, op="prefill", batch=_log(rng, 16, FP4_TOKENS), precision="split", layers=1)
    c = dict(zip(("hidden", "inter", "experts", "topk"), rng.choice(Q4_GEOMETRIES)), format="q4")
    if op == "chain":
        return dict(c, op=op, count=rng.randint(1, 16), group=_log(rng, 1, 8))
    if op == "block":
        return dict(c, op=op, batch=_log(rng, 1, 16), layers=1)
    if op == "prefill":
        return dict(c, op=op, batch=_log(rng, 128, 1999), precision=rng.choice(("split", "single")), layers=1)
    return dict(c, op=op, batch=_log(rng, 1, 64 if op == "decode" else 16), layers=rng.randint(1, Q4_LAYERS))


# ---- weights: made on the GPU, handed to the library as host arrays, once per process and geometry --------------
_kept = {}


def _once(key, make):
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _bf16_bytes(t):
    return t.to(torch.bfloat16).view(torch.uint8).reshape(t.shape[0], -1)


def _q4_tensors(g, count, rows, cols):
    """`count` affine-Q4 tensors, values | scales | biases: uniform codes, scale U(0.005, 0.02), and a bias that
    centres the weights up to a spread of half a step, as a min/max quantiser leaves it."""
    vb, gb = synth.q4_tensor_bytes(rows, cols)
    scale = (torch.rand(count, gb // 2, generator=g, device="cuda") * 0.015 + 0.005).to(torch.bfloat16).float()
    bias = -(7.5 + 0.5 * torch.randn(count, gb // 2, generator=g, device="cuda")) * scale
    codes = torch.randint(0, 256, (count, vb), generator=g, device="cuda", dtype=torch.uint8)
    return torch.cat((codes, _bf16_bytes(scale), _bf16_bytes(bias)), dim=1).cpu().numpy()


def _router(g, experts, hidden):
    return dict(router_w=(torch.randn(experts, hidden, generator=g, device="cuda") * 0.02).cpu().numpy(),
                router_scale=np.ones(hidden, np.float32), per_expert_scale=np.ones(experts, np.float32),
                norm_weight=(1.0 + 0.1 * torch.randn(hidden, generator=g, device="cuda")).cpu().numpy())


def _q4_layer(index, hidden, inter, experts, topk):
    g = _gen(1000 + index)
    pool = _q4_tensors(g, 3 * experts, inter, hidden)
    return synth.Q4MoeLayer(hidden, inter, experts, topk, 1e-6, pool=pool.reshape(-1), expert_stride=3 * pool.shape[1],
                            **_router(g, experts, hidden))


E2M1_STEPS = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0])


def _fp4_tensors(g, count, rows, cols):
    """`count` NVFP4 tensors quantised from N(0, 0.02) matrices: codes | block scales, and their weight divisors."""
    steps = E2M1_STEPS.cuda()
    out = np.empty((count, rows * cols // 2 + rows * cols // 16), np.uint8)
    divisors = np.empty(count, np.float32)
    for i in range(count):
        w = torch.randn(rows * cols // 16, 16, generator=g, device="cuda") * 0.02
        divisor = 448.0 * 6.0 / w.abs().max()
        scale = (w.abs().amax(dim=1) / 6.0 * divisor).to(torch.float8_e4m3fn)
        unit = scale.float() / divisor
        t = w / torch.where(unit == 0, 1.0, unit)[:, None]
        codes = (torch.bucketize(t.abs(), steps) | (torch.signbit(t).long() << 3)).to(torch.uint8).reshape(-1)
        packed = codes[0::2] | (codes[1::2] << 4)
        out[i] = torch.cat((packed, scale.view(torch.uint8))).cpu().numpy()
        divisors[i] = float(divisor)
    return out, divisors


def _fp4_layer(index, hidden, inter, experts, topk):
    g = _gen(2000 + index)
    pool, divisors = _fp4_tensors(g, 3 * experts, inter, hidden)
    return synth.Nvfp4MoeLayer(hidden, inter, experts, topk, 1e-6, pool=pool.reshape(-1),
                               expert_stride=3 * pool.shape[1], weight_divisors=divisors.reshape(experts, 3),
                               input_globals=np.full((experts, 3), 64.0, np.float32), **_router(g, experts, hidden))


def _dense_block(hidden):
    g = _gen(3000)
    w = [_q4_tensors(g, 1, r, c)[0] for r, c in ((DENSE_INTER, hidden), (DENSE_INTER, hidden), (hidden, DENSE_INTER))]
    norms = [(1.0 + 0.1 * torch.randn(hidden, generator=g, device="cuda")).cpu().numpy() for _ in range(5)]
    return synth.FfnBlock(DENSE_INTER, *w, *norms, layer_scalar=0.8125)


def _stack(case):
    geometry = tuple(case[k] for k in ("hidden", "inter", "experts", "topk"))
    q4 = case["format"] == "q4"

    def make():
        st = stack_mod.MoeStack(Q4_TOKENS if q4 else FP4_TOKENS, *geometry)
        for i in range(Q4_LAYERS if q4 else FP4_LAYERS):
            if q4:
                st.add_layer(_q4_layer(i, *geometry))
            else:
                st.add_nvfp4_layer(_fp4_layer(i, *geometry))
        if q4:
            _check(st.attach_ffn_block(0, _dense_block(geometry[0])))
        return st
    return _once(("stack", case["format"]) + geometry, make)


# ---- the operator surface with host pointers ---------------------------------------------------------------------
def _check(rc):
    if rc != 0:
        raise RuntimeError("the library refused a call of this case")


def _gpu():
    def make():
        g = backend.SaltGpu()
        _check(g.init())
        return g
    return _once("gpu", make)


def _next_id():
    _kept["ids"] = _kept.get("ids", 100) + 1
    return _kept["ids"]


def _projection(rows, cols):
    """One dense affine-Q4 projection in a trunk resource: (values, scales, biases)."""
    def make():
        buf = _q4_tensors(_gen(rows * 31 + cols), 1, rows, cols)[0]
        _check(_gpu().weight_resource_bind(backend.RESOURCE_TRUNK, _next_id(), buf))
        vb, gb = synth.q4_tensor_bytes(rows, cols)
        return buf[:vb].view(np.uint32), buf[vb:vb + gb].view(np.uint16), buf[vb + gb:].view(np.uint16)
    return _once(("projection", rows, cols), make)


def _fp4_projection(rows, cols):
    """One NVFP4 projection registered under a key."""
    def make():
        tensors, divisors = _fp4_tensors(_gen(rows * 37 + cols), 1, rows, cols)
        buf = np.concatenate((tensors[0], np.array([divisors[0], 64.0], np.float32).view(np.uint8)))
        codes, scales = buf[:rows * cols // 2], buf[rows * cols // 2:-8]
        rid, key = _next_id(), 0x4000000 + _next_id()
        g = _gpu()
        _check(g.weight_resource_bind(backend.RESOURCE_EXPERT_LAYER, rid, buf))
        _check(g.nvfp4_resource_slot(backend.RESOURCE_EXPERT_LAYER, rid, key, codes, scales, buf[-8:-4], buf[-4:], rows,
                                     cols))
        return key, buf
    return _once(("fp4", rows, cols), make)


def _experts(case):
    """The experts of one layer in an expert resource, as descriptors of the chain call (by expert)."""
    geometry = tuple(case[k] for k in ("hidden", "inter", "experts", "topk"))

    def make():
        layer, g, base = _q4_layer(50, *geometry), _gpu(), 0x8000000 + 0x10000 * _next_id()
        rid = _next_id()
        _check(g.expert_resource_bind(rid, layer.pool))
        found = []
        for e in range(layer.n_experts):
            fields = []
            for which in range(3):
                t = layer.tensor(e, which)
                r, c = (layer.inter, layer.hidden) if which < 2 else (layer.hidden, layer.inter)
                _check(g.expert_resource_slot(rid, base + 3 * e + which, *t, r, c))
                fields += [a.ctypes.data for a in t] + [base + 3 * e + which]
            found.append(fields)
        return layer, found
    return _once(("experts",) + geometry, make)


# ---- the cases -----------------------------------------------------------------------------------------------------
def _tokens(seed, batch, hidden):
    """Hidden states: independent N(0, 1) entries plus a component that all tokens share, which makes some experts
    more popular than others, as they are in a trained model."""
    g = _gen(seed)
    return torch.randn(batch, hidden, generator=g, device="cuda") + \
        0.5 * torch.randn(1, hidden, generator=g, device="cuda")


def prepare(case, seed):
    op = case["op"]
    if op == "matvec":
        x = _tokens(seed, 1, case["cols"])[0].cpu().numpy()
        return dict(case, gpu=_gpu(), weights=_projection(case["rows"], case["cols"]), x=x,
                    y=np.zeros(case["rows"], np.float32))
    if op == "fp4_batch":
        x = _tokens(seed, case["batch"], case["cols"]).cpu().numpy()
        return dict(case, gpu=_gpu(), key=_fp4_projection(case["rows"], case["cols"])[0], x=x,
                    y=np.zeros((case["batch"], case["rows"]), np.float32))
    if op == "chain":
        _, found = _experts(case)
        chosen = np.random.default_rng(seed).choice(len(found), case["count"], replace=False)
        x = _tokens(seed, case["count"] * case["group"], case["hidden"]).cpu().numpy()
        return dict(case, gpu=_gpu(), x=x, y=np.zeros_like(x),
                    chosen=[backend.MoeExpert(*found[e], case["group"], -1, 0) for e in sorted(chosen)])
    st = _stack(case)
    x = _tokens(seed, case["batch"], case["hidden"])
    if op == "decode_host":
        return dict(case, stack=st, x=x.cpu().numpy())
    return dict(case, stack=st, x=x, y=torch.zeros_like(x))


def run(s):
    op = s["op"]
    if op == "matvec":
        _check(s["gpu"].q4_matvec(*s["weights"], s["rows"], s["cols"], s["x"], s["y"]))
        return s["y"]
    if op == "fp4_batch":
        _check(s["gpu"].nvfp4_matvec_batch(s["key"], s["rows"], s["cols"], s["x"], s["y"]))
        return s["y"]
    if op == "chain":
        _check(s["gpu"].q4_moe_chain(s["chosen"], s["hidden"], s["inter"], s["x"], s["y"]))
        return s["y"]
    st = s["stack"]
    if op == "decode_host":
        return st.forward_host(s["x"], count=s["layers"])
    x, y, stream = s["x"].data_ptr(), s["y"].data_ptr(), torch.cuda.current_stream().cuda_stream
    if op == "decode":
        _check(st.forward_device(x, s["batch"], y, count=s["layers"], stream=stream))
    elif op == "block":
        _check(st.ffn_block_forward(0, x, s["batch"], y, stream=stream))
    else:
        _check(st.layer_experts(0, x, s["batch"], tensor_core=s["precision"], stream=stream))
        _check(st.layer_combine(0, s["batch"], y, apply_norm=True, stream=stream))
    return s["y"]


def work(case):
    """Bytes: the weights of every expert that gets a token (the expected number under even routing), the router and
    the activations, each once.  Operations: two per weight and token that meets it."""
    op = case["op"]          # both formats take 0.5625 bytes per weight: four bits and a share of the group's scales
    if op in ("matvec", "fp4_batch"):
        r, c, b = case["rows"], case["cols"], case.get("batch", 1)
        return {"bytes": r * c * 0.5625 + 4 * b * (r + c), "flops": 2 * r * c * b}
    h, m = case["hidden"], case["inter"]
    expert = 3 * h * m
    if op == "chain":
        n = case["count"] * case["group"]
        return {"bytes": case["count"] * expert * 0.5625 + 8 * n * h, "flops": 2 * n * expert}
    b, e, k = case["batch"], case["experts"], case["topk"]
    used = e * (1 - (1 - k / e) ** b)
    nbytes = used * expert * 0.5625 + 4 * e * h
    flops = 2 * b * (k * expert + e * h)
    if op == "block":
        nbytes += 3 * h * DENSE_INTER * 0.5625
        flops += 2 * b * 3 * h * DENSE_INTER
    return {"bytes": case["layers"] * nbytes + 8 * b * h, "flops": case["layers"] * flops}


def tolerance(case):
    """Everything is bit-exact except the tensor-core projections."""
    if case["op"] != "prefill":
        return "exact"
    if case["format"] == "nvfp4":
        # the quantiser between the two projections is discontinuous: a last-bit difference can move a code of about
        # one row in a few hundred, and such a row is off by its quantisation noise
        return {"rel": 5e-3, "max": 0.3}
    # fp16 operands carried as two halves: about 22 bits; rounded once: 11 bits in two projections in a row
    return {"rel": 2e-5, "max": 1e-3} if case["precision"] == "split" else {"rel": 2e-3, "max": 2e-2}
