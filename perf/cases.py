"""Performance cases of the quantised-matmul path: what a program that serves or prefills a quantised network has it do, through the
torch-tensor entry points (`torch_api.npu_quant_matmul`, `torch_api.npu_weight_quant_batchmatmul`) and `aclnn.dynamic_mx_quant`.

A case is a plain dict. `kind` says which operator it runs:

  wq     16-bit activations x int4 / int8 / e4m3 weight, per-group or per-channel antiquant scales (A16W4, A16W8, A16F8)
  token  int8 x int8 or e4m3 x e4m3, per-token x per-channel scales (A8W8)
  block  e4m3 x e4m3, scales per 1 x 128 block of the activations and per 128 x 128 block of the weight
  mx     MXFP8 or MXFP4 with e8m0 scales per 32 elements of k, batched; `dynamic` activations start as bf16 and are quantised in the call
  quant  the dynamic MX quantiser alone

`stored` is the weight's order in memory: "kn", or "nk" (an (n, k) tensor handed over as its transposed view, the usual torch layout).
m is the number of tokens: one to a few dozen while decoding, hundreds to thousands for a prompt.
"""
import importlib.util
import math
import os
import sys

import torch

DEV = "cuda:0"
GROUP_MX = (1 << 32) | (1 << 16) | 32
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def _package():
    if "ops_nn_b200" not in sys.modules:
        folder = os.path.join(os.getcwd(), "ops-nn_b200")
        spec = importlib.util.spec_from_file_location("ops_nn_b200", os.path.join(folder, "__init__.py"), submodule_search_locations=[folder])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["ops_nn_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["ops_nn_b200"]


def _wq(m, k, n, weight, act="bf16", group=128, offset=False, bias=False, stored="kn"):
    return {"kind": "wq", "m": m, "k": k, "n": n, "weight": weight, "act": act, "group": group, "offset": offset, "bias": bias, "stored": stored}


def _token(m, k, n, dtype, out="bf16", bias=True, stored="nk"):
    return {"kind": "token", "m": m, "k": k, "n": n, "dtype": dtype, "out": out, "bias": bias, "stored": stored}


def _block(m, k, n, out="bf16", stored="kn"):
    return {"kind": "block", "m": m, "k": k, "n": n, "out": out, "stored": stored}


def _mx(batch, m, k, n, dtype, dynamic, bias=False, stored="nk"):
    return {"kind": "mx", "batch": batch, "m": m, "k": k, "n": n, "dtype": dtype, "dynamic": dynamic, "bias": bias, "stored": stored}


def _quant(m, k, dtype):
    return {"kind": "quant", "m": m, "k": k, "dtype": dtype}


def listed():
    return [
        # one user's next token through a small projection: the smallest call there is, all latency
        dict(_wq(1, 4096, 4096, "int4", offset=True), name="w4 one token"),
        # a decoding step of sixteen users through a wide layer: the headline configuration
        dict(_wq(16, 8192, 28672, "int4", offset=True), name="w4 decode"),
        # an odd number of users in one step (continuous batching), symmetric fp16 weight in torch's own (n, k) order
        dict(_wq(77, 7168, 18432, "int4", act="fp16", stored="nk"), name="w4 many users"),
        # the prompt that precedes the decoding of the headline weight
        dict(_wq(2048, 8192, 28672, "int4", offset=True), name="w4 prompt"),
        # a few users against an 8-bit per-channel weight with bias
        dict(_wq(4, 4096, 14336, "int8", act="fp16", group=0, bias=True, stored="nk"), name="w8 decode"),
        # 8-bit activations and weight, a short prompt through a square layer
        dict(_token(128, 4096, 4096, "int8", stored="kn"), name="int8 short prompt"),
        # the same operator at its largest: a long prompt through a feed-forward layer
        dict(_token(4096, 7168, 18432, "int8", stored="kn"), name="int8 long prompt"),
        # a ragged prompt against one rank's share of a layer (n cut eight ways, no power of two left in it)
        dict(_token(717, 7168, 2304, "fp8", out="fp16", bias=False), name="fp8 ragged prompt"),
        # fp8 with block scales: a decoding step and a long prompt of the same layer
        dict(_block(24, 7168, 18432, stored="nk"), name="fp8 block decode"),
        dict(_block(4096, 7168, 18432), name="fp8 block prompt"),
        # MXFP4 on both sides, activations quantised by the layer before
        dict(_mx(8, 8192, 8192, 8192, "fp4", False), name="mxfp4 batch"),
        # MXFP8 with the activations quantised on the way in: the largest case
        dict(_mx(32, 2048, 4096, 14336, "fp8", True, bias=True, stored="kn"), name="mxfp8 dynamic"),
    ]


def draw(rng):
    def spread(lo, hi, step=1):
        return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step) * step))

    def layer(kstep, nstep):
        while True:
            k, n = spread(1024, 16384, kstep), spread(1024, 32768, nstep)
            if k * n <= 8192 * 28672:
                return k, n

    stored, out = rng.choice(["kn", "nk"]), rng.choice(["bf16", "bf16", "fp16"])
    kind = rng.choice(["wq", "wq", "token", "block", "mx", "quant"])
    if kind == "wq":
        weight = rng.choice(["int4", "int4", "int8", "fp8"])
        k, n = layer(128, 32)
        group = rng.choice([128, 128, 0] if weight == "int4" else [0, 0, 128])
        offset = weight != "fp8" and rng.random() < (0.5 if weight == "int4" else 0.2)
        m = spread(1, 32) if rng.random() < 0.5 else spread(1, 2048)
        return _wq(m, k, n, weight, out, group, offset, rng.random() < 0.25, stored)
    if kind == "token":
        k, n = layer(64, 16)
        return _token(spread(1, 4096), k, n, rng.choice(["int8", "fp8"]), out, rng.random() < 0.5, stored)
    if kind == "block":
        k, n = layer(128, 64)
        return _block(spread(1, 4096), k, n, out, stored)
    if kind == "mx":
        k, n = layer(64, 32)
        m = spread(1, 4096)
        most = min(32, int(5e12 / (2.0 * m * k * n)), (1 << 30) // (k * n))
        return _mx(spread(1, max(1, most)), m, k, n, rng.choice(["fp8", "fp4"]), rng.random() < 0.5, rng.random() < 0.5, stored)
    return _quant(spread(1, 65536), spread(1024, 16384, 32), rng.choice(["fp8", "fp4"]))


# ---- inputs ---------------------------------------------------------------------------------------------------------


def _mx_quantised(src, dtype, axis):
    """(payload bytes, e8m0 scale bytes) of a bf16 tensor, blocks of 32 along `axis` (-1 or -2)."""
    aclnn = _package().aclnn
    shape = list(src.shape)
    groups = -(-shape[axis] // 64)
    sshape = shape[:-1] + [groups, 2] if axis == -1 else shape[:-2] + [groups, shape[-1], 2]
    name = "float4_e2m1" if dtype == "fp4" else "float8_e4m3fn"
    q = torch.empty(shape[:-1] + [shape[-1] // 2 if dtype == "fp4" else shape[-1]], dtype=torch.uint8, device=src.device)
    s = torch.empty(sshape, dtype=torch.uint8, device=src.device)
    aclnn.dynamic_mx_quant(aclnn.from_torch(src), aclnn.from_torch(q, name, shape), aclnn.from_torch(s, "float8_e8m0"), name, axis=axis)
    return q, s


class _PreparedMx:
    """An MX weight that the program keeps, laid out once for the calls to come."""

    def __init__(self, w, scale, dtype, m):
        self.aclnn = _package().aclnn
        if dtype == "fp4":
            shape = list(w.shape)
            if w.stride(-1) == 1:
                shape[-1] *= 2
                strides = [2 * s for s in w.stride()[:-1]] + [1]
            else:
                shape[-2] *= 2
                strides = [2 * s for s in w.stride()[:-2]] + [1, 2 * w.stride(-1)]
            self.desc = self.aclnn.from_torch(w, "float4_e2m1", shape, strides)
        else:
            self.desc = self.aclnn.from_torch(w, "float8_e4m3fn")
        self.w, self.scale = w, scale
        self.storage = self.aclnn.prepare_x2(self.desc, self.aclnn.from_torch(scale, "float8_e8m0"), False, GROUP_MX, m_hint=m)

    def __del__(self):
        self.aclnn.release_x2(self.desc)


def _rand_e4m3(gen, shape):
    """What values of a normal distribution become once their largest has been scaled to e4m3's 448."""
    return torch.randn(shape, generator=gen, device=DEV).mul_(100).clamp_(-448, 448).to(torch.float8_e4m3fn)


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)

    def uniform(shape, lo, hi, dtype=torch.float32):
        return torch.empty(shape, device=DEV, dtype=torch.float32).uniform_(lo, hi, generator=gen).to(dtype)

    def ints(shape, lo, hi, dtype):
        return torch.randint(lo, hi, shape, generator=gen, device=DEV, dtype=dtype)

    kind, m, k = case["kind"], case["m"], case["k"]
    if kind == "quant":
        x = torch.randn((m, k), generator=gen, device=DEV, dtype=torch.bfloat16)
        x.view(-1)[ints((max(1, m * k // 1000),), 0, m * k, torch.int64)] *= 50
        return {"kind": kind, "x": x, "dtype": case["dtype"]}
    n, nk = case["n"], case["stored"] == "nk"
    wshape = (n, k) if nk else (k, n)
    if kind == "wq":
        act = DTYPES[case["act"]]
        x = torch.randn((m, k), generator=gen, device=DEV, dtype=act)
        if case["weight"] == "int4":  # eight values in a 32-bit word along the stored inner axis
            w = ints((wshape[0], wshape[1] // 8), -2**31, 2**31, torch.int32)
            scale = (0.005, 0.02)
        elif case["weight"] == "int8":
            w = ints(wshape, -127, 128, torch.int8)
            scale = (0.0003, 0.0012)
        else:
            w = _rand_e4m3(gen, wshape)
            scale = (0.0001, 0.0004)
        groups = k // case["group"] if case["group"] else 1
        sshape = (n, groups) if nk else (groups, n)
        scale = uniform(sshape, *scale, dtype=act)
        offset = uniform(sshape, -1, 1, dtype=act) if case["offset"] else None
        if nk:
            w, scale, offset = w.t(), scale.t(), None if offset is None else offset.t()
        if not case["group"]:
            scale, offset = scale.reshape(-1), None if offset is None else offset.reshape(-1)
        bias = uniform((n,), -1, 1, dtype=act) if case["bias"] else None
        return {"kind": kind, "x": x, "w": w, "scale": scale, "offset": offset, "bias": bias, "group": case["group"]}
    if kind == "token":
        if case["dtype"] == "int8":
            x, w = ints((m, k), -127, 128, torch.int8), ints(wshape, -127, 128, torch.int8)
            bias = ints((n,), -1000, 1001, torch.int32) if case["bias"] else None
        else:
            x, w = _rand_e4m3(gen, (m, k)), _rand_e4m3(gen, wshape)
            bias = uniform((n,), -1, 1) if case["bias"] else None
        return {"kind": kind, "x": x, "w": w.t() if nk else w, "s1": uniform((m,), 1e-3, 1e-2), "s2": uniform((n,), 1e-3, 1e-2), "bias": bias,
                "out": DTYPES[case["out"]]}
    if kind == "block":
        kb, nb = -(-k // 128), -(-n // 128)
        w, s2 = _rand_e4m3(gen, wshape), uniform((nb, kb) if nk else (kb, nb), 1e-4, 4e-4)  # the scale lies as the weight does
        return {"kind": kind, "x": _rand_e4m3(gen, (m, k)), "w": w.t() if nk else w, "s1": uniform((m, kb), 5e-3, 2e-2), "s2": s2,
                "out": DTYPES[case["out"]]}
    b, f4 = case["batch"], case["dtype"] == "fp4"
    act = torch.randn((b, m, k), generator=gen, device=DEV, dtype=torch.bfloat16)
    act.view(-1)[ints((max(1, act.numel() // 1000),), 0, act.numel(), torch.int64)] *= 50
    parts = [_mx_quantised(torch.randn(wshape, generator=gen, device=DEV, dtype=torch.bfloat16) * 0.02, case["dtype"], -1 if nk else -2) for _ in range(b)]
    w, ws = torch.stack([p[0] for p in parts]), torch.stack([p[1] for p in parts])
    del parts
    if not f4:
        w = w.view(torch.float8_e4m3fn)
    if nk:
        w = w.transpose(1, 2)
    x, xs = (act, None) if case["dynamic"] else _mx_quantised(act, case["dtype"], -1)
    if not f4 and not case["dynamic"]:
        x = x.view(torch.float8_e4m3fn)
    fp4 = "float4_e2m1" if f4 else None
    return {"kind": kind, "x": x, "xs": xs, "weight": _PreparedMx(w, ws, case["dtype"], m), "bias": uniform((n,), -1, 1) if case["bias"] else None,
            "x_dtype": None if case["dynamic"] else fp4, "w_dtype": fp4}


# ---- one pass -------------------------------------------------------------------------------------------------------


def run(state):
    pkg, kind = _package(), state["kind"]
    if kind == "wq":
        return pkg.torch_api.npu_weight_quant_batchmatmul(state["x"], state["w"], state["scale"], state["offset"], bias=state["bias"],
                                                          antiquant_group_size=state["group"])
    if kind == "token":
        return pkg.torch_api.npu_quant_matmul(state["x"], state["w"], state["s2"], pertoken_scale=state["s1"], bias=state["bias"], output_dtype=state["out"])
    if kind == "block":
        return pkg.torch_api.npu_quant_matmul(state["x"], state["w"], state["s2"], pertoken_scale=state["s1"], output_dtype=state["out"],
                                              group_sizes=[1, 128, 128])
    if kind == "mx":
        weight = state["weight"]
        return pkg.torch_api.npu_quant_matmul(state["x"], weight.w, weight.scale, pertoken_scale=state["xs"], bias=state["bias"],
                                              output_dtype=torch.bfloat16, group_sizes=[1, 1, 32], x1_dtype=state["x_dtype"], x2_dtype=state["w_dtype"],
                                              scale_dtype="float8_e8m0", pertoken_scale_dtype="float8_e8m0")
    return _mx_quantised(state["x"], state["dtype"], -1)


# ---- what a pass cannot do without ----------------------------------------------------------------------------------


def work(case):
    kind, m, k = case["kind"], case["m"], case["k"]
    if kind == "quant":
        return {"bytes": m * k * (2 + (1 if case["dtype"] == "fp8" else 0.5) + 1 / 32), "flops": 0}
    n, b = case["n"], case.get("batch", 1)
    if kind == "wq":
        groups = k // case["group"] if case["group"] else 1
        scales = 2 * groups * n * (2 if case["offset"] else 1)
        total = m * k * 2 + k * n * (0.5 if case["weight"] == "int4" else 1) + scales + m * n * 2 + (2 * n if case["bias"] else 0)
    elif kind == "token":
        total = m * k + k * n + 4 * (m + n) + m * n * 2 + (4 * n if case["bias"] else 0)
    elif kind == "block":
        total = m * k + k * n + 4 * (m * -(-k // 128) + -(-n // 128) * -(-k // 128)) + m * n * 2
    else:
        size = (1 if case["dtype"] == "fp8" else 0.5) + 1 / 32
        total = b * (m * k * (2 if case["dynamic"] else size) + k * n * size + m * n * 2) + (4 * n if case["bias"] else 0)
    return {"bytes": total, "flops": 2.0 * b * m * n * k}


def tolerance(case):
    """Sums are kept in 32 bits and rounded once to the output type (int8 products exactly until then): another order of the sum moves
    a value by at most one unit in its last place, 2^-8 (bf16) or 2^-11 (fp16), and most values by nothing. The quantiser's bytes
    are fully specified."""
    if case["kind"] == "quant":
        return "exact"
    out = case.get("act") or case.get("out") or "bf16"
    return {"rel": 4e-3 if out == "bf16" else 1e-3}
