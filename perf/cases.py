"""Timing cases of the MoE block: what a program that uses this library has it do.

A case names an entry point and sizes; `listed()` holds the fixed ones, `draw()`
more of the same ranges.  Layer shapes are the full-size layer of
synth.QWEN_CFG (hidden 2048, 256 experts, top-8, expert width 512, one shared
expert); weights, activations and the Zipf router bias have the distributions of
synth.py.

  stack  decode step of a server over a few chained layers: the first layer reads
         the step's token rows, the rest run in place on the residual stream
         (apus_cuda_moe_layer_dev, apus_cuda_moe_stack_dev)
  block  one block on device pointers (apus_cuda_moe_block_dev): prefill
  layer  the block with its norm and residual add (apus_cuda_moe_layer_dev)
  host   the block on host pointers, as the engine calls it (apus_cuda_moe_block)
  head   the output head as a device-pointer weight stream (apus_cuda_bf16_gemv_dev)
  hook   the engine's dense products on host pointers, bit-exact
         (apus_cuda_bf16_gemv for one row, apus_cuda_bf16_gemm for several)
"""
import ctypes as C
import importlib.util
import math
import os
import sys

import numpy as np
import torch

VOCAB = 248320          # rows of the output head
ZIPF_BETA = 0.27        # hottest expert about ten times the mean load


def listed():
    return [
        # one sequence generating: every layer waits for the one before
        {"name": "decode_t1", "op": "stack", "T": 1, "layers": 4},
        # a draft of three tokens verified at once
        {"name": "decode_t3", "op": "stack", "T": 3, "layers": 4},
        # a few sequences generating together
        {"name": "decode_t8", "op": "stack", "T": 8, "layers": 4},
        # a full decode batch, with the odd count that finished sequences leave
        {"name": "decode_t61", "op": "stack", "T": 61, "layers": 4},
        # a prompt of ordinary length (the T = 512 configuration of bench.py)
        {"name": "prefill_t512", "op": "block", "T": 512, "zipf": False},
        # a prefill chunk that ends where the prompt ends
        {"name": "prefill_t1999", "op": "layer", "T": 1999, "zipf": False},
        # the largest prefill, routed unevenly (bench.py's headline workload)
        {"name": "prefill_t8192_zipf", "op": "block", "T": 8192, "zipf": True},
        # the engine generating, block on its own malloc'd buffers
        {"name": "host_t1", "op": "host", "T": 1, "zipf": False, "pinned": False},
        # the engine's largest prefill from pinned buffers
        {"name": "host_t8192_zipf", "op": "host", "T": 8192, "zipf": True, "pinned": True},
        # the output head of a generating sequence on a server
        {"name": "head_m1", "op": "head", "M": 1, "O": VOCAB, "K": 2048},
        # the same product as the engine calls it, in its own summation order
        {"name": "hook_head", "op": "hook", "M": 1, "O": VOCAB, "K": 2048},
        # one of the engine's dense products over a prompt
        {"name": "hook_gemm_m512", "op": "hook", "M": 512, "O": 1024, "K": 2048},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(["stack", "stack", "block", "layer", "host", "head", "hook"])
    if op == "stack":
        return {"op": op, "T": _log_int(rng, 1, 64), "layers": rng.randint(2, 4)}
    if op in ("block", "layer"):
        return {"op": op, "T": _log_int(rng, 65, 8192), "zipf": rng.random() < 0.5}
    if op == "host":
        return {"op": op, "T": _log_int(rng, 1, 8192), "zipf": rng.random() < 0.5,
                "pinned": rng.random() < 0.5}
    if op == "head":
        return {"op": op, "M": rng.randint(1, 8), "O": _log_int(rng, 32768, VOCAB), "K": 2048}
    return {"op": op, "M": _log_int(rng, 1, 512), "O": _log_int(rng, 256, 4096),
            "K": rng.choice([512, 2048])}


# ---- the library ------------------------------------------------------------------

_lib = {}


def _backend():
    """(backend, synth module), loaded by path: the package directory's name is
    not an identifier."""
    if not _lib:
        root = os.path.join(os.getcwd(), "apus-qwen3.6-35b-a3b_b200")
        spec = importlib.util.spec_from_file_location(
            "apus_b200", os.path.join(root, "__init__.py"), submodule_search_locations=[root])
        pkg = importlib.util.module_from_spec(spec)
        sys.modules["apus_b200"] = pkg
        spec.loader.exec_module(pkg)
        import apus_b200.synth as synth
        torch.cuda.init()
        be = pkg.Backend()
        be.enable()
        _lib.update(be=be, synth=synth, pkg=pkg)
    return _lib["be"], _lib["synth"]


def _stream():
    return torch.cuda.current_stream().cuda_stream


class _Layer:
    """One resident layer with seeded weights; given back with the object."""

    def __init__(self, cfg, seed, index, zipf):
        be, synth = _backend()
        self.handle = be.layer_create(cfg)
        synth.device_weights(be, self.handle, cfg, seed=seed, layer=index, stream=_stream())
        if zipf:
            be.layer_upload(self.handle, "rtr_w", _zipf_router(cfg, seed, index))

    def __del__(self):
        _lib["be"].layer_destroy(self.handle)


def _zipf_router(cfg, seed, index):
    """The router matrix with the bias in the column of the constant-1 channel."""
    be, synth = _backend()
    E, H = cfg["experts"], cfg["hidden"]
    rtr = be.synth_fill_host(E * H, seed, index, synth.T_RTR, synth.W_SIGMA).reshape(E, H)
    bias = synth.zipf_bias(cfg, seed=seed, s=1.1, beta=ZIPF_BETA)
    rtr[:, -1] = synth.f32_to_bf16(np.asarray(bias, np.float32))
    return rtr


def _filled(shape, seed, index, tensor, sigma):
    """A device tensor of the approximately normal stream, BF16."""
    be, _ = _backend()
    t = torch.empty(shape, dtype=torch.bfloat16, device="cuda")
    be.synth_fill_dev(t.data_ptr(), t.numel(), seed, index, tensor, sigma, stream=_stream())
    return t


def _rows(T, H, seed, zipf):
    """Block inputs: rows of unit RMS, the last channel 1 where the bias rides on it."""
    _, synth = _backend()
    v = _filled((T, H), seed, 0, synth.T_X, 1.0).float()
    x = (v * torch.rsqrt(v.square().mean(dim=1, keepdim=True) + 1e-6)).bfloat16()
    if zipf:
        x[:, -1] = 1.0
    return x


# The engine's weights live as long as its process and are known to the library
# by their host addresses, so they are made once here too.
_host = {}


def _host_layer(cfg, zipf):
    be, synth = _backend()
    if "layer" not in _host:
        _host["layer"] = {
            name: _filled(shape, 1, 0, tid, synth.W_SIGMA).cpu().view(torch.int16).numpy()
            .view(np.uint16) for name, (tid, shape) in synth.weight_shapes(cfg).items()}
    if zipf and "zipf" not in _host:
        _host["zipf"] = dict(_host["layer"], rtr_w=_zipf_router(cfg, 1, 0))
    return _host["zipf" if zipf else "layer"]


def _host_matrix(O, K):
    if (O, K) not in _host:
        _, synth = _backend()
        _host[O, K] = _filled((O, K), 1, 0, synth.T_GU, synth.W_SIGMA).cpu()
    return _host[O, K]


def _u16p(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_uint16))


# ---- cases ------------------------------------------------------------------------


def prepare(case, seed):
    be, synth = _backend()
    cfg = synth.QWEN_CFG
    H = cfg["hidden"]
    s = {"case": case, "be": be}
    op = case["op"]
    if op in ("stack", "block", "layer"):
        T = case["T"]
        s["layers"] = [_Layer(cfg, seed, i, case.get("zipf", False))
                       for i in range(case.get("layers", 1))]
        s["handles"] = [layer.handle for layer in s["layers"]]
        s["x"] = _rows(T, H, seed, case.get("zipf", False))
        s["out"] = torch.empty_like(s["x"])
        s["gain"] = [_filled((H,), seed, i, synth.T_BIAS, 0.1) for i in range(len(s["layers"]))]
        s["gain_ptr"] = [g.data_ptr() for g in s["gain"]]
        be.reserve(cfg, T)
    elif op == "host":
        T = case["T"]
        W = _host_layer(cfg, case["zipf"])
        backend = _lib["pkg"].backend
        s["cfg"] = backend.MoeCfg.from_dict(cfg)
        s["w"] = backend.MoeW(*[W[k].ctypes.data for k in
                                ("rtr_w", "exp_gu", "exp_d", "sh_g", "sh_u", "sh_d", "sh_gate")])
        x = _rows(T, H, seed, case["zipf"]).cpu()
        s["x"] = x.pin_memory() if case["pinned"] else x
        s["out"] = torch.zeros_like(x)
        if case["pinned"]:
            s["out"] = s["out"].pin_memory()
        run(s)                  # the layer is resident from a program's first call on
    elif op == "head":
        M, O, K = case["M"], case["O"], case["K"]
        s["w"] = _filled((O, K), seed, 0, synth.T_GU, synth.W_SIGMA)
        s["x"] = _rows(M, K, seed, False)
        s["out"] = torch.empty((M, O), dtype=torch.bfloat16, device="cuda")
    else:
        M, O, K = case["M"], case["O"], case["K"]
        s["w"] = _host_matrix(O, K)
        s["x"] = _rows(M, K, seed, False).cpu()
        s["out"] = torch.zeros((M, O), dtype=torch.bfloat16)
        run(s)                  # likewise the matrix
    torch.cuda.synchronize()
    return s


def _ok(be, rc):
    if rc:
        raise RuntimeError(be.last_error())


def run(s):
    case, be = s["case"], s["be"]
    op = case["op"]
    if op == "stack":
        T, st = case["T"], _stream()
        be.moe_layer_dev(s["handles"][0], s["x"].data_ptr(), s["gain_ptr"][0],
                         s["out"].data_ptr(), T, stream=st)
        be.moe_stack_dev(s["handles"][1:], s["out"].data_ptr(), T, d_ln_w=s["gain_ptr"][1:],
                         stream=st)
    elif op == "block":
        be.moe_block_dev(s["handles"][0], s["x"].data_ptr(), s["out"].data_ptr(), case["T"],
                         stream=_stream())
    elif op == "layer":
        be.moe_layer_dev(s["handles"][0], s["x"].data_ptr(), s["gain_ptr"][0],
                         s["out"].data_ptr(), case["T"], stream=_stream())
    elif op == "host":
        _ok(be, be.lib.apus_cuda_moe_block(C.byref(s["cfg"]), C.byref(s["w"]), _u16p(s["x"]),
                                           _u16p(s["out"]), case["T"], None))
    elif op == "head":
        be.bf16_gemv_dev(s["w"].data_ptr(), s["x"].data_ptr(), s["out"].data_ptr(), case["M"],
                         case["O"], case["K"], stream=_stream())
    elif case["M"] == 1:
        _ok(be, be.lib.apus_cuda_bf16_gemv(_u16p(s["w"]), _u16p(s["x"]), _u16p(s["out"]),
                                           case["O"], case["K"]))
    else:
        _ok(be, be.lib.apus_cuda_bf16_gemm(_u16p(s["w"]), _u16p(s["x"]), _u16p(s["out"]),
                                           case["M"], case["O"], case["K"]))
    return s["out"]


def work(case):
    if case["op"] in ("head", "hook"):
        M, O, K = case["M"], case["O"], case["K"]
        return {"bytes": 2 * (O * K + M * K + M * O), "flops": 2 * M * O * K}
    H, E, I, TK = 2048, 256, 512, 8
    T, n = case["T"], case.get("layers", 1)
    # experts that at least one token picks, for an even router
    touched = E * (1.0 - (1.0 - TK / E) ** T)
    weights = 2 * (E * H + H + (touched + 1) * 3 * I * H)
    return {"bytes": n * (weights + 2 * T * H * 2),
            "flops": n * 2 * T * (E * H + H + (TK + 1) * 3 * I * H)}


def tolerance(case):
    if case["op"] == "hook":
        return "exact"
    # BF16 results of fp32 sums in any order.  In a chain of layers a last-bit
    # difference in one layer's output can turn a near-tie of the next router,
    # which moves a token by the difference of two experts' lightest shares
    # (about 0.02 of the residual row).
    return {"rel": 2e-2 if case["op"] == "stack" else 1e-2}
