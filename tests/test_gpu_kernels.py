"""GPU parity tests, kernel level, all through the C-ABI: the per-matmul
hooks, the router and the dispatch against the CPU checker.  Integer and
index results are compared bit for bit."""
import os

import numpy as np
import pytest

from test_oracle_cpu import rd, manifest, f32, tol_ok, rng_codes

pytestmark = pytest.mark.gpu


# ---- per-matmul hooks: bitwise the CPU anchor (tests/m10/test_kernels.c) ----

@pytest.mark.parametrize("O,K", [(1, 1), (3, 5), (7, 1), (33, 100), (64, 256),
                                 (256, 2048), (1024, 2048), (2048, 512),
                                 (512, 2048), (1, 2048)])
def test_hook_gemv_matvec_bitwise(gpu, orc, O, K):
    rng = np.random.default_rng(O * 131 + K)
    w, x = rng_codes(rng, (O, K), 0.5), rng_codes(rng, K, 1.0)
    assert np.array_equal(gpu.bf16_gemv(w, x), orc.gemv(w, x))
    assert np.array_equal(gpu.bf16_matvec_f32(w, x), orc.matvec_f32(w, x))


@pytest.mark.parametrize("M", [1, 2, 3, 5, 64, 300])
def test_hook_gemm_bitwise(gpu, orc, M):
    rng = np.random.default_rng(M)
    O, K = 96, 200
    w, x = rng_codes(rng, (O, K), 0.5), rng_codes(rng, (M, K), 1.0)
    assert np.array_equal(gpu.bf16_gemm(w, x), orc.gemm(w, x))


@pytest.mark.parametrize("M,O,K", [
    (1, 31, 8), (1, 33, 64), (2, 32, 72), (3, 5000, 136), (4, 95, 2048),   # rows per lane
    (5, 64, 8), (16, 65, 40), (17, 63, 96), (9, 130, 2048),                # 2-row tiles
    (50, 2300, 72), (51, 4000, 136), (300, 1000, 104),                     # 16-row tiles
    (129, 2560, 512), (513, 1500, 520)])                                   # the same, in parts
@pytest.mark.parametrize("scale", ["plain", "underflow", "overflow"])
def test_hook_exact_order_kernels(gpu, orc, M, O, K, scale):
    """Each kernel of the exact-order product at the edges of its tiles, with
    products that are exact in fp32 (fused chain) and with products that
    underflow or overflow (literal chain): bit for bit the anchor."""
    rng = np.random.default_rng(M * 131 + O * 7 + K)
    f = {"plain": 1.0, "underflow": 1e-20, "overflow": 1e19}[scale]
    w, x = rng_codes(rng, (O, K), 0.5 * f), rng_codes(rng, (M, K), f)
    exp = orc.gemm(w, x)
    got = gpu.bf16_gemm(w, x)
    nan = np.isnan(f32(exp))
    assert np.array_equal(np.isnan(f32(got)), nan)
    assert np.array_equal(got[~nan], exp[~nan])
    if M == 1:
        assert np.array_equal(gpu.bf16_gemv(w, x[0])[~nan[0]], exp[0][~nan[0]])
        assert np.array_equal(gpu.bf16_matvec_f32(w, x[0]), orc.matvec_f32(w, x[0]),
                              equal_nan=True)


@pytest.mark.parametrize("M,O,K", [
    (5, 127, 64), (7, 129, 136), (8, 4736, 64),        # tiles of 2 x 128
    (65, 640, 200), (97, 481, 64), (9, 4736, 64),      # 8 x 64
    (260, 300, 1016),                                  # the same in parts
    (67, 1217, 136), (130, 900, 72), (521, 2341, 72),  # 16 x 64
    (125, 3650, 72)])                                  # 32 x 128
@pytest.mark.parametrize("scale", ["plain", "underflow"])
def test_hook_exact_tiles_past_their_edges(gpu, orc, M, O, K, scale):
    """The tiles of the product of many rows, rows, outputs and k blocks left over; one row of
    underflowing products sends its tile, and only that, through the literal chain."""
    rng = np.random.default_rng(M + O + K)
    w, x = rng_codes(rng, (O, K), 0.5), rng_codes(rng, (M, K), 1.0)
    if scale == "underflow":
        w[::3] = rng_codes(rng, w[::3].shape, 1e-20)
        x[M // 2] = rng_codes(rng, (K,), 1e-20)
    assert np.array_equal(gpu.bf16_gemm(w, x), orc.gemm(w, x))


@pytest.mark.parametrize("M,O", [(5, 127), (97, 481), (130, 900), (125, 3650)])    # each tile
@pytest.mark.parametrize("block", [0, 1, 2, 5])
def test_hook_exact_tiles_turn_literal_on_the_way(gpu, orc, M, O, block):
    """The first product that is not exact in some block of 64 k: from there on the sums are
    the literal chain's, infinite past a product that overflows, where fused multiply-adds
    (-3e38 + 4e38) stay finite."""
    K, k = 328, 64 * block
    rng = np.random.default_rng(M + block)
    w, x = rng_codes(rng, (O, K), 0.5), rng_codes(rng, (M, K), 1.0)
    w[:, k:k + 2] = x[:, k + 1] = 0x5f8b                 # 2e19
    x[:, k] = 0xdf50                                     # -1.5e19
    exp = orc.gemm(w, x)
    assert np.isinf(f32(exp)).all()
    assert np.array_equal(gpu.bf16_gemm(w, x), exp)


@pytest.mark.parametrize("M", [1, 3])
@pytest.mark.parametrize("K", [15, 17, 31, 34, 1001])
@pytest.mark.parametrize("scale", ["plain", "underflow", "overflow"])
def test_hook_rows_of_unaligned_pieces(gpu, orc, M, K, scale):
    """K that is no multiple of eight, around the sixteen steps loaded ahead: bit for bit."""
    test_hook_exact_order_kernels(gpu, orc, M, 70, K, scale)


@pytest.mark.parametrize("M,O,K", [(4, 16000, 3008), (2, 14300, 6016)])
def test_hook_rows_that_fill_shared_memory(gpu, orc, M, O, K):
    """Rows of x and the rings of four warps are 232448 bytes here, all that a CTA may have,
    static tables included: fewer warps have to be taken."""
    rng = np.random.default_rng(K)
    w = rng.integers(0x3c00, 0x3d80, (O, K), dtype=np.uint16) ^ \
        (rng.integers(0, 2, (O, K), dtype=np.uint16) << 15)
    x = rng_codes(rng, (M, K), 1.0)
    assert np.array_equal(gpu.bf16_gemm(w, x), orc.gemm(w, x))


@pytest.mark.parametrize("mib", [1, 8, 32])
def test_hook_range_of_a_weight_covers_its_end(gpu, orc, mib):
    """The magnitude range that chooses between the fused and the literal chain is taken when
    a weight becomes resident; the values that decide lie in the last row, which arrives
    last.  (The rest of device memory holds ordinary values from the weight before.)"""
    import torch
    rng = np.random.default_rng(mib)
    K, O = 512, mib * 1024
    torch.full((mib << 20,), 0.5, device="cuda")
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    x = rng_codes(rng, (5, K), 1e-20)
    w = np.full((O, K), 0x3f00, np.uint16)
    w[-1] = rng_codes(rng, (K,), 0.5e-20)
    exp = orc.gemm(w, x)
    assert np.array_equal(gpu.bf16_gemm(w, x), exp)
    assert np.array_equal(gpu.bf16_gemv(w, x[0]), exp[0])


def test_hook_zero_dims_and_counters(gpu):
    assert gpu.lib.apus_cuda_bf16_gemv(None, None, None, 0, 8) != 0
    assert gpu.lib.apus_cuda_bf16_gemm(None, None, None, 1, 0, 8) != 0
    rng = np.random.default_rng(1)
    w, x = rng_codes(rng, (64, 64), 0.5), rng_codes(rng, 64, 1.0)
    up0, l0 = gpu.bytes_uploaded(), gpu.launches()
    gpu.bf16_gemv(w, x)
    gpu.bf16_gemv(w, x)      # second call reuses the resident copy
    assert gpu.bytes_uploaded() - up0 == w.nbytes
    assert gpu.launches() - l0 == 2


def test_hooks_inside_the_reference_engine(gpu, ref, be, synth):
    """Drop-in: the backend's three entry points installed into the
    reference's own hook table; the reference's MoE block, run through its own
    layer code, must reproduce its CPU result bit for bit (the per-op hooks
    keep the anchor's order)."""
    cfg = synth.MINI_CFG
    W = synth.host_weights(be, cfg, seed=21, sigma=0.08)
    x = synth.host_x(be, 5, cfg["hidden"], seed=21)
    cpu = ref.moe_block(cfg, W, x)
    l0 = gpu.launches()
    ref.set_hooks(gpu.lib.apus_cuda_bf16_gemv, gpu.lib.apus_cuda_bf16_gemm,
                  gpu.lib.apus_cuda_bf16_matvec_f32)
    try:
        for batched in (False, True):
            hooked = ref.moe_block(cfg, W, x, batched=batched)
            for k in ("idx", "w", "routed", "shared", "out"):
                assert np.array_equal(cpu[k], hooked[k]), (k, batched)
    finally:
        ref.set_hooks(None, None, None)
    assert gpu.launches() > l0       # the GPU really ran them


# ---- router ----------------------------------------------------------------------

def test_router_golden(gpu):
    m = manifest()
    E, K, TK = m["RTR_E"], m["RTR_K"], m["RTR_TK"]
    x = rd("moe_rtr_x.bin", np.uint16)
    wg = rd("moe_rtr_wg.bin", np.uint16).reshape(E, K)
    idx, w = gpu.moe_route(x, wg, TK)
    assert idx[0].tolist() == rd("moe_rtr_idx.bin", np.int64).tolist()
    assert tol_ok(f32(w[0]).astype(np.float64), rd("moe_rtr_w.bin", np.float64),
                  0.02, 0.008, 0.008).all()
    assert gpu.moe_route_topn(x, wg, TK).tolist() == idx[0].tolist()
    assert gpu.moe_route_topn(x, wg, TK + 4)[:TK].tolist() == idx[0].tolist()


def test_router_tie_kats(gpu):
    E, K, TK = 16, 4, 8
    x = np.array([0x3F80, 0, 0, 0], np.uint16)
    wg = np.zeros((E, K), np.uint16)
    wg[:, 0] = 0x3F00
    idx, w = gpu.moe_route(x, wg, TK)
    assert idx[0].tolist() == list(range(8))
    assert (w[0] == 0x3E00).all()
    wg[:, 0] = 0
    wg[:9, 0] = 0x3F80
    idx, _ = gpu.moe_route(x, wg, TK)
    assert idx[0].tolist() == list(range(8))


@pytest.mark.parametrize("T,E,K,TK,sx,sw", [
    (1, 256, 2048, 8, 1.0, 0.02), (2, 256, 2048, 8, 1.0, 0.02),
    (5, 16, 128, 4, 1.0, 0.08), (64, 256, 2048, 8, 1.0, 0.02),
    (300, 256, 2048, 8, 1.0, 0.02), (1111, 256, 2048, 8, 1.0, 0.02),
    (37, 100, 72, 6, 1.0, 0.1), (9, 33, 37, 5, 1.0, 0.1),
    (300, 256, 2048, 8, 1e-19, 1e-19),      # products underflow: literal chain
])
def test_router_bit_exact(gpu, orc, T, E, K, TK, sx, sw):
    """Selected ids, BF16 logits and BF16 routing weights against the CPU
    checker.  Logit ties are frequent here (256 BF16 logits per token), so
    the lowest-index rule is exercised on almost every token."""
    rng = np.random.default_rng(T * 7 + E)
    x = rng_codes(rng, (T, K), 0.4 * sx)
    wg = rng_codes(rng, (E, K), sw * 0.5)
    idx, w, lg = gpu.moe_route(x, wg, TK, want_logits=True)
    oi, ow, ol = orc.route_batch(x, wg, TK, want_logits=True)
    assert np.array_equal(lg, ol)            # logits: bit-exact chains
    assert np.array_equal(idx, oi)           # selection: bit-exact
    # weights: expf last-bit class only — at most one BF16 ulp, and rare
    d = np.abs(w.astype(np.int32) - ow.astype(np.int32))
    assert d.max() <= 1
    assert (d != 0).mean() <= 0.002


# ---- dispatch ------------------------------------------------------------------------

@pytest.mark.parametrize("T,TK,E,skew", [
    (1, 8, 256, False), (3, 8, 256, False), (5, 4, 16, False),
    (64, 8, 256, False), (300, 8, 256, False), (512, 8, 256, False),
    (513, 8, 256, True), (1000, 8, 256, True), (8192, 8, 256, True),
    (8448, 8, 256, False), (700, 6, 1000, False)])
def test_dispatch_bit_exact(gpu, orc, T, TK, E, skew):
    rng = np.random.default_rng(T + E)
    p = None
    if skew:
        p = np.arange(1, E + 1, dtype=np.float64) ** -1.1
        p = p[rng.permutation(E)]
        p /= p.sum()
    idx = np.stack([rng.choice(E, TK, replace=False, p=p) for _ in range(T)]
                   ).astype(np.int32)
    counts, offsets, perm = gpu.moe_dispatch(idx, E)
    oc, oo, op = orc.dispatch(idx, E)
    assert np.array_equal(counts, oc)
    assert np.array_equal(offsets, oo)
    assert np.array_equal(perm, op)


def test_dispatch_rejects_bad_expert_id(gpu):
    idx = np.array([[0, 1, 2, 999]], np.int32)
    with pytest.raises(Exception):
        gpu.moe_dispatch(idx, 16)
    # the context stays usable
    c, o, p = gpu.moe_dispatch(np.array([[3, 1, 2, 0]], np.int32), 16)
    assert p.tolist() == [3, 1, 2, 0]


# --- many-token router: fast logits + exact chains for the candidates ---------
def _route_dev(gpu, synth, cfg, W, x):
    """idx [T, TK], w [T, TK] from apus_cuda_route_dev on a resident layer."""
    import torch
    T = x.shape[0]
    layer = gpu.layer_create(cfg, W)
    d_x = torch.from_numpy(x.view(np.int16)).cuda()
    d_idx = torch.full((T, cfg["top_k"]), -1, dtype=torch.int32, device="cuda")
    d_w = torch.zeros((T, cfg["top_k"]), dtype=torch.int16, device="cuda")
    torch.cuda.synchronize()
    gpu.route_dev(layer, d_x.data_ptr(), T, d_idx.data_ptr(), d_w.data_ptr(),
                  stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return d_idx.cpu().numpy(), d_w.cpu().numpy().view(np.uint16)


CERT_CFG = dict(hidden=512, experts=128, moe_inter=128, shared_inter=128,
                top_k=8)


@pytest.mark.parametrize("T", [65, 257, 1000])
@pytest.mark.parametrize("case", ["plain", "tied_rows", "tiny_logits", "skewed"])
def test_router_certified_selection_is_exact(gpu, orc, be, synth, T, case):
    """Above 64 tokens the router scores all experts on the tensor cores and
    walks the exact chain only for experts that can still reach the top_k.
    The selection must equal the exact router's bit for bit, also when rows of
    the router matrix are identical (every logit tied with its neighbour), when
    all logits are tiny, and when a few experts dominate."""
    cfg = CERT_CFG
    W = synth.host_weights(be, cfg, seed=900 + T, sigma=0.05)
    x = synth.host_x(be, T, cfg["hidden"], seed=900 + T)
    rtr = W["rtr_w"]
    if case == "tied_rows":
        rtr[1::2] = rtr[0::2]
    elif case == "tiny_logits":
        rtr[:] = synth.f32_to_bf16(synth.bf16_to_f32(rtr) * 2.0 ** -20)
    elif case == "skewed":
        W, x = synth.apply_router_bias(W, x, synth.zipf_bias(cfg, seed=3))
        rtr = W["rtr_w"]
    before = gpu.router_exact_chains()
    idx, w = _route_dev(gpu, synth, cfg, W, x)
    chains = gpu.router_exact_chains() - before
    assert gpu.last_block_status() == 0          # includes the error-bound check
    eidx, ew = orc.route_batch(x, rtr, cfg["top_k"])
    assert np.array_equal(idx, eidx)
    d = np.abs(w.astype(np.int32) - ew.astype(np.int32))
    assert d.max() <= 1 and (d != 0).mean() <= 0.002
    # the certified path ran, and it ran far fewer chains than E per token
    assert cfg["top_k"] * T <= chains
    if case in ("plain", "skewed"):
        assert chains <= 4 * cfg["top_k"] * T


@pytest.mark.parametrize("T,E,K,kind", [
    (148, 256, 2048, "bias"), (149, 256, 2048, "bias"),        # a token to an SM, and one more
    (888, 256, 2048, "plain"), (889, 256, 2048, "bias"),       # whole CTAs of tokens, a rest
    (65, 1024, 256, "plain"), (66, 128, 768, "bias"), (67, 384, 2304, "plain"),
    (65, 128, 512, "subnormal"), (65, 128, 512, "ties"), (65, 1024, 512, "zero")])
def test_router_certified_kernel_edges(gpu, orc, be, synth, T, E, K, kind):
    """Both forms of the certifying router, up to 256 experts and more: selected logits that are
    small beside their terms, products that round, ties of all experts, tokens of zeros."""
    cfg = dict(hidden=K, experts=E, moe_inter=128, shared_inter=128, top_k=8)
    W = synth.host_weights(be, cfg, seed=T + K, sigma=0.05)
    x = synth.host_x(be, T, K, seed=T + E)
    rtr = W["rtr_w"]
    if kind == "bias":               # selected logits small beside their terms
        W, x = synth.apply_router_bias(W, x, synth.zipf_bias(cfg, seed=3))
        rtr = W["rtr_w"]
    elif kind == "subnormal":
        x = synth.f32_to_bf16(synth.bf16_to_f32(x) * np.float32(2.0 ** -120))
    elif kind == "ties":
        rtr[:] = rtr[:1]
    elif kind == "zero":
        x[::2] = 0
    idx, w = _route_dev(gpu, synth, cfg, W, x)
    assert gpu.last_block_status() == 0
    eidx, ew = orc.route_batch(x, rtr, cfg["top_k"])
    assert np.array_equal(idx, eidx)
    d = np.abs(w.astype(np.int32) - ew.astype(np.int32))
    assert d.max() <= 1 and (d != 0).mean() <= 0.002


@pytest.mark.parametrize("T,E,kind", [
    (65, 256, "plain"), (296, 256, "bias"), (297, 256, "bias"), (65, 128, "ties"),
    (66, 256, "ties"), (67, 256, "zero"), (68, 256, "subnormal"), (69, 256, "huge")])
def test_router_certified_chains_without_intervals(gpu, orc, be, synth, T, E, kind):
    """The one-kernel form on one to three tokens an SM: more candidates than lanes, products
    that round and logits of 2^110 (whose bound is out of the derivation's range)."""
    if kind != "huge":
        test_router_certified_kernel_edges(gpu, orc, be, synth, T, E, 2048, kind)
        return
    cfg = dict(hidden=2048, experts=E, moe_inter=128, shared_inter=128, top_k=8)
    W = synth.host_weights(be, cfg, seed=T, sigma=0.05)
    x = synth.host_x(be, T, 2048, seed=T)
    W["rtr_w"][:] = synth.f32_to_bf16(synth.bf16_to_f32(W["rtr_w"]) * np.float32(2.0 ** 110))
    idx, w = _route_dev(gpu, synth, cfg, W, x)
    assert gpu.last_block_status() == 0
    eidx, ew = orc.route_batch(x, W["rtr_w"], 8)
    assert np.array_equal(idx, eidx)
    assert np.abs(w.astype(np.int32) - ew.astype(np.int32)).max() <= 1


@pytest.mark.parametrize("T,E,K,kind", [
    (592, 256, 2048, "bias"), (593, 256, 2048, "bias"),        # one kernel, then lists
    (593, 384, 768, "plain"), (600, 1024, 256, "bias"),        # more than 256 experts
    (607, 128, 512, "ties"), (640, 128, 512, "zero"),          # every expert a candidate
    (600, 128, 512, "subnormal"), (600, 128, 512, "huge"),     # products that round, overflow
    (2049, 128, 256, "bias")])                                 # lists of many warps
def test_router_candidate_lists(gpu, orc, be, synth, T, E, K, kind):
    """Candidates' chains from lists per expert: both sides of four tokens an SM, lists that
    end inside a warp's 32 tokens, tokens with more candidates than lanes beside others."""
    if kind != "huge":
        test_router_certified_kernel_edges(gpu, orc, be, synth, T, E, K, kind)
        return
    cfg = dict(hidden=K, experts=E, moe_inter=128, shared_inter=128, top_k=8)
    W = synth.host_weights(be, cfg, seed=T, sigma=0.05)
    x = synth.host_x(be, T, K, seed=T)
    W["rtr_w"][:] = synth.f32_to_bf16(synth.bf16_to_f32(W["rtr_w"]) * np.float32(2.0 ** 110))
    idx, w = _route_dev(gpu, synth, cfg, W, x)
    assert gpu.last_block_status() == 0
    eidx, ew = orc.route_batch(x, W["rtr_w"], 8)
    assert np.array_equal(idx, eidx)
    assert np.abs(w.astype(np.int32) - ew.astype(np.int32)).max() <= 1


@pytest.mark.parametrize("T,E,K,topk", [
    (9, 256, 2048, 8), (52, 256, 2048, 8), (53, 256, 2048, 8), (64, 257, 2048, 8),
    (61, 300, 1032, 5), (64, 1024, 512, 32), (33, 37, 24, 1)])
@pytest.mark.parametrize("case", ["plain", "tied_rows", "tiny_logits"])
def test_router_few_tokens_edges(gpu, orc, be, synth, T, E, K, topk, case):
    """The few-token router where a second wave of CTAs would begin, with remainders of
    rows and tokens, and where code order may not decide."""
    cfg = dict(hidden=K, experts=E, moe_inter=128, shared_inter=128, top_k=topk)
    W = synth.host_weights(be, cfg, seed=T + K, sigma=0.05)
    x = synth.host_x(be, T, K, seed=T + E)
    rtr = W["rtr_w"]
    if case == "tied_rows":
        rtr[1::2] = rtr[0::2][:rtr[1::2].shape[0]]
    elif case == "tiny_logits":
        rtr[:] = synth.f32_to_bf16(synth.bf16_to_f32(rtr) * 2.0 ** -20)
    idx, w = _route_dev(gpu, synth, cfg, W, x)
    assert gpu.last_block_status() == 0
    eidx, ew = orc.route_batch(x, rtr, topk)
    assert np.array_equal(idx, eidx)
    d = np.abs(w.astype(np.int32) - ew.astype(np.int32))
    assert d.max() <= 1 and (d != 0).mean() <= 0.002


@pytest.mark.parametrize("T,E,K,topk", [(64, 256, 4736, 8), (64, 256, 4744, 8),
                                        (64, 256, 7104, 8), (64, 256, 7112, 8)])
def test_router_few_tokens_at_the_shared_memory_limit(gpu, orc, be, synth, T, E, K, topk):
    """The last sizes at which sixteen rows a CTA (4736) and eight (7104) fit beside the
    static tables, and the first at which they fit only without those."""
    cfg = dict(hidden=K, experts=E, moe_inter=8, shared_inter=8, top_k=topk)
    W = synth.host_weights(be, cfg, seed=K, sigma=0.02)
    x = synth.host_x(be, T, K, seed=T)
    idx, w = _route_dev(gpu, synth, cfg, W, x)
    assert gpu.last_block_status() == 0
    eidx, ew = orc.route_batch(x, W["rtr_w"], topk)
    assert np.array_equal(idx, eidx)
    assert np.abs(w.astype(np.int32) - ew.astype(np.int32)).max() <= 1


@pytest.mark.parametrize("T", [1184, 1185, 1776, 1777, 2368, 2369])
def test_router_certified_ring_and_chain_forms(gpu, orc, be, synth, T):
    """Candidate lists of eight to sixteen tokens an SM, tokens left over in the last CTA or
    not, with a router whose logits lie close together."""
    cfg = dict(hidden=2048, experts=256, moe_inter=8, shared_inter=8, top_k=8)
    W = synth.host_weights(be, cfg, seed=T, sigma=0.02)
    x = synth.host_x(be, T, 2048, seed=T)
    W, x = synth.apply_router_bias(W, x, synth.zipf_bias(cfg, seed=3, beta=0.27))
    idx, w = _route_dev(gpu, synth, cfg, W, x)
    assert gpu.last_block_status() == 0
    eidx, ew = orc.route_batch(x, W["rtr_w"], 8)
    assert np.array_equal(idx, eidx)
    d = np.abs(w.astype(np.int32) - ew.astype(np.int32))
    assert d.max() <= 1 and (d != 0).mean() <= 0.002


def _weights_at_midpoints(orc, synth, E, topk, n):
    """n logit vectors [n, E] (BF16 codes) whose weights differ between the engine's
    (q_i / S) / sum(q / S) and q_i / sum(q), with the engine's result for them."""
    rng = np.random.default_rng(E + topk)
    found, want = [], []
    while sum(len(v) for v in found) < n:
        z = synth.f32_to_bf16(rng.normal(0, 1, (200000, E)).astype(np.float32))
        v = f32(z)
        q = np.exp((v - v.max(1, keepdims=True)).astype(np.float64)).astype(np.float32)
        order = np.argsort(-v, axis=1, kind="stable")[:, :topk]
        S = np.zeros(len(q), np.float32)
        for e in range(E):
            S = S + q[:, e]
        qs = np.take_along_axis(q, order, 1)
        ps = np.take_along_axis(q / S[:, None], order, 1)
        sq, sp = np.zeros(len(q), np.float32), np.zeros(len(q), np.float32)
        for i in range(topk):
            sq, sp = sq + qs[:, i], sp + ps[:, i]
        w = synth.f32_to_bf16(ps / sp[:, None])
        diff = (w != synth.f32_to_bf16(qs / sq[:, None])).any(1)
        found.append(z[diff])
        want.append(w[diff])
    return np.concatenate(found)[:n], np.concatenate(want)[:n]


@pytest.mark.parametrize("E,topk", [(16, 8), (40, 3)])
def test_router_few_tokens_weights_follow_the_engines_steps(gpu, orc, be, synth, E, topk):
    """Weights that narrow differently when the softmax denominator is left out of the
    quotient; the logits are written into a router matrix that one-hot tokens read."""
    T = K = 64
    z, w = _weights_at_midpoints(orc, synth, E, topk, T)
    x = np.zeros((T, K), np.uint16)
    x[np.arange(T), np.arange(T)] = 0x3f80
    cfg = dict(hidden=K, experts=E, moe_inter=8, shared_inter=8, top_k=topk)
    W = synth.host_weights(be, cfg, seed=1, sigma=0.05)
    W["rtr_w"] = np.ascontiguousarray(z.T)
    eidx, ew = orc.route_batch(x, W["rtr_w"], topk)
    same = (ew == w).all(1)              # the rest: expf differs in a last bit
    assert same.mean() > 0.8
    for t0, n in ((0, 64), (0, 9), (30, 33)):
        gidx, gw = _route_dev(gpu, synth, cfg, W, x[t0:t0 + n])
        assert np.array_equal(gidx, eidx[t0:t0 + n])
        assert np.array_equal(gw[same[t0:t0 + n]], ew[t0:t0 + n][same[t0:t0 + n]])


@pytest.mark.parametrize("path,T,E,K", [("few", 64, 48, 64), ("certified", 256, 128, 256),
                                        ("one kernel", 8, 128, 128)])
@pytest.mark.parametrize("seed", range(3))
def test_router_small_logits_in_any_company(gpu, orc, be, synth, path, T, E, K, seed):
    """Logits around 2^-10, below which two of them may have the same probability: one small
    competitor among others, several, beside zeros of either sign, as the last one chosen and
    right below it.  One-hot tokens read the logits from the router matrix.  (2e-38 makes
    products round: above 64 tokens every token takes the softmax here.)"""
    rng = np.random.default_rng(seed)
    edge = 2.0 ** -10
    small = [0.0, -0.0, edge, -edge, edge * (1 + 2 ** -7), edge * (1 - 2 ** -8), 2 ** -11,
             -edge * (1 - 2 ** -8), 1e-5, 1.01e-5, -1e-5, 3e-20, -3e-20, 2e-38]
    z = rng.normal(-1.0, 1.0, (T, E))
    for t in range(T):
        n, top = int(rng.integers(0, 8)), int(rng.integers(0, 9))
        where = rng.permutation(E)
        z[t] = np.where(z[t] > -0.01, z[t] - 3.0, z[t])          # all others below
        z[t, where[:top]] = rng.uniform(0.01, 2.0, top)          # so many above
        z[t, where[top:top + n]] = rng.choice(small, n)
    z = synth.f32_to_bf16(z.astype(np.float32))
    x = np.zeros((T, K), np.uint16)
    x[np.arange(T), np.arange(T)] = 0x3f80
    cfg = dict(hidden=K, experts=E, moe_inter=16, shared_inter=16, top_k=8)
    W = synth.host_weights(be, cfg, seed=1, sigma=0.05)
    W["rtr_w"] = np.zeros((E, K), np.uint16)
    W["rtr_w"][:, :T] = z.T
    eidx, ew = orc.route_batch(x, W["rtr_w"], 8)
    if path == "one kernel":
        got = gpu.moe_block(cfg, W, x)
        assert gpu.last_block_path() == 0
        gidx, gw = got["idx"], got["w"]
    else:
        gidx, gw = _route_dev(gpu, synth, cfg, W, x)
    assert gpu.last_block_status() == 0
    assert np.array_equal(gidx, eidx)
    assert np.abs(gw.astype(np.int32) - ew.astype(np.int32)).max() <= 1


@pytest.mark.parametrize("T,K", [(256, 256), (640, 768)])
@pytest.mark.parametrize("seed", range(4))
def test_router_small_logits_where_code_order_decides(gpu, orc, be, synth, T, K, seed):
    """Logits around 2^-10 and far below, in both forms of the many-token router and with every
    product exact, so that the choice is made on codes: ties at the last place chosen with a
    neighbour below them that has their probability, zeros of either sign beside values that
    nothing tells from them, and logits that only the subtraction of the largest makes equal."""
    rng = np.random.default_rng(seed)
    E, edge = 128, 2.0 ** -10
    small = [0.0, -0.0, edge, -edge, edge * (1 + 2 ** -7), edge * (1 - 2 ** -8), 2 ** -11,
             -edge * (1 - 2 ** -8), 1e-5, 1.01e-5, -1e-5, 3e-20, -3e-20]
    z = rng.normal(-1.0, 1.0, (T, E))
    z = np.where(z > -0.01, z - 3.0, z)
    for t in range(T):
        n, top = int(rng.integers(0, 8)), int(rng.integers(0, 9))
        where = rng.permutation(E)
        z[t, where[:top]] = rng.uniform(0.01, 2.0, top)
        z[t, where[top:top + n]] = rng.choice(small, n)
    z[:3] = -2.0
    z[:3, 1:8] = np.linspace(0.5, 2.0, 7)
    z[0, [85, 97, 48]] = 1.0073e-05, 1.0073e-05, 1.0013e-05
    z[1, [60, 70, 9]] = 0.0, -0.0, -3e-20
    z[2, [7, 100, 50]] = 32.0, -131 * 2.0 ** -19, -133 * 2.0 ** -19
    z = synth.f32_to_bf16(z.astype(np.float32))
    x = np.zeros((T, K), np.uint16)
    x[np.arange(T), np.arange(T)] = 0x3f80
    cfg = dict(hidden=K, experts=E, moe_inter=16, shared_inter=16, top_k=8)
    W = synth.host_weights(be, cfg, seed=1, sigma=0.05)
    W["rtr_w"] = np.zeros((E, K), np.uint16)
    W["rtr_w"][:, :T] = z.T
    eidx, ew = orc.route_batch(x, W["rtr_w"], 8)
    assert eidx[:3, 7].tolist() == [48, 9, 50]           # the lowest number of its probability
    idx, w = _route_dev(gpu, synth, cfg, W, x)
    assert gpu.last_block_status() == 0
    assert np.array_equal(idx, eidx)
    assert np.abs(w.astype(np.int32) - ew.astype(np.int32)).max() <= 1


@pytest.mark.parametrize("T", [300, 640])                # one kernel, lists
def test_router_candidates_and_gate_fill_a_warp(gpu, orc, be, synth, T):
    """Tokens with 8 to 128 candidates side by side, the shared gate's chain the last that a
    warp's lanes hold, the first beyond them, or far beyond: ids, weights and the gate's code."""
    import torch
    K, E = 768, 128
    rng = np.random.default_rng(T)
    counts = np.resize([8, 30, 31, 32, 33, 63, 64, 127, 128], T)
    z = np.full((T, E), -1.0, np.float32)
    for t in range(T):
        z[t, rng.permutation(E)[:counts[t]]] = rng.choice([1.0, 1.0 + 2 ** -7], counts[t])
    x = np.zeros((T, K), np.uint16)
    x[np.arange(T), np.arange(T)] = 0x3f80               # each token reads its own column
    cfg = dict(hidden=K, experts=E, moe_inter=128, shared_inter=128, top_k=8)
    W = synth.host_weights(be, cfg, seed=1, sigma=0.05)
    W["rtr_w"] = np.zeros((E, K), np.uint16)
    W["rtr_w"][:, :T] = synth.f32_to_bf16(z).T
    layer = gpu.layer_create(cfg, W)
    d_x = torch.from_numpy(x.view(np.int16)).cuda()
    d_idx = torch.full((T, 8), -1, dtype=torch.int32, device="cuda")
    d_w = torch.zeros((T, 8), dtype=torch.int16, device="cuda")
    d_gate = torch.zeros(T, dtype=torch.int16, device="cuda")
    before = gpu.router_exact_chains()
    gpu.ep_route_dev(layer, d_x.data_ptr(), T, d_idx.data_ptr(), d_w.data_ptr(),
                     d_gate.data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert gpu.last_block_status() == 0
    assert gpu.router_exact_chains() - before == counts.sum() + T
    eidx, ew = orc.route_batch(x, W["rtr_w"], 8)
    w = d_w.cpu().numpy().view(np.uint16)
    assert np.array_equal(d_idx.cpu().numpy(), eidx)
    assert np.abs(w.astype(np.int32) - ew.astype(np.int32)).max() <= 1
    gate = W["sh_gate"].reshape(-1)[:T]
    assert np.array_equal(f32(d_gate.cpu().numpy().view(np.uint16)), f32(gate))
    gpu.layer_destroy(layer)


def test_router_certified_can_be_switched_off(be, orc, synth, monkeypatch):
    monkeypatch.setenv("APUS_CUDA_ROUTER_CERTIFY", "0")
    be.enable()
    try:
        cfg = CERT_CFG
        W = synth.host_weights(be, cfg, seed=77, sigma=0.05)
        x = synth.host_x(be, 130, cfg["hidden"], seed=77)
        before = be.router_exact_chains()
        idx, w = _route_dev(be, synth, cfg, W, x)
        assert be.router_exact_chains() == before
        eidx, _ = orc.route_batch(x, W["rtr_w"], cfg["top_k"])
        assert np.array_equal(idx, eidx)
    finally:
        be.disable()


# --- the callers either side of the block: rmsnorm before, residual add after ---
@pytest.mark.parametrize("T,N", [(1, 2048), (5, 2048), (149, 2048), (33, 512), (3, 130), (2, 24)])
def test_rmsnorm_and_residual_add_bitwise(gpu, orc, be, synth, T, N):
    """apus_cuda_rmsnorm_dev / apus_cuda_resadd_dev against the checker
    (c/attn.h:175-186 with its sequential sum of squares; c/layer.h:230-234):
    bit for bit, with and without a gain vector, rows that are not a multiple
    of the vector width included."""
    import torch
    x = synth.f32_to_bf16(
        synth.bf16_to_f32(be.synth_fill_host(T * N, 5, 0, 0, 1.0)).reshape(T, N) * 3.0)
    gw = be.synth_fill_host(N, 5, 1, 1, 0.3)
    sp = torch.cuda.current_stream().cuda_stream
    d_x = torch.from_numpy(x.view(np.int16)).cuda()
    d_w = torch.from_numpy(gw.view(np.int16)).cuda()
    d_y = torch.empty_like(d_x)
    for w_dev, w_host in ((d_w, gw), (None, None)):
        gpu.rmsnorm_dev(d_x.data_ptr(), w_dev.data_ptr() if w_dev is not None else None,
                        d_y.data_ptr(), T, N, stream=sp)
        torch.cuda.synchronize()
        assert np.array_equal(d_y.cpu().numpy().view(np.uint16), orc.rmsnorm(x, w_host))
    b = be.synth_fill_host(T * N, 6, 0, 0, 1.0).reshape(T, N)
    d_b = torch.from_numpy(b.view(np.int16)).cuda()
    gpu.resadd_dev(d_x.data_ptr(), d_b.data_ptr(), d_y.data_ptr(), T * N, stream=sp)
    torch.cuda.synchronize()
    assert np.array_equal(d_y.cpu().numpy().view(np.uint16), orc.resadd(x, b))


@pytest.mark.parametrize("N", [8, 128, 256, 768, 2048, 2560, 512, 576, 640, 1152, 1056, 4096,
                               1024, 1280, 2304])
def test_rmsnorm_sum_without_the_chain(gpu, orc, N):
    """The sum of squares composed from parity functions against the sequential
    chain, bit for bit, on rows made to go wrong: ties in every add, sums that sit
    on a binade's edge, one value that jumps several binades, descending and
    ascending magnitudes, zeros, subnormal squares, an overflow."""
    import torch
    rng = np.random.default_rng(N)
    rows = [rng.normal(0, s, N) for s in (1.0, 1e-3, 30.0, 1e-18)]
    rows += [np.ones(N), np.full(N, 1.5), np.full(N, 1.0 + 2 ** -7), np.zeros(N)]
    rows += [np.where(np.arange(N) == N // 2, 1e4, rng.normal(0, 1, N)),
             np.where(np.arange(N) == N - 1, 3e3, rng.normal(0, 1e-2, N)),
             np.exp2(np.linspace(6, -12, N)), np.exp2(np.linspace(-12, 6, N)),
             rng.integers(1, 4, N) * 0.5, np.where(np.arange(N) % 64 == 0, 8.0, 0.0),
             np.full(N, 1e20), np.sign(rng.normal(0, 1, N)) * 181.0]
    rows += [rng.normal(0, 2.0 ** rng.integers(-3, 4), N) for _ in range(40)]
    u = np.asarray(rows, np.float32).view(np.uint32).astype(np.uint64)
    x = ((u + 0x7fff + ((u >> 16) & 1)) >> 16).astype(np.uint16)
    d_x = torch.from_numpy(x.view(np.int16)).cuda()
    d_y = torch.empty_like(d_x)
    gpu.rmsnorm_dev(d_x.data_ptr(), None, d_y.data_ptr(), len(rows), N,
                    stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert np.array_equal(d_y.cpu().numpy().view(np.uint16), orc.rmsnorm(x, None))


@pytest.mark.parametrize("T,N", [(148, 2048), (9, 2048), (149, 2048), (148, 512)])
def test_rmsnorm_gains_from_the_kernel_before(gpu, orc, T, N):
    """A norm whose gains are a row of the norm in front of it: each kernel releases its successor
    early, so it has to wait for the gains as for the rows.  Buffers of their own for every link,
    so that a read too early finds zeros."""
    import torch
    rng = np.random.default_rng(T + N)
    links = 24
    x = rng_codes(rng, (links, T, N), 1.0)
    d_x = torch.from_numpy(x.view(np.int16)).cuda()
    d_y = torch.zeros_like(d_x)
    sp = torch.cuda.current_stream().cuda_stream
    torch.cuda.synchronize()
    for i in range(links):
        gpu.rmsnorm_dev(d_x[i].data_ptr(), d_y[i - 1, T - 1].data_ptr() if i else None,
                        d_y[i].data_ptr(), T, N, stream=sp)
    torch.cuda.synchronize()
    gains = None
    for i in range(links):
        y = orc.rmsnorm(x[i], gains)
        assert np.array_equal(d_y[i].cpu().numpy().view(np.uint16), y), i
        gains = y[T - 1]


@pytest.mark.parametrize("N,pieces,warps", [
    (512, 2, 1), (768, 4, 1), (1024, 4, 1), (1280, 8, 1), (1792, 8, 1), (2048, 8, 1),
    (1152, -1, 1), (2304, -1, 1), (2560, -1, 1),                    # rows of the row norm
    (512, 4, 2), (1536, 4, 2), (2048, 4, 2), (2560, 0, 2), (208, 0, 1), (144, 0, 1), (16, 4, 1), (1024, 4, 2),
    (2048, 2, 4), (2048, -2, 2), (2048, -2, 4)])
def test_sum_of_squares_is_the_chains(gpu, N, pieces, warps):
    """The fp32 sum itself, which a norm shows only through BF16, in every form that the row norm
    and the one-kernel path use: ties in every add, sums on a binade's edge, jumps over binades
    in either half of a row, falling and rising terms, subnormal squares, an overflow."""
    rng = np.random.default_rng(N + pieces + warps)
    at = np.arange(N)
    rows = [np.ones(N), np.full(N, 1.5), np.full(N, 1.0 + 2 ** -7), np.zeros(N),
            np.full(N, 1e20), np.sign(rng.normal(0, 1, N)) * 181.0, rng.integers(1, 4, N) * 0.5,
            np.exp2(np.linspace(6, -12, N)), np.exp2(np.linspace(-12, 6, N)),
            np.where(at % 64 == 0, 8.0, 0.0), rng.normal(0, 1e-18, N), rng.normal(0, 1e-22, N)]
    rows += [np.where(at == p, 1e3, rng.normal(0, 1, N))
             for p in (0, N // 4, N // 2 - 1, N // 2, N - 1)]
    rows += [rng.normal(0, 2.0 ** rng.uniform(-4, 4), N) for _ in range(200)]
    u = np.asarray(rows, np.float32).view(np.uint32).astype(np.uint64)
    x = ((u + 0x7fff + ((u >> 16) & 1)) >> 16).astype(np.uint16)
    with np.errstate(over="ignore", under="ignore"):
        q = f32(x) * f32(x)
        exp = np.zeros(len(rows), np.float32)
        for k in range(N):
            exp = exp + q[:, k]
    got = gpu.debug_sumsq(x, pieces, warps)
    assert np.array_equal(got.view(np.uint32), exp.view(np.uint32))


# ---- the dense weight stream on device pointers --------------------------------

@pytest.mark.parametrize("M,O,K,shift", [
    (1, 15, 256, 0), (5, 16, 512, 0), (7, 17, 2304, 0), (8, 148 * 16, 256, 0),
    (4, 148 * 16 * 8 + 5, 256, 0), (6, 148 * 16 * 8 * 2 - 1, 256, 0), (2, 31, 16384, 0),
    (8, 40, 7168, 0), (3, 100, 512, 1),
    # warps that share sixteen rows: eight, four and two of them, K that they do not divide
    (1, 148 * 16, 1280, 0), (3, 148 * 16 + 1, 2048, 0), (8, 148 * 32, 4096, 0),
    (2, 148 * 32 + 9, 768, 1), (5, 148 * 64 - 3, 2304, 0), (1, 148 * 64 + 1, 512, 0),
    (1, 9, 58112, 0), (8, 700, 7168, 0)])
def test_gemv_stream_edges(gpu, orc, M, O, K, shift):
    """Whole rounds, remainders and fewer rows than warps; x beside a smaller ring; x that
    is not 16-byte aligned.  Both sums are fp32 over K exact products: they differ by at
    most 2 K 2^-24 of the sum of magnitudes, and each narrows to BF16 (2^-8)."""
    import torch
    rng = np.random.default_rng(M * 1000 + O)
    w, x = rng_codes(rng, (O, K), 0.05), rng_codes(rng, (M, K), 1.0)
    d_w = torch.from_numpy(w.view(np.int16)).cuda()
    d_x = torch.zeros(M * K + 8, dtype=torch.int16, device="cuda")
    d_x[shift:shift + M * K] = torch.from_numpy(x.view(np.int16)).cuda().reshape(-1)
    d_y = torch.zeros((M + 1, O), dtype=torch.int16, device="cuda")
    gpu.bf16_gemv_dev(d_w.data_ptr(), d_x.data_ptr() + 2 * shift, d_y.data_ptr(), M, O, K,
                      stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    y = d_y.cpu().numpy().view(np.uint16)
    got, exp = f32(y[:M]).astype(np.float64), f32(orc.gemm(w, x)).astype(np.float64)
    mag = np.abs(f32(x).astype(np.float64)) @ np.abs(f32(w).astype(np.float64)).T
    assert (np.abs(got - exp) <= 2 * K * 2.0 ** -24 * mag + np.abs(exp) * 2.0 ** -7).all()
    assert not y[M].any()


@pytest.mark.parametrize("M,O,K,share", [(1, 65536, 2048, 0.97e-4), (8, 65536, 2048, 1.00e-4),
                                          (4, 16384, 8192, 1.68e-4)])
def test_gemv_stream_against_64_bit_sums(gpu, M, O, K, share):
    """How often a result narrows to another BF16 value than its 64-bit sum does, against
    `share`, what scalar multiply-adds in fp32 had there.  Bound: half as much again (six
    standard deviations of the 150 and more events in the three passes)."""
    import torch
    wrong = n = 0
    for seed in range(3 if M == 8 else 8):
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        w = (torch.randn(O, K, device="cuda", generator=gen) * 0.02).bfloat16()
        x = torch.randn(M, K, device="cuda", generator=gen).bfloat16()
        y = torch.empty((M, O), dtype=torch.bfloat16, device="cuda")
        gpu.bf16_gemv_dev(w.data_ptr(), x.data_ptr(), y.data_ptr(), M, O, K,
                          stream=torch.cuda.current_stream().cuda_stream)
        exp = (x.double() @ w.double().T).contiguous().view(torch.int64)
        exp = exp + ((1 << 44) - 1) + ((exp >> 45) & 1)          # one rounding to BF16
        wrong += int((y.double() != (exp >> 45 << 45).view(torch.float64)).sum())
        n += y.numel()
    assert wrong <= 1.5 * share * n, wrong / n


@pytest.mark.parametrize("M,O,K", [(1, 4096, 2048), (3, 1000, 512), (8, 777, 256),
                                   (1, 1, 256), (2, 33, 2048)])
def test_gemv_stream_dev(gpu, orc, M, O, K):
    """apus_cuda_bf16_gemv_dev against the CPU anchor: same products, another
    summation order, so BF16 tolerance (the hooks keep the exact bits)."""
    import torch
    rng = np.random.default_rng(M * 1000 + O)
    w, x = rng_codes(rng, (O, K), 0.05), rng_codes(rng, (M, K), 1.0)
    d_w = torch.from_numpy(w.view(np.int16)).cuda()
    d_x = torch.from_numpy(x.view(np.int16)).cuda()
    d_y = torch.zeros((M, O), dtype=torch.int16, device="cuda")
    gpu.bf16_gemv_dev(d_w.data_ptr(), d_x.data_ptr(), d_y.data_ptr(), M, O, K,
                      stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    got = f32(d_y.cpu().numpy().view(np.uint16))
    exp = f32(orc.gemm(w, x))
    scale = np.abs(exp).max() + 1e-9
    assert np.abs(got - exp).max() <= 1e-2 * scale
    assert (got.view(np.uint32) != exp.view(np.uint32)).mean() <= 0.2
