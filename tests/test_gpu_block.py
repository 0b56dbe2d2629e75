"""GPU parity tests for the MoE block operator, through the C-ABI, against
the CPU checker on the same seeded inputs and against the committed goldens.

Bar (the benchmark specification's): selected expert ids bit-exact; outputs
max-abs <= 2e-2 and relative L2 <= 1e-2 in BF16."""
import os

import numpy as np
import pytest

from conftest import rel_l2
from test_oracle_cpu import f32, G

pytestmark = pytest.mark.gpu

MAX_ABS, REL_L2 = 2e-2, 1e-2


def check_block(got, exp, tag=""):
    assert np.array_equal(got["idx"], exp["idx"]), tag + " idx"
    d = np.abs(got["w"].astype(np.int32) - exp["w"].astype(np.int32))
    assert d.max() <= 1 and (d != 0).mean() <= 0.002, tag + " rtr_w"
    for k in ("routed", "shared", "out"):
        a, b = f32(got[k]), f32(exp[k])
        assert np.isfinite(a).all(), tag + k
        assert np.abs(a - b).max() <= MAX_ABS, (tag, k, np.abs(a - b).max())
        assert rel_l2(a, b) <= REL_L2, (tag, k, rel_l2(a, b))


@pytest.mark.parametrize("name", ["block_mini_t1", "block_mini_t7",
                                  "block_qwen_t3"])
def test_block_goldens(gpu, be, synth, name):
    g = np.load(os.path.join(G, name + ".npz"))
    cfg = dict(zip(("hidden", "experts", "moe_inter", "shared_inter", "top_k"),
                   (int(v) for v in g["cfg"])))
    W = synth.host_weights(be, cfg, seed=int(g["seed"]), sigma=float(g["sigma"]))
    got = gpu.moe_block(cfg, W, g["x"])
    check_block(got, g, name)


@pytest.mark.parametrize("T", [1, 2, 3, 5, 64, 65, 300])
def test_block_mini(gpu, orc, be, synth, T):
    cfg = synth.MINI_CFG
    W = synth.host_weights(be, cfg, seed=300 + T, sigma=0.08)
    x = synth.host_x(be, T, cfg["hidden"], seed=300 + T)
    check_block(gpu.moe_block(cfg, W, x), orc.moe_block(cfg, W, x), f"T={T}")


@pytest.mark.parametrize("cfg", [
    dict(hidden=512, experts=64, moe_inter=128, shared_inter=64, top_k=8),
    dict(hidden=256, experts=8, moe_inter=64, shared_inter=128, top_k=2),
    # shapes the tensor-core path accepts (T > 64 takes it)
    dict(hidden=512, experts=64, moe_inter=128, shared_inter=128, top_k=8),
    dict(hidden=256, experts=8, moe_inter=256, shared_inter=256, top_k=3),
])
@pytest.mark.parametrize("T", [1, 40, 65, 200, 777])
def test_block_medium(gpu, orc, be, synth, cfg, T):
    W = synth.host_weights(be, cfg, seed=77, sigma=0.05)
    x = synth.host_x(be, T, cfg["hidden"], seed=77 + T)
    check_block(gpu.moe_block(cfg, W, x), orc.moe_block(cfg, W, x), f"T={T}")


@pytest.fixture(scope="module")
def qwen_weights(be, synth):
    return synth.host_weights(be, synth.QWEN_CFG, seed=0)


@pytest.mark.parametrize("T", [1, 8, 64, 512])
def test_block_qwen_dims(gpu, orc, be, synth, qwen_weights, T):
    """Benchmark configurations 0 (T=1), 2 (B=8, 64) and 1 (T=512) at the real
    dimensions, seed 0."""
    cfg = synth.QWEN_CFG
    x = synth.host_x(be, T, cfg["hidden"], seed=0)
    got = gpu.moe_block(cfg, qwen_weights, x)
    exp = orc.moe_block(cfg, qwen_weights, x)
    check_block(got, exp, f"qwen T={T}")
    assert gpu.last_block_status() == 0


FUSED_SMALL = dict(hidden=512, experts=64, moe_inter=128, shared_inter=64,
                   top_k=8)


@pytest.mark.parametrize("T", [1, 2, 3, 4])
@pytest.mark.parametrize("cfgname", ["small", "qwen"])
def test_block_one_kernel_path(gpu, orc, be, synth, qwen_weights, cfgname, T):
    """One to four tokens run as ONE cooperative launch; two calls in a row
    (the second reuses the self-resetting counters)."""
    cfg = FUSED_SMALL if cfgname == "small" else synth.QWEN_CFG
    W = (synth.host_weights(be, cfg, seed=5, sigma=0.05) if cfgname == "small"
         else qwen_weights)
    for seed in (11, 12):
        x = synth.host_x(be, T, cfg["hidden"], seed=seed + T)
        got = gpu.moe_block(cfg, W, x)
        assert gpu.last_block_launches() == 1
        assert gpu.last_block_status() == 0
        check_block(got, orc.moe_block(cfg, W, x), f"{cfgname} T={T}")


@pytest.mark.parametrize("T,H,E,I,Is,TK", [
    (5, 2048, 256, 512, 512, 8), (8, 2048, 256, 512, 512, 8),
    # rows of 2048: a logit's row cut over four warps (one and two tokens) and over two
    (1, 2048, 256, 256, 256, 8), (2, 2048, 256, 512, 512, 8), (3, 2048, 256, 256, 256, 8),
    (4, 2048, 256, 256, 256, 8), (4, 2048, 16, 256, 256, 4), (7, 208, 37, 48, 16, 3),
    (8, 1040, 300, 272, 144, 8), (3, 512, 1024, 128, 256, 2), (8, 16, 8, 16, 16, 8),
    (1, 128, 16, 32, 32, 1)])
@pytest.mark.parametrize("case", ["plain", "tied_rows", "tiny_logits", "opposite", "underflow"])
def test_block_one_kernel_edges(gpu, orc, be, synth, T, H, E, I, Is, TK, case):
    """The one-kernel path at the edges of its tiles (k slices, columns, expert
    changes inside a tile) and of its routing: logits tied with their neighbours,
    logits so small that probabilities decide, sums that cancel (wide intervals: the
    chains run), products that underflow (every chain runs)."""
    cfg = dict(hidden=H, experts=E, moe_inter=I, shared_inter=Is, top_k=TK)
    # gate and up of unit variance at most: outputs stay below 4, where one BF16 step
    # (2^-6), the difference two summation orders may show, is below MAX_ABS
    W = synth.host_weights(be, cfg, seed=700 + T + E, sigma=min(0.06, 0.9 / H ** 0.5))
    x = synth.host_x(be, T, H, seed=700 + T)
    rtr = W["rtr_w"]
    if case == "tied_rows":
        rtr[1::2] = rtr[0::2][:rtr[1::2].shape[0]]
    elif case == "tiny_logits":
        rtr[:] = synth.f32_to_bf16(synth.bf16_to_f32(rtr) * 2.0 ** -14)
    elif case == "opposite":
        rtr[:, 1::2] = rtr[:, 0::2] ^ 0x8000
        x[:, 1::2] = x[:, 0::2]
    elif case == "underflow":
        rtr[:] = synth.f32_to_bf16(synth.bf16_to_f32(rtr) * 1e-36)
    before = gpu.router_exact_chains()
    got = gpu.moe_block(cfg, W, x)
    assert gpu.last_block_launches() == 1 and gpu.last_block_status() == 0
    check_block(got, orc.moe_block(cfg, W, x), f"{case} T={T}")
    if case == "underflow":
        assert gpu.router_exact_chains() - before >= T * E


@pytest.mark.parametrize("T,H,E,I,Is,TK", [
    (1, 256, 64, 16, 32, 8), (1, 2048, 64, 16, 512, 8), (3, 208, 64, 16, 272, 8),
    (8, 512, 64, 16, 32, 8), (8, 256, 256, 16, 512, 8), (1, 256, 64, 32, 16, 8)])
def test_block_one_kernel_empty_halves(gpu, orc, be, synth, T, H, E, I, Is, TK):
    """Down rows are taken in halves of K.  Sixteen values have no second half; with eight
    distinct experts or more the same warp's next one (at last the shared expert's) does."""
    cfg = dict(hidden=H, experts=E, moe_inter=I, shared_inter=Is, top_k=TK)
    W = synth.host_weights(be, cfg, seed=40 + T, sigma=0.9 / H ** 0.5)
    for seed in (50, 51):          # the second call finds the first one's ring contents
        x = synth.host_x(be, T, H, seed=seed + T)
        got = gpu.moe_block(cfg, W, x)
        assert gpu.last_block_launches() == 1 and gpu.last_block_status() == 0
        check_block(got, orc.moe_block(cfg, W, x), f"I={I} Is={Is} T={T}")


@pytest.mark.parametrize("T,E,TK,skew", [
    (9, 128, 8, False), (65, 128, 1, True), (255, 128, 8, True), (256, 1024, 8, False),
    (257, 128, 8, True), (513, 256, 3, False), (300, 128, 32, True),     # counted by the router
    (301, 100, 5, False), (1030, 36, 8, True),         # another router: not counted
    (3100, 128, 8, True)])                             # two-SM kernels' lists
def test_block_placement_edges(gpu, orc, be, synth, T, E, TK, skew):
    """Sort, tile lists and permuted copy in one kernel: around its unit of 256 tokens,
    slots per token from one to 32, the most experts, remainders of every division, and
    the three-pass form where the router does not count."""
    H = 256
    cfg = dict(hidden=H, experts=E, moe_inter=128, shared_inter=128, top_k=TK)
    W = synth.host_weights(be, cfg, seed=T + E, sigma=0.9 / H ** 0.5)
    x = synth.host_x(be, T, H, seed=T)
    if skew:
        W, x = synth.apply_router_bias(W, x, synth.zipf_bias(cfg, seed=5))
    got = gpu.moe_block(cfg, W, x)
    assert gpu.last_block_status() == 0
    check_block(got, orc.moe_block(cfg, W, x), f"T={T} E={E} TK={TK}")


@pytest.mark.parametrize("sms", ["1", "2", "3"])
@pytest.mark.parametrize("T", [9, 65, 300])
def test_block_on_a_few_sms(be, orc, synth, monkeypatch, sms, T):
    """APUS_CUDA_SMS: grids for fewer SMs than there are, down to one (the placement kernel
    then has no CTA to spare for the copy; the expert kernels run side by side)."""
    cfg = dict(hidden=512, experts=64, moe_inter=128, shared_inter=128, top_k=8)
    W = synth.host_weights(be, cfg, seed=77, sigma=0.05)
    x = synth.host_x(be, T, cfg["hidden"], seed=T)
    monkeypatch.setenv("APUS_CUDA_SMS", sms)
    be.enable()
    try:
        got = be.moe_block(cfg, W, x)
        assert be.last_block_status() == 0
        check_block(got, orc.moe_block(cfg, W, x), f"T={T} on {sms} SMs")
    finally:
        be.disable()


@pytest.mark.parametrize("T", [1, 3, 4, 8])
def test_block_one_kernel_on_fewer_sms(be, orc, synth, monkeypatch, T):
    """128 SMs have three router rows each, which warps then take one by one, and columns of
    the down rows without a remainder."""
    cfg = dict(hidden=2048, experts=256, moe_inter=256, shared_inter=256, top_k=8)
    W = synth.host_weights(be, cfg, seed=78, sigma=0.02)
    W["rtr_w"][1::2] = W["rtr_w"][0::2]
    x = synth.host_x(be, T, cfg["hidden"], seed=T)
    monkeypatch.setenv("APUS_CUDA_SMS", "128")
    be.enable()
    try:
        got = be.moe_block(cfg, W, x)
        assert be.last_block_status() == 0 and be.last_block_launches() == 1
        check_block(got, orc.moe_block(cfg, W, x), f"T={T} on 128 SMs")
    finally:
        be.disable()


def test_block_batched_equals_per_token(gpu, be, synth):
    """tests/m9c of the reference: the batched body equals the per-token body.
    Here: selected ids are identical and outputs agree to BF16 tolerance when
    the same tokens go through one call or one call each."""
    cfg = synth.MINI_CFG
    W = synth.host_weights(be, cfg, seed=5, sigma=0.08)
    x = synth.host_x(be, 9, cfg["hidden"], seed=5)
    whole = gpu.moe_block(cfg, W, x)
    for t in range(9):
        one = gpu.moe_block(cfg, W, x[t:t + 1])
        assert np.array_equal(one["idx"][0], whole["idx"][t])
        assert np.array_equal(one["w"][0], whole["w"][t])
        assert np.abs(f32(one["out"][0]) - f32(whole["out"][t])).max() <= MAX_ABS


def test_block_skewed_router(gpu, orc, be, synth):
    """Configuration 3's skew, at a size the CPU checker finishes quickly: a
    Zipf(1.1) router bias realised through a constant-1 input channel."""
    cfg = dict(hidden=512, experts=64, moe_inter=128, shared_inter=128, top_k=8)
    W = synth.host_weights(be, cfg, seed=3, sigma=0.05)
    x = synth.host_x(be, 400, cfg["hidden"], seed=3)
    W, x = synth.apply_router_bias(W, x, synth.zipf_bias(cfg, seed=3, beta=1.0))
    got, exp = gpu.moe_block(cfg, W, x), orc.moe_block(cfg, W, x)
    check_block(got, exp, "skew")
    load = np.bincount(exp["idx"].ravel(), minlength=64)
    assert load.max() > 4 * load.mean()


@pytest.mark.parametrize("T,skew", [(8192, False), (8192, True), (8448, False)])
def test_block_full_size_rows_match_the_checker(gpu, orc, be, synth,
                                                qwen_weights, T, skew):
    """Benchmark configuration 3's shape on one GPU: 8192 tokens at the real
    dimensions, uniform and Zipf(1.1)-skewed routing.  Every token's result
    depends on that token alone, so the CPU checker runs on a seeded sample of
    rows (the full batch would take it minutes) and must agree with the rows of
    the full-size GPU call; the dispatch of the full batch is checked through
    its defining property."""
    cfg = synth.QWEN_CFG
    W = qwen_weights
    x = synth.host_x(be, T, cfg["hidden"], seed=31)
    if skew:
        W, x = synth.apply_router_bias(W, x, synth.zipf_bias(cfg, seed=31, beta=0.27))
    got = gpu.moe_block(cfg, W, x)
    assert gpu.last_block_status() == 0
    # the router's result for EVERY token (the CPU checker routes the whole
    # batch in under a second); full rows on a seeded sample
    ridx, rw = orc.route_batch(x, W["rtr_w"], cfg["top_k"])
    assert np.array_equal(got["idx"], ridx)
    assert (got["w"] != rw).mean() <= 0.002
    rows = np.sort(np.random.default_rng(31).choice(T, 96, replace=False))
    exp = orc.moe_block(cfg, W, x[rows])
    check_block({k: got[k][rows] for k in ("idx", "w", "routed", "shared", "out")},
                exp, f"T={T} skew={skew}")
    load = np.bincount(got["idx"].ravel(), minlength=cfg["experts"])
    assert load.sum() == T * cfg["top_k"]
    if skew:
        assert load.max() > 8 * load.mean()
    counts, offsets, perm = gpu.moe_dispatch(got["idx"], cfg["experts"])
    assert np.array_equal(perm, np.argsort(got["idx"].ravel(), kind="stable"))
    assert np.array_equal(counts, load)


def test_block_rejects_bad_arguments(gpu, be, synth):
    cfg = dict(synth.MINI_CFG)
    W = synth.host_weights(be, cfg, seed=1, sigma=0.08)
    x = synth.host_x(be, 2, cfg["hidden"], seed=1)
    bad = dict(cfg, hidden=cfg["hidden"] + 1)
    with pytest.raises(Exception):
        gpu.moe_block(bad, W, x)
    with pytest.raises(Exception):
        gpu.moe_block(dict(cfg, top_k=64), W, x)
    # still usable afterwards
    gpu.moe_block(cfg, W, x)


@pytest.mark.parametrize("T", [1, 3, 64, 300])
def test_block_replays_from_a_cuda_graph(gpu, orc, be, synth, qwen_weights, T):
    """The block on device pointers captured once and replayed: every counter
    the kernels hand work over with (decode barrier, per-expert completion
    counts of the expert GEMMs, router tickets) must be back in its initial
    state after a run, so the third replay equals the eager call bit for bit
    and the checker within tolerance."""
    import torch
    cfg = synth.QWEN_CFG
    x = synth.host_x(be, T, cfg["hidden"], seed=70 + T)
    layer = gpu.layer_create(cfg, qwen_weights)
    gpu.reserve(cfg, T)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        d_x = torch.from_numpy(x.view(np.int16)).cuda()
        d_eager = torch.empty_like(d_x)
        d_out = torch.empty_like(d_x)
        sp = stream.cuda_stream
        gpu.moe_block_dev(layer, d_x.data_ptr(), d_eager.data_ptr(), T, stream=sp)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            gpu.moe_block_dev(layer, d_x.data_ptr(), d_out.data_ptr(), T,
                              stream=torch.cuda.current_stream().cuda_stream)
        for _ in range(3):
            d_out.zero_()
            g.replay()
        torch.cuda.synchronize()
    assert gpu.last_block_status() == 0
    assert torch.equal(d_out, d_eager)
    exp = orc.moe_block(cfg, qwen_weights, x)
    a, b = f32(d_out.cpu().numpy().view(np.uint16)), f32(exp["out"])
    assert np.abs(a - b).max() <= MAX_ABS and rel_l2(a, b) <= REL_L2


@pytest.mark.parametrize("knob", ["APUS_CUDA_GEMM_OVERLAP", "APUS_CUDA_GEMM_DYNAMIC",
                                  "APUS_CUDA_PDL"])
def test_block_with_overlap_knobs_off(be, orc, synth, qwen_weights, knob, monkeypatch):
    """The plain kernel boundary between the two expert GEMMs, tiles assigned
    to CTAs by index instead of by an atomic counter, and no programmatic
    dependent launches at all, give the same block."""
    monkeypatch.setenv(knob, "0")
    be.enable()
    try:
        cfg = synth.QWEN_CFG
        x = synth.host_x(be, 200, cfg["hidden"], seed=91)
        check_block(be.moe_block(cfg, qwen_weights, x),
                    orc.moe_block(cfg, qwen_weights, x), knob + "=0")
        assert be.last_block_status() == 0
    finally:
        be.disable()


@pytest.mark.parametrize("T", [5, 16, 31, 32, 33, 64])
def test_block_few_tokens_without_gathered_rows(be, orc, synth, qwen_weights, T,
                                                monkeypatch):
    """Up to 64 tokens the gate_up kernel multiplies every expert's weights
    with all tokens of the block input and picks each row's column in its
    epilogue, instead of reading a gathered copy of the rows.  Same block as
    with the gathered copy, bit for bit, and within tolerance of the checker."""
    cfg = synth.QWEN_CFG
    x = synth.host_x(be, T, cfg["hidden"], seed=300 + T)
    outs = {}
    for knob in ("1", "0"):
        monkeypatch.setenv("APUS_CUDA_GEMM_DIRECT", knob)
        be.enable()
        try:
            outs[knob] = be.moe_block(cfg, qwen_weights, x)
            assert be.last_block_status() == 0
        finally:
            be.disable()
    for k in ("idx", "w", "routed", "shared", "out"):
        assert np.array_equal(outs["1"][k], outs["0"][k]), k
    check_block(outs["1"], orc.moe_block(cfg, qwen_weights, x), f"direct T={T}")


@pytest.mark.parametrize("T,E,TK,skew", [(300, 8, 4, False), (257, 8, 4, False),
                                         (1000, 8, 4, False), (1500, 16, 8, True),
                                         (129, 4, 4, False)])
@pytest.mark.parametrize("swap", ["0", "192", "256"])
def test_block_two_sm_gemm_path(be, orc, synth, monkeypatch, T, E, TK, skew, swap):
    """Many rows per expert: the GEMMs in which a pair of SMs shares a tile
    (tokens as the MMA's M, 256 per pair).  Checked against the CPU checker and,
    bit for bit, against the one-SM kernels on the same inputs (a row's result
    must not depend on the tiling).  swap: last chunks of fewer rows than this are
    multiplied with the rows as N — 0 none, 192 the default, 256 all."""
    monkeypatch.setenv("APUS_CUDA_PAIR_SWAP_BELOW", swap)
    cfg = dict(hidden=512, experts=E, moe_inter=128, shared_inter=128, top_k=TK)
    W = synth.host_weights(be, cfg, seed=60 + T, sigma=0.05)
    x = synth.host_x(be, T, cfg["hidden"], seed=60 + T)
    if skew:
        W, x = synth.apply_router_bias(W, x, synth.zipf_bias(cfg, seed=3, beta=0.6))
    exp = orc.moe_block(cfg, W, x)
    res = {}
    monkeypatch.setenv("APUS_CUDA_PAIR_MIN_ROWS", "64")   # default: 120 rows per expert
    for pair in ("1", "0"):
        monkeypatch.setenv("APUS_CUDA_PAIR", pair)
        be.enable()
        try:
            res[pair] = be.moe_block(cfg, W, x)
            assert be.last_block_status() == 0
            assert be.last_block_path() == (3 if pair == "1" else 2)
        finally:
            be.disable()
        check_block(res[pair], exp, f"pair={pair} T={T}")
    for k in ("idx", "w", "shared", "routed", "out"):
        assert np.array_equal(res["1"][k], res["0"][k]), k


def test_one_kernel_products_against_64_bit_sums(gpu, synth):
    """How often a product of the one-kernel path narrows to another BF16 value than its
    64-bit sum does: a measure of the fp32 sum's error that the narrowing does not hide.
    Scalar multiply-adds in fp32 gave 1.04e-4 (gate/up rows, K 2048) and 0.78e-4 (down rows,
    K 512); the bounds are five standard deviations of the counted events above that
    (4e6 x 1.04e-4 = 426 +- 21, 16e6 x 0.78e-4 = 1280 +- 36).

    One expert a token and weight 1; gate rows hold 64 for the constant channel, so that
    silu(g) = 64 exactly; down rows that pick one activation show 64 * bf16(u) itself."""
    import torch
    H, I, E, N, T = 2048, 512, 8, 8000, 8
    cfg = dict(hidden=H, experts=E, moe_inter=I, shared_inter=I, top_k=1)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)

    def rand(*s):
        return torch.randn(*s, device="cuda", generator=gen)

    def codes(t):
        return t.bfloat16().cpu().view(torch.int16).numpy().view(np.uint16)

    def narrowed(v):                    # fp64 -> BF16, one rounding
        b = v.contiguous().view(torch.int64)
        b = b + ((1 << 44) - 1) + ((b >> 45) & 1)
        return (b >> 45 << 45).view(torch.float64)

    gate = torch.zeros(E, I, H, device="cuda")
    gate[:, :, -1] = 64
    gu = torch.cat([gate, rand(E, I, H) * 0.02], 1).bfloat16()
    pick = torch.zeros(E, H, I, device="cuda")
    rows = torch.arange(H, device="cuda")
    pick[:, rows, rows % I] = 1
    down = (rand(E, H, I) * 0.02).bfloat16()
    none = np.zeros((I, H), np.uint16)
    W = dict(rtr_w=codes(rand(E, H) * 0.02), exp_gu=codes(gu), sh_g=none, sh_u=none,
             sh_d=none.reshape(H, I), sh_gate=np.zeros((1, H), np.uint16))
    x = rand(N, H)
    x = (x * torch.rsqrt(x.square().mean(1, keepdim=True))).bfloat16()
    x[:, -1] = 1
    idx = torch.empty((N, 1), dtype=torch.int32, device="cuda")

    def run(exp_d):
        layer = gpu.layer_create(cfg, dict(W, exp_d=codes(exp_d)))
        out = torch.empty_like(x)
        st = torch.cuda.current_stream().cuda_stream
        for t in range(0, N, T):
            gpu.moe_block_dev(layer, x[t].data_ptr(), out[t].data_ptr(), T, stream=st,
                              d_trace={"idx": idx[t].data_ptr()})
        torch.cuda.synchronize()
        assert gpu.last_block_path() == 0 and gpu.last_block_status() == 0
        gpu.layer_destroy(layer)
        return out.double()

    act, y = run(pick)[:, :I], run(down)
    wrong_u = wrong_y = 0
    for e in range(E):
        m = idx[:, 0] == e
        u = narrowed(x[m].double() @ gu[e, I:].double().T)
        wrong_u += int((act[m] / 64 != u).sum())
        wrong_y += int((y[m] != narrowed(act[m] @ down[e].double().T)).sum())
    assert wrong_u <= 1.30e-4 * N * I, wrong_u / (N * I)
    assert wrong_y <= 0.89e-4 * N * H, wrong_y / (N * H)
