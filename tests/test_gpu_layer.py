"""The block with its two neighbours folded in (c/layer.h:386-388):
res_out = rnd(res + moe_block(rmsnorm(res, 1 + ln_w))), one entry point, and a
stack of such layers in place on one residual stream.  Must equal, bit for bit,
the three separate calls (rmsnorm, block, residual add), which are themselves
checked against the CPU checker; and the CPU checker's chain directly."""
import numpy as np
import pytest

from test_gpu_block import check_block

pytestmark = pytest.mark.gpu

MID = dict(hidden=512, experts=64, moe_inter=128, shared_inter=128, top_k=8)


def f32(c):
    return (np.asarray(c, np.uint16).astype(np.uint32) << 16).view(np.float32)


def _dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int16)).cuda()


def _three_calls(gpu, torch, layer, d_res, d_w, T, H):
    ln = torch.empty_like(d_res)
    moe = torch.empty_like(d_res)
    out = torch.empty_like(d_res)
    gpu.rmsnorm_dev(d_res.data_ptr(), d_w.data_ptr() if d_w is not None else None,
                    ln.data_ptr(), T, H)
    gpu.moe_block_dev(layer, ln.data_ptr(), moe.data_ptr(), T)
    gpu.resadd_dev(d_res.data_ptr(), moe.data_ptr(), out.data_ptr(), T * H)
    torch.cuda.synchronize()
    return moe.cpu().numpy().view(np.uint16), out.cpu().numpy().view(np.uint16)


@pytest.mark.parametrize("T", [1, 2, 4, 5, 9, 80, 300])
@pytest.mark.parametrize("gains", [False, True])
def test_layer_equals_three_calls_and_the_checker(gpu, orc, be, synth, T, gains):
    import torch
    cfg, H = MID, MID["hidden"]
    W = synth.host_weights(be, cfg, seed=80, sigma=0.05)
    layer = gpu.layer_create(cfg, W)
    rng = np.random.default_rng(T)
    res = synth.f32_to_bf16(rng.normal(0, 1.7, (T, H)).astype(np.float32))
    lnw = synth.f32_to_bf16(rng.normal(0, 0.1, H).astype(np.float32)) if gains else None
    d_res = _dev(torch, res)
    d_w = _dev(torch, lnw) if gains else None
    moe3, out3 = _three_calls(gpu, torch, layer, d_res, d_w, T, H)
    d_out = torch.empty_like(d_res)
    d_tr = torch.empty_like(d_res)
    gpu.moe_layer_dev(layer, d_res.data_ptr(), d_w.data_ptr() if gains else None,
                      d_out.data_ptr(), T, d_trace={"out": d_tr.data_ptr()})
    torch.cuda.synchronize()
    assert gpu.last_block_status() == 0
    assert gpu.last_block_launches() == (1 if T <= 4 else gpu.last_block_launches())
    assert np.array_equal(d_out.cpu().numpy().view(np.uint16), out3)
    assert np.array_equal(d_tr.cpu().numpy().view(np.uint16), moe3)
    # the CPU checker's chain
    ln = orc.rmsnorm(res, lnw)
    exp = orc.resadd(res, orc.moe_block(cfg, W, ln)["out"])
    assert np.abs(f32(out3) - f32(exp)).max() <= 4e-2      # a BF16 step of |res + moe| ~ 4
    # in place
    d_in = d_res.clone()
    gpu.moe_layer_dev(layer, d_in.data_ptr(), d_w.data_ptr() if gains else None,
                      d_in.data_ptr(), T)
    torch.cuda.synchronize()
    assert np.array_equal(d_in.cpu().numpy().view(np.uint16), out3)


@pytest.mark.parametrize("T", [1, 3, 40])
def test_stack_in_place_equals_the_chain_of_calls(gpu, be, synth, T):
    import torch
    cfg, H, L = MID, MID["hidden"], 3
    layers = [gpu.layer_create(cfg, synth.host_weights(be, cfg, seed=81, layer=l, sigma=0.05))
              for l in range(L)]
    res = synth.host_x(be, T, H, seed=81)
    d = _dev(torch, res)
    ref = d.clone()
    for lay in layers:
        _, out = _three_calls(gpu, torch, lay, ref, None, T, H)
        ref = _dev(torch, out)
    gpu.moe_stack_dev(layers, d.data_ptr(), T)
    torch.cuda.synchronize()
    assert gpu.last_block_status() == 0
    assert np.array_equal(d.cpu().numpy(), ref.cpu().numpy())
    if T <= 4:
        assert gpu.last_block_launches() == L          # one kernel per layer


@pytest.mark.parametrize("T,E,I,TK,L", [
    (1, 64, 256, 8, 3), (8, 37, 256, 8, 2), (4, 256, 512, 8, 2), (5, 256, 256, 8, 3),
    (3, 8, 256, 8, 35), (8, 16, 512, 1, 2), (2, 5, 256, 3, 4)])
def test_stack_of_wide_rows_in_one_launch(gpu, be, synth, T, E, I, TK, L):
    """Layers of 2048 values, up to 32 to a launch: the bits of a call per step and layer.  Few
    and many experts a token shares, two and four slices of a down row, more items than places in
    the ring and fewer, a second launch for the layers left over."""
    import torch
    cfg = dict(hidden=2048, experts=E, moe_inter=I, shared_inter=I, top_k=TK)
    some = [gpu.layer_create(cfg, synth.host_weights(be, cfg, seed=82, layer=l, sigma=0.02))
            for l in range(min(L, 3))]
    layers = [some[l % len(some)] for l in range(L)]
    H = cfg["hidden"]
    gains = [_dev(torch, synth.f32_to_bf16(np.random.default_rng(l).normal(0, 0.1, H)
                                           .astype(np.float32))) for l in range(L)]
    ref = _dev(torch, synth.host_x(be, T, H, seed=82 + T))
    d = ref.clone()
    for lay, g in zip(layers, gains):
        _, out = _three_calls(gpu, torch, lay, ref, g, T, H)
        ref = _dev(torch, out)
    for _ in range(2):                       # the second call finds the first one's words
        x = d.clone()
        gpu.moe_stack_dev(layers, x.data_ptr(), T, d_ln_w=[g.data_ptr() for g in gains])
        torch.cuda.synchronize()
        assert gpu.last_block_status() == 0
        assert gpu.last_block_launches() == (L + 31) // 32
        assert np.array_equal(x.cpu().numpy(), ref.cpu().numpy())
    for lay in some:
        gpu.layer_destroy(lay)


@pytest.mark.parametrize("T,E,I,TK", [(1, 64, 256, 8), (8, 37, 256, 8), (5, 256, 256, 8),
                                      (3, 8, 256, 8), (8, 16, 512, 1), (2, 5, 256, 3)])
def test_stack_kernels_block_is_the_checkers(gpu, orc, be, synth, T, E, I, TK):
    """The comparison above is with block calls that run the same kernel at these shapes: here
    against the CPU checker, two calls in a row.  (Outputs stay below 4, where one BF16 step,
    2^-6, is below the largest difference allowed.)"""
    cfg = dict(hidden=2048, experts=E, moe_inter=I, shared_inter=I, top_k=TK)
    W = synth.host_weights(be, cfg, seed=82, sigma=0.02)
    for seed in (21, 22):
        x = synth.host_x(be, T, 2048, seed=seed)
        exp = orc.moe_block(cfg, W, x)
        assert np.abs(f32(exp["out"])).max() < 4
        got = gpu.moe_block(cfg, W, x)
        assert gpu.last_block_status() == 0 and gpu.last_block_launches() == 1
        check_block(got, exp, f"T={T} E={E} I={I}")


@pytest.fixture(scope="module")
def loud_weights(be, synth):
    """Three layers of a shape, made once: down rows four times as large as the others."""
    made = {}

    def get(E, I):
        if (E, I) not in made:
            cfg = dict(hidden=2048, experts=E, moe_inter=I, shared_inter=I, top_k=8)
            made.clear()
            made[E, I] = cfg, [synth.host_weights(be, cfg, seed=86, layer=l, sigma=0.02)
                               for l in range(3)]
            for W in made[E, I][1]:
                for name in ("exp_d", "sh_d"):
                    W[name] += np.where(W[name] & 0x7f80, 0x100, 0).astype(np.uint16)
        return made[E, I]
    return get


@pytest.mark.parametrize("T,E,I", [(1, 64, 256), (2, 160, 256), (3, 32, 512), (4, 48, 256),
                                   (8, 64, 256)])
@pytest.mark.parametrize("case", ["tied_rows", "tiny_logits", "opposite", "underflow"])
def test_stack_of_hard_routers_is_the_checkers(gpu, orc, be, synth, loud_weights, T, E, I, case):
    """Routers that leave the selection open, in the first layer of a launch and the ones behind it,
    which find the lists, masks and chains of the layer before.  The stack of n layers starts from
    what the stack of n - 1 gave, bit for bit, so each layer is checked by itself.

    The block's norm is 0.2 of the stream's and more here (asserted), of which each side's last
    narrowing is 2^-9 / sqrt(3) at most, 0.6 % of the block; with the block's own tolerance of 1 %
    2e-2 bounds the difference.  One of a token's experts left out is 0.08 of the block and more
    (the checker, these inputs), another in its place 1.4 times that."""
    import torch
    H, L = 2048, 3
    cfg, base = loud_weights(E, I)
    layers, weights = [], []
    for l in range(L):
        W = dict(base[l], rtr_w=base[l]["rtr_w"].copy())
        rtr = W["rtr_w"]
        if case == "tied_rows":
            rtr[1::2] = rtr[0::2]
        elif case == "tiny_logits":
            rtr[:] = synth.f32_to_bf16(synth.bf16_to_f32(rtr) * 2.0 ** -14)
        elif case == "opposite":            # the stream stays in pairs, so that every sum cancels
            rtr[:, 1::2] = rtr[:, 0::2] ^ 0x8000
            W["exp_d"] = np.repeat(W["exp_d"].reshape(E, H, I)[:, 0::2], 2, axis=1)
            W["sh_d"] = np.repeat(W["sh_d"].reshape(H, I)[0::2], 2, axis=0)
        else:
            rtr[:] = synth.f32_to_bf16(synth.bf16_to_f32(rtr) * 1e-36)
        weights.append(W)
        layers.append(gpu.layer_create(cfg, W))
    first = synth.host_x(be, T, H, seed=86 + T)
    if case == "opposite":
        first[:, 1::2] = first[:, 0::2]
    res = first
    for n in range(1, L + 1):
        y = _dev(torch, first)
        before = gpu.router_exact_chains()
        gpu.moe_stack_dev(layers[:n], y.data_ptr(), T)
        torch.cuda.synchronize()
        if case in ("opposite", "underflow"):       # (half of them at least, in every layer)
            assert gpu.router_exact_chains() - before >= n * T * E // (
                1 if case == "underflow" else 2)
        assert gpu.last_block_status() == 0 and gpu.last_block_launches() == 1
        got = y.cpu().numpy().view(np.uint16)
        exp = orc.resadd(res, orc.moe_block(cfg, weights[n - 1], orc.rmsnorm(res, None))["out"])
        diff = np.linalg.norm(f32(got) - f32(exp), axis=1)
        block = np.linalg.norm(f32(exp) - f32(res), axis=1)
        assert (block >= 0.2 * np.linalg.norm(f32(res), axis=1)).all()
        assert (diff <= 2e-2 * block).all(), (n, diff / block)
        res = got
    for lay in layers:
        gpu.layer_destroy(lay)


def test_stack_at_the_end_of_the_round_counter(gpu, be, synth):
    """The words that CTAs exchange carry the round counter as their tag, and the counter wraps:
    what eight tokens left there a turn ago is not this call's, in no row and at no place of the
    lists of chains.  (The middle layer's products underflow: all its logits are chains.)"""
    import torch
    T, H, L, END = 8, 2048, 3, 1 << 24
    cfg = dict(hidden=H, experts=64, moe_inter=256, shared_inter=256, top_k=8)
    layers = []
    for l in range(L):
        W = synth.host_weights(be, cfg, seed=83, layer=l, sigma=0.02)
        if l == 1:
            W["rtr_w"][:] = synth.f32_to_bf16(synth.bf16_to_f32(W["rtr_w"]) * 1e-36)
        layers.append(gpu.layer_create(cfg, W))

    def run(x, T, stack=layers):
        y = x.clone()
        gpu.moe_stack_dev(stack, y.data_ptr(), T)
        torch.cuda.synchronize()
        assert gpu.last_block_status() == 0
        return y

    a, b = (_dev(torch, synth.host_x(be, T, H, seed=s)) for s in (83, 84))
    want_a, want_b, want_1, want_32 = run(a, T), run(b, T), run(a, 1), run(b, 3, layers[::2] * 16)
    gpu.debug_decode_rounds(1000)
    assert torch.equal(run(a, T), want_a)
    gpu.debug_decode_rounds(END - 530)          # a launch of three layers takes five rounds
    for i in range(60):
        assert torch.equal(run(a, 1), want_1), i
    assert torch.equal(run(b, T), want_b)
    gpu.debug_decode_rounds(END - 30)
    assert torch.equal(run(b, 3, layers[::2] * 16), want_32)    # its tags on both sides
    assert torch.equal(run(a, 1), want_1)
    gpu.debug_decode_rounds(1000)
    assert torch.equal(run(b, T), want_b)       # the rounds, so the tags, of `a` above
    for lay in layers:
        gpu.layer_destroy(lay)


@pytest.mark.parametrize("T,L,cta", [(1, 1, 0), (3, 6, 5), (8, 32, 64), (8, 3, 147)])
def test_stack_with_a_part_that_never_comes(gpu, be, synth, T, L, cta):
    """A CTA that leaves at once, with router rows of its own (up to 64 here) and without: the
    others' waits for its logits run out, once for the whole launch, whatever its layers, tiles
    and cells; the status says so, and the next calls are right."""
    import time
    import torch
    H = 2048
    cfg = dict(hidden=H, experts=64, moe_inter=512, shared_inter=512, top_k=8)
    layer = gpu.layer_create(cfg, synth.host_weights(be, cfg, seed=85, sigma=0.02))
    d = _dev(torch, synth.host_x(be, T, H, seed=85))

    def run():
        y = d.clone()
        torch.cuda.synchronize()
        t = time.monotonic()
        gpu.moe_stack_dev([layer] * L, y.data_ptr(), T)
        torch.cuda.synchronize()
        return y, time.monotonic() - t

    want, _ = run()
    assert gpu.last_block_status() == 0
    gpu.debug_decode_absent(cta)
    _, took = run()
    assert gpu.last_block_status() == 4
    assert took < 10, took                   # 32 layers would wait for 32 and more
    for _ in range(3):
        got, _ = run()
        assert gpu.last_block_status() == 0 and torch.equal(got, want)
    gpu.layer_destroy(layer)


def test_layer_at_the_real_dimensions_one_token(gpu, orc, be, synth):
    import torch
    cfg = synth.QWEN_CFG
    layer = gpu.layer_create(cfg, None)
    synth.device_weights(gpu, layer, cfg, seed=5, layer=0)
    H = cfg["hidden"]
    res = synth.f32_to_bf16(np.random.default_rng(5).normal(0, 2.0, (1, H)).astype(np.float32))
    d_res = _dev(torch, res)
    moe3, out3 = _three_calls(gpu, torch, layer, d_res, None, 1, H)
    d_out = torch.empty_like(d_res)
    gpu.moe_layer_dev(layer, d_res.data_ptr(), None, d_out.data_ptr(), 1)
    torch.cuda.synchronize()
    assert gpu.last_block_launches() == 1
    assert np.array_equal(d_out.cpu().numpy().view(np.uint16), out3)


@pytest.mark.parametrize("H,I", [(208, 16), (512, 16), (768, 16), (1280, 16), (1536, 16),
                                 (2048, 16), (2048, 256)])
def test_one_kernel_norm_on_rows_made_to_go_wrong(gpu, be, synth, H, I):
    """The one-kernel path's norm, one warp or two to a row and lane chunks in registers or not,
    against the row kernel's in the layer's output: sums on the edge of a binade, ties in every
    add, a jump over binades, rising and falling terms.  (Last bits of the sum seldom show here:
    test_sum_of_squares_is_the_chains compares them.)"""
    import torch
    cfg = dict(hidden=H, experts=64, moe_inter=I, shared_inter=I, top_k=8)
    layer = gpu.layer_create(cfg, synth.host_weights(be, cfg, seed=H, sigma=0.05))
    rng = np.random.default_rng(H)
    rows = [np.ones(H), np.full(H, 1.0 + 2 ** -7), rng.integers(1, 4, H) * 0.5,
            np.where(np.arange(H) == H // 2, 1e3, rng.normal(0, 1, H)),
            np.exp2(np.linspace(6, -12, H)), np.exp2(np.linspace(-12, 6, H)),
            np.sign(rng.normal(0, 1, H)) * 181.0, rng.normal(0, 3, H)]
    rows += [rng.normal(0, 2.0 ** s, H) for s in range(-4, 4)]
    x = synth.f32_to_bf16(np.asarray(rows, np.float32))
    for at, T in ((0, 8), (8, 8), (2, 1), (5, 3)):
        d_res = _dev(torch, x[at:at + T])
        _, expected = _three_calls(gpu, torch, layer, d_res, None, T, H)
        d_out = torch.empty_like(d_res)
        gpu.moe_layer_dev(layer, d_res.data_ptr(), None, d_out.data_ptr(), T)
        torch.cuda.synchronize()
        assert gpu.last_block_launches() == 1 and gpu.last_block_status() == 0
        assert np.array_equal(d_out.cpu().numpy().view(np.uint16), expected)
    gpu.layer_destroy(layer)
