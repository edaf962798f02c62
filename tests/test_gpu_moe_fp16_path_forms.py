"""The batched layer's path "fp16" in both its forms, E4M3 terms on block-scaled MMAs and fp16 MMAs, at the edges of the rule that chooses
between them and of the tiles of the first, against 64 bits and against each other."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
LUT = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6, -0., -.5, -1, -1.5, -2, -3, -4, -6], dtype=torch.float64)


def dense(p, s):
    v = torch.stack([LUT.to(p.device)[(p & 15).long()], LUT.to(p.device)[(p >> 4).long()]], -1).flatten(-2)
    return v * torch.ldexp(torch.ones(s.shape, dtype=torch.float64, device=p.device), s.int() - 127).repeat_interleave(32, -1)


def layer64(bank, x, ids, w):
    out = torch.zeros(x.shape[0], bank["w2p"].shape[1], dtype=torch.float64, device=x.device)
    for e in range(bank["w1p"].shape[0]):
        t, j = (ids == e).nonzero(as_tuple=True)
        if len(t):
            a, b = (x[t].double() @ dense(bank[n + "p"][e], bank[n + "s"][e]).T for n in ("w1", "w3"))
            out.index_add_(0, t, ((a * torch.sigmoid(a) * b) @ dense(bank["w2p"][e], bank["w2s"][e]).T) * w[t, j].double()[:, None])
    return out


def beside_rounding(out, ref):
    """The largest error of a token beside the rounding of its values to bf16, of its norm."""
    rounding = (ref.to(torch.bfloat16).double() - ref).norm(dim=1)
    return (((out.double() - ref).norm(dim=1) ** 2 - rounding ** 2).clamp(min=0).sqrt() / (ref.norm(dim=1) + 1e-300)).max().item()


# What the intermediate is held in beside the output's rounding: three terms of four bits, which leave 2^-13 of a value; or 11 bits (fp16, and
# one bit more where a row lies low in its range).
TERMS, HALF = 2.0 ** -13, 2 * 2.0 ** -11 / 3 ** 0.5


@pytest.mark.parametrize("counts,K,H,O", [
    ([1, 0, 15, 16], 256, 256, 256),             # two stages a tile, one run of scale bytes cut short
    ([24, 24, 24, 24], 1280, 512, 1280),         # the most pairs for tiles of 32 tokens
    ([25, 24, 24, 24], 1280, 512, 1280),         # one more
    ([17, 31, 32, 33] + [0] * 4, 2304, 768, 2304),
    ([64, 65, 1, 30] + [0] * 4, 4096, 2048, 4096),          # three tokens tiles of an expert
    ([80, 80, 80, 80], 768, 1280, 768),          # the most for the E4M3 form
    ([112, 97, 48, 62], 512, 256, 640),          # a quarter tile of output rows
    ([130, 33, 96, 49], 4096, 512, 4096),
    ([81, 80, 80, 80], 512, 256, 512),           # fp16 MMAs
    ([40, 9], 256, 1280, 256),                   # no room for the terms of the intermediate
    ([40, 9], 1280, 256, 384),                   # nor of x
    # 64 experts with 320 tiles in either GEMM: four or five for each of 74 CTA pairs, of differing token widths, the last of an expert's down
    # tiles half empty; of 32 and of 112 tokens, and with fp16 MMAs of 64 and of 128
    ([i * 7 % 41 for i in range(64)], 2304, 1280, 2304),
    ([i * 37 % 121 for i in range(64)], 2304, 1280, 2304),
])
def test_forms_agree(rt, qz, odd_bank, counts, K, H, O):
    g = torch.Generator(device=DEV).manual_seed(sum(counts) + K)
    E, T = len(counts), sum(counts)
    bank = qz.make_expert_bank(E, K, H, DEV, seed=K)
    if O != K:
        bank["w2p"], bank["w2s"] = qz.quantize_mxfp4((torch.randn(E, O, H, generator=g, device=DEV) * 0.02).to(torch.bfloat16))
    bank["w1s"] += (torch.arange(bank["w1s"].numel(), device=DEV).view(bank["w1s"].shape) % 5).to(torch.uint8)        # scales that differ along K
    ids = torch.repeat_interleave(torch.arange(E, device=DEV), torch.tensor(counts, device=DEV))
    ids = ids[torch.randperm(T, generator=g, device=DEV)].to(torch.int32)[:, None].contiguous()
    w = torch.rand(T, 1, generator=g, device=DEV) + 0.5
    x = (torch.randn(T, K, generator=g, device=DEV) * torch.exp2(torch.randn(T, 1, generator=g, device=DEV) * 3)).to(torch.bfloat16)
    x[T // 2, :64] = 0
    one = rt.moe_forward(bank, x, ids, w, path="fp16")
    other = rt.moe_forward(odd_bank(bank), x, ids, w, path="fp16")
    again = rt.moe_forward(bank, x, ids, w, path="fp16")
    assert rt.moe_device_status() == 0
    assert torch.equal(one.view(torch.int16), again.view(torch.int16))
    ref = layer64(bank, x, ids, w)
    terms = T <= 80 * E and 99 * (K // 32) <= 128 * (O // 32) and 99 * H <= 64 * (K + H)
    for out, bound in ((one, TERMS if terms else HALF), (other, HALF)):
        worst = beside_rounding(out, ref)
        assert worst <= bound, f"{counts} {K} {H} {O}: {worst:.2e} of a token's norm beside the rounding, {bound:.2e} allowed"


@pytest.mark.parametrize("counts", [[24] * 4, [60] * 4])
def test_wide_range_of_x(rt, qz, counts):
    """Elements 2^14 below the largest of their 32 keep their eight bits: one channel of 32 that much larger, its weights zero."""
    g = torch.Generator(device=DEV).manual_seed(len(counts))
    K, H, E, T = 1024, 512, len(counts), sum(counts)
    bank = qz.make_expert_bank(E, K, H, DEV, seed=3)
    x = torch.randn(T, K, generator=g, device=DEV)
    x[:, 5::32] *= 2.0 ** 14
    x = x.to(torch.bfloat16)
    for n in ("w1p", "w3p"):
        bank[n][:, :, 2::16] &= 0x0f                       # odd elements are the high nibbles
    ids = torch.repeat_interleave(torch.arange(E, device=DEV), torch.tensor(counts, device=DEV)).to(torch.int32)[:, None].contiguous()
    w = torch.ones(T, 1, device=DEV)
    out = rt.moe_forward(bank, x, ids, w, path="fp16").double()
    ref = layer64(bank, x, ids, w)
    rounding = (ref.to(torch.bfloat16).double() - ref).norm() / ref.norm()
    assert ((out - ref).norm() / ref.norm()) ** 2 <= rounding ** 2 + 2.0 ** -26


@pytest.mark.parametrize("n", [24, 60])
@pytest.mark.parametrize("up,down,of_x", [
    (64, -100, [0]), (0, -110, [66]), (100, -110, [-30]),       # silu(G) * U beyond FP32,
    (0, -110, [100]), (-70, 100, [0]), (-30, 100, [-40]), (0, 110, [-90]),      # and below its smallest normal value
    (8, 0, [30, -30, 0, 17, -17, 16]),                          # normalised tokens beside others
])
def test_range_of_the_intermediate(rt, qz, odd_bank, n, up, down, of_x):
    """Scales of x (powers of two, token by token) and of W1 and W3 that take silu(G) * U out of the range of FP32, and scales of W2 that
    bring the result back into that of bf16."""
    E, K, H = 4, 1024, 512
    T = E * n
    g = torch.Generator(device=DEV).manual_seed(n)
    bank = qz.make_expert_bank(E, K, H, DEV, seed=5)
    for name, d in (("w1s", up), ("w3s", up), ("w2s", down)):
        bank[name] = (bank[name].int() + d).to(torch.uint8)
    ids = torch.repeat_interleave(torch.arange(E, device=DEV), n).to(torch.int32)[:, None].contiguous()
    w = torch.rand(T, 1, generator=g, device=DEV) + 0.5
    e = torch.tensor(of_x, device=DEV)[torch.arange(T, device=DEV) % len(of_x)]
    x = (torch.randn(T, K, generator=g, device=DEV) * torch.exp2(e.float())[:, None]).to(torch.bfloat16)
    ref = layer64(bank, x, ids, w)
    assert 1e-37 < ref.norm(dim=1).min() and ref.abs().max() < 2.0 ** 127
    for b, bound in ((bank, TERMS), (odd_bank(bank), HALF)):
        out = rt.moe_forward(b, x, ids, w, path="fp16")
        assert torch.isfinite(out).all()
        worst = beside_rounding(out, ref)
        assert worst <= bound, f"{worst:.2e} of a token's norm beside the rounding, {bound:.2e} allowed"
    assert rt.moe_device_status() == 0


@pytest.mark.parametrize("T,K,E,k,O", [
    (80, 1024, 36, 33, 1024),                    # more pairs per token than a warp has lanes
    (1800, 4096, 32, 1, 4096),                   # a row to a block, the blocks three rows each
    (9000, 768, 128, 1, 768),                    # four rows to a block, the same
    (1000, 5120, 16, 1, 5120), (700, 9472, 10, 1, 9472),          # two and four pieces of a row a lane, the last cut short
])
def test_terms_of_many_tokens(rt, qz, T, K, E, k, O):
    """x as three E4M3 terms where a block of the quantiser takes one row after another, and rows longer than it takes at once."""
    H = 256
    g = torch.Generator(device=DEV).manual_seed(T + K)
    bank = qz.make_expert_bank(E, K, H, DEV, seed=K)
    ids = torch.stack([torch.randperm(E, generator=g, device=DEV)[:k] for _ in range(T)]).to(torch.int32) if k > 1 else \
        (torch.randperm(T, generator=g, device=DEV) % E).to(torch.int32)[:, None].contiguous()
    w = torch.rand(T, k, generator=g, device=DEV) + 0.5
    x = (torch.randn(T, K, generator=g, device=DEV) * torch.exp2(torch.randn(T, 1, generator=g, device=DEV) * 9)).to(torch.bfloat16)
    x[3, :64], x[4] = 0, 0
    x[T - 1, K - 1] = float("inf")
    out = rt.moe_forward(bank, x, ids, w, path="fp16")
    assert rt.moe_device_status() == 0
    assert torch.isnan(out[T - 1]).all() and torch.isfinite(out[:T - 1]).all() and not out[4].any()
    worst = beside_rounding(out[:T - 1], layer64(bank, x[:T - 1], ids[:T - 1], w[:T - 1]))
    assert worst <= TERMS, f"{worst:.2e} of a token's norm beside the rounding, {TERMS:.2e} allowed"


@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("counts,K,H", [([12] * 4, 1280, 512), ([33, 1, 0, 60], 2304, 768), ([40] * 4, 512, 256), ([0] * 7 + [97], 256, 256)])
def test_unusual_values_in_both_forms(rt, qz, odd_bank, odd, counts, K, H):
    """Scale bytes 0xFF, some blocks and all of a row, which contribute nothing; pairs that are skipped, some and all of a token's; tokens
    2^20 and 2^-20 the size of others, of zeros, and not finite."""
    E, n = len(counts), sum(counts)
    g = torch.Generator(device=DEV).manual_seed(n + K)
    bank = qz.make_expert_bank(E, K, H, DEV, seed=K)
    clean = {name: t.clone() for name, t in bank.items()}
    for name, rows in (("w1", slice(1, None, 5)), ("w3", slice(2, None, 7)), ("w2", slice(0, None, 7))):
        bank[name + "s"][:, rows, 1] = 255
        bank[name + "s"][:, 3] = 255
        clean[name + "p"][(bank[name + "s"] == 255).repeat_interleave(16, -1)] = 0
    ids = torch.repeat_interleave(torch.arange(E, device=DEV), torch.tensor(counts, device=DEV)).to(torch.int32)[:, None]
    ids = torch.cat([ids, (ids + 1) % E], 1)                   # two pairs a token (80 an expert at most), a third of them skipped
    ids[torch.rand(n, 2, generator=g, device=DEV) < 0.33] = -1
    ids[7] = -1
    w = torch.rand(n, 2, generator=g, device=DEV) + 0.5
    x = torch.randn(n, K, generator=g, device=DEV)
    x[1::5] *= 2.0 ** 20
    x[2::5] *= 2.0 ** -20
    x = x.to(torch.bfloat16)
    x[6], x[n // 2, 7], ids[n // 2, 0] = 0, float("inf"), 0
    out = rt.moe_forward(odd_bank(bank) if odd else bank, x, ids.contiguous(), w, path="fp16")
    assert rt.moe_device_status() == 0
    assert not torch.isfinite(out[n // 2]).all() and not out[6].any() and not out[7].any()
    rest = torch.arange(n, device=DEV) != n // 2
    worst = beside_rounding(out[rest], layer64(clean, x[rest], ids[rest], w[rest]))
    bound = HALF if odd else TERMS
    assert worst <= bound, f"{worst:.2e} of a token's norm beside the rounding, {bound:.2e} allowed"
