"""GPU parity of the row-streaming kernels where their copies and splits can go wrong: scale rows at every alignment and
with gaps between them, row counts around the number of SMs, the shortest and longest reduction lengths, tile scales that
change inside a CTA's rows, and stages that run over the end of an expert."""
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def close(got, ref, what):
    got = got.float().cpu().numpy()
    err, cos = oracle.max_abs_rel(got, ref), oracle.cosine(got, ref)
    # bf16 output rounding (2^-9 of a value) and fp16 sums of four products inside a block
    assert err <= 5e-3 and cos >= 0.99999, f"{what}: max-abs/inf {err:.3e} cosine {cos:.7f}"


def vec(K, seed):
    return torch.randn(K, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16)


@pytest.mark.parametrize("K,N", [(32, 1), (32, 700), (1056, 147), (1056, 149), (2912, 1009), (8192, 5), (8192, 333), (512, 20000)])
def test_mxfp4_rows_and_lengths(rt, qz, K, N):
    p, s = qz.quantize_mxfp4(torch.randn(N, K, generator=torch.Generator().manual_seed(K + N)) * 0.02)
    x = vec(K, N)
    close(rt.mxfp4_gemv(p.to(DEV), s.to(DEV), x.to(DEV)), oracle.mxfp4_gemv_ref(p, s, x), f"{N}x{K}")


@pytest.mark.parametrize("shift", [0, 1, 7, 15])
@pytest.mark.parametrize("gap", [0, 3, 16])
def test_mxfp4_scale_rows_at_any_address(rt, qz, shift, gap):
    N, K = 401, 1312                                    # 41 scale bytes per row
    p, s = qz.quantize_mxfp4(torch.randn(N, K, generator=torch.Generator().manual_seed(gap)) * 0.02)
    x = vec(K, shift)
    buf = torch.full((shift + N * (K // 32 + gap) + 16,), 255, dtype=torch.uint8, device=DEV)
    view = buf[shift:shift + N * (K // 32 + gap)].view(N, K // 32 + gap)[:, : K // 32]
    view.copy_(s.to(DEV))
    close(rt.mxfp4_gemv(p.to(DEV), view, x.to(DEV)), oracle.mxfp4_gemv_ref(p, s, x), f"shift {shift} gap {gap}")


@pytest.mark.parametrize("kind", ["e8m0", "f32"])
@pytest.mark.parametrize("K,N", [(128, 384), (640, 128 * 160), (8192, 640), (8320, 256), (16384, 1280)])
def test_fp8_tile_scales(rt, qz, K, N, kind):
    w, s = qz.quantize_fp8_block128(torch.randn(N, K, generator=torch.Generator().manual_seed(K)) * 0.02, kind)
    s = (s.int() + torch.arange(s.numel()).view(s.shape) % 3).to(torch.uint8) if kind == "e8m0" else s * (1 + torch.arange(s.numel()).view(s.shape) % 3)
    x = vec(K, N)
    call = rt.fp8_e4m3_gemv if kind == "e8m0" else rt.fp8_e4m3_gemv_f32scale
    scale = torch.ldexp(torch.ones(s.shape), s.int() - 127) if kind == "e8m0" else s
    full = torch.repeat_interleave(torch.repeat_interleave(scale, 128, 0), 128, 1)
    ref = ((w.view(torch.float8_e4m3fn).float() * full) @ x.float()).numpy()
    close(call(w.to(DEV), s.to(DEV), x.to(DEV)), ref, f"{kind} {N}x{K}")


@pytest.mark.parametrize("E,K,H,O", [(1, 32, 32, 7), (8, 32, 32, 32), (5, 4096, 32, 300), (8, 1056, 480, 1056), (3, 96, 4096, 1), (7, 2880, 1440, 2880)])
def test_grouped_experts_across_stage_ends(rt, qz, E, K, H, O):
    g = torch.Generator().manual_seed(E + K)
    n = E + 3
    bank = {}
    for name, shape in (("w1", (n, H, K)), ("w3", (n, H, K)), ("w2", (n, O, H))):
        bank[name + "p"], bank[name + "s"] = qz.quantize_mxfp4(torch.randn(shape, generator=g) * 0.05)
    x, ids, r = vec(K, E), torch.randperm(n, generator=g)[:E], torch.rand(E, generator=g) + 0.1
    out = rt.mxfp4_grouped_gemv_ids({k: v.to(DEV) for k, v in bank.items()}, ids.to(torch.int32).to(DEV), x.to(DEV), r.to(DEV))
    sub = {k: v[ids] for k, v in bank.items()}
    close(out, oracle.grouped_gemv_ref(x, sub["w1p"], sub["w3p"], sub["w2p"], sub["w1s"], sub["w3s"], sub["w2s"], r), f"E={E} K={K} H={H}")
    assert rt.device_status() == 0


@pytest.mark.parametrize("K,N,G,S,gap", [
    (128, 128, 2, 2, 0),               # one K step: one warp per row tile
    (896, 2048, 8, 40, 0),             # 7 K steps over warps that do not divide them, several items per CTA, a last pass of 8 of 16 tokens
    (1152, 128, 200, 3, 16),           # 9 K steps, items of different groups, rows apart in memory
    (16384, 512, 1, 16, 0),            # activations in ranges
    (4224, 2176, 1, 9, 128),           # 33 K steps, tiles that do not fill the last item
    (1024, 4736, 1, 8, 0),
])
def test_fp8_several_tokens(rt, qz, K, N, G, S, gap):
    g = torch.Generator().manual_seed(K + N)
    w, s = qz.quantize_fp8_block128(torch.randn(G * N, K, generator=g) * 0.02, "e8m0")
    s = (s.int() + torch.arange(s.numel()).view(s.shape) % 3).to(torch.uint8)
    x = torch.randn(S, G * K, generator=g).to(torch.bfloat16)
    wide = torch.zeros(G * N, K + gap, dtype=w.dtype, device=DEV)
    wide[:, :K].copy_(w.to(DEV))
    y = rt.fp8_e4m3_gemv_batched(wide[:, :K], s.to(DEV), x.to(DEV), n_groups=G)
    scale = torch.ldexp(torch.ones(s.shape), s.int() - 127)
    for grp in {0, G // 2, G - 1}:
        r, b = slice(grp * N, (grp + 1) * N), slice(grp * N // 128, (grp + 1) * N // 128)
        full = w[r].view(torch.float8_e4m3fn).float() * torch.repeat_interleave(torch.repeat_interleave(scale[b], 128, 0), 128, 1)
        close(y[:, r], (x[:, grp * K:(grp + 1) * K].float() @ full.T).numpy(), f"group {grp} of {G}x{N}x{K}, {S} tokens")


@pytest.mark.parametrize("G,N,K", [
    (2, 1024, 512), (37, 128, 512),    # groups that divide 148 SMs
    (3, 2048, 896), (3, 2048, 1024),   # others, either side of 40 KB per SM
    (8, 1024, 4096), (147, 128, 512), (149, 128, 512), (300, 128, 384),
])
def test_fp8_groups_one_token(rt, qz, G, N, K):
    """One launch over G groups equals the G single calls bit for bit (the split of the reduction depends on K alone)."""
    g = torch.Generator().manual_seed(G)
    w, s = qz.quantize_fp8_block128(torch.randn(G * N, K, generator=g) * 0.02, "e8m0")
    s = (s.int() + torch.arange(s.numel()).view(s.shape) % 3).to(torch.uint8)
    x = torch.randn(G * K, generator=g).to(torch.bfloat16)
    w, s, x = w.to(DEV), s.to(DEV), x.to(DEV)
    y = rt.fp8_e4m3_gemv_batched(w, s, x, n_groups=G)
    single = [rt.fp8_e4m3_gemv(w[i * N:(i + 1) * N], s[i * N // 128:(i + 1) * N // 128], x[i * K:(i + 1) * K]) for i in range(G)]
    assert torch.equal(y.view(torch.int16), torch.cat(single).view(torch.int16))
    full = w[:N].cpu().view(torch.float8_e4m3fn).float()
    tiles = torch.ldexp(torch.ones(N // 128, K // 128), s[:N // 128].cpu().int() - 127)
    full = full * torch.repeat_interleave(torch.repeat_interleave(tiles, 128, 0), 128, 1)
    close(y[:N], (full @ x[:K].float().cpu()).numpy(), f"group 0 of {G}x{N}x{K}")
