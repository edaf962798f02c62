"""Two contracts of the single-kernel decode path (csrc/decode_stream.cuh) that parity tests do not reach:

* re-entrancy: what its CTAs wait on lives in the caller's workspace, so two calls on two streams with two
  workspaces may overlap on the device and still give the bits of the same calls run one after the other;
* the give-up path of its bounded waits: a wait that cannot be satisfied ends after its poll budget, the kernel
  returns, the status is reported, the output rows are NaN, and the next ordinary call is bit-exact again.
  The unsatisfiable wait is made on the host side of the call (the service warps are told to expect tags that no
  producer writes); nothing faults, traps or spins without a limit.
"""
import importlib

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

K, H, E, k = 4096, 2048, 24, 6


@pytest.fixture(scope="module")
def case(qz):
    dev = torch.device("cuda:0")
    bank = qz.make_expert_bank(E, K, H, dev, seed=321)
    g = torch.Generator(device=dev).manual_seed(7)
    xs = [torch.randn(K, generator=g, device=dev).to(torch.bfloat16) for _ in range(8)]
    logits = [torch.randn(E, generator=g, device=dev) for _ in range(8)]
    return dev, bank, xs, logits


def test_two_streams_two_workspaces_equal_serial_calls(rt, case):
    """Default launch mode.  The two streams are released together by an event, so their grids are in flight at
    the same time; each call has its own workspace, which is all the entry's contract asks for."""
    dev, bank, xs, logits = case
    gb = importlib.import_module("dsv4_b200.runtime.mxfp4_grouped_gemv_binding")
    n = len(xs)
    serial = [rt.moe_decode_layer(bank, logits[i], xs[i], k=k, score_func="softmax").clone() for i in range(n)]
    torch.cuda.synchronize()
    ws = [torch.empty(rt.decode_workspace_bytes(k, H, K), dtype=torch.uint8, device=dev) for _ in range(2)]
    outs = [torch.empty(K, dtype=torch.bfloat16, device=dev) for _ in range(n)]
    streams = [torch.cuda.Stream(device=dev) for _ in range(2)]
    for rep in range(3):
        go = torch.cuda.Event()
        blocker = torch.empty(1 << 26, dtype=torch.float32, device=dev)
        blocker.normal_()                       # some work on the default stream in front of the event
        go.record()
        for s, stream in enumerate(streams):
            with torch.cuda.stream(stream):
                stream.wait_event(go)
                for i in range(s, n, 2):        # stream 0: even calls, stream 1: odd calls, each with its own workspace
                    rt.moe_decode_layer(bank, logits[i], xs[i], k=k, score_func="softmax", out=outs[i], workspace=ws[s])
        torch.cuda.synchronize()
        for i in range(n):
            assert torch.equal(outs[i].view(torch.int16), serial[i].view(torch.int16)), (rep, i)
    assert gb.device_status() == 0


def test_bounded_wait_gives_up_reports_and_recovers(rt, case):
    dev, bank, xs, logits = case
    gb = importlib.import_module("dsv4_b200.runtime.mxfp4_grouped_gemv_binding")
    ws = torch.empty(rt.decode_workspace_bytes(k, H, K), dtype=torch.uint8, device=dev)
    good = rt.moe_decode_layer(bank, logits[0], xs[0], k=k, score_func="softmax", workspace=ws).clone()
    torch.cuda.synchronize()
    assert gb.device_status() == 0
    gb.debug_wait_limits(2000, 1)               # 2000 polls, and tags that no producer writes
    try:
        bad = rt.moe_decode_layer(bank, logits[0], xs[0], k=k, score_func="softmax", workspace=ws).clone()
        torch.cuda.synchronize()                # the kernel has returned: its waits ran out, it did not hang
    finally:
        gb.debug_wait_limits(0, 0)
    assert gb.device_status() == 3              # reported ...
    assert gb.device_status() == 0              # ... and cleared by the read
    assert torch.isnan(bad.float()).all()       # the damage is visible in the output, not silent
    again = rt.moe_decode_layer(bank, logits[0], xs[0], k=k, score_func="softmax", workspace=ws)
    torch.cuda.synchronize()
    assert torch.equal(again.view(torch.int16), good.view(torch.int16))
    ids, w = oracle.route_softmax(logits[0].cpu().numpy()[None], k)
    sub = {n_: v[torch.from_numpy(ids[0].astype(np.int64)).to(dev)].cpu() for n_, v in bank.items()}
    ref = oracle.moe_layer_ref(xs[0].cpu()[None], sub, np.arange(k)[None], w)[0]
    got = again.float().cpu().numpy()
    assert oracle.max_abs_rel(got, ref) <= 1e-2 and oracle.cosine(got, ref) >= 0.9999
    assert gb.device_status() == 0


def test_row_streaming_gives_up_with_nan_rows(rt, qz):
    """The dense GEMVs and the routed FFN of the other shapes (csrc/row_stream.cuh): the last stage of every CTA is not
    requested, so the wait for it runs out; the status is reported, the rows that depend on it are NaN, the others right, and
    the next call is bit-exact."""
    capi = importlib.import_module("dsv4_b200.runtime._capi")
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(5)

    def act(n):
        return torch.randn(n, generator=g, device=dev).to(torch.bfloat16)

    x4, p4 = act(2912), qz.quantize_mxfp4((torch.randn(3000, 2912, generator=g, device=dev) * 0.02).to(torch.bfloat16))
    x8, p8 = act(4096), qz.quantize_fp8_block128(torch.randn(2048, 4096, generator=g, device=dev) * 0.02)
    shared = {}
    for name, n, k_ in (("w1", 1024, 2048), ("w3", 1024, 2048), ("w2", 2048, 1024)):
        shared[name], shared[name + "s"] = qz.quantize_fp8_block128(torch.randn(n, k_, generator=g, device=dev) * 0.02)
    xs, bank, xg = act(2048), qz.make_expert_bank(6, 2880, 1440, dev, seed=3), act(2880)
    stacked = [{"packed": bank[n + "p"], "scale": bank[n + "s"]} for n in ("w1", "w3", "w2")]
    r = torch.rand(6, generator=g, device=dev) + 0.1
    mxfp4, fp8, grouped = capi.load("mxfp4"), capi.load("fp8"), capi.load("grouped")
    cases = [
        ("mxfp4", lambda: rt.mxfp4_gemv(*p4, x4), mxfp4.mxfp4_gemv_test_wait_limits, mxfp4.mxfp4_gemv_device_status, (2,)),
        ("fp8", lambda: rt.fp8_e4m3_gemv(*p8, x8), fp8.fp8_e4m3_gemv_test_wait_limits, fp8.fp8_e4m3_gemv_device_status, (2,)),
        ("fp8 groups", lambda: rt.fp8_e4m3_gemv_batched(*p8, torch.cat((x8, x8)).view(1, -1), n_groups=2),
         fp8.fp8_e4m3_gemv_test_wait_limits, fp8.fp8_e4m3_gemv_device_status, (2,)),
        ("shared expert", lambda: rt.fp8_shared_swiglu(shared, xs), fp8.fp8_e4m3_gemv_test_wait_limits,
         fp8.fp8_e4m3_gemv_device_status, (2,)),
        ("stacked experts", lambda: rt.mxfp4_grouped_gemv(*stacked, None, xg, r), grouped.dsv4_b200_test_wait_limits,
         grouped.dsv4_b200_device_status, (1, 2)),
    ]
    for what, call, limits, status, codes in cases:
        good = call().clone()
        torch.cuda.synchronize()
        assert status() == 0, what
        try:
            assert limits(-1, 0) == -1 and limits(0, -1) == -1
            assert limits(2000, 1) == 0
            bad = call().clone()
            assert status() in codes, what      # (synchronises: the kernel has returned)
            assert status() == 0, what
            nan = torch.isnan(bad.float())      # the last stage's rows, or all where they feed a second product; no row is silently wrong
            assert nan.any() and torch.equal(bad[~nan].view(torch.int16), good[~nan].view(torch.int16)), what
            assert limits(2000, 64) == 0        # every stage
            bad = call().clone()
            assert status() in codes, what
            assert torch.isnan(bad.float()).all(), what
        finally:
            limits(0, 0)
        again = call()
        torch.cuda.synchronize()
        assert torch.equal(again.view(torch.int16), good.view(torch.int16)) and status() == 0, what
