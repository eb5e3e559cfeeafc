"""The persistent CTA-pair contractions at the sizes where their tiling can go wrong: token counts
around the 32-token batches and the 256-token tiles, weight rows that end inside a pair tile, a
reduction that ends inside a stage, K split over the pairs of a cluster, several tiles per pair
(accumulator rotation, overlapping accumulators), outputs that are not 16-byte aligned.  Expectation: the
f64 oracle on the codes the kernel read; bound: one BF16 rounding (2^-8 relative) plus fp32 summation,
asked for as 1e-2 of max(|expected|, floor) like the other projection tests."""
import numpy as np
import pytest
import torch

from gpu_util import assert_inactive_untouched, dev, graph_replay, host, max_relative_error, sentinel_plane

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tk():
    import tuiskollm_b200 as tk
    return tk


def _u16(t):
    return host(t.view(torch.int16)).view(np.uint16)


def _nvfp4_planes(tk, rows, k):
    return (torch.zeros((rows, k // 2), dtype=torch.uint8, device="cuda"),
            torch.zeros((tk.ops.nvfp4_scale_plane_bytes(rows, k),), dtype=torch.uint8, device="cuda"))


@pytest.mark.parametrize("out_rows,k,rows,tok,splits", [
    (256, 128, 33, 0, 0),      # one stage, one pair tile
    (1040, 1024, 64, 0, 0),    # weight rows end inside a pair tile
    (512, 1024, 301, 0, 0),    # ragged tokens, two tiles of 160
    (512, 1024, 257, 32, 1),   # smallest token tile
    (768, 2048, 100, 0, 2),    # K split in two
    (512, 4096, 130, 160, 4),  # K split in four, odd number of batches
    (40000, 256, 70, 64, 1),   # more tiles than pairs: three rounds of the two accumulators
    (512, 1024, 64, 0, 5),     # a split count no cluster has: the plan's own
])
def test_fp8_projection(tk, oracle, monkeypatch, out_rows, k, rows, tok, splits):
    from tuiskollm_b200 import synth

    monkeypatch.setenv("TK100_PAIR_TOK", str(tok))
    monkeypatch.setenv("TK100_PAIR_SPLITS", str(splits))
    c = tk.Context(device=0)
    xb = synth.normal_bf16(61, rows, (rows, k))
    w, s = synth.torch_fp8_weights(61, out_rows, out_rows, k, "cuda")
    codes = torch.zeros((rows, k), dtype=torch.uint8, device="cuda")
    scales = torch.zeros((rows,), dtype=torch.float32, device="cuda")
    out = sentinel_plane((rows + 1, out_rows), torch.int16)
    op = tk.ops.Fp8ProjectionOp(c)
    op.launch(None, rows, out_rows, k, dev(xb.view(np.int16)), codes, scales, w, s, out)
    torch.cuda.synchronize()
    assert c.last_kernel.startswith("pair_gemm_kernel"), c.last_kernel
    assert f"splits={splits if 1 <= splits <= 4 else 1}" in c.last_kernel, c.last_kernel
    assert c.device_status() == 0
    oc, os_ = oracle.quantize_e4m3(xb)
    assert np.array_equal(host(codes), oc)
    exp = oracle.fp8_projection(oc, os_, host(w), _u16(s))
    assert max_relative_error(_u16(out)[:rows], exp, 4 * float(np.abs(exp).mean())) <= 1e-2
    assert_inactive_untouched(out, rows)
    # an output plane that starts 2 bytes off a 16-byte boundary takes the narrow stores: same bits
    flat = sentinel_plane((rows * out_rows + 1,), torch.int16)
    op.launch(None, rows, out_rows, k, None, codes, scales, w, s, flat[1:])
    torch.cuda.synchronize()
    assert torch.equal(flat[1:].view(rows, out_rows), out[:rows])
    assert c.device_status() == 0


@pytest.mark.parametrize("tok,splits", [(64, 1), (160, 1), (256, 1), (160, 2), (256, 3), (224, 4)])
def test_one_tile_per_pair_has_the_bits_of_one_cta_tiles(tk, monkeypatch, tok, splits):
    """One tile per pair, more stages than the ring holds (which then reaches over the epilogue's transposition
    space), every place of a split's own values in the sum: the kernel of one-CTA tiles cuts K at the same places
    and adds the parts in the same order, so every output bit agrees."""
    from tuiskollm_b200 import synth

    out_rows, k, rows = 768, 5120, tok - 3
    xb = synth.normal_bf16(66, tok, (rows, k))
    w, s = synth.torch_fp8_weights(66, 1, out_rows, k, "cuda")
    outs = []
    for env in ({"TK100_PAIR_TOK": tok, "TK100_PAIR_SPLITS": splits}, {"TK100_SPLITS": splits, "TK100_BLOCK_TOK": 64}):
        for name in ("TK100_PAIR_TOK", "TK100_PAIR_SPLITS", "TK100_SPLITS", "TK100_BLOCK_TOK"):
            monkeypatch.setenv(name, str(env.get(name, 0)))
        c = tk.Context(device=0)
        codes = torch.zeros((rows, k), dtype=torch.uint8, device="cuda")
        scales = torch.zeros((rows,), dtype=torch.float32, device="cuda")
        out = sentinel_plane((rows + 1, out_rows), torch.int16)
        tk.ops.Fp8ProjectionOp(c).launch(None, rows, out_rows, k, dev(xb.view(np.int16)), codes, scales, w, s, out)
        torch.cuda.synchronize()
        kernel = "pair_gemm_kernel" if "TK100_PAIR_TOK" in env else "fp8_projection_kernel<64"
        assert c.last_kernel.startswith(kernel) and f"splits={splits}" in c.last_kernel, c.last_kernel
        assert c.device_status() == 0
        assert_inactive_untouched(out, rows)
        outs.append(out[:rows])
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("out_rows,k,rows,kernel", [
    (1040, 3072, 48, "fp8_projection_kernel<64"),    # three splits planned: one-CTA tiles up to 48 tokens
    (1040, 3072, 49, "pair_gemm_kernel"),
    (1040, 2048, 48, "pair_gemm_kernel"),     # two splits planned
    (1040, 4096, 64, "fp8_projection_kernel<64"),    # four splits planned: up to 64
    (1040, 4096, 65, "pair_gemm_kernel"),
    (768, 4096, 64, "pair_gemm_kernel"),
    (4096, 6144, 64, "fp8_projection_kernel<64"),    # three splits, but a long K
    (4096, 3072, 33, "fp8_projection_kernel<64"),    # most rows of the rule
    (4112, 3072, 33, "pair_gemm_kernel"),
    (5120, 256, 641, "fp8_pair_kernel"),             # 60 tiles in one wave, planned at 224 tokens
    (5120, 256, 576, "pair_gemm_kernel"),     # ... at 192
    (5136, 256, 700, "pair_gemm_kernel"),     # weight rows end inside a tile
    (8192, 2176, 256, "fp8_pair_kernel"),            # two splits planned
    (12288, 256, 256, "fp8_pair_kernel"),            # one wave where the plan takes two
    (8192, 512, 630, "fp8_pair_kernel"),             # 96 tiles in two waves of 160 tokens: K up to 512
    (8192, 640, 630, "pair_gemm_kernel"),
    (2560, 512, 2048, "pair_gemm_kernel"),    # a second wave mostly empty
    (8192, 256, 1281, "pair_gemm_kernel"),    # more tiles than two waves hold
])
def test_fp8_projection_route_rules(tk, oracle, out_rows, k, rows, kernel):
    """Both sides of each line between the pair kernel and the kernels it leaves a launch to."""
    from tuiskollm_b200 import synth

    c = tk.Context(device=0)
    xb = synth.normal_bf16(64, rows, (rows, k))
    w, s = synth.torch_fp8_weights(64, out_rows, out_rows, k, "cuda")
    codes = torch.zeros((rows, k), dtype=torch.uint8, device="cuda")
    scales = torch.zeros((rows,), dtype=torch.float32, device="cuda")
    out = sentinel_plane((rows + 1, out_rows), torch.int16)
    tk.ops.Fp8ProjectionOp(c).launch(None, rows, out_rows, k, dev(xb.view(np.int16)), codes, scales, w, s, out)
    torch.cuda.synchronize()
    assert c.last_kernel.startswith(kernel), c.last_kernel
    oc, os_ = oracle.quantize_e4m3(xb)
    exp = oracle.fp8_projection(oc, os_, host(w), _u16(s))
    assert max_relative_error(_u16(out)[:rows], exp, 4 * float(np.abs(exp).mean())) <= 1e-2
    assert_inactive_untouched(out, rows)
    assert c.device_status() == 0


@pytest.mark.parametrize("rows,tok,splits", [(33, 0, 0), (96, 0, 0), (129, 0, 0), (257, 0, 0), (300, 32, 0), (40, 0, 3)])
def test_fp8_swiglu(tk, oracle, monkeypatch, rows, tok, splits):
    from tuiskollm_b200 import synth

    monkeypatch.setenv("TK100_PAIR_TOK", str(tok))
    monkeypatch.setenv("TK100_PAIR_SPLITS", str(splits))  # gate/up does not split: its plan ignores it
    hidden, inter = 1024, 1280
    c = tk.Context(device=0, hidden=hidden, intermediate=inter)
    xb = synth.normal_bf16(62, rows, (rows, hidden))
    wc, ws = synth.fp8_weights(62, 1, 2 * inter, hidden)
    codes = torch.zeros((rows, hidden), dtype=torch.uint8, device="cuda")
    scales = torch.zeros((rows,), dtype=torch.float32, device="cuda")
    out = sentinel_plane((rows + 1, inter), torch.int16)
    tk.Fp8SwiGluOp(c).launch(None, rows, dev(xb.view(np.int16)), codes, scales, dev(wc), dev(ws.view(np.int16)), out)
    torch.cuda.synchronize()
    assert c.last_kernel.startswith("pair_gemm_kernel"), c.last_kernel
    assert c.device_status() == 0
    oc, os_ = oracle.quantize_e4m3(xb)
    dots = oracle.fp8_projection(oc, os_, wc, ws)
    exp = oracle.silu_mul(dots[:, :inter], dots[:, inter:])
    assert max_relative_error(_u16(out)[:rows], exp, 4 * float(np.abs(exp).mean())) <= 1e-2
    assert_inactive_untouched(out, rows)


@pytest.mark.parametrize("hidden,inter,rows,tok,splits", [
    (1024, 512, 33, 0, 0),
    (1024, 1664, 97, 0, 0),     # down: K = 1664 ends half-way into its last stage
    (1024, 1536, 160, 0, 0),
    (1024, 1536, 301, 128, 1),
    (1024, 512, 500, 256, 1),
    (256, 12800, 520, 256, 1),  # several tiles per pair on overlapping accumulators
    (256, 9728, 700, 128, 1),   # and on disjoint ones
    (512, 9472, 70, 0, 4),      # down: K split in four over 37 stages
])
def test_nvfp4_mlp(tk, oracle, monkeypatch, hidden, inter, rows, tok, splits):
    """gate/up + SwiGLU with the NVFP4 form of its output, then the down projection in both output
    types; codes and scales of the intermediate are the quantiser's bit for bit."""
    from tuiskollm_b200 import synth

    monkeypatch.setenv("TK100_PAIR_TOK", str(tok))
    xb = synth.normal_bf16(63, rows, (rows, hidden))
    gu, gus, gud = synth.nvfp4_weights(63, 1, 2 * inter, hidden)
    dn, dns, dnd = synth.nvfp4_weights(63, 2, hidden, inter)
    a_div, m_div = float(np.float32(448.0 * 6.0 / 5.0)), float(np.float32(448.0 * 6.0 / 8.0))
    monkeypatch.setenv("TK100_PAIR_SPLITS", str(splits))  # gate/up does not split: its plan ignores it
    c = tk.Context(device=0, hidden=hidden, intermediate=inter)
    a_codes, a_scales = _nvfp4_planes(tk, rows, hidden)
    m_codes, m_scales = _nvfp4_planes(tk, rows, inter)
    mid = sentinel_plane((rows + 1, inter), torch.int16)
    out = sentinel_plane((rows + 1, hidden), torch.int16)
    part = sentinel_plane((rows + 1, hidden), torch.float32)
    tk.Nvfp4SwiGluOp(c).launch_quantize(None, rows, dev(xb.view(np.int16)), dev(gu), dev(gus), float(gud), mid,
                                        activation_codes=a_codes, activation_scales=a_scales,
                                        input_global_divisor=a_div, output_global_divisor=m_div,
                                        output_codes=m_codes, output_scales=m_scales)
    assert c.last_kernel.startswith("pair_gemm_kernel") and "splits=1" in c.last_kernel, c.last_kernel
    down = tk.Nvfp4DownOp(c)
    kw = dict(activation_codes=m_codes, activation_scales=m_scales, input_global_divisor=m_div)
    down.launch(None, rows, None, dev(dn), dev(dns), float(dnd), out, **kw)
    if splits:
        assert f"splits={splits}" in c.last_kernel, c.last_kernel
    down.launch_partial(None, rows, None, dev(dn), dev(dns), float(dnd), part, **kw)
    torch.cuda.synchronize()
    assert c.device_status() == 0
    oc, osc = oracle.nvfp4_quantize(xb, a_div)
    dots = oracle.nvfp4_w4a4_dot(oc, osc, a_div, gu, gus, float(gud))
    exp_mid = oracle.silu_mul(dots[:, :inter], dots[:, inter:])
    got_mid = _u16(mid)[:rows]
    assert max_relative_error(got_mid, exp_mid, 4 * float(np.abs(exp_mid).mean())) <= 1e-2
    mc, msc = oracle.nvfp4_quantize(got_mid, m_div)
    assert np.array_equal(host(m_codes), mc)
    assert np.array_equal(host(m_scales), msc)
    exp = oracle.nvfp4_w4a4_dot(mc, msc, m_div, dn, dns, float(dnd))
    floor = 4 * float(np.abs(exp).mean())
    got = _u16(out)[:rows]
    assert max_relative_error(got, exp, floor) <= 1e-2
    got32 = host(part)[:rows]
    assert (np.abs(got32 - exp) / np.maximum(np.abs(exp), floor)).max() <= 2e-3
    assert np.array_equal(oracle.f32_to_bf16(got32), got)
    for plane in (mid, out, part):
        assert_inactive_untouched(plane, rows)


@pytest.mark.parametrize("hidden,inter,rows,kernel", [
    (5120, 6144, 33, "nvfp4_gemm_kernel"),      # three splits planned
    (5120, 6144, 64, "nvfp4_gemm_kernel"),
    (5120, 6144, 65, "pair_gemm_kernel"),
    (5120, 4352, 33, "pair_gemm_kernel"),   # two
    (1024, 2176, 80, "nvfp4_gemm_kernel"),      # few weight rows
    (1024, 2176, 81, "pair_gemm_kernel"),
    (1024, 2048, 64, "pair_gemm_kernel"),
    (1280, 2176, 64, "pair_gemm_kernel"),
])
def test_nvfp4_down_route_rules(tk, oracle, hidden, inter, rows, kernel):
    """Both sides of each line between the pair kernel and the one-CTA kernel, in both output types."""
    from tuiskollm_b200 import synth

    xb = synth.normal_bf16(65, rows, (rows, inter))
    dn, dns, dnd = synth.torch_nvfp4_weights(65, 2, hidden, inter, "cuda")
    div = float(np.float32(448.0 * 6.0 / 8.0))
    c = tk.Context(device=0, hidden=hidden, intermediate=inter)
    codes, scales = _nvfp4_planes(tk, rows, inter)
    out = sentinel_plane((rows + 1, hidden), torch.int16)
    part = sentinel_plane((rows + 1, hidden), torch.float32)
    down = tk.Nvfp4DownOp(c)
    kw = dict(activation_codes=codes, activation_scales=scales, input_global_divisor=div)
    down.launch(None, rows, dev(xb.view(np.int16)), dn, dns, float(dnd), out, **kw)
    assert c.last_kernel.startswith(kernel), c.last_kernel
    down.launch_partial(None, rows, None, dn, dns, float(dnd), part, **kw)
    assert c.last_kernel.startswith(kernel), c.last_kernel
    torch.cuda.synchronize()
    oc, osc = oracle.nvfp4_quantize(xb, div)
    exp = oracle.nvfp4_w4a4_dot(oc, osc, div, host(dn), host(dns), float(dnd))
    floor = 4 * float(np.abs(exp).mean())
    assert max_relative_error(_u16(out)[:rows], exp, floor) <= 1e-2
    got32 = host(part)[:rows]
    assert (np.abs(got32 - exp) / np.maximum(np.abs(exp), floor)).max() <= 2e-3
    for plane in (out, part):
        assert_inactive_untouched(plane, rows)
    assert c.device_status() == 0


@pytest.mark.parametrize("hidden,rows,inter,tok,rounds", [
    (5120, 1000, 6208, 0, 1),    # 80 tiles: a round of whole ones, 14 left over; a last stage of one step
    (5120, 1930, 4160, 0, 2),    # 160 tiles: two rounds, then split ones on the other accumulator's turn
    (5120, 1000, 3840, 0, 0),    # fewer than eight stages a split
    (5120, 700, 6208, 0, 0),     # 60 tiles in one round
    (24576, 100, 4160, 0, 1),    # 128-token tiles, whose accumulators are disjoint: 96 of them
    (19200, 200, 6208, 128, 2),  # 150: the split ones come when the first accumulator has been read twice
    (22528, 50, 6208, 0, 1),     # 88, three splits: up to 64 tokens too, where few tiles go to one-CTA tiles
])
def test_nvfp4_down_whole_tiles_then_split_ones(tk, oracle, monkeypatch, hidden, rows, inter, tok, rounds):
    """Tiles left over by the rounds of whole tiles are split over the pairs of a cluster (counts for 148 SMs: 74
    pairs, 33 clusters of two, 22 of three).  Against the unsplit plan: K / 64 accumulations on either side, each
    within 2^-23 of a partial sum, and partial sums within twice the largest result."""
    from tuiskollm_b200 import synth

    monkeypatch.setenv("TK100_PAIR_TOK", str(tok))
    xb = synth.normal_bf16(67, rows, (rows, inter))
    dn, dns, dnd = synth.torch_nvfp4_weights(67, 2, hidden, inter, "cuda")
    div = float(np.float32(448.0 * 6.0 / 8.0))
    codes, scales = _nvfp4_planes(tk, rows, inter)
    kw = dict(activation_codes=codes, activation_scales=scales, input_global_divisor=div)
    got = []
    for forced in (0, 1):
        monkeypatch.setenv("TK100_PAIR_SPLITS", str(forced))
        c = tk.Context(device=0, hidden=hidden, intermediate=inter)
        out = sentinel_plane((rows + 1, hidden), torch.int16)
        part = sentinel_plane((rows + 1, hidden), torch.float32)
        down = tk.Nvfp4DownOp(c)
        down.launch(None, rows, dev(xb.view(np.int16)), dn, dns, float(dnd), out, **kw)
        assert c.last_kernel.startswith("pair_gemm_kernel"), c.last_kernel
        assert c.last_kernel.endswith(f" rounds={rounds}") == (forced == 0 and rounds > 0), c.last_kernel
        assert ("splits=1" in c.last_kernel) == (forced == 1 or rounds == 0), c.last_kernel
        down.launch_partial(None, rows, None, dn, dns, float(dnd), part, **kw)
        torch.cuda.synchronize()
        first = out.clone()
        replay = graph_replay(lambda: down.launch(None, rows, None, dn, dns, float(dnd), out, **kw))
        replay.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, first)
        assert_inactive_untouched(out, rows)
        assert_inactive_untouched(part, rows)
        assert c.device_status() == 0
        assert np.array_equal(oracle.f32_to_bf16(host(part)[:rows]), _u16(out)[:rows])
        got.append(host(part)[:rows].astype(np.float64))
    bound = 2 * 2 * (inter / 64) * 2.0 ** -23 * np.abs(got[1]).max()
    assert np.abs(got[0] - got[1]).max() <= bound
    oc, osc = oracle.nvfp4_quantize(xb, div)
    tile = 128 * (inter // 16)  # scales of the last 128 weight rows
    exp = oracle.nvfp4_w4a4_dot(oc, osc, div, host(dn)[-128:], host(dns).reshape(-1)[-tile:], float(dnd))
    floor = 4 * float(np.abs(exp).mean())
    assert (np.abs(got[0][:, -128:] - exp) / np.maximum(np.abs(exp), floor)).max() <= 2e-3


def test_launches_on_two_streams_of_one_context_are_independent(tk):
    """A split tile meets in the cluster's shared memory, not in the context's scratch: launches that
    overlap on two streams leave the bits of launches one after the other."""
    from tuiskollm_b200 import synth

    out_rows, k, rows, count = 5120, 6144, 100, 12
    c = tk.Context(device=0)
    op = tk.ops.Fp8ProjectionOp(c)
    planes = []
    for i in range(2):
        w, s = synth.torch_fp8_weights(66, i, out_rows, k, "cuda")
        x = synth.torch_normal_bf16(66, 10 + i, (rows, k), "cuda")
        codes = torch.empty((rows, k), dtype=torch.uint8, device="cuda")
        scales = torch.empty((rows,), dtype=torch.float32, device="cuda")
        op.quantize(None, rows, k, x, codes, scales)
        planes.append((codes, scales, w, s, torch.empty((count, rows, out_rows), dtype=torch.int16, device="cuda")))

    def launch(i, n):
        codes, scales, w, s, out = planes[i]
        op.launch(None, rows, out_rows, k, None, codes, scales, w, s, out[n])

    want = []
    for i in range(2):
        launch(i, 0)
        assert "splits=3" in c.last_kernel and c.last_kernel.startswith("pair_gemm_kernel"), c.last_kernel
        want.append(planes[i][4][0].clone())
        planes[i][4].zero_()
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for n in range(count):
        for i in range(2):
            with torch.cuda.stream(streams[i]):
                launch(i, n)
    torch.cuda.synchronize()
    for i in range(2):
        assert bool((planes[i][4] == want[i]).all())
    assert c.device_status() == 0


def test_quantised_output_planes_are_held_to_the_quantisers_alignment(tk):
    """More than 32 rows: what the quantiser launch refuses, the epilogue's quantisation refuses."""
    rows, hidden, inter = 40, 256, 256
    c = tk.Context(device=0, hidden=hidden, intermediate=inter)
    codes, scales = _nvfp4_planes(tk, rows, hidden)
    w = torch.zeros((2 * inter, hidden // 2), dtype=torch.uint8, device="cuda")
    ws = torch.zeros((tk.ops.nvfp4_scale_plane_bytes(2 * inter, hidden),), dtype=torch.uint8, device="cuda")
    mid = torch.zeros((rows * inter + 8,), dtype=torch.bfloat16, device="cuda")
    m_codes = torch.zeros((rows * inter // 2 + 16,), dtype=torch.uint8, device="cuda")
    m_scales = torch.zeros((tk.ops.nvfp4_scale_plane_bytes(rows, inter) + 16,), dtype=torch.uint8, device="cuda")
    op = tk.Nvfp4SwiGluOp(c)
    for planes in ((mid[8:], m_codes, m_scales), (mid, m_codes[16:], m_scales), (mid, m_codes, m_scales[16:])):
        with pytest.raises(tk.GpuError) as info:
            op.launch_quantize(None, rows, None, w, ws, 1.0, planes[0], activation_codes=codes, activation_scales=scales,
                               input_global_divisor=1.0, output_global_divisor=1.0, output_codes=planes[1],
                               output_scales=planes[2])
        assert info.value.code == "gpu.launch"
    op.launch_quantize(None, rows, None, w, ws, 1.0, mid, activation_codes=codes, activation_scales=scales,
                       input_global_divisor=1.0, output_global_divisor=1.0, output_codes=m_codes, output_scales=m_scales)
    torch.cuda.synchronize()
    assert c.last_kernel.startswith("pair_gemm_kernel") and c.device_status() == 0
