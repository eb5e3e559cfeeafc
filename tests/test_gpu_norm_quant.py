"""GPU parity: fused residual-add + RMSNorm + per-token E4M3 quantisation against the CPU
oracle, following qual/src/residual_norm.rs (exact batches, sentinels, graph replay)."""
import ctypes

import numpy as np
import pytest
import torch

import fixtures_ref as F
from gpu_util import (assert_inactive_untouched, check_close, dev, graph_replay, host,
                      sentinel_plane)

pytestmark = pytest.mark.gpu

MAX_ROWS = 8


@pytest.fixture(scope="module")
def tk():
    import tuiskollm_b200 as tk
    return tk


@pytest.fixture(scope="module")
def ctx(tk):
    return tk.Context(device=0)


def _u16(t):
    return host(t.view(torch.int16)).view(np.uint16)


def run_all(tk, ctx, x, b, w, rows, max_rows, hidden):
    op = tk.ResidualNormOp(ctx)
    plain = sentinel_plane((max_rows, hidden), torch.int16)
    res = sentinel_plane((max_rows, hidden), torch.int16)
    norm = sentinel_plane((max_rows, hidden), torch.int16)
    fres = sentinel_plane((max_rows, hidden), torch.int16)
    fnorm = sentinel_plane((max_rows, hidden), torch.int16)
    codes = sentinel_plane((max_rows, hidden), torch.uint8)
    scales = sentinel_plane((max_rows,), torch.float32)
    pcodes = sentinel_plane((max_rows, hidden), torch.uint8)
    pscales = sentinel_plane((max_rows,), torch.float32)
    pnorm = sentinel_plane((max_rows, hidden), torch.int16)

    def launch():
        op.launch_plain(None, rows, x, w, plain)
        op.launch_residual(None, rows, x, b, w, res, norm)
        op.launch_quantize(None, rows, x, b, w, fres, fnorm, codes, scales)
        op.launch_quantize(None, rows, x, None, w, None, pnorm, pcodes, pscales)

    planes = dict(plain=plain, res=res, norm=norm, fres=fres, fnorm=fnorm, codes=codes,
                  scales=scales, pcodes=pcodes, pscales=pscales, pnorm=pnorm)
    return launch, planes


def verify(oracle, planes, xb, bb, wb, rows, eps):
    res_o, norm_o = oracle.residual_rms_norm(xb[:rows], bb[:rows], wb, eps)
    _, plain_o = oracle.residual_rms_norm(xb[:rows], None, wb, eps)
    plain = _u16(planes["plain"])
    res, norm = _u16(planes["res"]), _u16(planes["norm"])
    fres, fnorm, pnorm = _u16(planes["fres"]), _u16(planes["fnorm"]), _u16(planes["pnorm"])
    # residual publication is bit exact (qual/src/residual_norm.rs:236-243)
    assert np.array_equal(res[:rows], res_o)
    assert np.array_equal(fres[:rows], res_o)
    # norm within max(1/64, 0.5 %) of the f64 oracle (qual/src/residual_norm.rs:364)
    f64 = lambda bits: oracle.bf16_to_f32(bits).astype(np.float64)
    worst = max(check_close(plain[:rows], f64(plain_o), 1 / 64, 0.005, "plain RMSNorm"),
                check_close(norm[:rows], f64(norm_o), 1 / 64, 0.005, "residual RMSNorm"))
    # the fused producer writes the same normalised words as the unfused launches
    assert np.array_equal(fnorm[:rows], norm[:rows]) and np.array_equal(pnorm[:rows], plain[:rows])
    # codes and scales are bit exact against the oracle applied to the row the device wrote
    for cplane, splane, nplane in (("codes", "scales", fnorm), ("pcodes", "pscales", pnorm)):
        oc, os_ = oracle.quantize_e4m3(nplane[:rows])
        assert np.array_equal(host(planes[cplane])[:rows], oc), cplane
        assert np.array_equal(host(planes[splane])[:rows].view(np.uint32), os_.view(np.uint32)), splane
    for name, p in planes.items():
        assert_inactive_untouched(p, rows)
    differing = int((norm[:rows] != norm_o).sum())
    return worst, differing


@pytest.mark.parametrize("rows", list(range(1, MAX_ROWS + 1)))
def test_reference_fixture_exact_batches(tk, ctx, oracle, rows):
    hidden = 5120
    xb, bb, wb = F.norm_fixture(MAX_ROWS, hidden)
    x, b, w = dev(xb.view(np.int16)), dev(bb.view(np.int16)), dev(wb.view(np.int16))
    launch, planes = run_all(tk, ctx, x, b, w, rows, MAX_ROWS, hidden)
    launch()
    torch.cuda.synchronize()
    worst, differing = verify(oracle, planes, xb, bb, wb, rows, 1e-6)
    assert worst <= 1 / 64
    eager = {k: host(v.view(torch.uint8)).copy() for k, v in planes.items()}
    # eager == two graph replays, bit for bit (qual/src/residual_norm.rs:116-123)
    for p in planes.values():
        p.view(torch.uint8).fill_(0xA5)
    g = graph_replay(launch)
    for p in planes.values():
        p.view(torch.uint8).fill_(0xA5)
    g.replay()
    g.replay()
    torch.cuda.synchronize()
    for k, v in planes.items():
        assert np.array_equal(host(v.view(torch.uint8)), eager[k]), k
    assert ctx.device_status() == 0


@pytest.mark.parametrize("rows", [1, 5, 32, 256, 512])
def test_random_rows_match_oracle(tk, oracle, rows):
    from tuiskollm_b200 import synth

    hidden = 5120
    ctx = tk.Context(device=0, max_rows=512)
    xb = synth.normal_bf16(2024, 1, (rows, hidden))
    bb = synth.normal_bf16(2024, 2, (rows, hidden))
    wb = synth.normal_bf16(2024, 3, (hidden,), std=0.1)
    x, b, w = dev(xb.view(np.int16)), dev(bb.view(np.int16)), dev(wb.view(np.int16))
    launch, planes = run_all(tk, ctx, x, b, w, rows, rows + 3, hidden)
    launch()
    torch.cuda.synchronize()
    worst, differing = verify(oracle, planes, xb, bb, wb, rows, 1e-6)
    # the device row differs from the f64 oracle's BF16 rounding in a handful of words at most
    assert differing <= max(4, rows * hidden // 2000), differing
    assert ctx.device_status() == 0


def test_small_geometry_and_edge_rows(tk, oracle):
    """The reference's test geometry (hidden 1024, eps 1e-5: tuisko-kernels-sm120/src/lib.rs:24-52)
    plus all-zero and signed-zero rows."""
    from tuiskollm_b200 import synth

    hidden, rows = 1024, 6
    ctx = tk.Context(device=0, hidden=hidden, rms_norm_epsilon=1e-5, max_rows=8)
    xb = synth.normal_bf16(7, 1, (rows, hidden))
    bb = synth.normal_bf16(7, 2, (rows, hidden))
    xb[2] = 0
    bb[2] = 0
    bb[2, 7] = 0x8000  # 0 + (-0) = +0 in round-to-nearest
    xb[3] = bb[3] ^ 0x8000  # x + branch cancels exactly
    wb = synth.normal_bf16(7, 3, (hidden,), std=0.1)
    x, b, w = dev(xb.view(np.int16)), dev(bb.view(np.int16)), dev(wb.view(np.int16))
    launch, planes = run_all(tk, ctx, x, b, w, rows, 8, hidden)
    launch()
    torch.cuda.synchronize()
    verify(oracle, planes, xb, bb, wb, rows, 1e-5)
    scales = host(planes["scales"])
    assert scales[2] == 1.0 and scales[3] == 1.0
    assert not host(planes["codes"])[2].any()


def test_in_place_residual_and_aliasing(tk, ctx, oracle):
    """x and branch may alias (tuisko-kernels-sm120/src/residual_norm.rs:463-465); the residual
    stream may be updated in place."""
    from tuiskollm_b200 import synth

    hidden, rows = 5120, 4
    xb = synth.normal_bf16(99, 1, (rows, hidden))
    wb = synth.normal_bf16(99, 3, (hidden,), std=0.1)
    x, w = dev(xb.view(np.int16)), dev(wb.view(np.int16))
    norm = sentinel_plane((rows, hidden), torch.int16)
    tk.ResidualNormOp(ctx).launch_residual(None, rows, x, x, w, x, norm)
    torch.cuda.synchronize()
    res_o, norm_o = oracle.residual_rms_norm(xb, xb, wb, 1e-6)
    assert np.array_equal(_u16(x), res_o)
    check_close(_u16(norm), oracle.bf16_to_f32(norm_o).astype(np.float64), 1 / 64, 0.005)


def test_standalone_quantiser_wide_rows(tk, ctx, oracle):
    """quantize_activation_e4m3 on 17408-wide rows (the dense-FP8 down input width,
    tuisko-kernels-sm120/src/fp8/down.rs:35-60) and on the reference fixture tokens."""
    from tuiskollm_b200 import synth

    for cols, xb in ((17408, synth.normal_bf16(5, 1, (3, 17408))), (5120, F.fp8_input(16, 5120))):
        rows = xb.shape[0]
        codes = sentinel_plane((rows + 1, cols), torch.uint8)
        scales = sentinel_plane((rows + 1,), torch.float32)
        tk.Fp8ProjectionOp(ctx).quantize(None, rows, cols, dev(xb.view(np.int16)), codes, scales)
        torch.cuda.synchronize()
        oc, os_ = oracle.quantize_e4m3(xb, search=(cols == 5120))
        assert np.array_equal(host(codes)[:rows], oc)
        assert np.array_equal(host(scales)[:rows].view(np.uint32), os_.view(np.uint32))
        assert_inactive_untouched(codes, rows)
        assert_inactive_untouched(scales, rows)


def test_rejected_launches_report_gpu_launch(tk, ctx):
    hidden = 5120
    x = torch.zeros((8, hidden), dtype=torch.int16, device="cuda")
    w = torch.zeros((hidden,), dtype=torch.int16, device="cuda")
    op = tk.ResidualNormOp(ctx)
    for rows in (0, -1, 100000):
        with pytest.raises(tk.GpuError) as info:
            op.launch_plain(None, rows, x, w, x)
        assert info.value.code == "gpu.launch" and "admitted" in str(info.value)
    with pytest.raises(tk.GpuError) as info:
        op.launch_plain(None, 1, x.data_ptr() + 2, w, x)
    assert info.value.code == "gpu.launch" and "aligned" in str(info.value)
    with pytest.raises(tk.GpuError) as info:
        op.launch_residual(None, 1, x, None, w, x, x)
    assert info.value.code == "gpu.launch" and "null" in str(info.value)
    with pytest.raises(tk.GpuError):
        tk.Context(device=0, hidden=1000)
    with pytest.raises(tk.GpuError) as info:
        tk.Context(device=99)
    assert info.value.code == "gpu.context"


@pytest.mark.parametrize("cols,rows", [(256, 64), (5120, 3), (5120, 500)])
def test_quotients_of_every_scale_round_as_the_division(tk, oracle, cols, rows):
    """E4M3 and NVFP4 codes come from products with a two-part reciprocal per row or block: rows whose maximum
    runs through the whole BF16 range (the E4M3 route divides below 2^-60 and above 2^97), quotients on the
    rounding boundaries, signed zeros, and a NaN that must not disturb its neighbours' E4M3 codes."""
    rng = np.random.default_rng(cols + rows)
    exps = rng.integers(-130, 120, rows)
    x = rng.standard_normal((rows, cols)) * np.exp2(exps.astype(np.float64))[:, None]
    # small integers over a power of two: quotients that are, or are next to, halves of a code step
    grid = rows // 2
    x[:grid] = rng.integers(-28, 29, (grid, cols)) * np.exp2(exps[:grid].astype(np.float64))[:, None] / 4
    x[:, 5::16] = np.where(rng.random(x[:, 5::16].shape) < 0.5, 0.0, -0.0)
    bits = oracle.f32_to_bf16(np.clip(x, -3e38, 3e38).astype(np.float32))
    codes, scales = (torch.zeros((rows, cols), dtype=torch.uint8, device="cuda"),
                     torch.zeros((rows,), dtype=torch.float32, device="cuda"))
    c = tk.Context(device=0)
    op = tk.ops.Fp8ProjectionOp(c)
    op.quantize(None, rows, cols, dev(bits.view(np.int16)), codes, scales)
    oc, os_ = oracle.quantize_e4m3(bits)
    assert np.array_equal(host(scales), os_) and np.array_equal(host(codes), oc)
    c4 = torch.zeros((rows, cols // 2), dtype=torch.uint8, device="cuda")
    s4 = torch.zeros((tk.ops.nvfp4_scale_plane_bytes(rows, cols),), dtype=torch.uint8, device="cuda")
    for divisor in (1.0, 448.0, 448.0 * 6.0 / 5.0):
        tk.Nvfp4SwiGluOp(c).quantize(None, rows, cols, dev(bits.view(np.int16)), divisor, c4, s4)
        qc, qs = oracle.nvfp4_quantize(bits, float(np.float32(divisor)))
        assert np.array_equal(host(c4), qc) and np.array_equal(host(s4), qs), divisor
    assert c.device_status() == 0
    bits[:, 7] = 0x7FC0
    op.quantize(None, rows, cols, dev(bits.view(np.int16)), codes, scales)
    clean = bits.copy()
    clean[:, 7] = 0
    oc, os_ = oracle.quantize_e4m3(clean)
    oc[:, 7] = 0x7F
    assert np.array_equal(host(scales), os_) and np.array_equal(host(codes), oc)


@pytest.mark.parametrize("exponent", [-66, -60, 0, 96, 97, 110])
def test_every_pair_of_significands_rounds_as_the_division(tk, oracle, exponent):
    """E4M3 scales and codes come from products with a two-part reciprocal: all 128 significands a row maximum
    can have (exponents inside and on both sides of the range the products are used in; at 97 the power of two
    alone is still inside) against all 128 of a value, down to 2^-20 of the maximum."""
    mant = 1.0 + np.arange(128) / 128.0
    values = np.concatenate([mant * 2.0 ** -e for e in range(20)])
    x = np.minimum(values[None, :], mant[:, None])
    x[:, 1::2] *= -1.0
    x[:, 0] = mant
    bits = oracle.f32_to_bf16((x * 2.0 ** exponent).astype(np.float32))
    codes, scales = (torch.zeros(bits.shape, dtype=torch.uint8, device="cuda"),
                     torch.zeros((128,), dtype=torch.float32, device="cuda"))
    c = tk.Context(device=0)
    tk.ops.Fp8ProjectionOp(c).quantize(None, 128, bits.shape[1], dev(bits.view(np.int16)), codes, scales)
    oc, os_ = oracle.quantize_e4m3(bits)
    assert np.array_equal(host(scales), os_) and np.array_equal(host(codes), oc)
    assert c.device_status() == 0


def _nonfinite_columns(bits):
    """NaN in a low and in a high half of a pair, infinities in blocks of their own, and a block of NaN alone."""
    bits[..., 5] = 0x7FC0
    bits[..., 22] = 0xFFC0
    bits[..., 40] = 0x7F80
    bits[..., 57] = 0xFF80
    bits[..., 64:80] = 0x7FC0
    return bits


@pytest.mark.parametrize("cols", [256, 5120])
def test_nonfinite_values_stay_in_their_place(tk, oracle, cols):
    """NVFP4: a NaN is left out of its block's maximum and codes as the largest magnitude, an infinity saturates
    the block's scale and its own code; neighbours code as without them.  E4M3: an infinity makes the row's
    scale infinite and sets the status bit, a NaN alone does not."""
    from tuiskollm_b200 import _lib, synth

    rows = 3
    bits = _nonfinite_columns(synth.normal_bf16(77, 1, (rows, cols)))
    nan = (bits & 0x7FFF) > 0x7F80
    c = tk.Context(device=0)
    c4 = torch.zeros((rows, cols // 2), dtype=torch.uint8, device="cuda")
    s4 = torch.zeros((tk.ops.nvfp4_scale_plane_bytes(rows, cols),), dtype=torch.uint8, device="cuda")
    tk.Nvfp4SwiGluOp(c).quantize(None, rows, cols, dev(bits.view(np.int16)), 448.0, c4, s4)
    qc, qs = oracle.nvfp4_quantize(np.where(nan, 0, bits).astype(np.uint16), 448.0)
    nibbles = np.stack([qc & 15, qc >> 4], axis=-1).reshape(rows, cols)
    nibbles[nan] = 7
    nibbles[:, 64:80] = 0  # no finite value: scale 0, zeros with the sign of the value
    got = host(c4)
    assert np.array_equal(np.stack([got & 15, got >> 4], axis=-1).reshape(rows, cols), nibbles)
    assert np.array_equal(host(s4), qs)

    codes, scales = (torch.zeros((rows, cols), dtype=torch.uint8, device="cuda"),
                     torch.zeros((rows,), dtype=torch.float32, device="cuda"))
    tk.ops.Fp8ProjectionOp(c).quantize(None, rows, cols, dev(bits.view(np.int16)), codes, scales)
    assert c.device_status() == _lib.DEVICE_NONFINITE_INPUT
    nonfinite = (bits & 0x7F80) == 0x7F80
    want = np.where(nonfinite, 0x7F, (bits >> 8) & 0x80).astype(np.uint8)
    assert np.isinf(host(scales)).all() and np.array_equal(host(codes), want)


def test_nonfinite_values_behind_the_norm(tk, oracle):
    """The fused producer's two quantised forms of a row with NaN and infinities (from the norm weight) are those
    of the stand-alone quantisers on the row that it wrote."""
    from tuiskollm_b200 import synth

    rows, hidden = 3, 5120
    x, branch = (dev(synth.normal_bf16(78, i, (rows, hidden)).view(np.int16)) for i in (1, 2))
    weight = dev(_nonfinite_columns(synth.normal_bf16(78, 3, (hidden,), std=0.1)).view(np.int16))
    c = tk.Context(device=0)
    i16 = lambda: torch.zeros((rows, hidden), dtype=torch.int16, device="cuda")
    forms = lambda: (torch.zeros((rows, hidden), dtype=torch.uint8, device="cuda"),
                     torch.zeros((rows,), dtype=torch.float32, device="cuda"),
                     torch.zeros((rows, hidden // 2), dtype=torch.uint8, device="cuda"),
                     torch.zeros((tk.ops.nvfp4_scale_plane_bytes(rows, hidden),), dtype=torch.uint8, device="cuda"))
    residual, normed, got, want = i16(), i16(), forms(), forms()
    tk.ResidualNormOp(c).launch_quantize_nvfp4(None, rows, x, branch, weight, residual, normed, got[0], got[1],
                                               448.0, got[2], got[3])
    tk.ops.Fp8ProjectionOp(c).quantize(None, rows, hidden, normed, want[0], want[1])
    tk.Nvfp4SwiGluOp(c).quantize(None, rows, hidden, normed, 448.0, want[2], want[3])
    row = _u16(normed)
    assert ((row[:, 5] & 0x7FFF) > 0x7F80).all() and ((row[:, 40] & 0x7FFF) == 0x7F80).all()
    for a, b in zip(got, want):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))


@pytest.mark.parametrize("cols,ctas", [(2048, 8), (2560, 6), (5120, 3), (6144, 4), (10240, 2)])
def test_quantiser_on_both_sides_of_a_wave(tk, ctx, oracle, cols, ctas):
    """Rows beyond one wave of CTAs (`ctas` to an SM) are quantised by four chunks a thread: the last count of one
    side, the first of the other, and a ragged one further on."""
    from tuiskollm_b200 import synth

    wave = torch.cuda.get_device_properties(0).multi_processor_count * ctas
    bits = synth.normal_bf16(79, cols, (min(wave + 37, 2048), cols))
    want_codes, want_scales = oracle.quantize_e4m3(bits)
    x = dev(bits.view(np.int16))
    for rows in sorted({min(wave, 2048), min(wave + 1, 2048), bits.shape[0]}):
        codes = sentinel_plane((rows + 1, cols), torch.uint8)
        scales = sentinel_plane((rows + 1,), torch.float32)
        tk.Fp8ProjectionOp(ctx).quantize(None, rows, cols, x, codes, scales)
        torch.cuda.synchronize()
        assert np.array_equal(host(codes)[:rows], want_codes[:rows])
        assert np.array_equal(host(scales)[:rows], want_scales[:rows])
        assert_inactive_untouched(codes, rows)
        assert_inactive_untouched(scales, rows)


@pytest.mark.parametrize("hidden,ctas", [(2560, 6), (8192, 4)])
def test_norm_on_both_sides_of_a_wave(tk, oracle, hidden, ctas):
    """The fused producer doubles its chunks beyond a wave, from one to two and from two to four."""
    from tuiskollm_b200 import synth

    wave = torch.cuda.get_device_properties(0).multi_processor_count * ctas
    xb, bb = (synth.normal_bf16(80, i, (wave + 1, hidden)) for i in (1, 2))
    wb = synth.normal_bf16(80, 3, (hidden,), std=0.1)
    want_res, want_norm = oracle.residual_rms_norm(xb, bb, wb, 1e-6)
    x, branch, weight = (dev(a.view(np.int16)) for a in (xb, bb, wb))
    op = tk.ResidualNormOp(tk.Context(device=0, hidden=hidden))
    for rows in (wave, wave + 1):
        residual, normed = (sentinel_plane((rows + 1, hidden), torch.int16) for _ in range(2))
        codes, scales = sentinel_plane((rows + 1, hidden), torch.uint8), sentinel_plane((rows + 1,), torch.float32)
        op.launch_quantize(None, rows, x, branch, weight, residual, normed, codes, scales)
        torch.cuda.synchronize()
        assert np.array_equal(_u16(residual)[:rows], want_res[:rows])
        check_close(_u16(normed)[:rows], oracle.bf16_to_f32(want_norm[:rows]).astype(np.float64), 1 / 64, 0.005)
        oc, os_ = oracle.quantize_e4m3(_u16(normed)[:rows])
        assert np.array_equal(host(codes)[:rows], oc) and np.array_equal(host(scales)[:rows], os_)
        for plane in (residual, normed, codes, scales):
            assert_inactive_untouched(plane, rows)


def _tiled_scale_offsets(rows, hidden):
    """Byte of each (row, block) in a scale plane: tiles of 128 rows x 4 blocks, 16 bytes per row of a tile's quarter."""
    r = torch.arange(rows, device="cuda")[:, None]
    g = torch.arange(hidden // 16, device="cuda")[None, :]
    return ((r >> 7) * (hidden // 64) + (g >> 2)) * 512 + (r & 31) * 16 + ((r & 127) >> 5) * 4 + (g & 3)


@pytest.mark.parametrize("hidden", [2048, 5120, 6144, 17408])
@pytest.mark.parametrize("with_branch", [True, False])
def test_rows_in_clusters_have_the_bits_of_rows_alone(tk, hidden, with_branch):
    """A cluster changes nothing but a row's place: every plane has the bits of launches of four rows, which have none,
    on both sides of each line and with one to three rows in the last cluster, and nothing behind the rows."""
    from tuiskollm_b200 import ops, synth

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    c = tk.Context(device=0, hidden=hidden)
    most = 2 * sms + 4
    x, branch = (synth.torch_normal_bf16(95, i, (most, hidden), "cuda") for i in (1, 2))
    weight = synth.torch_normal_bf16(95, 3, (hidden,), "cuda", std=0.1)
    op = tk.ResidualNormOp(c)

    def planes(rows):
        return ([sentinel_plane((rows + 1, hidden), torch.int16) for _ in range(2)] +
                [sentinel_plane((rows + 1, hidden), torch.uint8), sentinel_plane((rows + 1,), torch.float32),
                 sentinel_plane((rows + 1, hidden // 2), torch.uint8),
                 torch.zeros((ops.nvfp4_scale_plane_bytes(rows, hidden),), dtype=torch.uint8, device="cuda")])

    def launch(rows, first, out):
        op.launch_quantize_nvfp4(None, rows, x[first:first + rows], branch[first:first + rows] if with_branch else None,
                                 weight, out[0], out[1], out[2], out[3], 448.0, out[4], out[5])

    offsets = _tiled_scale_offsets(most, hidden)
    want = planes(most)
    for first in range(0, most, 4):
        four = planes(4)
        launch(4, first, four)
        for w, f in zip(want[:5], four[:5]):
            w[first:first + 4] = f[:4]
        want[5][offsets[first:first + 4]] = four[5][offsets[:4]]
    for rows in (4, 12, 13, 14, 15, 16, 29, 32, 33, sms, sms + 1, 3 * sms // 2 + 1, 2 * sms + 1):
        got = planes(rows)
        launch(rows, 0, got)
        torch.cuda.synchronize()
        for i, (w, g) in enumerate(zip(want[:5], got[:5])):
            if i == 0 and not with_branch:
                continue  # no residual plane is written
            assert torch.equal(w[:rows].view(torch.uint8), g[:rows].view(torch.uint8)), (rows, i)
            assert_inactive_untouched(g, rows)
        scales = torch.zeros_like(got[5])  # zero behind the rows
        scales[offsets[:rows]] = want[5][offsets[:rows]]
        assert torch.equal(scales, got[5]), rows
    assert c.device_status() == 0


class _KernelNode(ctypes.Structure):
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3),
                ("shared_bytes", ctypes.c_uint), ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p),
                ("kern", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]


def test_norms_hold_no_shared_memory_that_they_do_not_use(tk, ctx):
    """Beside a kernel of another stream that has most of an SM's shared memory a norm must find room: its launch asks
    for none beyond the few bytes of its reductions (those are static), whatever the number of rows."""
    from tuiskollm_b200 import synth

    driver = ctypes.CDLL("libcuda.so.1")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    most, hidden = 2 * sms, 5120
    x, branch = (synth.torch_normal_bf16(96, i, (most, hidden), "cuda") for i in (1, 2))
    weight = synth.torch_normal_bf16(96, 3, (hidden,), "cuda", std=0.1)
    residual, normed = (torch.zeros((most, hidden), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    codes = torch.zeros((most, hidden), dtype=torch.uint8, device="cuda")
    scales = torch.zeros((most,), dtype=torch.float32, device="cuda")
    op = tk.ResidualNormOp(ctx)
    for rows in (1, 4, 5, 12, 13, 30, 32, 33, 100, sms, sms + 1, most):
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(graph):
            op.launch_quantize(None, rows, x, branch, weight, residual, normed, codes, scales)
        raw, count = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(1)
        nodes = (ctypes.c_void_p * 1)()
        assert driver.cuGraphGetNodes(raw, nodes, ctypes.byref(count)) == 0 and count.value == 1
        node = _KernelNode()
        assert driver.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(nodes[0]), ctypes.byref(node)) == 0
        assert node.grid[0] == ((rows + 3) // 4 * 4 if 13 <= rows <= 32 else rows), rows
        assert node.shared_bytes == 0, rows
