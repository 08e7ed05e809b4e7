"""Resident P6 layout: lossless on the codes, GEMV equal to the oracle."""
import os

import numpy as np
import pytest
import torch

from oracle import ixb_oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(64, 5120), (48, 5120), (40, 17408), (96, 2176), (7, 4352), (33, 96), (1, 32), (3, 1024), (300, 512),
          (10, 96), (5, 100), (17, 72), (512, 17408), (16, 64)]


def bits_to_bf16(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int16)).view(torch.bfloat16)


def rel_err(y, ref):
    return float(np.abs(y.astype(np.float64) - ref).max() / max(float(np.abs(ref).max()), 1e-30))


def make(out_f, in_f, seed, codes=None):
    from ixrun_b200.p6 import P6Packed

    if codes is None:
        codes = O.laplace_codes(out_f, in_f, seed)
    scale = torch.tensor(0.00251, dtype=torch.bfloat16)
    return codes, scale, P6Packed(torch.from_numpy(codes).cuda(), scale, out_f, in_f)


@pytest.mark.parametrize("out_f,in_f", SHAPES)
def test_p6_roundtrip_is_lossless(out_f, in_f):
    codes, scale, p6 = make(out_f, in_f, out_f + in_f)
    assert np.array_equal(p6.decode(kind="codes").cpu().numpy().reshape(-1), codes)
    sc_bits = int(scale.view(torch.int16).item()) & 0xFFFF
    w = p6.decode(kind="bf16").cpu().view(torch.int16).numpy().view(np.uint16).reshape(-1)
    assert np.array_equal(w, O.codes_to_bf16(codes, sc_bits))


@pytest.mark.parametrize("out_f,in_f", SHAPES)
@pytest.mark.parametrize("m", [1, 2, 5, 8])
def test_p6_gemv_matches_oracle(out_f, in_f, m):
    codes, scale, p6 = make(out_f, in_f, out_f * 5 + in_f + m)
    sc_bits = int(scale.view(torch.int16).item()) & 0xFFFF
    xb = O.f32_to_bf16_bits(np.random.default_rng(m).standard_normal((m, in_f)).astype(np.float32))
    ref = O.gemm_f32(codes, sc_bits, xb, out_f, in_f).astype(np.float64)
    x = bits_to_bf16(xb).cuda()
    bias = torch.randn(out_f).bfloat16().cuda()
    y32 = p6.gemv(x, out_dtype=torch.float32)
    assert rel_err(y32.cpu().numpy(), ref) < 2e-5
    assert torch.equal(p6.gemv(x), y32.bfloat16())
    assert torch.equal(p6.gemv(x, bias=bias), p6.gemv(x) + bias)
    assert torch.equal(p6.gemv(x, out_dtype=torch.float32), y32)


def test_p6_one_scratch_buffer_serves_layers_of_any_shape():
    """Layers whose row tiles are shared by three or more CTAs, by two, and by none run back to back on ONE scratch
    buffer (the library leaves it all zero after every launch), in both orders, and still match the oracle."""
    from ixrun_b200.p6 import GemvScratch

    shapes = [(16, 17408), (256, 17408), (5120, 2176), (64, 5120), (16, 17408), (5120, 2176), (300, 512)]
    scratch = GemvScratch("cuda")
    cases = []
    for i, (out_f, in_f) in enumerate(shapes):
        codes, scale, p6 = make(out_f, in_f, 100 + i)
        p6.scratch = scratch
        sc_bits = int(scale.view(torch.int16).item()) & 0xFFFF
        xb = O.f32_to_bf16_bits(np.random.default_rng(i).standard_normal((1, in_f)).astype(np.float32))
        cases.append((p6, bits_to_bf16(xb).cuda(), O.gemm_f32(codes, sc_bits, xb, out_f, in_f).astype(np.float64)))
    for order in (range(len(cases)), reversed(range(len(cases)))):
        for i in order:
            p6, x, ref = cases[i]
            assert rel_err(p6.gemv(x, out_dtype=torch.float32).cpu().numpy(), ref) < 2e-5
    assert int(scratch.buf.max().item()) == 0       # every launch left the scratch all zero


def test_p6_extreme_level_mixes_and_from_packed(golden_dir):
    from ixrun_b200.p6 import P6Packed

    out_f, in_f = 8, 1024
    n = out_f * in_f
    rng = np.random.default_rng(0)
    xb = O.f32_to_bf16_bits(rng.standard_normal((2, in_f)).astype(np.float32))
    for codes in (rng.choice(np.r_[-127:-16, 32:128], size=n).astype(np.int8),
                  rng.integers(-16, 32, size=n).astype(np.int8),
                  rng.integers(-3, 4, size=n).astype(np.int8),
                  np.where(np.arange(n) % 2 == 0, 1, 100).astype(np.int8),
                  np.zeros(n, dtype=np.int8)):
        c, scale, p6 = make(out_f, in_f, 0, codes=codes)
        assert np.array_equal(p6.decode(kind="codes").cpu().numpy().reshape(-1), codes)
        sc_bits = int(scale.view(torch.int16).item()) & 0xFFFF
        ref = O.gemm_f32(codes, sc_bits, xb, out_f, in_f).astype(np.float64)
        y = p6.gemv(bits_to_bf16(xb).cuda(), out_dtype=torch.float32).cpu().numpy()
        assert float(np.abs(y - ref).max()) <= 2e-5 * max(float(np.abs(ref).max()), 1e-30)
    # from the reference's packed streams (fixture written by the reference's own quantiser)
    g = dict(np.load(os.path.join(golden_dir, "heavy_64x1024.npz")))
    packed = {"level_bits": (3, 5, 8), "out_f": 64, "in_f": 1024, "N": 65536, "scale": bits_to_bf16(g["scale_bits"]).reshape(()),
              "bitmaps": [torch.from_numpy(g["b1"]), torch.from_numpy(g["b2"])],
              "streams": [torch.from_numpy(g["l1"]), torch.from_numpy(g["l2"]), torch.from_numpy(g["l3"])],
              "counts": [int(c) for c in g["counts"]], "total_bytes": int(g["total_bytes"][0])}
    p6 = P6Packed.from_packed(packed)
    assert np.array_equal(p6.decode(kind="codes").cpu().numpy().reshape(-1), g["codes"])
    y = p6.gemv(bits_to_bf16(g["x_bits"]).cuda(), out_dtype=torch.float32).cpu().numpy()
    assert rel_err(y, g["y_f32"].astype(np.float64)) < 2e-5


@pytest.mark.parametrize("out_f,in_f", [(5120, 17408), (17408, 5120), (5120, 5120), (1024, 5120), (2048, 2048)])
def test_p6_full_size_against_the_oracle(out_f, in_f):
    """The five benchmark shapes at full size, batch 1: the GEMV on the resident layout against the CPU oracle's
    fp32-accumulated product of the same codes, the decoded codes against the codes that were packed; twice for
    reproducibility; 8 rows against the fused kernel on the reference's streams (itself checked against the
    oracle)."""
    from ixrun_b200.p6 import P6Packed
    from ixrun_b200.packed import DevicePacked
    from ixrun_b200.synth import laplace_codes, synthetic_packed

    dp = DevicePacked(synthetic_packed(out_f, in_f, seed=3))
    codes = laplace_codes(out_f, in_f, seed=3)
    p6 = P6Packed.from_packed(dp)
    got = p6.decode(kind="codes")
    assert torch.equal(got, dp.decode(kind="codes"))
    assert np.array_equal(got.cpu().numpy().reshape(-1), codes.reshape(-1))
    sc_bits = int(dp.scale.view(torch.int16).item()) & 0xFFFF
    xb = O.f32_to_bf16_bits(np.random.default_rng(7).standard_normal((1, in_f)).astype(np.float32))
    ref = O.gemm_f32(codes.reshape(-1), sc_bits, xb, out_f, in_f).astype(np.float64)
    y = p6.gemv(bits_to_bf16(xb).cuda(), out_dtype=torch.float32)
    assert rel_err(y.cpu().numpy(), ref) < 2e-5
    assert torch.equal(p6.gemv(bits_to_bf16(xb).cuda(), out_dtype=torch.float32), y)
    x8 = torch.randn(8, in_f, device="cuda").bfloat16()
    ref8 = dp.gemv(x8, out_dtype=torch.float32)
    y8 = p6.gemv(x8, out_dtype=torch.float32)
    assert float((y8 - ref8).abs().max() / ref8.abs().max()) < 2e-5
    assert torch.equal(p6.gemv(x8, out_dtype=torch.float32), y8)
    assert p6.resident_bytes < 1.2 * dp.total_bytes


@pytest.mark.parametrize("out_f,in_f", [(512, 5120), (512, 8256), (2400, 5120), (100, 2052)])
def test_p6_programmatic_dependent_launch_gives_the_same_result(out_f, in_f):
    """Back-to-back launches with programmatic dependent launch on (eagerly and replayed from a CUDA graph):
    every launch must still see the activations written just before it and produce the bits of a plain launch.  Two layers of few
    blocks per warp, one of many between such ones, two of many (tiles shared by CTAs), and two whose rows are no multiple of 16 bytes."""
    from ixrun_b200.p6 import set_pdl

    _, _, a = make(out_f, in_f, 11)
    _, _, b = make(in_f, out_f, 12)
    x = torch.randn(1, in_f, device="cuda").bfloat16()
    h_ref = a.gemv(x)
    y_ref = b.gemv(h_ref)
    torch.cuda.synchronize()
    prev = set_pdl(True)
    try:
        h = torch.empty_like(h_ref)
        y = torch.empty_like(y_ref)
        for _ in range(3):
            h.zero_()
            y.zero_()
            a.gemv(x, out=h)
            b.gemv(h, out=y)          # reads what the launch just ahead of it wrote
            assert torch.equal(h, h_ref) and torch.equal(y, y_ref)
        st = torch.cuda.Stream()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.stream(st):
            with torch.cuda.graph(g, stream=st):
                for _ in range(4):
                    a.gemv(x, out=h)
                    b.gemv(h, out=y)
        h.zero_()
        y.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(h, h_ref) and torch.equal(y, y_ref)
    finally:
        set_pdl(prev)


@pytest.mark.parametrize("in_f,rows", [(512, (48, 100, 256)), (5120, (1536, 256, 6, 6)), (2048, (2048, 1024, 1024))])
def test_p6_fused_tensor_gives_every_part_its_own_result(in_f, rows):
    """Tensors fused row-wise keep their own per-tensor scales: decoding gives every part's weights bit for bit, the
    GEMV every part's outputs (the fp32 sums may be added in another order than in the part alone: 1e-6 of the
    largest output; the tile layout and the products are the same)."""
    from ixrun_b200.p6 import P6Packed
    from ixrun_b200.synth import synthetic_packed

    parts = [synthetic_packed(r, in_f, seed=11 + i) for i, r in enumerate(rows)]
    for i, p in enumerate(parts):                       # clearly different scales
        p["scale"] = (p["scale"].float() * (1.0 + 0.37 * i)).to(torch.bfloat16)
    alone = [P6Packed.from_packed(p) for p in parts]
    fused = P6Packed.fuse(parts)
    assert [n for _, n in fused.sections] == list(rows) and all(a % 16 == 0 for a, _ in fused.sections)
    w = fused.decode(kind="bf16")
    c = fused.decode(kind="codes").view(fused.out_f, in_f)
    for (a, n), one in zip(fused.sections, alone):
        assert torch.equal(w[a:a + n], one.decode(kind="bf16"))
        assert torch.equal(c[a:a + n], one.decode(kind="codes").view(n, in_f))
    for m in (1, 3):
        x = torch.randn(m, in_f, device="cuda").bfloat16()
        y = fused.gemv(x, out_dtype=torch.float32)
        yb = fused.gemv(x)
        for (a, n), one in zip(fused.sections, alone):
            ref = one.gemv(x, out_dtype=torch.float32)
            assert float((y[:, a:a + n] - ref).abs().max()) <= 1e-6 * float(ref.abs().max())
            assert float((yb[:, a:a + n].float() - ref).abs().max()) <= 2.0 ** -8 * float(ref.abs().max())
    if len(rows) == 3:
        q, k, v = fused.split(fused.gemv(torch.randn(1, in_f, device="cuda").bfloat16()))
        assert q.numel() == rows[0] and k.numel() == rows[1] and v.numel() == rows[2]


@pytest.mark.parametrize("out_f,in_f,m", [(128, 512, 16), (16, 1024, 64), (40, 5120, 33), (100, 1024, 9), (300, 512, 64),
                                          (512, 5120, 64), (1000, 2176, 17), (3, 3072, 1), (2048, 2048, 32)])
def test_p6_gemm_small_m_against_the_oracle(out_f, in_f, m):
    """GEMM on the resident layout (1..64 rows) against the oracle's fp32 result; bias, bf16 output and
    repeatability; within fp32 summation-order rounding of the GEMV for the rows both take."""
    codes, scale, p6 = make(out_f, in_f, out_f * 3 + m)
    sc_bits = int(scale.view(torch.int16).item()) & 0xFFFF
    xb = O.f32_to_bf16_bits(np.random.default_rng(m).standard_normal((m, in_f)).astype(np.float32))
    ref = O.gemm_f32(codes, sc_bits, xb, out_f, in_f).astype(np.float64)
    x = bits_to_bf16(xb).cuda()
    bias = torch.randn(out_f).bfloat16().cuda()
    y32 = p6.gemm(x, out_dtype=torch.float32)
    assert rel_err(y32.cpu().numpy(), ref) < 2e-5
    assert torch.equal(p6.gemm(x), y32.bfloat16())
    assert torch.equal(p6.gemm(x, bias=bias), p6.gemm(x) + bias)
    assert torch.equal(p6.gemm(x, out_dtype=torch.float32), y32)          # deterministic
    if m <= 8:
        assert rel_err(p6.gemv(x, out_dtype=torch.float32).cpu().numpy(), y32.cpu().numpy().astype(np.float64)) < 2e-5


@pytest.mark.parametrize("out_f,in_f", [(17408, 5120), (5120, 17408)])
@pytest.mark.parametrize("m", [16, 32, 64])
def test_p6_gemm_full_size(out_f, in_f, m):
    """The batched-serving shapes at full size: against an fp32 matmul on the decoded weights (the reference's
    decode + dense matmul in fp32; 1e-3 is the path's stated tolerance, the observed error is fp32 rounding)."""
    from ixrun_b200.p6 import P6Packed
    from ixrun_b200.synth import synthetic_packed

    p6 = P6Packed.from_packed(synthetic_packed(out_f, in_f, seed=3))
    x = torch.randn(m, in_f, device="cuda").bfloat16()
    w = p6.decode(kind="bf16")
    ref = x.double() @ w.double().t()
    y = p6.gemm(x, out_dtype=torch.float32)
    err = float((y.double() - ref).abs().max() / ref.abs().max())
    assert err < 2e-5, err
    assert torch.equal(p6.gemm(x), y.bfloat16())


@pytest.mark.parametrize("m", [9, 16, 17, 24, 25, 33, 40, 41, 48, 49, 64])
@pytest.mark.parametrize("out_f,in_f,outliers", [(129, 64, False), (272, 192, True), (2064, 2240, False)])
def test_p6_gemm_row_counts(out_f, in_f, outliers, m):
    """Every variant of the kernel at the edges of its row counts; one column block, three (a part without work), 35 over
    several splits; a last row group of one tile; blocks with up to 800 outliers.  fp32 against float64 sums of exact
    products: the metric and bound of the tests above."""
    from ixrun_b200.p6 import P6Packed

    gen = torch.Generator(device="cuda").manual_seed(out_f + m)
    if outliers:
        codes = torch.randint(-127, 128, (out_f, in_f), generator=gen, device="cuda").to(torch.int8)
    else:
        codes = (torch.randn(out_f, in_f, generator=gen, device="cuda") * 12).round().clamp(-127, 127).to(torch.int8)
    p6 = P6Packed(codes, torch.tensor(0.007, dtype=torch.bfloat16), out_f, in_f)
    x = torch.randn(m, in_f, generator=gen, device="cuda").bfloat16()
    w = p6.decode(kind="bf16").double()
    assert torch.equal(w, (codes.float() * p6.scale.float()).bfloat16().double())
    ref = x.double() @ w.t()
    y = p6.gemm(x, out_dtype=torch.float32)
    assert float((y.double() - ref).abs().max() / ref.abs().max()) < 2e-5
    bias = torch.randn(out_f, generator=gen, device="cuda").bfloat16()
    assert torch.equal(p6.gemm(x, bias=bias), y.bfloat16() + bias)


@pytest.mark.parametrize("m", [33, 47, 48, 49, 64])
@pytest.mark.parametrize("out_f,in_f,outliers", [(129, 8192, False), (40, 17408, True), (300, 16384, False)])
def test_p6_gemm_few_row_groups(out_f, in_f, outliers, m):
    """More than 32 rows on layers of few row groups and many columns: a last row group of one tile, many K splits of unequal
    length, blocks with up to 800 outliers.  Bound as above.  ixb_p6_gemm asks for 256 bytes of scratch, leaves them alone and gives
    what ixb_p6_rows gives, bit for bit."""
    from ixrun_b200 import _lib
    from ixrun_b200.p6 import P6Packed

    gen = torch.Generator(device="cuda").manual_seed(out_f + m)
    if outliers:
        codes = torch.randint(-127, 128, (out_f, in_f), generator=gen, device="cuda").to(torch.int8)
    else:
        codes = (torch.randn(out_f, in_f, generator=gen, device="cuda") * 12).round().clamp(-127, 127).to(torch.int8)
    p6 = P6Packed(codes, torch.tensor(0.007, dtype=torch.bfloat16), out_f, in_f)
    x = torch.randn(m, in_f, generator=gen, device="cuda").bfloat16()
    ref = x.double() @ (codes.float() * p6.scale.float()).bfloat16().double().t()
    L = _lib.lib()
    assert L.ixb_p6_gemm_scratch_bytes(out_f, in_f, m) == 256
    y = p6.gemm(x, out_dtype=torch.float32)
    assert float((y.double() - ref).abs().max() / ref.abs().max()) < 2e-5
    assert torch.equal(p6.gemm(x, out_dtype=torch.float32), y)
    bias = torch.randn(out_f, generator=gen, device="cuda").bfloat16()
    assert torch.equal(p6.gemm(x, bias=bias), y.bfloat16() + bias)
    small, out = torch.full((256,), 7, dtype=torch.uint8, device="cuda"), torch.empty(m, out_f, dtype=torch.bfloat16, device="cuda")
    _lib.check(L.ixb_p6_gemm(p6._ref, x.data_ptr(), m, None, out.data_ptr(), 0, small.data_ptr(), 256, _lib.stream_ptr(x.device)))
    assert torch.equal(out, p6.rows(x)) and bool((small == 7).all())


@pytest.mark.parametrize("out_f,in_f,dense", [(48, 6464, False), (48, 6464, True), (16, 64, True), (2500, 96, True), (5120, 320, False),
                                              (48, 16448, False), (48, 16448, True), (2500, 4200, True), (2500, 100, True),
                                              (5120, 2180, False), (14800, 16448, False)])
def test_p6_gemv_rows_get_the_bits_they_get_alone(out_f, in_f, dense):
    """Layers of few blocks per warp (the first five) and of many.  There outliers go through the tensor core 32 at a time for all
    activation rows: more steps than blocks (every second code an outlier), segments shorter than the pipeline, several row tiles
    per run, runs of more than 64 blocks (the last); up to 8 rows, with activations in shared memory and (eight wide rows) from
    global memory.  Against float64 sums of exact products."""
    from ixrun_b200.p6 import P6Packed

    gen = torch.Generator(device="cuda").manual_seed(out_f + in_f)
    codes = (torch.randn(out_f, in_f, generator=gen, device="cuda") * (40 if dense else 12)).round().clamp(-127, 127).to(torch.int8)
    p6 = P6Packed(codes, torch.tensor(0.007, dtype=torch.bfloat16), out_f, in_f)
    x = torch.randn(8, in_f, generator=gen, device="cuda").bfloat16()
    ref = x.double() @ (codes.float() * p6.scale.float()).bfloat16().double().t()
    alone = torch.cat([p6.gemv(x[i:i + 1].clone(), out_dtype=torch.float32) for i in range(8)])      # (16-byte aligned)
    assert float((alone.double() - ref).abs().max() / ref.abs().max()) < 2e-5
    for m in (2, 3, 7, 8):
        assert torch.equal(p6.gemv(x[:m], out_dtype=torch.float32), alone[:m])


@pytest.mark.parametrize("in_f", [256, 8264, 100])
def test_p6_gemv_infinite_activation_reaches_only_its_rows(in_f):
    """An infinite activation in one of three rows: the other rows keep their bits, and a weight row without an outlier in
    that column gets what the dense product gives (an infinity of the weight's sign, NaN for weight 0).  On the kernel for few
    blocks per warp (256 columns) and on the other one."""
    from ixrun_b200.p6 import P6Packed

    gen = torch.Generator(device="cuda").manual_seed(2)
    out_f, col = 64, 77
    codes = torch.randint(1, 32, (out_f, in_f), generator=gen, device="cuda").to(torch.int8)
    codes[::2] = -torch.randint(1, 17, (out_f // 2, in_f), generator=gen, device="cuda").to(torch.int8)
    codes[5, col], codes[21, col], codes[3, 5], codes[8, col] = 100, -90, 120, 0
    p6 = P6Packed(codes, torch.tensor(0.01, dtype=torch.bfloat16), out_f, in_f)
    x = torch.randn(3, in_f, generator=gen, device="cuda").bfloat16()
    clean = p6.gemv(x)
    x[1, col] = float("inf")
    y = p6.gemv(x)
    assert torch.equal(y[0], clean[0]) and torch.equal(y[2], clean[2])
    for got in (y[1], p6.gemv(x[1:2].clone())[0]):
        for r in range(out_f):
            if r in (5, 21):
                assert not bool(torch.isfinite(got[r]))               # an outlier there: not finite either
            elif r == 8:
                assert bool(torch.isnan(got[r]))
            else:
                assert bool(torch.isinf(got[r])) and bool(got[r] > 0) == bool(codes[r, col] > 0), r


@pytest.mark.parametrize("out_f,in_f", [(48, 64), (33, 72), (50, 2176), (16, 8)])
@pytest.mark.parametrize("shift,scale", [(0, 0.0071), (8, 0.0071), (0, 2.0 ** -131), (0, 2.0 ** 120)])
def test_p6_decode_stores(out_f, in_f, shift, scale):
    """Sector stores and 16-byte ones (rows or an output that is only 16-byte aligned), blocks with none, one, two and many
    outliers; subnormal and huge weights; the streams' decoder on the same codes.  Bit for bit, and nothing beside the output is written."""
    from ixrun_b200.p6 import P6Packed
    from ixrun_b200.gpu_pack import pack_codes_gpu

    gen = torch.Generator(device="cuda").manual_seed(in_f)
    codes = torch.randint(-32, 32, (out_f, in_f), generator=gen, device="cuda").to(torch.int8)
    n_kb = (in_f + 63) // 64
    for kb, n in zip(range(n_kb), (0, 1, 2, 3, 40) * n_kb):
        for k in range(n):
            codes[(5 * k) % min(out_f, 16), min(64 * kb + (7 * k) % 64, in_f - 1)] = 100 - k
    scale = torch.tensor(scale, dtype=torch.bfloat16)
    want = (codes.float() * scale.float().cuda()).bfloat16()
    buf = torch.full((out_f * in_f + 64,), 7.0, dtype=torch.bfloat16, device="cuda")
    for src in (P6Packed(codes.reshape(-1), scale, out_f, in_f), pack_codes_gpu(codes, scale, out_f, in_f)):
        buf.fill_(7.0)
        got = src.decode(out=buf[16 + shift:16 + shift + out_f * in_f], kind="bf16")
        assert torch.equal(got.view(torch.int16), want.view(torch.int16))
        assert bool((buf[:16 + shift] == 7).all()) and bool((buf[16 + shift + out_f * in_f:] == 7).all())


@pytest.mark.parametrize("in_f", [192, 200])
def test_p6_negative_scale(in_f):
    """A scale below zero: code 0 becomes +0.0 (the product would be -0.0, which has the same value), outliers of either
    sign keep theirs, in the decoder and at every row count of the kernels (fp32 sums against float64: the bound of the
    tests above)."""
    from ixrun_b200.p6 import P6Packed

    gen = torch.Generator(device="cuda").manual_seed(in_f)
    out_f = 50
    codes = torch.randint(-127, 128, (out_f, in_f), generator=gen, device="cuda").to(torch.int8)
    codes[:16] = torch.randint(-32, 32, (16, in_f), generator=gen, device="cuda").to(torch.int8)
    codes[3, 5], codes[4, 6], codes[5, 80] = -100, 90, -33         # blocks with one, two outliers
    scale = torch.tensor(-0.0071, dtype=torch.bfloat16, device="cuda")
    want = (codes.float() * scale.float()).bfloat16()
    p6 = P6Packed(codes.reshape(-1), scale, out_f, in_f)
    got = p6.decode(kind="bf16")
    assert torch.equal(got, want)
    assert torch.equal(got.view(torch.int16), torch.where(codes == 0, 0.0, want).bfloat16().view(torch.int16))
    x = torch.randn(50, in_f, generator=gen, device="cuda").bfloat16()
    ref = x.double() @ want.double().t()
    near = lambda y, m: float((y.double() - ref[:m]).abs().max() / ref.abs().max()) < 2e-5
    assert near(p6.gemv(x[:8], out_dtype=torch.float32), 8)
    if in_f % 64 == 0:
        assert near(p6.gemm(x[:23], out_dtype=torch.float32), 23)
    y = p6.rows(x)
    assert bool(((y.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-5 * ref.abs().max()).all())


@pytest.mark.parametrize("m", [9, 16, 17, 33, 64])
@pytest.mark.parametrize("out_f,in_f,per_block", [(16, 64, 0), (16, 64, 2), (144, 1000, 4), (2064, 128, 2), (300, 4160, 49),
                                                  (300, 4160, 51), (129, 17408, 1)])
def test_p6_rows_edges(out_f, in_f, per_block, m):
    """9..64 rows where their kernels can go wrong: one column block, an odd number of them, a ragged last one, a last row group
    of one tile, both sides of the rule on outliers per block (3 and 50), an activation of infinity.  Bound: fp32 sums of at most
    17408 exact products in chains, 2e-5 of the largest result as above."""
    from ixrun_b200.p6 import P6Packed

    gen = torch.Generator(device="cuda").manual_seed(out_f + in_f + m)
    codes = (torch.randn(out_f, in_f, generator=gen, device="cuda") * 8).round().clamp(-31, 31)
    rt, kb = (out_f + 15) // 16, (in_f + 63) // 64
    at = torch.randperm(out_f * in_f, generator=gen, device="cuda")[:per_block * rt * kb]
    codes.view(-1)[at] = torch.where(codes.view(-1)[at] < 0, -127.0, 100.0)
    p6 = P6Packed(codes.to(torch.int8), torch.tensor(0.007, dtype=torch.bfloat16), out_f, in_f)
    w = (codes * p6.scale.float()).bfloat16().double()
    x = torch.randn(m, in_f, generator=gen, device="cuda").bfloat16()
    call = p6.gemm if in_f % 64 == 0 else p6.rows
    ref = x.double() @ w.t()
    assert float((call(x).double() - ref).abs().max() / ref.abs().max()) < 2e-5 + 2.0 ** -8
    if in_f % 64 == 0:
        y = p6.gemm(x, out_dtype=torch.float32)
        assert float((y.double() - ref).abs().max() / ref.abs().max()) < 2e-5
    # infinity times a weight is infinity of its sign, or NaN for a weight of 0; it reaches only its own row of activations
    x[3, in_f // 2] = float("inf")
    y, ref = call(x), (x.double() @ w.t()).bfloat16()
    assert torch.equal(y[3].nan_to_num(nan=7.0, posinf=1.0, neginf=-1.0), ref[3].nan_to_num(nan=7.0, posinf=1.0, neginf=-1.0))
    assert torch.isfinite(y[torch.arange(m, device="cuda") != 3]).all()


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("out_f,in_f", [(16, 8), (40, 1000), (2384, 128), (300, 2176), (2048, 8192), (2048, 8256), (18944, 512),
                                        (19000, 512)])
def test_p6_gemv_few_blocks(out_f, in_f, dense):
    """1..8 rows on layers of few blocks per warp, and both sides of the rule (8 blocks): fewer column blocks than warps, slices
    of unequal length, a ragged last block, CTAs with fewer tiles than others, more outliers than lanes, an infinite activation.
    Bound: fp32 sums of at most 8256 exact products, 2e-5 of the largest result as above."""
    from ixrun_b200.p6 import P6Packed

    gen = torch.Generator(device="cuda").manual_seed(out_f + in_f)
    codes = torch.randn(out_f, in_f, generator=gen, device="cuda") * (60 if dense else 10)
    codes = codes.round().clamp(-127, 127).to(torch.int8)
    p6 = P6Packed(codes, torch.tensor(-0.007, dtype=torch.bfloat16), out_f, in_f)
    w = (codes.float() * p6.scale.float()).bfloat16().double()
    x = torch.randn(8, in_f, generator=gen, device="cuda").bfloat16()
    ref = x.double() @ w.t()
    bias = torch.randn(out_f, generator=gen, device="cuda").bfloat16()
    y8 = p6.gemv(x, out_dtype=torch.float32)
    assert float((y8.double() - ref).abs().max() / ref.abs().max()) < 2e-5
    for m in (1, 2, 5):
        assert torch.equal(p6.gemv(x[:m], out_dtype=torch.float32), y8[:m])
    assert torch.equal(p6.gemv(x[:3], bias=bias), y8[:3].bfloat16() + bias)
    if (out_f, in_f) in ((2048, 8256), (19000, 512)):
        return                                       # the other kernel: an infinity that meets an outlier is NaN there (see above)
    x[1, in_f // 2] = float("-inf")
    y, ref = p6.gemv(x), (x.double() @ w.t()).bfloat16()
    assert torch.equal(y[1].nan_to_num(nan=7.0, posinf=1.0, neginf=-1.0), ref[1].nan_to_num(nan=7.0, posinf=1.0, neginf=-1.0))
    assert torch.equal(y[[0, 2, 3, 4, 5, 6, 7]], y8[[0, 2, 3, 4, 5, 6, 7]].bfloat16())


@pytest.mark.parametrize("m", [16, 64])
@pytest.mark.parametrize("out_f,in_f", [(256, 32768), (19000, 1280)])
def test_p6_rows_behind_a_kernel_that_takes_long(out_f, in_f, m):
    """Dependent launch: the kernel ahead (attention over four million positions by one CTA, a tenth of a second and more) lets the
    launch begin at once, and however long it takes counts against none of the launch's bounded waits: the bits of a launch
    with nothing ahead.  K split over a cluster and not, more stages than are in flight."""
    from ixrun_b200.glue import AttnDecode
    from ixrun_b200.p6 import P6Packed, set_pdl

    gen = torch.Generator(device="cuda").manual_seed(m)
    codes = (torch.randn(out_f, in_f, generator=gen, device="cuda") * 12).round().clamp(-127, 127).to(torch.int8)
    p6 = P6Packed(codes, torch.tensor(0.007, dtype=torch.bfloat16), out_f, in_f)
    x = torch.randn(m, in_f, generator=gen, device="cuda").bfloat16()
    n = 1 << 22
    cache = torch.zeros(n, 1, 64, dtype=torch.bfloat16, device="cuda")
    cache[-1] = 1
    attn = AttnDecode(2, 1, 64, "cuda", splits=1)
    q, pos = torch.ones(128, device="cuda").bfloat16(), torch.tensor([n - 1], dtype=torch.int32, device="cuda")
    a, y = torch.empty(128, dtype=torch.bfloat16, device="cuda"), torch.empty(m, out_f, device="cuda")
    torch.cuda.synchronize()
    before = set_pdl(True)
    try:
        alone = p6.gemm(x, out_dtype=torch.float32)
        torch.cuda.synchronize()
        for _ in range(2):
            y.zero_()
            attn(q, cache, cache, pos, out=a)
            p6.gemm(x, out=y)
            torch.cuda.synchronize()
            assert torch.equal(y, alone)
    finally:
        set_pdl(before)
    ref = x.double() @ (codes.float() * p6.scale.float()).bfloat16().double().t()
    assert float((alone.double() - ref).abs().max() / ref.abs().max()) < 2e-5


@pytest.mark.parametrize("m", [9, 23, 48, 64])
@pytest.mark.parametrize("out_f,in_f", [(4096, 2048), (2048, 6144), (1024, 5120), (640, 1536), (320, 512), (8224, 200)])
def test_p6_rows_have_the_same_bits_with_dependent_launches(out_f, in_f, m):
    """9..64 rows called one by one, with dependent launches and in a captured chain of them: the same bits of every layer,
    whatever its K splits; the second launch of the chain reads what the first one wrote.  (9 rows: hardly an outlier a block,
    the other kernel than at 23.)"""
    from ixrun_b200.p6 import P6Packed, set_pdl

    gen = torch.Generator(device="cuda").manual_seed(out_f + m)
    codes = (torch.randn(out_f, in_f, generator=gen, device="cuda") * (8 if m == 9 else 12)).round().clamp(-127, 127).to(torch.int8)
    a = P6Packed(codes, torch.tensor(0.007, dtype=torch.bfloat16), out_f, in_f)
    b = P6Packed(codes.t().contiguous(), torch.tensor(0.004, dtype=torch.bfloat16), in_f, out_f)
    x = torch.randn(m, in_f, generator=gen, device="cuda").bfloat16()
    call = (lambda p, t: p.gemm(t)) if in_f % 64 == 0 else (lambda p, t: p.rows(t))
    h = call(a, x)
    y = call(b, h)
    torch.cuda.synchronize()
    before = set_pdl(True)
    try:
        h1 = call(a, x)
        y1 = call(b, h1)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(3):
                h2 = call(a, x)
                y2 = call(b, h2)
        graph.replay()
        torch.cuda.synchronize()
    finally:
        set_pdl(before)
    for got in (h1, h2):
        assert torch.equal(got, h)
    for got in (y1, y2):
        assert torch.equal(got, y)


@pytest.mark.parametrize("m", [9, 32, 64])
def test_p6_rows_join_many_sums_in_pairs(m):
    """A layer of few rows and many columns: its fp32 outputs are 64 to 128 partial sums.  A rounding to the nearest has a relative
    error of 0.25e-7 (2^-23 / sqrt(12), the mantissa's mean 0.72), and so has each of the seven levels of a sum in pairs, as random
    partial sums keep their 2-norm from level to level: sqrt(7) of it, 0.66e-7.  Two levels' worth more for the short chains in the
    tensor core; one after the other the sums lose sqrt(12.8) of it."""
    from ixrun_b200.p6 import P6Packed

    gen = torch.Generator(device="cuda").manual_seed(m)
    codes = (torch.randn(300, 16384, generator=gen, device="cuda") * 6).round().clamp(-31, 31).to(torch.int8)
    p6 = P6Packed(codes, torch.tensor(2.0 ** -9, dtype=torch.bfloat16), 300, 16384)
    x = torch.randn(m, 16384, generator=gen, device="cuda").bfloat16()
    ref = x.double() @ (codes.double() * 2.0 ** -9).t()
    assert float((p6.gemm(x, out_dtype=torch.float32).double() - ref).norm() / ref.norm()) < 0.75e-7
