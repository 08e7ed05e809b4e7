"""Packed-linear modules and functional entry points (the reference's API
surface for this path) on the GPU, checked against the CPU oracle."""
import os

import numpy as np
import pytest
import torch
import torch.nn as nn

from oracle import ixb_oracle as O

pytestmark = pytest.mark.gpu


def bf16(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int16)).view(torch.bfloat16)


def bits(t):
    return t.detach().cpu().contiguous().view(torch.int16).numpy().view(np.uint16)


def oracle_y(codes, scale_t, x, out_f, in_f):
    sc = int(bits(scale_t.reshape(1))[0])
    return O.gemm_f32(codes, sc, bits(x.reshape(-1, in_f)), out_f, in_f)


def make_layer(out_f, in_f, seed, bias=False):
    from ixrun_b200.quantize import int8x_quantize

    torch.manual_seed(seed)
    # heavy-tail weights like the reference's parity scripts (tests/test_fused.py:17-22)
    w = torch.randn(out_f, in_f) * 0.005
    flat = w.view(-1)
    idx = torch.randperm(flat.numel())[: int(flat.numel() * 0.04)]
    flat[idx] = torch.randn(len(idx)) * 0.05
    w = w.bfloat16()
    p = int8x_quantize(w)
    b = (torch.randn(out_f) * 0.1).bfloat16() if bias else None
    codes = O.quantize_bf16(bits(w))[0]
    return w, p, b, codes


@pytest.mark.parametrize("out_f,in_f", [(1536, 1536), (512, 4608), (300, 96)])
def test_streaming_linear_single_token(out_f, in_f):
    from ixrun_b200.engine import StreamingLinear

    w, p, b, codes = make_layer(out_f, in_f, 0, bias=True)
    x = torch.randn(1, 1, in_f).bfloat16().cuda()
    ref = torch.from_numpy(oracle_y(codes, p["scale"], x, out_f, in_f)).bfloat16() + b
    # the default keeps one copy of the weights (the resident layout); keep_streams=True keeps the reference's
    # buffers beside it; resident="streams" runs the fused kernel on the streams themselves
    for kw in ({}, {"keep_streams": True}, {"resident": "streams"}):
        sl = StreamingLinear(p, bias=b, **kw)
        assert sl.out_features == out_f and sl.in_features == in_f
        if kw:
            assert sl._use_fused == (in_f % 32 == 0) and sl._b1.is_cuda and sl._l3.is_cuda
            if sl._use_fused:
                assert sl._q1.numel() == (out_f * (in_f // sl._split_chunk) if sl._split_chunk else out_f)
        else:
            assert not hasattr(sl, "_b1") and sl._dp is None and sl.resident_bytes == sl._res.resident_bytes
        y = sl(x)
        assert y.shape == (1, 1, out_f) and y.dtype == torch.bfloat16
        # one bf16 ulp of slack for sums that sit on a rounding boundary
        assert (y.cpu().float().reshape(-1) - ref.float().reshape(-1)).abs().max() <= 2.0 ** -7 * ref.float().abs().max()


def test_streaming_linear_many_tokens_uses_decode_buffer():
    from ixrun_b200.engine import StreamingLinear

    out_f, in_f = 256, 1024
    w, p, b, codes = make_layer(out_f, in_f, 1, bias=True)
    sl = StreamingLinear(p, bias=b, keep_streams=True)
    x = torch.randn(2, 16, in_f).bfloat16().cuda()
    ref = oracle_y(codes, p["scale"], x, out_f, in_f).reshape(2, 16, out_f) + b.float().numpy()
    # 9..64 rows: the tensor-core GEMM on the resident layout, no decode buffer involved (the fused paths round the
    # sum to bf16 and then add the bias in bf16, ixrun/engine.py:166-168: up to one more bf16 ulp than the dense path)
    y_gemm = sl(x)
    assert np.abs(y_gemm.float().cpu().numpy() - ref).max() / np.abs(ref).max() < 1e-2
    assert torch.equal(y_gemm.reshape(32, out_f), sl._res.gemm(x.reshape(32, in_f)) + b.cuda())
    # more than 64 rows (or the GEMM switched off): decode into the shared buffer + dense matmul
    sl._use_p6_gemm = False
    with pytest.raises(RuntimeError):
        sl(x)                                  # no shared buffer yet
    buf = torch.empty(out_f * in_f + 100, dtype=torch.bfloat16, device="cuda")
    sl._set_shared_buf(buf)
    y = sl(x)
    x_many = torch.randn(100, in_f).bfloat16().cuda()
    sl._use_p6_gemm = True
    assert sl(x_many).shape == (100, out_f)    # beyond the GEMM's row count: the decode path
    sl._use_p6_gemm = False
    w_dec = bf16(O.decode_bf16({**p, "scale": int(bits(p["scale"].reshape(1))[0]),
                                "bitmaps": [t.numpy() for t in p["bitmaps"]],
                                "streams": [t.numpy() for t in p["streams"]]}))
    assert torch.equal(sl._decode().cpu(), w_dec)
    err = np.abs(y.float().cpu().numpy() - ref).max() / np.abs(ref).max()
    assert err < 5e-3
    # the same input through the tensor-core fused kernel (opt-in)
    sl._use_tc = True
    y_tc = sl(x)
    # the fused paths round the sum to bf16 and then add the bias in bf16 (ixrun/engine.py:166-168):
    # up to one more bf16 ulp than the dense path, which adds the bias before rounding
    assert np.abs(y_tc.float().cpu().numpy() - ref).max() / np.abs(ref).max() < 1e-2
    assert torch.equal(y_tc.reshape(32, out_f), sl._dp.gemm(x.reshape(32, in_f)) + b.cuda())


def test_fused_gemv_and_prefix_functions_golden(golden_dir):
    from ixrun_b200.fused import compute_row_prefixes, fused_gemv

    g = dict(np.load(os.path.join(golden_dir, "heavy_64x1024.npz")))
    out_f, in_f = g["w_bits"].shape
    p = {"level_bits": (3, 5, 8), "out_f": out_f, "in_f": in_f, "N": out_f * in_f,
         "scale": bf16(g["scale_bits"]).reshape(()), "bitmaps": [torch.from_numpy(g["b1"]), torch.from_numpy(g["b2"])],
         "streams": [torch.from_numpy(g["l1"]), torch.from_numpy(g["l2"]), torch.from_numpy(g["l3"])],
         "counts": [int(c) for c in g["counts"]]}
    q1, q2 = compute_row_prefixes(p)
    assert q1.device.type == "cpu" and np.array_equal(q1.numpy(), g["row_q1"]) and np.array_equal(q2.numpy(), g["row_q2"])
    chunk = int(g["chunk"][0])
    q1c, q2c = compute_row_prefixes(p, chunk)
    assert np.array_equal(q1c.numpy(), g["chunk_q1"]) and np.array_equal(q2c.numpy(), g["chunk_q2"])
    dev = "cuda"
    x = bf16(g["x_bits"])[0].to(dev)
    gb = [t.to(dev) for t in (*p["bitmaps"], *p["streams"])]
    y = fused_gemv(x, *gb, q1.to(dev), q2.to(dev), p["scale"].to(dev), out_f, in_f)
    ref = g["y_f32"][0]
    assert y.shape == (out_f,) and y.dtype == torch.bfloat16
    assert np.abs(y.float().cpu().numpy() - ref).max() / np.abs(ref).max() < 5e-3
    y32 = torch.full((out_f,), 7.0, dtype=torch.float32, device=dev)      # stale contents must not matter
    r = fused_gemv(x, *gb, q1c.to(dev), q2c.to(dev), p["scale"].to(dev), out_f, in_f, chunk=chunk, y32=y32)
    assert r is y32
    assert np.abs(y32.cpu().numpy() - ref).max() / np.abs(ref).max() < 2e-5


def test_decode_functions_and_cached_linear():
    from ixrun_b200.kernels import decode_codes, decode_weight_triton, precompute_block_offsets
    from ixrun_b200.linear import Int8XLinear

    out_f, in_f = 128, 256
    w, p, b, codes = make_layer(out_f, in_f, 2, bias=True)
    wd = decode_weight_triton(p, device="cuda")
    assert torch.equal(decode_codes(p).cpu().reshape(-1), torch.from_numpy(codes))
    sc = p["scale"].float()
    assert torch.equal(wd.cpu(), (torch.from_numpy(codes).float() * sc).bfloat16().view(out_f, in_f))
    a, c = precompute_block_offsets(p, 1024)
    np_p = {**p, "scale": 0, "bitmaps": [t.numpy() for t in p["bitmaps"]], "streams": [t.numpy() for t in p["streams"]]}
    q1, q2 = O.prefixes(np_p, 1024)
    assert np.array_equal(a.cpu().numpy(), q1) and np.array_equal(c.cpu().numpy(), q2)
    a2, c2 = precompute_block_offsets(p, 4096)
    q1, q2 = O.prefixes(np_p, 4096)
    assert np.array_equal(a2.cpu().numpy(), q1) and np.array_equal(c2.cpu().numpy(), q2)
    for cache in ("full", "none"):
        lin = Int8XLinear(p, bias=b, cache=cache)
        x = torch.randn(4, in_f).bfloat16().cuda()
        y = lin(x)
        ref = torch.nn.functional.linear(x, wd, b.cuda())
        assert torch.equal(y, ref)


class ToyBlock(nn.Module):
    def __init__(self, h=256, f=768):
        super().__init__()
        self.gate_proj = nn.Linear(h, f, bias=False)
        self.up_proj = nn.Linear(h, f, bias=False)
        self.down_proj = nn.Linear(f, h, bias=True)
        self.lm_head = nn.Linear(h, 64, bias=False)      # skipped by name
        self.tiny = nn.Linear(8, 8)                      # skipped by size

    def forward(self, x):
        return self.down_proj(torch.nn.functional.silu(self.gate_proj(x)) * self.up_proj(x))


@pytest.mark.parametrize("mode", ["cached", "streaming", "graph"])
def test_engine_deploy_modes_agree(mode, tmp_path):
    from ixrun_b200.engine import GraphLinear, Int8XEngine, StreamingLinear
    from ixrun_b200.linear import Int8XLinear, iter_quantizable_linears

    torch.manual_seed(0)
    ref_model = ToyBlock().bfloat16()
    names = [n for n, _ in iter_quantizable_linears(ref_model)]
    assert names == ["gate_proj", "up_proj", "down_proj"]
    # ground truth: the same block with weights replaced by their decoded int8 values
    from ixrun_b200.kernels import decode_weight
    from ixrun_b200.quantize import int8x_quantize

    gt = ToyBlock().bfloat16()
    gt.load_state_dict(ref_model.state_dict())
    for n in names:
        lin = getattr(gt, n)
        lin.weight.data = decode_weight(int8x_quantize(lin.weight.data)).cpu()
    gt = gt.cuda()
    model = ToyBlock().bfloat16()
    model.load_state_dict(ref_model.state_dict())
    replay = None
    if mode == "cached":
        model = model.cuda()
        stats = Int8XEngine._deploy_cached(model, (3, 5, 8), verbose=False)
        assert isinstance(model.gate_proj, Int8XLinear) and stats["n_layers"] == 3
    elif mode == "streaming":
        cache = str(tmp_path / "packed.pt")
        stats = Int8XEngine._deploy_streaming(model, (3, 5, 8), verbose=False, cache_path=cache)
        assert os.path.exists(cache) and isinstance(model.down_proj, StreamingLinear)
        # second deploy loads the cache file; a wrong scheme is rejected
        m2 = ToyBlock().bfloat16()
        Int8XEngine._deploy_streaming(m2, (3, 5, 8), verbose=False, cache_path=cache)
        with pytest.raises(ValueError):
            Int8XEngine._deploy_streaming(ToyBlock().bfloat16(), (2, 5, 8), verbose=False, cache_path=cache)
        model = model.cuda()
    else:
        stats, replay = Int8XEngine._deploy_graph(model, (3, 5, 8), verbose=False)
        assert isinstance(model.up_proj, GraphLinear)
        model = model.cuda()
        for n in names:                       # buffers are only valid after a replay
            getattr(model, n)._w_buf.zero_()
        replay()
    assert stats["total_bytes"] > 0
    for shape in [(1, 1, 256), (1, 5, 256), (2, 9, 256)]:
        x = torch.randn(*shape).bfloat16().cuda()
        y, y_gt = model(x), gt(x)
        tol = 2e-2 * y_gt.float().abs().max()
        assert (y.float() - y_gt.float()).abs().max() <= tol, (mode, shape)


def test_graphed_layer_sequence_matches_eager():
    """CUDA-graph capture of a per-layer sequence of fused launches"""
    from ixrun_b200.engine import GraphedCall, StreamingLinear

    h, f = 512, 1536
    layers = [StreamingLinear(make_layer(f, h, 10)[1]), StreamingLinear(make_layer(f, h, 11)[1]),
              StreamingLinear(make_layer(h, f, 12)[1])]

    def mlp(x):
        return layers[2](torch.nn.functional.silu(layers[0](x)) * layers[1](x))

    x = torch.randn(1, h).bfloat16().cuda()
    gc = GraphedCall(mlp, x)
    for _ in range(3):
        x = torch.randn(1, h).bfloat16().cuda()
        assert torch.equal(gc(x), mlp(x))


def test_graphed_call_with_host_buffers_is_one_launch_per_call():
    """host_io=True: the copies from and to pinned host memory are part of the graph; run_host returns the result
    in host memory, equal to the eager module call on the same input."""
    from ixrun_b200.engine import GraphedCall, StreamingLinear

    lay = StreamingLinear(make_layer(768, 1024, 21)[1])
    gc = GraphedCall(lay, torch.zeros(1, 1024).bfloat16().cuda(), host_io=True)
    for i in range(3):
        x = torch.randn(1, 1024, generator=torch.Generator().manual_seed(i)).bfloat16()
        y = gc.run_host(x)
        assert not y.is_cuda and y.is_pinned()
        assert torch.equal(y, lay(x.cuda()).cpu())
    with pytest.raises(RuntimeError):
        GraphedCall(lay, torch.zeros(1, 1024).bfloat16().cuda()).run_host(x)


@pytest.mark.parametrize("in_f,rows", [(512, 65), (512, 128), (512, 129), (1056, 24), (1056, 64), (1056, 100)])
def test_streaming_linear_passes_keep_what_a_dense_matmul_gives(in_f, rows):
    """9..64 rows without a bias in one pass of the resident kernel, whatever in_f: values against float64 (one bf16
    rounding, 2^-8), an unaligned input, gradients and forward-mode tangents as from the matmul that took these calls
    before, and takes the ones with more rows."""
    import torch.autograd.forward_ad as fwAD

    from ixrun_b200.engine import StreamingLinear

    out_f = 200
    gen = torch.Generator(device="cuda").manual_seed(rows)
    w = (torch.randn(out_f, in_f, generator=gen, device="cuda") * 0.05).bfloat16()
    lin = StreamingLinear.from_weight(w)
    x = torch.randn(rows, in_f, generator=gen, device="cuda").bfloat16()
    if rows > 64 or in_f % 64:
        with pytest.raises(RuntimeError):
            lin(x)                                             # no decode buffer: refused, as always
    lin._set_shared_buf(torch.empty(out_f * in_f, dtype=torch.bfloat16, device="cuda"))
    wd = lin._res.decode(kind="bf16").double()
    ref = x.double() @ wd.t()
    ok = lambda y, r: bool(((y.double() - r).abs() <= r.abs() * 2.0 ** -8 + 1e-5 * r.abs().max()).all())
    assert ok(lin(x), ref) and lin(x).shape == (rows, out_f)
    odd = torch.empty(rows * in_f + 1, dtype=torch.bfloat16, device="cuda")[1:].view(rows, in_f)
    odd.copy_(x)
    if rows <= 64:
        assert ok(lin(odd), ref)
    else:                                                      # the dense matmul, which may reduce such an input in bf16
        assert torch.equal(lin(odd), torch.nn.functional.linear(odd, lin._decode()))
    xg = x.clone().requires_grad_()
    lin(xg).sum().backward()
    assert ok(xg.grad, wd.sum(0).expand(rows, in_f))
    t = torch.ones_like(x)
    with fwAD.dual_level():
        y, tangent = fwAD.unpack_dual(lin(fwAD.make_dual(x, t)))
        assert ok(y, ref) and ok(tangent, t.double() @ wd.t())


@pytest.mark.parametrize("in_f", [1024, 1056])
def test_streaming_linear_refuses_host_activations(monkeypatch, in_f):
    """No host pointer reaches a kernel: refused by the wrapper, or by the dense matmul where that took the call before.  (The
    library is replaced by one that fails the test when a kernel on the activations is asked for.)"""
    from ixrun_b200 import _lib
    from ixrun_b200.engine import StreamingLinear

    w = (torch.randn(64, in_f, device="cuda") * 0.05).bfloat16()
    lin = StreamingLinear.from_weight(w)
    lin._set_shared_buf(torch.empty(64 * in_f, dtype=torch.bfloat16, device="cuda"))
    real = _lib.lib()

    class NoLaunch:
        def __getattr__(self, name):
            if name in ("ixb_p6_gemv", "ixb_p6_gemm", "ixb_p6_rows"):
                return lambda *a: pytest.fail(f"{name} was called")
            return getattr(real, name)

    monkeypatch.setattr(_lib, "lib", lambda: NoLaunch())
    for rows in (1, 8, 9, 64, 65):
        with pytest.raises((ValueError, RuntimeError)):
            lin(torch.zeros(rows, in_f).bfloat16())


def test_streaming_linear_leaves_autocast_and_modes_to_the_dense_matmul():
    """9..64 rows with in_f not a multiple of 64: the result's type under autocast, what dispatch and function modes see, and
    an input with a pending negation, as with decode + dense matmul."""
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    from ixrun_b200.engine import StreamingLinear

    lin = StreamingLinear.from_weight((torch.randn(64, 1056, device="cuda") * 0.05).bfloat16())
    lin._set_shared_buf(torch.empty(64 * 1056, dtype=torch.bfloat16, device="cuda"))
    x = torch.randn(24, 1056, device="cuda").bfloat16()
    with torch.no_grad():
        y = lin(x)
        with torch.autocast("cuda", dtype=torch.float16):
            assert lin(x).dtype == torch.float16
        seen = []

        class Dispatch(TorchDispatchMode):
            def __torch_dispatch__(self, func, types, args=(), kwargs=None):
                seen.append(str(func))
                return func(*args, **(kwargs or {}))

        class Function(TorchFunctionMode):
            def __torch_function__(self, func, types, args=(), kwargs=None):
                seen.append(func.__name__)
                return func(*args, **(kwargs or {}))

        with Dispatch():
            lin(x)
        assert any("mm" in s for s in seen)
        seen.clear()
        with Function():
            lin(x)
        assert "linear" in seen
        assert (lin(torch._neg_view(x)).float() + y.float()).abs().max() <= 2.0 ** -7 * y.float().abs().max()


@pytest.mark.parametrize("in_f,bias", [(128, False), (128, True), (200, False)])
def test_call_through_the_extension_is_the_python_path(in_f, bias):
    """The extension's call takes ordinary activations and leaves the rest: every form gives what the Python path gives."""
    from ixrun_b200.engine import StreamingLinear

    class Sub(torch.Tensor):
        pass

    gen = torch.Generator(device="cuda").manual_seed(3)
    w = (torch.randn(96, in_f, generator=gen, device="cuda") * 0.02).bfloat16()
    b = torch.randn(96, generator=gen, device="cuda").bfloat16() if bias else None
    lin = StreamingLinear.from_weight(w, bias=b)
    lin._set_shared_buf(torch.empty(96 * in_f, dtype=torch.bfloat16, device="cuda"))
    big = torch.randn(4, 64, 2 * in_f + 8, generator=gen, device="cuda").bfloat16()
    forms = [big[0, 0, :in_f].clone(), big[:1, 0, :in_f], big[0, :8, :in_f].contiguous(), big[0, :9, :in_f].contiguous(),
             big[0, :64, :in_f].contiguous(), big[0, :64, :in_f], big[:, :2, :in_f].contiguous(), big[:, :3, :in_f].contiguous(),
             big[:2, :, :in_f].contiguous(), big[0, ::2, 8:8 + in_f],
             big[0, :2, :in_f].contiguous().requires_grad_(), big[0, :2, :in_f].contiguous().as_subclass(Sub),
             big[0, :in_f, :3].t().contiguous() if in_f <= 64 else big[0, :3, :in_f].t().contiguous().t()]
    stream = torch.cuda.Stream()
    for many in (True, False):
        lin._use_p6_gemm = many
        for x in forms:
            lin._res._call = None
            torch.cuda.synchronize()
            with torch.cuda.stream(stream):
                y = lin(x)
            lin._res._call = lambda *a: None
            ref = lin(x)
            torch.cuda.synchronize()
            assert type(y) is type(ref) and y.shape == ref.shape and y.dtype == ref.dtype and torch.equal(y, ref)
    lin._res._call = None
    for bad in (torch.randn(2, in_f).bfloat16(), torch.randn(2, in_f + 8, device="cuda").bfloat16()):
        with pytest.raises(Exception):
            lin(bad)
    assert lin(torch.randn(2, in_f, device="cuda")).dtype == torch.float32          # another type: the dense matmul


def test_a_scratch_that_is_replaced_serves_the_next_call():
    """Launches that may overlap need separate scratch instances: one that is set on a layer in use is the one that its next
    call takes, through the module as through `gemv`."""
    from ixrun_b200.engine import StreamingLinear
    from ixrun_b200.p6 import GemvScratch

    gen = torch.Generator(device="cuda").manual_seed(4)
    lin = StreamingLinear.from_weight((torch.randn(96, 8256, generator=gen, device="cuda") * 0.02).bfloat16())
    x = torch.randn(2, 8256, generator=gen, device="cuda").bfloat16()
    y = lin(x)
    for _ in range(2):
        own = lin._res.scratch = GemvScratch("cuda")
        assert own.buf.numel() == 0 and lin._res.scratch is own
        assert torch.equal(lin(x), y)
        assert own.buf.numel() > 0                       # the call asked this one
        torch.cuda.synchronize()
        assert not bool(own.buf.any())                   # (zero between launches)
        assert torch.equal(lin._res.gemv(x), y)


def test_the_packed_call_lets_other_threads_run():
    """The interpreter lock is free while the extension allocates and launches (a launch waits where the queue is full): the C
    library's sleep takes the place of the launch, and another thread goes on meanwhile."""
    import ctypes as C
    import threading
    import time

    from ixrun_b200 import _lib

    class Timespec(C.Structure):
        _fields_ = [("s", C.c_long), ("ns", C.c_long)]

    host, L = _lib.host(), _lib.lib()
    sleep = C.cast(C.CDLL(None).nanosleep, C.c_void_p).value
    for rows in (1, 64):
        nap = Timespec(1, 0)                             # in the place of the tensor's structure: the first argument
        call = host.p6(C.addressof(nap), 64, 128, 0, torch.zeros(1024, dtype=torch.uint8, device="cuda"))
        x = torch.zeros(rows, 128, dtype=torch.bfloat16, device="cuda")
        torch.cuda.synchronize()
        done = []
        host.bind(sleep, sleep, _lib.check)
        try:
            t = threading.Thread(target=lambda: (call(x, None, True), done.append(time.perf_counter())))
            t0 = time.perf_counter()
            t.start()
            while time.perf_counter() - t0 < 0.3:        # (with the lock held: not before the sleep is over)
                time.sleep(0.01)
            seen = time.perf_counter() - t0
            t.join()
        finally:
            host.bind(C.cast(L.ixb_p6_gemv, C.c_void_p).value, C.cast(L.ixb_p6_rows, C.c_void_p).value, _lib.check)
        assert seen < 0.9 and done[0] - t0 >= 1.0


def test_errors_of_the_extension_keep_their_type():
    """Memory that is not there and what a mode raises reach the caller as torch's functions raise them."""
    from torch.utils._python_dispatch import TorchDispatchMode

    from ixrun_b200 import _lib

    class Refuse(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            raise KeyError("refused")

    with pytest.raises(torch.OutOfMemoryError):
        _lib.host().empty(0, (16, "i"), (1 << 50, "B"))
    with Refuse(), pytest.raises(KeyError):
        _lib.host().empty(0, (16, "i"))
    a, b, c = _lib.host().empty(0, (16, "i"), (-1, "h"), (0, "b"))
    assert (a.dtype, a.shape, b.dtype, b.shape, c.dtype, c.shape) == (torch.int32, (16,), torch.bfloat16, (), torch.int8, (0,))


@pytest.mark.filterwarnings("ignore:the host extension")
def test_without_the_extension_the_python_path_serves(monkeypatch):
    """No compiler and no built file: deployment and calls go through Python, with the same results."""
    from ixrun_b200 import _lib
    from ixrun_b200 import build as b
    from ixrun_b200.engine import StreamingLinear

    gen = torch.Generator(device="cuda").manual_seed(6)
    w, bias = (torch.randn(96, 128, generator=gen, device="cuda") * 0.02).bfloat16(), torch.randn(96, device="cuda").bfloat16()
    xs = [torch.randn(m, 128, generator=gen, device="cuda").bfloat16() for m in (1, 8, 23, 64, 65)]

    def all_of():
        lin = StreamingLinear.from_weight(w, bias=bias)
        lin._set_shared_buf(torch.empty(96 * 128, dtype=torch.bfloat16, device="cuda"))
        return [lin(x) for x in xs] + [lin._res.plane[:-960], lin._res.esc[:lin._res.n_esc], lin._res.blk_off]

    want = all_of()

    def refuse(force=False):
        raise RuntimeError("no compiler")

    monkeypatch.setattr(_lib, "_host", None)
    monkeypatch.setattr(b, "host_is_stale", lambda: True)
    monkeypatch.setattr(b, "build_host", refuse)
    for got, ref in zip(all_of(), want):
        assert torch.equal(got, ref)


def test_a_prompt_asks_nothing_of_the_extension(monkeypatch):
    """More rows than the fused kernels take: no object of the extension is made for the layer, and none is called."""
    from ixrun_b200.engine import StreamingLinear
    from ixrun_b200.p6 import P6Packed

    lin = StreamingLinear.from_weight((torch.randn(96, 128, device="cuda") * 0.02).bfloat16())
    lin._set_shared_buf(torch.empty(96 * 128, dtype=torch.bfloat16, device="cuda"))
    calls = []
    monkeypatch.setattr(P6Packed, "make_call", lambda self: calls.append(1) or (lambda *a: None))
    for rows in (65, 1000):
        assert lin(torch.randn(rows, 128, device="cuda").bfloat16()).shape == (rows, 96)
    assert not calls and lin._res._call is None
    assert lin(torch.randn(64, 128, device="cuda").bfloat16()).shape == (64, 96) and calls
