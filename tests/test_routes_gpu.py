"""Launch routes chosen by size, alignment and magnitude, at the edges where each begins.

References: the float64 product on the device, and for values that a route must not change the
CUDA-core kernel's own result, bit for bit.  Tolerances are the bounds of fp32 accumulation
(k 2^-24 sum |a||b|, the factor 3 of the other parity tests) plus one rounding of the output."""
import hashlib
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

import tensilelite_gb300 as tl

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

LAYOUTS = ["NN", "NT", "TN", "TT"]
MANT = {torch.float32: 23, torch.float16: 10, torch.bfloat16: 7}


@pytest.fixture(scope="module")
def h():
    handle = tl.Handle()
    yield handle
    handle.close()


def _mat(g, rows, cols, ld, batch, dtype, dist="normal"):
    n = batch * ld * cols
    x = torch.randn(n, device="cuda", generator=g) if dist == "normal" else torch.rand(n, device="cuda", generator=g) * 2 - 1
    x = x.to(dtype)
    return x, x.view(batch, cols, ld)[:, :, :rows].transpose(1, 2).double()


class Case:
    def __init__(self, dtype, layout, m, n, k, *, beta=0.0, batch=1, pad=0, seed=0, dist="normal"):
        self.ta, self.tb = layout[0] == "T", layout[1] == "T"
        g = torch.Generator(device="cuda").manual_seed(seed)
        ra, ca = (k, m) if self.ta else (m, k)
        rb, cb = (n, k) if self.tb else (k, n)
        self.m, self.n, self.k, self.batch, self.beta = m, n, k, batch, beta
        self.lda, self.ldb, self.ldc = ra + pad, rb + pad, m + pad
        self.A, a = _mat(g, ra, ca, self.lda, batch, dtype, dist)
        self.B, b = _mat(g, rb, cb, self.ldb, batch, dtype, dist)
        self.C, c = _mat(g, m, n, self.ldc, batch, dtype)
        self.a, self.b = (a.transpose(1, 2) if self.ta else a), (b.transpose(1, 2) if self.tb else b)
        self.c, self.dtype = c, dtype

    def run(self, h, kernel="auto", in_place=False, stream=None):
        D = self.C.clone() if in_place else torch.full_like(self.C, float("nan"))
        p = tl.Problem.make(self.m, self.n, self.k, dtype=tl.torch_dtype_code(self.dtype), trans_a=self.ta,
                            trans_b=self.tb, beta=self.beta, lda=self.lda, ldb=self.ldb, ldc=self.ldc, ldd=self.ldc,
                            batch=self.batch, kernel=kernel)
        h.gemm(p, D, D if in_place else self.C, self.A, self.B, stream=stream)
        return D

    def view(self, D):
        return D.view(self.batch, self.n, self.ldc)[:, :, :self.m].transpose(1, 2)

    def check(self, D):
        ref = self.a @ self.b + self.beta * self.c
        bound = 3.0 * self.k * 2.0 ** -24 * (self.a.abs() @ self.b.abs()) + 2.0 ** -MANT[self.dtype] * ref.abs() + \
            2.0 ** -23 * (self.beta * self.c).abs() + 1e-30
        got = self.view(D).double()
        assert torch.isfinite(got).all()
        assert bool(((got - ref).abs() <= bound).all())
        return float((got - ref).norm() / ref.norm())


# ---- shared pieces of the fp32 split: more than one wave of 256 x 128 tiles (here by batch), sizes at the
# edges of the 256 x 256 tile and of a k-block ----
@pytest.mark.parametrize("kernel,most", [("bf16x3", 6e-6), ("bf16x6", 4e-7)])
@pytest.mark.parametrize("layout,m,n,k,beta", [("NN", 136, 256, 64, 0.0), ("TN", 256, 264, 72, 0.5),
                                               ("NT", 264, 200, 256, 0.0), ("TT", 520, 520, 200, 0.5)])
def test_shared_pieces_edges(h, kernel, most, layout, m, n, k, beta):
    c = Case(torch.float32, layout, m, n, k, beta=beta, batch=40, dist="uniform")
    D = c.run(h, kernel)
    h.device_status()
    ref = c.a @ c.b + beta * c.c
    err = float((c.view(D).double() - ref).norm() / ref.norm())
    assert err < most      # 2^-18 class for two pieces, fp32 accumulation for three


@pytest.mark.parametrize("m,n,k", [(3000, 2000, 1096), (4096, 2560, 64)])
def test_shared_pieces_last_wave(h, m, n, k):
    c = Case(torch.float32, "TN", m, n, k, dist="uniform")
    assert c.check(c.run(h, "bf16x6")) < 4e-7
    h.device_status()


# ---- promoted chains of an NN problem that runs as its transposed view ----
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,n,k,mt1", [(136, 72, 2048, 128), (520, 392, 2056, 256), (256, 512, 2112, 256)])
def test_promoted_chains_of_the_transposed_view(h, dtype, m, n, k, mt1):
    c = Case(dtype, "NN", m, n, k)
    p = tl.Problem.make(m, n, k, dtype=tl.torch_dtype_code(dtype), lda=c.lda, ldb=c.ldb, ldc=c.ldc, ldd=c.ldc)
    s = tl.Solution(kernel=tl.KERNEL_TCGEN05, macro_tile0=128, macro_tile1=mt1, stages=4, split_k=1, promote_k=256)
    D = torch.full_like(c.C, float("nan"))
    h.gemm(p, D, None, c.A, c.B, solution=s)
    c.check(D)
    h.device_status()


# ---- plain fp32 left to the library: the tensor cores from 3e8 multiply-adds on ----
@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("m,n,k,beta,batch,pad", [(1024, 1024, 320, 0.0, 1, 0), (711, 653, 701, 0.5, 1, 3),
                                                  (64, 5000, 1003, 0.0, 1, 0), (333, 257, 129, 0.5, 40, 1),
                                                  (2048, 1000, 64, 0.0, 5, 64)])
def test_fp32_auto_matches_fp64_as_the_cuda_cores(h, layout, m, n, k, beta, batch, pad):
    c = Case(torch.float32, layout, m, n, k, beta=beta, batch=batch, pad=pad)
    l0 = h.launch_count()
    D = c.run(h)
    assert h.launch_count() - l0 == 4          # two splits, tensor cores, CUDA cores (returning at once)
    err = c.check(D)
    h.device_status()
    assert err <= max(1.5 * c.check(c.run(h, "simt")), 3e-7)
    if pad:                                     # the gap between columns is not written
        assert torch.isnan(D.view(batch, n, c.ldc)[:, :, m:]).all()
    if beta:
        assert torch.equal(c.run(h, in_place=True).view(torch.int32).view(batch, n, c.ldc)[:, :, :m],
                           D.view(torch.int32).view(batch, n, c.ldc)[:, :, :m])


@pytest.mark.parametrize("where,value", [("A", float("inf")), ("B", float("-inf")), ("A", float("nan")), ("B", 3e38),
                                         ("A", 1e-40), ("B", 1e-33), ("A", 1e25)])
def test_fp32_auto_out_of_range_is_the_cuda_core_result(h, where, value):
    c = Case(torch.float32, "TN", 720, 700, 640, beta=0.5)
    (c.A if where == "A" else c.B)[12345] = value
    if value == 1e25:
        c.B.mul_(1e13)
    got, want = c.run(h), c.run(h, "simt")
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    # in place, where a first launch that wrote anything would be seen by the second
    got, want = c.run(h, in_place=True), c.run(h, "simt", in_place=True)
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    h.device_status()


def test_fp32_auto_zero_operands(h):
    c = Case(torch.float32, "NN", 700, 700, 700, beta=0.5)
    c.A.zero_()
    assert torch.equal(c.run(h).view(torch.int32), c.run(h, "simt").view(torch.int32))


def test_fp32_auto_streams_and_threads_are_independent(h):
    cases = [Case(torch.float32, "TN", 900 + 64 * i, 1100, 512, seed=i) for i in range(4)]
    want = [c.run(h) for c in cases]
    torch.cuda.synchronize()
    got = [None] * 4

    def work(i):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for _ in range(6):
                got[i] = cases[i].run(h, stream=s)
        s.synchronize()

    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    for g, w in zip(got, want):
        assert torch.equal(g.view(torch.int32), w.view(torch.int32))
    h.device_status()


def test_fp32_auto_under_capture_runs_the_cuda_cores():
    h = tl.Handle()
    c = Case(torch.float32, "NN", 800, 800, 800)
    want = c.run(h, "simt")
    s = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        with torch.cuda.graph(g, stream=s):
            D = c.run(h, stream=s)
        g.replay()
    s.synchronize()
    assert torch.equal(D.view(torch.int32), want.view(torch.int32))
    h.close()


# ---- 16-bit operands off 16-byte boundaries: aligned copies and the tensor cores from 1.5e8 on ----
@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,n,k,beta,batch,pad", [(1001, 515, 433, 0.5, 1, 0), (520, 640, 678, 0.0, 1, 3),
                                                  (64, 1601, 2051, 0.0, 1, 0), (130, 129, 337, 0.5, 40, 1),
                                                  (777, 65, 3001, 0.0, 1, 0), (2040, 1999, 2049, 0.0, 1, 1)])
def test_unaligned_half_matches_fp64_as_the_cuda_cores(h, dtype, layout, m, n, k, beta, batch, pad):
    c = Case(dtype, layout, m, n, k, beta=beta, batch=batch, pad=pad)
    assert any(ld % 8 for ld in (c.lda, c.ldb))
    l0 = h.launch_count()
    D = c.run(h)
    # copies, tensor cores, and from 2e5 outputs that are not whole vectors a copy back
    assert h.launch_count() - l0 == 2 + (m * n * batch >= 2e5 and (m % 8 or c.ldc % 8) != 0)
    err = c.check(D)
    h.device_status()
    assert err <= 1.02 * c.check(c.run(h, "simt"))      # both are one output rounding away
    if pad:
        assert torch.isnan(D.view(batch, n, c.ldc)[:, :, m:]).all()
    if beta:
        assert torch.equal(c.run(h, in_place=True).view(torch.int16).view(batch, n, c.ldc)[:, :, :m],
                           D.view(torch.int16).view(batch, n, c.ldc)[:, :, :m])


@pytest.mark.parametrize("off_a,off_b", [(1, 0), (0, 3), (2, 5), (7, 4)])
def test_unaligned_half_bases(h, off_a, off_b):
    c = Case(torch.float16, "TN", 640, 768, 512)
    want = c.run(h, "tcgen05")
    for name, off in (("A", off_a), ("B", off_b)):
        x = getattr(c, name)
        y = torch.full((x.numel() + off,), float("nan"), device="cuda", dtype=x.dtype)[off:]
        y.copy_(x)
        setattr(c, name, y)
    D = c.run(h)
    c.check(D)
    assert float((D.double() - want.double()).norm() / want.double().norm()) < 2e-4
    h.device_status()


def test_unaligned_half_capture_and_streams():
    h = tl.Handle()
    c = Case(torch.bfloat16, "TN", 801, 700, 515, beta=0.5)
    want = c.run(h, "simt")
    D = torch.empty_like(want)
    p = tl.Problem.make(c.m, c.n, c.k, dtype="bf16", trans_a=True, beta=0.5, lda=c.lda, ldb=c.ldb, ldc=c.ldc, ldd=c.ldc)
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        h.gemm(p, D, c.C, c.A, c.B, stream=s)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(D.view(torch.int16), want.view(torch.int16))      # captured: the CUDA-core kernel
    cases = [Case(torch.bfloat16, "NN", 301 + 64 * i, 1100, 1011, seed=i) for i in range(4)]      # split k
    alone = [x.run(h) for x in cases]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in cases]
    for _ in range(5):
        got = []
        for x, st in zip(cases, streams):
            with torch.cuda.stream(st):
                got.append(x.run(h, stream=st))
        torch.cuda.synchronize()
        for a, b in zip(got, alone):
            assert torch.equal(a.view(torch.int16), b.view(torch.int16))
    h.device_status()
    h.close()


# ---- CUDA-core kernel, small tiles: slabs read by lines, at the edges of the 64 x 32 tile and the slab ----
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("m,n,k,beta,pad", [(64, 32, 64, 0.0, 0), (65, 33, 67, 0.5, 0), (63, 31, 1, 0.0, 4), (1, 100, 130, 0.5, 3),
                                            (200, 96, 316, 0.0, 4)])
def test_cuda_core_small_tiles(h, dtype, layout, m, n, k, beta, pad):
    c = Case(dtype, layout, m, n, k, beta=beta, batch=2, pad=pad)
    D = c.run(h, "simt")
    c.check(D)
    if pad:
        assert torch.isnan(D.view(2, n, c.ldc)[:, :, m:]).all()


# ---- output path: whole lines through shared memory, or element by element ----
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("layout", ["TN", "NT"])
@pytest.mark.parametrize("m,n,k,beta,pad", [(256, 256, 64, 0.0, 0), (264, 129, 128, 0.5, 0), (257, 300, 136, 0.5, 7),
                                            (1000, 600, 520, 0.5, 0), (8, 1, 64, 0.0, 8), (72, 513, 64, 0.5, 8)])
def test_output_lines_and_elements(h, dtype, layout, m, n, k, beta, pad):
    c = Case(dtype, layout, m, n, k, beta=beta, batch=2)
    # padded leading dimensions of C and D only: operands stay 16-byte aligned
    if c.ta is False and m % 8:
        c = Case(dtype, "TN", m, n, k, beta=beta, batch=2)
    D = c.run(h)
    c.check(D)
    if beta:
        assert torch.equal(c.run(h, in_place=True).view(torch.int16), D.view(torch.int16))
    if pad:
        ld = m + pad
        W = torch.full((2 * n * ld,), float("nan"), dtype=dtype, device="cuda")
        Cp = torch.zeros(2, n, ld, dtype=dtype, device="cuda")
        Cp[:, :, :m] = c.C.view(2, n, m)
        p = tl.Problem.make(m, n, k, dtype=tl.torch_dtype_code(dtype), trans_a=c.ta, trans_b=c.tb, beta=beta, lda=c.lda,
                            ldb=c.ldb, ldc=ld, ldd=ld, batch=2)
        h.gemm(p, W, Cp, c.A, c.B)
        W = W.view(2, n, ld)
        assert torch.equal(W[:, :, :m].contiguous().view(torch.int16), D.view(2, n, m).view(torch.int16))
        assert torch.isnan(W[:, :, m:]).all()
    h.device_status()


# ---- quantisation: vector and element paths, sources and destinations off the 16-byte grid ----
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("n,so,do", [(1, 0, 0), (15, 1, 0), (16, 0, 0), (17, 0, 1), (4097, 3, 3), (100003, 1, 1),
                                     (1 << 20, 0, 0), ((1 << 20) + 5, 0, 8)])
def test_quantize_alignments(h, dtype, n, so, do):
    g = torch.Generator(device="cuda").manual_seed(n)
    src = (torch.randn(n + so, device="cuda", generator=g) * 3).to(dtype)[so:]
    buf = torch.full((n + do + 32,), 0xAA, dtype=torch.uint8, device="cuda")
    scale, amax = torch.zeros(1, device="cuda"), torch.full((1,), 7e9, device="cuda")
    h.quantize_fp8(src, n, buf[do:], scale, amax, src_dtype=tl.torch_dtype_code(dtype))
    a = src.float().abs().max()
    want = (src.float() * (torch.tensor(448.0, device="cuda") / a)).clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)
    assert float(amax) == float(a) and np.float32(float(scale)) == np.float32(float(a)) / np.float32(448.0)
    assert torch.equal(buf[do:do + n], want)
    assert bool((buf[do + n:] == 0xAA).all()) and bool((buf[:do] == 0xAA).all())


# ---- FP8 outputs: tiles that are no whole number of 128-column groups (192 wide), and the tile that the
# library picks by itself.  D starts as E4M3's NaN, which a saturating store never writes ----
@pytest.mark.parametrize("dtype,layout,m,n,k,tile", [
    ("bf16", "NN", 192, 129, 192, 192), ("fp16", "NT", 400, 128, 64, 192), ("fp8", "TN", 176, 300, 256, 192),
    ("bf16", "TN", 784, 257, 320, 192), ("bf16", "TN", 1152, 2752, 2624, 0), ("fp8", "TN", 1344, 4608, 1472, 0),
    ("bf16", "NN", 384, 8192, 1024, 0), ("fp8", "TN", 128, 200, 256, 128), ("bf16", "NT", 320, 200, 128, 64)])
def test_fp8_output_covers_every_tile(h, dtype, layout, m, n, k, tile):
    ta, tb = layout[0] == "T", layout[1] == "T"
    (ra, ca), (rb, cb) = ((k, m) if ta else (m, k)), ((n, k) if tb else (k, n))
    g = torch.Generator(device="cuda").manual_seed(m + n)
    to = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp8": torch.float8_e4m3fn}[dtype]
    A, B = (torch.randn(r * c, device="cuda", generator=g).to(to) for r, c in ((ra, ca), (rb, cb)))
    a, b = (x.double().view(c, r).T for x, r, c in ((A, ra, ca), (B, rb, cb)))
    ref = (a.T if ta else a) @ (b.T if tb else b)
    bound = 3.0 * k * 2.0 ** -24 * ((a.T if ta else a).abs() @ (b.T if tb else b).abs())      # fp32 accumulation
    p = tl.Problem.make(m, n, k, dtype=dtype, out_dtype="fp8", trans_a=ta, trans_b=tb)
    sol = tl.Solution(kernel=tl.KERNEL_TCGEN05, macro_tile0=tile, macro_tile1=128, stages=4, split_k=1) if tile else None
    assert tile or h.default_solution(p).macro_tile0 == 192
    D = torch.full((m * n + 64,), 0x7f, dtype=torch.uint8, device="cuda")
    amax = torch.zeros(1, device="cuda")
    scale = 2.0
    h.gemm_ex(p, D, None, A, B, amax=amax, d_scale=scale, solution=sol)
    h.device_status()
    got = D[:m * n].view(torch.float8_e4m3fn).double().view(n, m).T
    assert torch.isfinite(got).all() and bool((D[m * n:] == 0x7f).all())
    want = (ref * scale).clamp(-448, 448)
    # half a step of E4M3 (three bits; 2^-9 below 2^-6) beside the accumulation's error
    assert bool(((got - want).abs() <= 2.0 ** -4 * want.abs() + 2.0 ** -10 + scale * bound).all())
    assert abs(float(amax) - float(ref.abs().max())) <= float(bound.max())
    if not tile:
        E = torch.full((m * n,), 0x7f, dtype=torch.uint8, device="cuda")
        h.gemm(p, E, None, A, B)
        got = E.view(torch.float8_e4m3fn).double().view(n, m).T
        want = ref.clamp(-448, 448)
        assert bool(((got - want).abs() <= 2.0 ** -4 * want.abs() + 2.0 ** -10 + bound).all())


# ---- magnitudes whose leading bf16 piece is infinite, beside operands small enough for finite sums ----
@pytest.mark.parametrize("where,bits", [("A", 0x7f7fffff), ("A", 0xff7fffff), ("B", 0x7f7fffff), ("B", 0x7f7f8000),
                                        ("A", 0x7f7f7fff)])
def test_fp32_auto_next_to_the_largest_float(h, where, bits):
    c = Case(torch.float32, "TN", 720, 700, 640)
    other = c.B if where == "A" else c.A
    other.mul_(1e-5)
    x = c.A if where == "A" else c.B
    x[12345] = float(np.uint32(bits).view(np.float32))
    got, want = c.run(h), c.run(h, "simt")
    assert torch.isfinite(want).all() and torch.isfinite(got).all()
    if bits & 0x7fffffff >= 0x7f7f8000:
        assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    else:                           # the largest magnitude whose pieces are finite
        c.a = c.A.view(1, c.m, c.lda)[:, :, :c.k].double()
        c.b = c.B.view(1, c.n, c.ldb)[:, :, :c.k].transpose(1, 2).double()
        c.check(got)
    h.device_status()


# ---- shared pieces: as exact as the tiles that load every product's pieces.  Largest error, 2-norm and mean
# signed error against float64, each within a tenth of those of the one-SM tile's (the same chains) ----
@pytest.mark.parametrize("kernel", ["bf16x3", "bf16x6"])
@pytest.mark.parametrize("k", [64, 512, 8192])
@pytest.mark.parametrize("dist", ["normal", "uniform", "positive"])
def test_shared_pieces_are_as_exact_as_single_products(h, kernel, k, dist):
    c = Case(torch.float32, "TN", 3072, 3072, k, dist="normal" if dist == "normal" else "uniform")
    if dist == "positive":
        for x in (c.A, c.B, c.a, c.b):
            x.abs_()
    p = tl.Problem.make(c.m, c.n, k, dtype="fp32", trans_a=True, kernel=kernel)
    one_sm = h.default_solution(p)
    assert one_sm.macro_tile1 == 256
    one_sm.macro_tile1, one_sm.stages = 128, 4
    ref = c.a @ c.b
    errs = []
    for sol in (None, one_sm):
        D = torch.full_like(c.C, float("nan"))
        h.gemm(p, D, None, c.A, c.B, solution=sol)
        e = c.view(D).double() - ref
        errs.append((float(e.abs().max() / ref.abs().max()), float(e.norm() / ref.norm()),
                     abs(float((e * ref.sign()).mean() / ref.abs().mean()))))
    h.device_status()
    for got, want in zip(*errs):
        assert got <= 1.1 * want


# ---- splits of a call with scratch of its own: whoever sums a chunk, the same bits.  Waiting as by default, not at
# all (every share is left to the last split) and by the last split alone ----
SPLIT_CASES = [(torch.float32, "TN", 300, 400, 4096, 0.5), (torch.float32, "NN", 700, 700, 700, 0.0),
               (torch.bfloat16, "NN", 129, 257, 8191, 0.0), (torch.float16, "TN", 301, 1100, 1011, 0.5)]


def split_digests(h):
    out = []
    for dtype, layout, m, n, k, beta in SPLIT_CASES:
        c = Case(dtype, layout, m, n, k, beta=beta)
        for _ in range(3):
            D = c.run(h)
        h.device_status()
        c.check(D)
        out.append(hashlib.sha256(c.view(D).contiguous().view(torch.uint8).cpu().numpy().tobytes()).hexdigest())
    return out


@pytest.mark.parametrize("env", [{"TL_SPLIT_WAIT_NS": "0"}, {"TL_SPLIT_WAIT_NS": "700"}, {"TL_PAR_REDUCE": "0"}])
def test_split_shares_left_to_the_last(h, env):
    here = os.path.dirname(os.path.abspath(__file__))
    code = ("import sys; sys.path[:0] = %r\nimport test_routes_gpu as t\nh = t.tl.Handle()\nprint(' '.join(t.split_digests(h)))"
            % [os.path.dirname(here), here])
    r = subprocess.run([sys.executable, "-c", code], env={**os.environ, **env}, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stdout.split() == split_digests(h)


# ---- plain fp32, the sizes at which the CUDA cores would sum in eight groups of k: the relative 2-norm against
# float64 is no larger than theirs.  Values of one sign with short k, where a chain's two truncations (3.3e-8
# together) add up instead of averaging out, may take a fifth more ----
@pytest.mark.parametrize("dist", ["normal", "uniform", "positive"])
@pytest.mark.parametrize("m,n,k", [(1024, 1024, 320), (2304, 1024, 256), (2048, 1024, 160), (1024, 600, 512), (700, 700, 700),
                                   (64, 5000, 1003), (1024, 1024, 2048), (300, 400, 4096)])
def test_fp32_auto_is_as_exact_as_the_cuda_cores(h, m, n, k, dist):
    c = Case(torch.float32, "TN", m, n, k, dist="normal" if dist == "normal" else "uniform")
    if dist == "positive":
        for x in (c.A, c.B, c.a, c.b):
            x.abs_()
    ref = c.a @ c.b
    errs = [float((c.view(c.run(h, kernel)).double() - ref).norm() / ref.norm()) for kernel in ("auto", "simt")]
    h.device_status()
    assert errs[0] <= (1.2 if dist == "positive" and k < 512 else 1.0) * errs[1]


# ---- tuning: no slower than no solution ----
def _median_us(run, reps=7):
    run(), run()
    times = []
    for _ in range(reps):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(5):
            run()
        e1.record()
        torch.cuda.synchronize()
        times.append(e0.elapsed_time(e1) * 200)
    return sorted(times)[reps // 2]


@pytest.mark.parametrize("kernel", ["bf16x3", "bf16x6"])
def test_tuned_split_products_keep_the_shared_pieces(kernel):
    h = tl.Handle()
    c = Case(torch.float32, "TN", 4096, 4096, 2048)
    p = tl.Problem.make(4096, 4096, 2048, dtype="fp32", trans_a=True, kernel=kernel)
    D = torch.empty_like(c.C)
    run = lambda: h.gemm(p, D, None, c.A, c.B)
    before = _median_us(run)
    h.tune(p, D, None, c.A, c.B, max_candidates=3, reps=3)
    assert _median_us(run) <= 1.2 * before
    # the ring's depth does not choose the algorithm: a deeper ring is no slower
    s = h.default_solution(p)
    s.stages = 8
    assert _median_us(lambda: h.gemm(p, D, None, c.A, c.B, solution=s)) <= 1.2 * before
    h.close()


@pytest.mark.parametrize("dtype,kernel", [("fp32", "bf16x6"), ("bf16", "auto"), ("fp8", "auto")])
def test_the_first_candidate_is_the_default(dtype, kernel):
    h = tl.Handle()
    m, n, k = 1152, 2048, 1024
    t = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp8": torch.float8_e4m3fn}[dtype]
    A, B = torch.randn(m * k, device="cuda").to(t), torch.randn(n * k, device="cuda").to(t)
    D = torch.empty(m * n, device="cuda", dtype=torch.bfloat16 if dtype == "fp8" else t)
    p = tl.Problem.make(m, n, k, dtype=dtype, out_dtype="bf16" if dtype == "fp8" else dtype, trans_a=True, kernel=kernel)
    best, ms = h.tune(p, D, None, A, B, max_candidates=1, reps=2)
    want = h.default_solution(p)
    assert ms > 0 and best.as_dict() == want.as_dict()
    h.close()


def test_tuned_fp32_keeps_the_tensor_cores(tmp_path):
    h = tl.Handle()
    c = Case(torch.float32, "TN", 1024, 1024, 1024)
    p = tl.Problem.make(1024, 1024, 1024, dtype="fp32", trans_a=True)
    D = torch.empty_like(c.C)
    run = lambda handle=h, **kw: handle.gemm(p, D, None, c.A, c.B, **kw)

    def launches(handle):
        l0 = handle.launch_count()
        run(handle)
        return handle.launch_count() - l0

    assert launches(h) == 4
    want = D.clone()
    path = str(tmp_path / "tuned.json")
    best, ms = h.tune(p, D, None, c.A, c.B, reps=5, cache_path=path)
    h.check_solution(p, best)
    simt = _median_us(lambda: run(solution=best))
    assert best.kernel == tl.KERNEL_SIMT and ms * 1e3 < 0.75 * simt
    assert launches(h) == 4 and torch.equal(D.view(torch.int32), want.view(torch.int32))
    h2 = tl.Handle()
    assert h2.load_solutions(path) == 1 and launches(h2) == 4
    h2.close()
    h.close()


def test_tuned_for_aligned_operands_leaves_unaligned_ones_their_route():
    h = tl.Handle()
    c = Case(torch.bfloat16, "TN", 640, 768, 512)
    p = tl.Problem.make(640, 768, 512, dtype="bf16", trans_a=True)
    D = torch.empty_like(c.C)
    h.tune(p, D, None, c.A, c.B, max_candidates=2, reps=2)
    A = torch.empty(c.A.numel() + 1, dtype=c.A.dtype, device="cuda")[1:]
    A.copy_(c.A)
    l0 = h.launch_count()
    h.gemm(p, D, None, A, c.B)
    assert h.launch_count() - l0 == 2          # aligned copies, tensor cores
    c.check(D)
    h.device_status()
    h.close()


# ---- kernel timing of a plain fp32 GEMM: the launch that did the work, whichever it was ----
def test_kernel_timing_of_out_of_range_operands():
    h = tl.Handle()
    c = Case(torch.float32, "TN", 2048, 2048, 1024)
    c.A[77] = float("inf")
    c.run(h), c.run(h, "simt")
    h.set_kernel_timing(True)
    h.kernel_timing(reset=True)
    for _ in range(4):
        c.run(h)
    auto, n = h.kernel_timing(reset=True)
    assert n == 4
    for _ in range(4):
        c.run(h, "simt")
    simt, n = h.kernel_timing(reset=True)
    assert n == 4 and auto >= 0.9 * simt
    h.close()


# ---- one matrix for a whole batch (stride 0): its pieces and aligned copies are made once ----
@pytest.mark.parametrize("which", ["A", "B"])
@pytest.mark.parametrize("dtype,kernel,k", [(torch.float32, "bf16x3", 1024), (torch.float32, "bf16x6", 1024), (torch.float32, "auto", 1024),
                                            (torch.bfloat16, "auto", 1023)])
def test_one_matrix_for_a_whole_batch(dtype, kernel, k, which):
    h = tl.Handle()
    batch, big, small = 48, 2048, 64
    m, n = (big, small) if which == "A" else (small, big)
    g = torch.Generator(device="cuda").manual_seed(3)
    one = lambda r: torch.randn(r * k, device="cuda", generator=g).to(dtype)
    many = lambda r: torch.randn(batch * r * k, device="cuda", generator=g).to(dtype)
    A, B = (one(m), many(n)) if which == "A" else (many(m), one(n))
    D = torch.full((batch * m * n,), float("nan"), dtype=dtype, device="cuda")
    p = tl.Problem.make(m, n, k, dtype=tl.torch_dtype_code(dtype), trans_a=True, kernel=kernel, batch=batch)
    setattr(p, "stride_a" if which == "A" else "stride_b", 0)
    h.gemm(tl.Problem.make(64, 64, 64, dtype="bf16", trans_a=True), torch.empty(4096, device="cuda", dtype=torch.bfloat16), None,
           torch.zeros(4096, device="cuda", dtype=torch.bfloat16), torch.zeros(4096, device="cuda", dtype=torch.bfloat16))
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    h.gemm(p, D, None, A, B)
    h.device_status()
    used = free - torch.cuda.mem_get_info()[0]
    # six bytes an element and pieces or copies of every other operand's matrix, partial sums, allocation granules
    assert used <= 6 * (A.numel() + B.numel()) + (160 << 20)
    a = A.view(-1, m, k).double()
    b = B.view(-1, n, k).double().transpose(1, 2)
    ref = a @ b
    bound = (3.0 * k * 2.0 ** -24 if kernel != "bf16x3" else 2.0 ** -15) * (a.abs() @ b.abs()) + 2.0 ** -MANT[dtype] * ref.abs()
    got = D.view(batch, n, m).transpose(1, 2).double()
    assert bool(((got - ref).abs() <= bound).all())
    h.close()


# ---- the two-piece split of a vector: counts that are no multiple of four are read by vectors as well ----
def test_split_of_a_ragged_vector(h):
    n = (1 << 26) + 3
    x = torch.randn(n, device="cuda")
    hi, lo = (torch.empty(n, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    split = lambda count: h.split_bf16x2(x, count, hi, lo)
    split(n)
    want = x.bfloat16()
    assert torch.equal(hi.view(torch.int16), want.view(torch.int16))
    assert torch.equal(lo.view(torch.int16), (x - want.float()).bfloat16().view(torch.int16))
    assert _median_us(lambda: split(n)) <= 1.3 * _median_us(lambda: split(n - 3))


# ---- the call scratch's pool keeps a bounded amount ----
def test_call_scratch_is_given_back():
    h = tl.Handle()
    m, k = 8192, 24576                        # 2.4 GB of pieces
    A, B = (torch.ones(m * k, device="cuda") for _ in range(2))
    D = torch.empty(m * m, device="cuda")
    p = tl.Problem.make(m, m, k, dtype="fp32", trans_a=True)
    h.gemm(tl.Problem.make(1024, 1024, 1024, dtype="fp32", trans_a=True), D, None, A, B)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    h.gemm(p, D, None, A, B)
    torch.cuda.synchronize()
    h.gemm(tl.Problem.make(1024, 1024, 1024, dtype="fp32", trans_a=True), D, None, A, B)
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] <= (1 << 30) + (64 << 20)
    h.device_status()
    h.close()


# ---- fused activations with an fp32 output: as exact as plain fp32 arithmetic with a correctly rounded quotient ----
@pytest.mark.parametrize("scale", [0.1, 1.0, 6.0])
@pytest.mark.parametrize("act", ["gelu", "silu"])
def test_activation_of_fp32_outputs(h, act, scale):
    m, n, k = 1024, 512, 64
    g = torch.Generator(device="cuda").manual_seed(1)
    A = (torch.randn(m * k, device="cuda", generator=g) * scale).bfloat16()
    B = (torch.randn(n * k, device="cuda", generator=g) / 8).bfloat16()
    x, D = torch.empty(m * n, device="cuda"), torch.empty(m * n, device="cuda")
    p = tl.Problem.make(m, n, k, dtype="bf16", out_dtype="fp32", trans_a=True)
    h.gemm(p, x, None, A, B)
    h.gemm_ex(p, D, None, A, B, activation=act)
    h.device_status()
    f = (lambda v: 0.7978845608028654 * 2 * (v + 0.044715 * v * v * v)) if act == "gelu" else (lambda v: v)
    ref = x.double() / (1 + torch.exp(-f(x.double())))
    plain = x / (1 + torch.exp(-f(x)))
    err = lambda v: float((v.double() - ref).norm() / ref.norm())
    assert err(D) <= 1.05 * err(plain)
    edge = torch.tensor([float("inf"), float("nan"), -87.9, -1e4, 0.0, -0.0], device="cuda")
    A1, B1 = torch.zeros(64 * 64, device="cuda").bfloat16(), torch.zeros(64 * 64, device="cuda").bfloat16()
    E, bias = torch.empty(64 * 64, device="cuda"), torch.zeros(64, device="cuda")
    bias[:6] = edge
    h.gemm_ex(tl.Problem.make(64, 64, 64, dtype="bf16", out_dtype="fp32", trans_a=True), E, None, A1, B1, bias=bias,
              activation=act)
    e = E[:6]
    assert float(e[0]) == float("inf") and bool(torch.isnan(e[1])) and abs(float(e[2])) < 1e-35 and not e[3:].any()
