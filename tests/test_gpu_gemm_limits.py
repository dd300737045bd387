"""ci_gemm_bf16 where its kernels and copies meet their limits: length of the chains that the
tensor core sums, sizes of launch grids, captured streams.  Operands and reference as in
tests/test_gpu_gemm_shapes.py.

The tensor core's FP32 sums lose about 1.1e-9 of the result per product of a chain (7.3e-6
after 6,591 products), sums of a few chains add the rounding of one FP32 addition each,
6e-8 at most: 1.2e-9 times the longest chain, and 2e-8, hold for chains of 192 products and
more."""
import numpy as np
import pytest

from test_gpu_gemm_shapes import product

pytestmark = pytest.mark.gpu


def error(c, ref):
    return float(np.linalg.norm(c - ref) / np.linalg.norm(ref))


@pytest.mark.parametrize("M,N,K,chain", [(2048, 2048, 512, 256), (4096, 1024, 704, 256),
                                         (8192, 320, 896, 320), (10000, 64, 520, 192),
                                         (9800, 100, 896, 320), (19000, 256, 640, 320),
                                         (8190, 515, 521, 320)])
@pytest.mark.parametrize("form", [dict(), dict(bias=True, act=1, alpha=0.02, copy=True, ldc_pad=3),
                                  dict(beta=0.5, ldc_pad=4)])
def test_chains_of_short_products(cilib, M, N, K, chain, form):
    """Products of K from 512 to 896 whose tiles fill more than half of the GPU are summed in the
    chains of split K (512 products in one chain would be 4.7e-7, 896 8.6e-7)."""
    torch = pytest.importorskip("torch")
    c, ref = product(cilib, torch, M, N, K, lda_pad=(-K) % 8 if N != 515 else 0,
                     ldb_pad=(-K) % 8 if N != 515 else 0, seed=K, **form)
    assert error(c, ref) <= 1.2e-9 * chain + 2e-8


@pytest.mark.parametrize("M,N,K,form", [(8192, 96, 1031, dict()), (8192, 200, 1031, dict(ta=1)),
                                        (4096, 16, 2048, dict()), (1024, 33, 4096, dict(tb=0)),
                                        (8192, 256, 1024, dict()), (5000, 100, 1100, dict(bias=True))])
def test_chains_of_streamed_products(cilib, M, N, K, form):
    """The kernel that streams a long A past a narrow B sums chains of 256 products (of 512,
    up to 3.8e-7 here)."""
    torch = pytest.importorskip("torch")
    c, ref = product(cilib, torch, M, N, K, seed=N, **form)
    assert error(c, ref) <= 1.2e-9 * 256 + 2e-8


@pytest.mark.parametrize("M,N,K", [(25001, 40, 1031), (25000, 72, 1024), (40000, 32, 1024),
                                   (39001, 100, 1096), (39000, 200, 1032), (1024, 256, 4160),
                                   (1030, 130, 6600), (300, 48, 20000), (4224, 97, 1024)])
@pytest.mark.parametrize("form", [dict(), dict(bias=True, act=1, alpha=0.02, copy=True, ldc_pad=3),
                                  dict(beta=0.5, ldc_pad=(4), c_off=4)])
def test_streamed_tiles(cilib, M, N, K, form):
    """Long products in whole tiles (304 tiles and more), in ranges that cut them, with fewer and
    with more tiles than ranges, column tiles of 64 to 256.  Beside the chains of at most 512 the
    sums of K / 256 of them round in FP32, 3e-8 of the result each, at random."""
    torch = pytest.importorskip("torch")
    c, ref = product(cilib, torch, M, N, K, seed=M, **form)
    assert error(c, ref) <= 1.2e-9 * 512 + 3e-8 * (K / 256) ** 0.5
    again, _ = product(cilib, torch, M, N, K, seed=M, **form)
    assert np.array_equal(c, again)


@pytest.mark.parametrize("M,N,K,ta,tb", [(2097121, 20, 12, 0, 1), (2200000, 8, 48, 1, 1),
                                         (8, 2200000, 10, 0, 0), (1, 9, 8400000, 1, 0)])
def test_copies_of_many_rows(cilib, M, N, K, ta, tb):
    """Operands to be copied with more than 32 * 65,535 rows, and more than 128 * 65,535 columns,
    checked in 64 bits on the device."""
    torch = pytest.importorskip("torch")
    import ctypes as C
    g = torch.Generator(device="cuda").manual_seed(K)
    a = torch.randn((K, M) if ta else (M, K), generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn((N, K) if tb else (K, N), generator=g, device="cuda").to(torch.bfloat16)
    c = torch.full((M, N), float("nan"), device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    rc = cilib.lib().ci_gemm_bf16(a.data_ptr(), a.shape[1], ta, b.data_ptr(), b.shape[1], tb,
                                  c.data_ptr(), N, None, M, N, K, 1.0, 0.0, None, 0,
                                  err.data_ptr(), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, cilib.lib().ci_last_error()
    assert int(err.item()) == 0
    ref = (a.t() if ta else a).double() @ (b.t() if tb else b).double()
    assert float((c.double() - ref).norm() / ref.norm()) <= 1e-5


def test_captured_workspace_outlives_larger_calls(cilib):
    """A graph keeps the partial sums' address of its split product: a later call on the same
    stream that needs more memory must leave that memory alone.  (This one also captures behind
    a copy and behind a joined stream.)"""
    torch = pytest.importorskip("torch")
    import ctypes as C
    g = torch.Generator(device="cuda").manual_seed(1)
    rand = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)
    s, side = torch.cuda.Stream(), torch.cuda.Stream()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")

    def call(a, b, c, tb=1):
        rc = cilib.lib().ci_gemm_bf16(a.data_ptr(), a.shape[1], 0, b.data_ptr(), b.shape[1], tb,
                                      c.data_ptr(), c.shape[1], None, a.shape[0], c.shape[1],
                                      a.shape[1], 1.0, 0.0, None, 0, err.data_ptr(),
                                      C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0, cilib.lib().ci_last_error()

    a, b = rand(256, 2048), rand(300, 2048)
    a2, c, d = torch.empty_like(a), *(torch.empty((256, 300), device="cuda") for _ in range(2))
    big_a, big_b = rand(2000, 8008), rand(8008, 500)
    big_c = torch.empty((2000, 500), device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        call(a, b, c)   # the workspace exists before the capture
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        graph.capture_begin()
        a2.copy_(a)
        call(a2, b, c)
        side.wait_stream(s)
        with torch.cuda.stream(side):
            e = c + 0.0
        call(a2, b, d)
        s.wait_stream(side)
        call(a2, b, d)
        graph.capture_end()
        ref = a.double() @ b.double().t()
        for _ in range(3):
            call(big_a, big_b, big_c, tb=0)
            torch.cuda.synchronize()
            # whatever was freed is somebody else's now
            other = [torch.zeros(1 << 20, device="cuda") for _ in range(64)]
            c.zero_(), d.zero_(), a2.zero_()
            graph.replay()
            torch.cuda.synchronize()
            for x in (c, d, e):
                assert float((x.double() - ref).norm() / ref.norm()) <= 1e-6
            assert all(not bool(o.any()) for o in other)
    big = big_a.double() @ big_b.double()
    assert float((big_c.double() - big).norm() / big.norm()) <= 1e-6 and int(err.item()) == 0


def test_workspaces_are_bounded_and_given_back(cilib):
    """Copies of 126 MB on eight streams hold 512 MB together, not 1 GB; a stream that goes on
    with small split products gives its 130 MB back."""
    torch = pytest.importorskip("torch")
    import ctypes as C
    g = torch.Generator(device="cuda").manual_seed(2)
    a = torch.randn((327680, 96), generator=g, device="cuda").to(torch.bfloat16)
    sa, sb = (torch.randn((256, 2048), generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    c, d = torch.empty((96, 96), device="cuda"), torch.empty((256, 256), device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    streams = [torch.cuda.Stream() for _ in range(8)]
    L = cilib.lib()

    def big(s):
        assert L.ci_gemm_bf16(a.data_ptr(), 96, 1, a.data_ptr(), 96, 0, c.data_ptr(), 96, None, 96, 96,
                              327680, 1.0, 0.0, None, 0, err.data_ptr(), C.c_void_p(s.cuda_stream)) == 0
        torch.cuda.synchronize()

    def small(s):
        assert L.ci_gemm_bf16(sa.data_ptr(), 2048, 0, sb.data_ptr(), 2048, 1, d.data_ptr(), 256, None,
                              256, 256, 2048, 1.0, 0.0, None, 0, err.data_ptr(),
                              C.c_void_p(s.cuda_stream)) == 0
        torch.cuda.synchronize()

    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    for s in streams:
        big(s)
    ref = a.double().t() @ a.double()
    assert float((c.double() - ref).norm() / ref.norm()) <= 1e-6
    assert free0 - torch.cuda.mem_get_info()[0] <= 600 << 20
    big(streams[0])
    held = torch.cuda.mem_get_info()[0]
    for _ in range(70):
        small(streams[0])
    assert torch.cuda.mem_get_info()[0] - held >= 100 << 20
    assert int(err.item()) == 0
