"""Forms of ci_gemm_bf16 beside tests/test_gpu_gemm.py: leading dimensions of C, C alone or
with its BF16 copy, at the edges of the kernels' tiles.  Reference: a float64 product of the
same BF16 operands.  FP32 accumulation of K products rounds to about sqrt(K) 2^-24 of the
result (7e-6 at K = 16,384; the tensor core's sums may truncate, twice that): 2e-5 holds
everywhere here."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def product(cilib, torch, M, N, K, ta=0, tb=1, lda_pad=0, ldb_pad=0, ldc_pad=0, a_off=0, b_off=0,
            c_off=0, bias=False, act=0, beta=0.0, copy=False, alpha=1.0, seed=0, a_edit=None):
    """C = alpha op(A) op(B) + ... with operands inside larger buffers (NaN around them, so
    that a read outside shows); returns C, the untouched surroundings' check and the reference."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def place(rows, cols, pad, off):
        buf = torch.full((off + rows * (cols + pad) + 16,), float("nan"), device="cuda",
                         dtype=torch.bfloat16)
        v = buf[off:off + rows * (cols + pad)].view(rows, cols + pad)[:, :cols]
        v.copy_(torch.randn((rows, cols), generator=g, device="cuda"))
        return buf, v

    ba, a = place(K if ta else M, M if ta else K, lda_pad, a_off)
    bb, b = place(N if tb else K, K if tb else N, ldb_pad, b_off)
    if a_edit:
        a_edit(a)
    ldc = N + ldc_pad
    cbuf = torch.full((c_off + M * ldc + 8,), 7.0, device="cuda")
    c = cbuf[c_off:c_off + M * ldc].view(M, ldc)
    if beta:
        c[:, :N] = torch.randn((M, N), generator=g, device="cuda")
    c0 = c[:, :N].double().clone()
    cb = torch.zeros((M, ldc), device="cuda", dtype=torch.bfloat16) if copy else None
    bi = torch.randn(N, generator=g, device="cuda") if bias else None
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    rc = cilib.lib().ci_gemm_bf16(ba.data_ptr() + 2 * a_off, a.stride(0), ta,
                                  bb.data_ptr() + 2 * b_off, b.stride(0), tb, c.data_ptr(), ldc,
                                  None if cb is None else cb.data_ptr(), M, N, K, alpha, beta,
                                  None if bi is None else bi.data_ptr(), act, err.data_ptr(),
                                  C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, cilib.lib().ci_last_error()
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    A = (a.t() if ta else a).double()
    B = (b.t() if tb else b).double()
    ref = alpha * (A @ B) + (beta * c0 if beta else 0.0) + (bi.double() if bias else 0.0)
    if act:
        ref = torch.tanh(ref)
    # the gap between C's rows and the ends of its buffer are as they were
    assert bool((c[:, N:] == 7.0).all()) and bool((cbuf[:c_off] == 7.0).all())
    assert bool((cbuf[c_off + M * ldc:] == 7.0).all())
    if copy:
        assert bool(torch.equal(cb[:, :N], c[:, :N].to(torch.bfloat16)))
    return c[:, :N].double().cpu().numpy(), ref.cpu().numpy()


def close(c, ref, tol=2e-5):
    return np.linalg.norm(c - ref) <= tol * np.linalg.norm(ref)


@pytest.mark.parametrize("M,N,K", [(128, 16, 64), (129, 65, 64), (160, 67, 512), (300, 131, 576),
                                   (257, 259, 72), (20000, 40, 64)])
@pytest.mark.parametrize("form", [dict(), dict(ldc_pad=1), dict(ldc_pad=4, c_off=4, bias=True),
                                  dict(c_off=1, bias=True, copy=True, ldc_pad=3),
                                  dict(beta=0.5, act=1, alpha=0.01, ldc_pad=2)])
def test_epilogue_forms(cilib, M, N, K, form):
    """The persistent kernel's stores (K of 512 and less and above): aligned and odd rows of C,
    whole and ragged 32 x 32 blocks, C alone, with bias, beta, tanh and the BF16 copy."""
    torch = pytest.importorskip("torch")
    c, ref = product(cilib, torch, M, N, K, lda_pad=(-K) % 8, ldb_pad=(-K) % 8, seed=M + N, **form)
    assert close(c, ref)


@pytest.mark.parametrize("M,N,K", [(4096, 16, 1024), (4103, 96, 1031), (5000, 64, 2050),
                                   (8200, 65, 1100), (4097, 131, 1999), (4099, 256, 1027),
                                   (96, 96, 50001), (300, 30, 15000)])
@pytest.mark.parametrize("form", [dict(), dict(lda_pad=1), dict(lda_pad=2, a_off=3), dict(a_off=8),
                                  dict(lda_pad=4, ldc_pad=3, bias=True, copy=True),
                                  dict(ldb_pad=3, b_off=5, beta=0.5, alpha=0.01, act=1)])
def test_streaming_products(cilib, M, N, K, form):
    """A long A past a narrow B: one unit range per SM, cut tiles, rows of every offset to a
    16-byte boundary (row classes), B copied; NaN around the operands; repeats to the bit."""
    torch = pytest.importorskip("torch")
    c, ref = product(cilib, torch, M, N, K, seed=M + K, **form)
    assert close(c, ref)
    c2, _ = product(cilib, torch, M, N, K, seed=M + K, **form)
    assert np.array_equal(c, c2)


@pytest.mark.parametrize("lda_pad", [0, 1, 2, 4, 7])
def test_an_infinite_row_end_stays_in_its_row(cilib, lda_pad):
    """Row classes read the end of the row before; an infinity there reaches its own row only."""
    torch = pytest.importorskip("torch")

    def edit(a):
        a[17, -1] = float("inf")
        a[4000, -3:] = float("nan")

    M, N, K = 4099, 40, 1025
    c, ref = product(cilib, torch, M, N, K, lda_pad=lda_pad, a_edit=edit, seed=5)
    bad = ~np.isfinite(c).all(axis=1)
    assert sorted(np.flatnonzero(bad)) == [17, 4000]
    assert close(c[~bad], ref[~bad])


@pytest.mark.parametrize("M,N,K", [(40, 70, 1000), (1000, 17, 130), (20000, 96, 96), (129, 300, 67),
                                   (700, 9, 1500), (2000, 1000, 40), (5, 3000, 3000)])
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (1, 1), (0, 1)])
@pytest.mark.parametrize("form", [dict(), dict(lda_pad=3, ldb_pad=1, a_off=1, b_off=2)])
def test_copied_operands(cilib, M, N, K, ta, tb, form):
    """Products whose operands TMA cannot read go through aligned copies, in every transpose
    form, M, N and K below a tile among them."""
    torch = pytest.importorskip("torch")
    c, ref = product(cilib, torch, M, N, K, ta=ta, tb=tb, bias=True, seed=M + N, **form)
    assert close(c, ref)


def test_captured_product(cilib):
    """While its stream is captured a product takes no workspace: replays read the operands."""
    torch = pytest.importorskip("torch")
    M, N, K = 300, 100, 131
    a = torch.randn((M, K), device="cuda").to(torch.bfloat16)
    b = torch.randn((N, K), device="cuda").to(torch.bfloat16)
    c = torch.zeros((M, N), device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")

    def call():
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert cilib.lib().ci_gemm_bf16(a.data_ptr(), K, 0, b.data_ptr(), K, 1, c.data_ptr(), N,
                                        None, M, N, K, 1.0, 0.0, None, 0, err.data_ptr(), st) == 0

    call()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call()
    a.mul_(0.5)
    g.replay()
    torch.cuda.synchronize()
    ref = (a.double() @ b.double().t()).cpu().numpy()
    assert close(c.double().cpu().numpy(), ref)
