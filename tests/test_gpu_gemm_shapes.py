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
