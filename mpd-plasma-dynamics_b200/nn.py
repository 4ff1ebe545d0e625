"""Host side of the surrogate network's device kernels: thin wrappers that
pass torch-allocated device buffers (torch only provides memory and the
stream) to the library's own kernels through the C ABI."""
from __future__ import annotations

import ctypes as C

from . import _native as N


def _stream():
    import torch
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def gemm(A, B, Cout, M, N_, K, batch=1, sa=None, sb=None, sc=None, alpha=1.0, beta=0.0,
         work=None):
    """Cout[b](m,n) = alpha * sum_k A[b](m,k) B[b](n,k) + beta * Cout[b](m,n) on the
    tcgen05 tensor cores (operands rounded to BF16, FP32 accumulate).
    sa = (row, k, batch) element strides of A (default: row-major M x K
    contiguous), likewise sb for B (N x K) and sc for Cout (M x N).  work: an
    optional float32 device buffer for split-K partial sums."""
    lib = N.load()
    sa = sa or (K, 1, M * K)
    sb = sb or (K, 1, N_ * K)
    sc = sc or (N_, 1, M * N_)
    d = N.GemmDesc(M, N_, K, batch, A.data_ptr(), sa[0], sa[1], sa[2], B.data_ptr(), sb[0],
                   sb[1], sb[2], Cout.data_ptr(), sc[0], sc[1], sc[2], float(alpha), float(beta),
                   work.data_ptr() if work is not None else None,
                   work.numel() if work is not None else 0)
    N.check(lib.mpd_nn_gemm(C.byref(d), _stream()), lib)
    return Cout


FORWARD, ACT_BWD, PLAIN = 0, 1, 2   # epilogues of layer()
MIX_GRAD_MAX_B = 32                 # samples up to which spectral() also makes dR


def basis_image(A, rows, K, s_row, s_k, block_k=256):
    """The (rows x K) float32 operand at A[row * s_row + k * s_k], rounded to
    BF16 in the tensor core's layout (blocks of block_k columns)."""
    import torch
    lib = N.load()
    n = -(-K // block_k) * -(-rows // 128) * 128 * block_k
    img = torch.empty(n, dtype=torch.bfloat16, device=A.device)
    N.check(lib.mpd_nn_basis_image(C.c_void_p(A.data_ptr()), s_row, s_k, rows, K, block_k,
                                   C.c_void_p(img.data_ptr()), _stream()), lib)
    return img


def spectral(h, basis, R, r_sn, r_sk, V, U, u_image, P, B, work=None, V_fwd=None,
             dR=None):
    """V[b] = basis h[b], U[b, q] = V[b, q] R[q], u_image = U as layer() reads it,
    dR[q] = sum over b of V_fwd[b, q]^T V[b, q]: mpd_nn_spectral in
    include/mpd_b200.h."""
    lib = N.load()
    d = N.SpectralDesc(P, B, h.data_ptr(), basis.data_ptr(), R.data_ptr(), r_sn, r_sk,
                       V.data_ptr(), U.data_ptr(), u_image.data_ptr(),
                       work.data_ptr() if work is not None else None,
                       work.numel() if work is not None else 0,
                       V_fwd.data_ptr() if V_fwd is not None else None,
                       dR.data_ptr() if dR is not None else None)
    N.check(lib.mpd_nn_spectral(C.byref(d), _stream()), lib)


def layer(h, w, w_sn, w_sk, out0, P, B, n_out=64, epilogue=FORWARD, basis=None, u_image=None,
          bias=None, z_in=None, out1=None, w2=None, bias2=None, out2=None,
          w2_sn=0, w2_sk=0):
    """out0 = h W + basis U[b] (+ bias), out1 = GELU(out0); or the backward forms
    of it; or the projection (n_out 128) and the product after it, out2:
    mpd_nn_layer in include/mpd_b200.h."""
    lib = N.load()
    ptr = lambda t: None if t is None else t.data_ptr()
    d = N.LayerDesc(P, B, n_out, epilogue, h.data_ptr(), w.data_ptr(), w_sn, w_sk, ptr(basis),
                    ptr(u_image), ptr(bias), ptr(z_in), out0.data_ptr(), ptr(out1),
                    ptr(w2), ptr(bias2), w2_sn, w2_sk, ptr(out2))
    N.check(lib.mpd_nn_layer(C.byref(d), _stream()), lib)


def lift(x, w, bias, z):
    """z = x W + bias (rows x 6 to rows x 64), rounded as gemm() rounds."""
    lib = N.load()
    x = x.contiguous()
    N.check(lib.mpd_nn_lift(C.c_void_p(x.data_ptr()), C.c_void_p(w.data_ptr()),
                            C.c_void_p(bias.data_ptr()), C.c_void_p(z.data_ptr()), x.shape[0],
                            _stream()), lib)


def wgrad(a, g, P, B, dw, db, work, colwork):
    """dw = a^T g and db = column sums of g over B samples of P rows:
    mpd_nn_wgrad in include/mpd_b200.h."""
    lib = N.load()
    a, g = a.contiguous(), g.contiguous()
    N.check(lib.mpd_nn_wgrad(C.c_void_p(a.data_ptr()), C.c_void_p(g.data_ptr()), a.shape[1],
                             g.shape[1], P, B, C.c_void_p(dw.data_ptr()),
                             C.c_void_p(db.data_ptr()), C.c_void_p(work.data_ptr()), work.numel(),
                             C.c_void_p(colwork.data_ptr()), _stream()), lib)


def wait_status():
    lib = N.load()
    N.check(lib.mpd_nn_wait_status(_stream()), lib)
