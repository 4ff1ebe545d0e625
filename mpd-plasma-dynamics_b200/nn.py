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
# the widths the kernels behind spectral(), layer(), lift() and wgrad() are made
# for (MPD_NN_* in include/mpd_b200.h)
INPUTS, WIDTH, BASIS, HIDDEN, OUTPUTS = 6, 64, 256, 128, 8

# These check their operands' sizes, types and layout (3 us a call) unless told
# check=False, as the network does for the buffers it has made itself.

def _dense(**tensors):
    """Each name=(tensor, elements needed, dtype), a None tensor aside: dense, of
    that type, large enough, on the GPU."""
    for name, (t, n, dtype) in tensors.items():
        if t is None:
            continue
        if t.numel() < n or t.dtype != dtype or not t.is_contiguous() or not t.is_cuda:
            raise ValueError(f"{name}: needs a dense CUDA tensor of at least {n} {dtype} elements, "
                             f"got shape {tuple(t.shape)}, strides {t.stride()}, {t.dtype} on "
                             f"{t.device}")


def _strided(name, t, n, sn, k, sk, first=0):
    """A float32 operand whose element (i, j), i < n, j < k, lies at
    t[first + i * sn + j * sk]."""
    if t is None:
        return
    import torch
    room = t.untyped_storage().nbytes() // 4 - t.storage_offset()
    last = first + (n - 1) * sn + (k - 1) * sk
    if t.dtype != torch.float32 or not t.is_cuda or sn < 0 or sk < 0 or last >= room:
        raise ValueError(f"{name}: needs a float32 CUDA tensor with element {last}, got "
                         f"{tuple(t.shape)} {t.dtype} on {t.device}")


def basis_image(A, rows, K, s_row, s_k, block_k=256):
    """The (rows x K) float32 operand at A[row * s_row + k * s_k], rounded to
    BF16 in the tensor core's layout (blocks of block_k columns)."""
    import torch
    lib = N.load()
    _strided("A", A, rows, s_row, K, s_k)
    n = -(-K // block_k) * -(-rows // 128) * 128 * block_k
    img = torch.empty(n, dtype=torch.bfloat16, device=A.device)
    N.check(lib.mpd_nn_basis_image(C.c_void_p(A.data_ptr()), s_row, s_k, rows, K, block_k,
                                   C.c_void_p(img.data_ptr()), _stream()), lib)
    return img


def spectral(h, basis, R, r_sn, r_sk, V, U, u_image, P, B, work=None, V_fwd=None,
             dR=None, check=True):
    """V[b] = basis h[b], U[b, q] = V[b, q] R[q], u_image = U as layer() reads it,
    dR[q] = sum over b of V_fwd[b, q]^T V[b, q]: mpd_nn_spectral in
    include/mpd_b200.h."""
    lib = N.load()
    if check:
        import torch
        f32, v = torch.float32, B * BASIS * WIDTH
        _dense(h=(h, B * P * WIDTH, f32), V=(V, v, f32), U=(U, v, f32), V_fwd=(V_fwd, v, f32),
               basis=(basis, -(-P // 32) * BASIS * 32, torch.bfloat16),
               u_image=(u_image, v, torch.bfloat16), dR=(dR, BASIS * WIDTH * WIDTH, f32),
               work=(work, 0, f32))
        _strided("R", R, WIDTH, r_sn, WIDTH, r_sk, first=(BASIS - 1) * WIDTH * WIDTH)
    d = N.SpectralDesc(P, B, h.data_ptr(), basis.data_ptr(), R.data_ptr(), r_sn, r_sk,
                       V.data_ptr(), U.data_ptr(), u_image.data_ptr(),
                       work.data_ptr() if work is not None else None,
                       work.numel() if work is not None else 0,
                       V_fwd.data_ptr() if V_fwd is not None else None,
                       dR.data_ptr() if dR is not None else None)
    N.check(lib.mpd_nn_spectral(C.byref(d), _stream()), lib)


def layer(h, w, w_sn, w_sk, out0, P, B, n_out=64, epilogue=FORWARD, basis=None, u_image=None,
          bias=None, z_in=None, out1=None, w2=None, bias2=None, out2=None,
          w2_sn=0, w2_sk=0, check=True):
    """out0 = h W + basis U[b] (+ bias), out1 = GELU(out0); or the backward forms
    of it; or the projection (n_out 128) and the product after it, out2:
    mpd_nn_layer in include/mpd_b200.h."""
    lib = N.load()
    if check:
        import torch
        f32, rows, n2 = torch.float32, B * P, OUTPUTS if epilogue == FORWARD else WIDTH
        k1 = OUTPUTS if basis is None and epilogue == ACT_BWD else WIDTH
        _dense(h=(h, rows * k1, f32), out0=(out0, rows * n_out, f32),
               out1=(out1, rows * n_out, f32), z_in=(z_in, rows * n_out, f32),
               bias=(bias, n_out, f32), bias2=(bias2, n2, f32), out2=(out2, rows * n2, f32),
               basis=(basis, -(-P // 128) * 128 * BASIS, torch.bfloat16),
               u_image=(u_image, B * BASIS * WIDTH, torch.bfloat16))
        _strided("w", w, n_out, w_sn, k1, w_sk)
        _strided("w2", w2, n2, w2_sn, HIDDEN, w2_sk)
    ptr = lambda t: None if t is None else t.data_ptr()
    d = N.LayerDesc(P, B, n_out, epilogue, h.data_ptr(), w.data_ptr(), w_sn, w_sk, ptr(basis),
                    ptr(u_image), ptr(bias), ptr(z_in), out0.data_ptr(), ptr(out1),
                    ptr(w2), ptr(bias2), w2_sn, w2_sk, ptr(out2))
    N.check(lib.mpd_nn_layer(C.byref(d), _stream()), lib)


def lift(x, w, bias, z, check=True):
    """z = x W + bias (rows x 6 to rows x 64), rounded as gemm() rounds."""
    lib = N.load()
    x = x.contiguous()
    if check:
        import torch
        f32, rows = torch.float32, x.shape[0]
        _dense(x=(x, rows * INPUTS, f32), w=(w, INPUTS * WIDTH, f32), bias=(bias, WIDTH, f32),
               z=(z, rows * WIDTH, f32))
    N.check(lib.mpd_nn_lift(C.c_void_p(x.data_ptr()), C.c_void_p(w.data_ptr()),
                            C.c_void_p(bias.data_ptr()), C.c_void_p(z.data_ptr()), x.shape[0],
                            _stream()), lib)


def wgrad(a, g, P, B, dw, db, work, colwork, check=True):
    """dw = a^T g and db = column sums of g over B samples of P rows:
    mpd_nn_wgrad in include/mpd_b200.h."""
    lib = N.load()
    a, g = a.contiguous(), g.contiguous()
    if check:
        import torch
        f32, k, n = torch.float32, a.shape[1], g.shape[1]
        _dense(a=(a, B * P * k, f32), g=(g, B * P * n, f32), dw=(dw, k * n, f32), db=(db, n, f32),
               work=(work, 0, f32), colwork=(colwork, 128 * n, f32))
    N.check(lib.mpd_nn_wgrad(C.c_void_p(a.data_ptr()), C.c_void_p(g.data_ptr()), a.shape[1],
                             g.shape[1], P, B, C.c_void_p(dw.data_ptr()),
                             C.c_void_p(db.data_ptr()), C.c_void_p(work.data_ptr()), work.numel(),
                             C.c_void_p(colwork.data_ptr()), _stream()), lib)


def wait_status():
    lib = N.load()
    N.check(lib.mpd_nn_wait_status(_stream()), lib)
