"""The fused layer kernel against the separate launches it stands for (products
by the general GEMM, bias + activation and its derivative as element-wise
kernels): the same roundings in the same order, so the same bits.  Sizes around
its tiles of 128 rows, tiles shared by several samples and by several CTAs."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def _operands(P, B, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    return dict(h=rnd(B * P, 64), W=rnd(64, 64) / 8, G=rnd(P, 256), U=rnd(B, 256, 64) / 16,
                bias=rnd(64), z=2 * rnd(B * P, 64))


def _u_image(U):
    """U[b] (256 x 64) in 16-byte units of 8 coefficients, unit (q / 8, column)."""
    import torch
    return U.to(torch.bfloat16).view(-1, 32, 8, 64).transpose(2, 3).contiguous()


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _sum(nn, o, P, B, trans):
    """h W + G U[b] by the general GEMM (trans: W transposed)."""
    import torch
    s = torch.empty(B * P, 64, device="cuda")
    nn.gemm(o["h"], o["W"], s, B * P, 64, 64, 1, sa=(64, 1, 0),
            sb=(64, 1, 0) if trans else (1, 64, 0), sc=(64, 1, 0))
    nn.gemm(o["G"], o["U"], s, P, 64, 256, B, sa=(256, 1, 0), sb=(1, 64, 256 * 64),
            sc=(64, 1, P * 64), beta=1.0)
    return s


@pytest.mark.parametrize("P,B", [(1, 1), (127, 2), (128, 1), (129, 3), (400, 60), (19000, 1)])
def test_layer_is_the_separate_launches(pkg, P, B):
    import torch
    nn, lib, o = pkg.nn, pkg._native.load(), _operands(P, B, P + B)
    img = nn.basis_image(o["G"], P, 256, 256, 1)
    stream = nn._stream()
    z = _sum(nn, o, P, B, False)
    out = torch.empty_like(z)
    assert lib.mpd_nn_bias_act(_ptr(z), _ptr(o["bias"]), _ptr(out), B * P, 64, 1, stream) == 0
    got0, got1 = torch.full_like(z, 7.0), torch.full_like(z, 7.0)
    args = dict(basis=img, u_image=_u_image(o["U"]))
    nn.layer(o["h"], o["W"], 1, 64, got0, P, B, bias=o["bias"], out1=got1, **args)
    assert torch.equal(got0, z) and torch.equal(got1, out)
    got0.fill_(7.0)
    nn.layer(o["h"], o["W"], 1, 64, got0, P, B, bias=o["bias"], **args)
    assert torch.equal(got0, z)
    # backward: the transposed weight, G^T's image read from its transpose
    img_t = nn.basis_image(o["G"].t().contiguous(), P, 256, 1, P)
    assert torch.equal(img_t, img)
    gh = _sum(nn, o, P, B, True)
    gz = torch.empty_like(gh)
    assert lib.mpd_nn_act_bwd(_ptr(gh), _ptr(o["z"]), _ptr(gz), gh.numel(), stream) == 0
    nn.layer(o["h"], o["W"], 64, 1, got0, P, B, epilogue=nn.PLAIN, **args)
    assert torch.equal(got0, gh)
    nn.layer(o["h"], o["W"], 64, 1, got0, P, B, epilogue=nn.ACT_BWD, z_in=o["z"], **args)
    assert torch.equal(got0, gz)
    nn.wait_status()


@pytest.mark.parametrize("rows", [1, 128, 1001, 40000])
def test_projection_is_the_separate_launches(pkg, rows):
    import torch
    nn, lib, o = pkg.nn, pkg._native.load(), _operands(rows, 1, rows)
    W = torch.randn(64, 128, device="cuda") / 8
    bias = torch.randn(128, device="cuda")
    z, out = torch.empty(rows, 128, device="cuda"), torch.empty(rows, 128, device="cuda")
    nn.gemm(o["h"], W, z, rows, 128, 64, 1, sa=(64, 1, 0), sb=(1, 128, 0), sc=(128, 1, 0))
    assert lib.mpd_nn_bias_act(_ptr(z), _ptr(bias), _ptr(out), rows, 128, 1, nn._stream()) == 0
    W2, bias2 = torch.randn(128, 8, device="cuda") / 11, torch.randn(8, device="cuda")
    zo, y = torch.empty(rows, 8, device="cuda"), torch.empty(rows, 8, device="cuda")
    nn.gemm(out, W2, zo, rows, 8, 128, 1, sa=(128, 1, 0), sb=(1, 8, 0), sc=(8, 1, 0))
    assert lib.mpd_nn_bias_act(_ptr(zo), _ptr(bias2), _ptr(y), rows, 8, 0, nn._stream()) == 0
    got0, got1, got2 = (torch.full_like(t, 7.0) for t in (z, out, y))
    nn.layer(o["h"], W, 1, 128, got0, rows, 1, n_out=128, bias=bias, out1=got1, w2=W2,
             w2_sn=1, w2_sk=8, bias2=bias2, out2=got2)
    assert torch.equal(got0, z) and torch.equal(got1, out) and torch.equal(got2, y)
    # backward: from the gradient of the 8 outputs to the 64 columns of h
    gz, gh = torch.empty_like(z), torch.empty(rows, 64, device="cuda")
    nn.gemm(y, W2, out, rows, 128, 8, 1, sa=(8, 1, 0), sb=(8, 1, 0), sc=(128, 1, 0))
    assert lib.mpd_nn_act_bwd(_ptr(out), _ptr(z), _ptr(gz), gz.numel(), nn._stream()) == 0
    nn.gemm(gz, W, gh, rows, 64, 128, 1, sa=(128, 1, 0), sb=(128, 1, 0), sc=(64, 1, 0))
    got2 = torch.full_like(gh, 7.0)
    nn.layer(y, W2, 8, 1, got0, rows, 1, n_out=128, epilogue=nn.ACT_BWD, z_in=z, w2=W,
             w2_sn=128, w2_sk=1, out2=got2)
    assert torch.equal(got0, gz) and torch.equal(got2, gh)
    nn.wait_status()


@pytest.mark.parametrize("rows", [1, 127, 129, 75777, 300000])
def test_lift_is_the_separate_launches(pkg, rows):
    import torch
    nn, lib = pkg.nn, pkg._native.load()
    x, W = torch.randn(rows, 6, device="cuda"), torch.randn(6, 64, device="cuda")
    bias = torch.randn(64, device="cuda")
    z, h = torch.empty(rows, 64, device="cuda"), torch.empty(rows, 64, device="cuda")
    nn.gemm(x, W, z, rows, 64, 6, 1, sa=(6, 1, 0), sb=(1, 64, 0), sc=(64, 1, 0))
    assert lib.mpd_nn_bias_act(_ptr(z), _ptr(bias), _ptr(h), rows, 64, 0, nn._stream()) == 0
    got = torch.full_like(z, 7.0)
    nn.lift(x, W, bias, got)
    assert torch.equal(got, z)
    nn.wait_status()


@pytest.mark.parametrize("k_in,n_out", [(6, 64), (64, 64), (64, 128), (128, 8)])
@pytest.mark.parametrize("P,B,room", [(1, 1, 1), (63, 2, 64), (257, 3, 64), (1300, 16, 64),
                                      (4100, 2, 3), (1001, 9, 1)])
def test_weight_gradients_are_the_separate_launches(pkg, k_in, n_out, P, B, room):
    import torch
    nn, lib = pkg.nn, pkg._native.load()
    a, g = torch.randn(B * P, k_in, device="cuda"), torch.randn(B * P, n_out, device="cuda")
    mn = k_in * n_out
    work = torch.empty(room * B * mn, device="cuda")
    colwork = torch.empty(128 * n_out, device="cuda")
    parts, dw = torch.empty(B * mn, device="cuda"), torch.empty(k_in, n_out, device="cuda")
    db = torch.empty(n_out, device="cuda")
    nn.gemm(a, g, parts, k_in, n_out, P, B, sa=(1, k_in, P * k_in), sb=(1, n_out, P * n_out),
            sc=(n_out, 1, mn), work=work)
    assert lib.mpd_nn_sum_parts(_ptr(parts), B, mn, _ptr(dw), 0, nn._stream()) == 0
    assert lib.mpd_nn_colsum(_ptr(g), B * P, n_out, _ptr(db), _ptr(colwork), nn._stream()) == 0
    got_w, got_b = torch.full_like(dw, 7.0), torch.full_like(db, 7.0)
    work.fill_(7.0), colwork.fill_(7.0)
    nn.wgrad(a, g, P, B, got_w, got_b, work, colwork)
    assert torch.equal(got_w, dw) and torch.equal(got_b, db)
    nn.wait_status()


def test_refused_operands(pkg):
    import torch
    nn, o = pkg.nn, _operands(8, 1, 0)
    out = torch.empty(8, 64, device="cuda")
    img = nn.basis_image(o["G"], 8, 256, 256, 1)
    for bad in (dict(basis=img), dict(basis=img, u_image=_u_image(o["U"])),
                dict(bias=o["bias"])):
        with pytest.raises(pkg._native.MpdError):
            nn.layer(o["h"], o["W"], 1, 64, out, 8, 1, **bad)


@pytest.mark.parametrize("P,B,room", [(1, 1, 16), (31, 2, 16), (33, 3, 16), (255, 2, 16),
                                      (300, 2, 0), (1001, 16, 16), (4100, 1, 16), (70, 130, 2),
                                      (40000, 2, 16), (90, 17, 16), (90, 32, 16), (4100, 16, 16),
                                      (500, 150, 1)])
def test_spectral_half_is_the_separate_launches(pkg, P, B, room):
    """Both directions (R and R^T), split and unsplit K, more samples than a tile."""
    import torch
    nn, o = pkg.nn, _operands(P, B, 7 * P + B)
    Fq = o["G"].t().contiguous()
    R = torch.randn(256, 64, 64, device="cuda") / 8
    n = B * 256 * 64
    work = torch.empty(room * n, device="cuda") if room else None
    img = nn.basis_image(Fq, 256, P, P, 1, block_k=32)
    assert torch.equal(img, nn.basis_image(o["G"], 256, P, 1, 256, block_k=32))
    new = lambda: torch.full((B, 256, 64), 7.0, device="cuda")
    for r_sn, r_sk in ((1, 64), (64, 1)):
        V, U, gV, gU = new(), new(), new(), new()
        nn.gemm(Fq, o["h"], V, 256, 64, P, B, sa=(P, 1, 0), sb=(1, 64, P * 64),
                sc=(64, 1, 256 * 64), work=work)
        nn.gemm(V, R, U, B, 64, 64, 256, sa=(256 * 64, 1, 64), sb=(r_sn, r_sk, 4096),
                sc=(256 * 64, 1, 64))
        image = torch.zeros(n, dtype=torch.bfloat16, device="cuda")
        nn.spectral(o["h"], img, R, r_sn, r_sk, gV, gU, image, P, B, work=work)
        assert torch.equal(gV, V) and torch.equal(gU, U)
        assert torch.equal(image, _u_image(U).view(-1))
        if B <= nn.MIX_GRAD_MAX_B:
            Vf = torch.randn(B, 256, 64, device="cuda")
            dR, gR = torch.empty_like(R), torch.full_like(R, 7.0)
            nn.gemm(Vf, V, dR, 64, 64, B, 256, sa=(1, 256 * 64, 64), sb=(1, 256 * 64, 64),
                    sc=(64, 1, 4096))
            nn.spectral(o["h"], img, R, r_sn, r_sk, gV, gU, image, P, B, work=work, V_fwd=Vf,
                        dR=gR)
            assert torch.equal(gR, dR) and torch.equal(gV, V) and torch.equal(gU, U)
    nn.wait_status()
