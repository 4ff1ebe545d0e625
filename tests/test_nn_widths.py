"""The network kernels are made for one set of widths: the header's, the binding's
and the network's are the same, another network is refused before anything is
allocated, and the binding refuses operands too small, of another type or layout
instead of letting a kernel read past them."""
import pathlib
import re

import pytest

import __graft_entry__

pkg = __graft_entry__.load_package()
nn, S = pkg.nn, pkg.surrogate
HEADER = pathlib.Path(__file__).resolve().parent.parent / "include" / "mpd_b200.h"


def test_header_and_binding_agree():
    macros = dict(re.findall(r"#define MPD_NN_(\w+) (\d+)", HEADER.read_text()))
    for name in ("INPUTS", "WIDTH", "BASIS", "HIDDEN", "OUTPUTS", "MIX_GRAD_MAX_B"):
        assert int(macros[name]) == getattr(nn, name)


@pytest.mark.parametrize("name,value", [("WIDTH", 32), ("WIDTH", 128), ("MODES", 6), ("MODES", 10),
                                        ("HIDDEN", 64), ("N_OUT", 7), ("N_IN", 8)])
def test_other_networks_are_refused(monkeypatch, name, value):
    monkeypatch.setattr(S, name, value)
    with pytest.raises(ValueError, match="made for"):
        S.SpectralOperator(4, 4, 1, params={})


def _operands(P=5, B=2):
    import torch
    f = lambda *s: torch.zeros(*s)
    bf = lambda n: torch.zeros(n, dtype=torch.bfloat16)
    spectral = dict(h=f(B * P, 64), basis=bf(-(-P // 32) * 256 * 32), R=f(256, 64, 64), r_sn=1,
                    r_sk=64, V=f(B, 256, 64), U=f(B, 256, 64), u_image=bf(B * 256 * 64), P=P, B=B,
                    V_fwd=f(B, 256, 64), dR=f(256, 64, 64))
    layer = dict(h=f(B * P, 64), w=f(64, 64), w_sn=1, w_sk=64, out0=f(B * P, 64), P=P, B=B,
                 basis=bf(128 * 256), u_image=bf(B * 256 * 64), bias=f(64), out1=f(B * P, 64))
    head = dict(h=f(B * P, 64), w=f(64, 128), w_sn=1, w_sk=128, out0=f(B * P, 128), P=B * P, B=1,
                n_out=128, bias=f(128), out1=f(B * P, 128), w2=f(128, 8), w2_sn=1, w2_sk=8,
                bias2=f(8), out2=f(B * P, 8))
    wgrad = dict(a=f(B * P, 64), g=f(B * P, 128), P=P, B=B, dw=f(64, 128), db=f(128),
                 work=f(B * 64 * 128), colwork=f(128 * 128))
    lift = dict(x=f(P, 6), w=f(6, 64), bias=f(64), z=f(P, 64))
    return [(nn.spectral, spectral), (nn.layer, layer), (nn.layer, head), (nn.wgrad, wgrad),
            (nn.lift, lift)]


class OnGpu:
    """A CPU tensor that says it lies on the GPU: what is refused is what is wrong."""

    def __init__(self, t):
        self.t = t

    is_cuda = True

    def __getattr__(self, name):
        return getattr(self.t, name)

    def contiguous(self):
        return OnGpu(self.t.contiguous())


@pytest.mark.parametrize("which", range(5))
def test_wrong_operands_are_refused(monkeypatch, which):
    import torch
    calls = []

    class Lib:
        def __getattr__(self, name):
            return lambda *a: calls.append(name) or 0
    monkeypatch.setattr(nn.N, "load", Lib)
    monkeypatch.setattr(nn, "_stream", lambda: None)
    fn, good = _operands()[which]
    tensors = {k: v for k, v in good.items() if isinstance(v, torch.Tensor)}
    args = {**good, **{k: OnGpu(t) for k, t in tensors.items()}}
    fn(**args)
    assert len(calls) == 1
    rows = ("a", "g", "x")          # made dense, their rows the call's size
    for k, t in tensors.items():
        bad = [OnGpu(t.to(torch.float64)), t]                   # another type, not on the GPU
        if k not in ("work", "x"):                              # (scratch has no least size)
            cut = t[:-1].clone() if k in rows else t.flatten()[:-1].clone()
            bad.append(OnGpu(cut))                              # too small
        if t.dim() > 1 and k not in ("w", "w2", "R", *rows):
            bad.append(OnGpu(t.transpose(0, 1).contiguous().transpose(0, 1)))   # not dense
        for b in bad:
            with pytest.raises(ValueError):
                fn(**{**args, k: b})
    assert len(calls) == 1


def test_attributes_are_set_once_on_each_device():
    """A kernel's shared-memory opt-in: again on another device, and after a failure."""
    import ctypes as C
    calls = [(0, 0, 1), (0, 0, 0), (1, 5, 1), (1, 0, 1), (1, 0, 0), (0, 0, 0), (63, 0, 1),
             (63, 0, 0), (64, 0, 1), (64, 0, 1)]
    arr = lambda v: (C.c_int * len(calls))(*v)
    ran, ret = arr([9] * len(calls)), arr([9] * len(calls))
    pkg._native.load_emu().mpd_emu_once_per_device(arr(c[0] for c in calls),
                                                   arr(c[1] for c in calls), len(calls), ran, ret)
    assert list(ran) == [c[2] for c in calls]
    assert list(ret) == [c[1] for c in calls]
