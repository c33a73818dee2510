"""The training kernels where their work is split: weight gradients over fewer
and more tiles than SMs and a dz that starts off 16 bytes, against the float64
oracle; the fused data gradient against the three launches it replaces, bit for
bit; ten tensors of Adam in one launch against ten launches, bit for bit.

Weight-gradient tolerance: products of BF16 values are exact in FP32, so the
error is that of adding K of them (at most a few thousand a CTA, then the
partials) in FP32: below 1e-5 of the largest sum, as for one tile."""
import ctypes

import numpy as np
import pytest
import torch

import nn_oracle as O
from classic_b200 import _lib

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _bf(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float32)).to(torch.bfloat16).cuda().contiguous()


@pytest.mark.parametrize("n,h,w", [(1, 16, 16), (1, 16, 48), (3, 112, 64), (10, 64, 64)])
@pytest.mark.parametrize("cin,cout", [(16, 32), (32, 32), (32, 16)])
@pytest.mark.parametrize("shift", [0, 1])
def test_weight_gradient(n, h, w, cin, cout, shift):
    rng = np.random.default_rng(n + w + cin)
    x = O.bf16(rng.standard_normal((n, h, w, cin)))
    dz = O.bf16(rng.standard_normal((n, h, w, cout)))
    blocks = n * (h // 16) * (w // 16)
    partial = torch.full((blocks * cout * 9 * cin + shift,), float("nan"), device="cuda")[shift:]
    pdb = torch.full((blocks * cout + shift,), float("nan"), device="cuda")[shift:]
    dw = torch.full((cout * 9 * cin + shift,), float("nan"), device="cuda")[shift:]
    db = torch.full((cout + shift,), float("nan"), device="cuda")[shift:]
    xd = _bf(x)
    dzd = torch.cat([torch.zeros(shift, dtype=torch.bfloat16, device="cuda"), _bf(dz).flatten()])[shift:]
    rc = _lib.load().nn_conv3x3_wgrad(_p(xd), _p(dzd), _p(partial), _p(pdb), _p(dw), _p(db), n, h, w, cin,
                                      cout, None)
    assert rc == 0
    torch.cuda.synchronize()
    dwr, dbr = O.conv3x3_wgrad(x, dz)
    for got, ref in ((dw.cpu().numpy().reshape(dwr.shape), dwr), (db.cpu().numpy(), dbr)):
        assert np.max(np.abs(got - ref)) <= 1e-5 * np.max(np.abs(ref))


@pytest.mark.parametrize("cin,cout", [(32, 32), (32, 16)])
@pytest.mark.parametrize("n,h,w", [(1, 16, 16), (5, 80, 64)])
@pytest.mark.parametrize("act", [False, True])
def test_data_gradient(cin, cout, n, h, w, act):
    g = torch.Generator(device="cuda").manual_seed(n + cout)
    dz = torch.randn((n, h, w, cout), generator=g, device="cuda").to(torch.bfloat16)
    wt = (0.2 * torch.randn((cout, 9, cin), generator=g, device="cuda")).to(torch.bfloat16)
    z = torch.randn((n, h, w, cin), generator=g, device="cuda")
    lib = _lib.load()
    flip = torch.empty((cin, 9, cout), dtype=torch.bfloat16, device="cuda")
    zero = torch.zeros(cin, device="cuda")
    ref, got = (torch.empty((n, h, w, cin), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    assert lib.nn_flip_weights(_p(wt), _p(flip), cout, cin, None) == 0
    assert lib.nn_conv3x3_forward(_p(dz), _p(flip), _p(zero), _p(ref), None, n, h, w, cout, cin, 0, 0, None) == 0
    if act:
        assert lib.nn_gelu_backward(_p(ref), _p(z), _p(ref), ref.numel(), None) == 0
    assert lib.nn_conv3x3_dgrad(_p(dz), _p(wt), _p(z) if act else None, _p(got), n, h, w, cin, cout, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(ref.view(torch.int16), got.view(torch.int16))


def test_adam_multi():
    g = torch.Generator(device="cuda").manual_seed(3)
    sizes = [9216, 4608, 1, 32, 300]
    lib, runs = _lib.load(), []
    base = [[torch.rand(s, generator=g, device="cuda") for s in sizes] for _ in range(4)]
    for multi in (False, True):
        w, gr, m, v = ([t.clone() for t in lst] for lst in base)
        w16 = [torch.zeros(s, dtype=torch.bfloat16, device="cuda") if k != 2 else None for k, s in enumerate(sizes)]
        ptr = [[None if t is None else t.data_ptr() for t in lst] for lst in (w, gr, m, v, w16)]
        if multi:
            arrs = [(ctypes.c_void_p * len(sizes))(*q) for q in ptr]
            ns = (ctypes.c_longlong * len(sizes))(*sizes)
            assert lib.nn_adam_multi(len(sizes), *arrs, ns, 1e-3, 0.9, 0.999, 1e-8, 3, None) == 0
        else:
            for k, s in enumerate(sizes):
                assert lib.nn_adam(*(q[k] for q in ptr), s, 1e-3, 0.9, 0.999, 1e-8, 3, None) == 0
        torch.cuda.synchronize()
        runs.append(w + m + v + [t for t in w16 if t is not None])
    for a, b in zip(*runs):
        assert torch.equal(a, b)
