"""The 32-bit precision that csrc/attn_tc.cu and the product of the latents (csrc/layered_tc.cu, tc_gemm_split) state, on fp32 data against 64 bits: every
instance of the head sizes, masks, sink, softcap, gates, paged rows.

Bounds, of a row's size: the norm of the same weights over the values' magnitudes (a row's own norm may come out near zero by chance, four values wide
above all).  Scores: an operand in two f16 parts is off by 2^-23 at most and 2^-25 as a root mean square, the product of the two small parts that
is left out by as much, and a dozen additions that are cut by 2^-24 each of their partial sum; weighted by |q||k| scale (3 to 8 here) a score is off by some
4e-7, which is the relative error of its weight, and the values' sum is off by as much again: under 1e-6.  A softcap takes
2^-24 of its 20 more.  (Without the small parts of one operand it would be 1e-4.)"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest
import torch

from conftest import ROOT
from nano_b200 import build as nb_build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    lib = os.environ.get("NB200_ENGINE_SO", nb_build.ENGINE_SO)
    so = str(tmp_path_factory.mktemp("probe") / "tc_probe.so")
    subprocess.run([nb_build.NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I" + nb_build.CSRC, os.path.join(ROOT, "tests", "tc_probe.cu"), lib, "-Xlinker",
                    "-rpath," + os.path.dirname(os.path.abspath(lib)), "-o", so], check=True)
    torch.zeros(1, device="cuda")
    return C.CDLL(so)


def ptr(t):
    return C.c_void_p(t.data_ptr() if t is not None else None)


def attention(probe, q, k, v, H, G, pos0, scale, softcap=0.0, block=0, window=0, sink=None, gate=None, mul=None, paged=False):
    T, D, VD = q.shape[0], q.shape[2], v.shape[2]
    n = k.shape[0]
    rows = torch.zeros((n + 31) // 32 * 32, G * (D + VD), device="cuda")
    table = None
    if paged:
        pages = torch.randperm(rows.shape[0] // 32, generator=torch.Generator().manual_seed(1)).cuda()
        place = (pages[torch.arange(n, device="cuda") // 32] * 32 + torch.arange(n, device="cuda") % 32).long()
        table = pages.to(torch.int32)
    else:
        place = torch.arange(n, device="cuda")
    rows[place] = torch.cat([k.reshape(n, -1), v.reshape(n, -1)], 1)
    out = torch.full((T, H, VD), float("nan"), device="cuda")
    a = np.array([T, H, G, D, VD, pos0, block, window, H * D, D, G * (D + VD), G * (D + VD), D, VD, H, H * VD], np.uint32)
    torch.cuda.synchronize()
    rc = probe.probe_attention(ptr(q), ptr(rows), C.c_void_p(rows.data_ptr() + 4 * G * D), ptr(table), ptr(out), a.ctypes.data_as(C.c_void_p), C.c_float(scale), C.c_float(softcap), ptr(sink), ptr(gate), ptr(mul))
    assert rc == 0, rc
    return out


def attention64(q, k, v, H, G, pos0, scale, softcap=0.0, block=0, window=0, sink=None, gate=None, mul=None):
    scale, softcap = float(np.float32(scale)), float(np.float32(softcap))
    pos, key = pos0 + torch.arange(q.shape[0], device="cuda")[:, None], torch.arange(k.shape[0], device="cuda")[None]
    seen = key <= pos
    if block:
        seen &= key >= pos - pos % block
    if window:
        seen &= key > pos - window
    out = []
    for h in range(H):
        s = q[:, h].double() @ k[:, h * G // H].double().T * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        s = s.masked_fill(~seen, -torch.inf)
        top = s.amax(1, keepdim=True)
        e = torch.exp(s - top)
        den = e.sum(1, keepdim=True) + (torch.exp(sink[h].double() - top) if sink is not None else 0.0)
        o = (e / den) @ v[:, h * G // H].double()
        if gate is not None:
            o = o * torch.sigmoid(gate[:, h:h + 1].double())
        out.append(o * mul[:, h].double() if mul is not None else o)
    return torch.stack(out, 1)


def randn(seed, *shape):
    return torch.randn(*shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")


OPTIONS = {"plain": {}, "block": {"block": 200}, "window": {"window": 130}, "sink gate": {"sink": True, "gate": True}, "softcap": {"softcap": 20.0}, "negative": {"negative": True}, "mul": {"mul": True}}


@pytest.mark.parametrize("option", OPTIONS)
@pytest.mark.parametrize("D,VD", [(64, 64), (48, 48), (48, 128), (128, 60), (128, 128), (68, 4)])
def test_attention(probe, D, VD, option):
    o = dict(OPTIONS[option])
    T, H, G, pos0 = 333, 6, 2, 177
    q, k, v = randn(1, T, H, D), randn(2, pos0 + T, G, D), randn(3, pos0 + T, G, VD)
    scale = D ** -0.5 * (-1.0 if o.pop("negative", None) else 1.0)
    if o.pop("sink", None):
        o["sink"] = randn(4, H)
    if o.pop("gate", None):
        o["gate"] = randn(5, T, H)
    if o.pop("mul", None):
        o["mul"] = randn(6, T, H, VD)
    got = attention(probe, q, k, v, H, G, pos0, scale, paged=option in ("block", "sink gate"), **o).double()
    want = attention64(q, k, v, H, G, pos0, scale, **o)
    size = attention64(q, k, v.abs(), H, G, pos0, scale, **dict(o, mul=o["mul"].abs() if "mul" in o else None)).norm(dim=2)
    err = (got - want).norm(dim=2) / size
    print("%d %d %s: worst row %.2e, all %.2e" % (D, VD, option, err.max(), (got - want).norm() / size.norm()))
    assert err.max() < 1e-6 + 2.0 ** -24 * o.get("softcap", 0.0)


@pytest.mark.parametrize("D,VD", [(48, 48), (64, 64), (128, 128)])
def test_what_the_sums_lose(probe, D, VD):
    """Values near 1 under nearly equal weights: what the tensor cores cut off is always of the same sign.  An addition of 16 keys loses half of a last place
    on average, 2^-24 of a sum just above a power of two: two of them for heads of up to 64 values (a sum per 32 keys), eight above (one per 128)."""
    T, H, G, pos0 = 256, 4, 4, 768
    q, k, v = 0.1 * randn(1, T, H, D), randn(2, pos0 + T, G, D), 1.0 + 0.1 * randn(3, pos0 + T, G, VD)
    got, want = attention(probe, q, k, v, H, G, pos0, D ** -0.5).double(), attention64(q, k, v, H, G, pos0, D ** -0.5)
    lost = float(((want - got) / want).mean())
    print("%d %d: lost %.2e" % (D, VD, lost))
    assert lost < (2 if VD <= 64 else 8) * 2.0 ** -24


@pytest.mark.parametrize("first,rows,N,K", [(0, 128, 128, 64), (0, 333, 200, 40), (130, 517, 1000, 256), (32, 129, 136, 520)])
def test_product_of_latents(probe, first, rows, N, K):
    """fp32 rows in three bfloat16 parts (all 24 bits) times bfloat16 weights: fp32 sums that are cut, 2^-24 for each 16 of the 3 K."""
    n, ld = first + rows, K + 8
    cache = torch.zeros((n + 31) // 32 * 32, ld, device="cuda")
    pages = torch.randperm(cache.shape[0] // 32, generator=torch.Generator().manual_seed(1)).cuda()
    at = torch.arange(n, device="cuda")
    x = randn(1, n, K) * torch.exp2(torch.randint(-20, 20, (n, 1), generator=torch.Generator(device="cuda").manual_seed(3), device="cuda").float())
    cache[(pages[at // 32] * 32 + at % 32).long(), :K] = x
    w = randn(2, N, K).bfloat16()
    out = torch.full((rows, N), float("nan"), device="cuda")
    table = pages.to(torch.int32)
    torch.cuda.synchronize()
    assert probe.probe_split(ptr(cache), ptr(table), ld, first, rows, ptr(w), N, K, ptr(out), N) == 0
    want = x[first:].double() @ w.double().T
    err = (out.double() - want).norm(dim=1) / want.norm(dim=1)
    print("%d %d %d: worst row %.2e" % (rows, N, K, err.max()))
    assert err.max() < 2.0 ** -23 * max(4.0, (K / 16) ** 0.5)
