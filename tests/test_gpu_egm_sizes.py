"""The electrogram's kernels at the edges of their tiles, copies and alignments,
against the same sums in plain torch FP64."""
import ctypes

import numpy as np
import pytest

from pyheartsim_b200 import _lib

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


# 128 x 64 output tiles, K-steps of 16, at least 256 of K per split; odd leading
# dimensions and bases off a 16-byte boundary take the 8-byte copies
@pytest.mark.parametrize("T,n_e,n_v,pad,shift", [(1, 1, 1, 0, 0), (127, 63, 15, 1, 0), (128, 64, 16, 0, 0),
                                                 (129, 65, 17, 1, 1), (100, 16, 20001, 0, 0), (257, 130, 4096, 2, 1),
                                                 (300, 70, 1001, 3, 0)])
def test_fp64_contraction_edges(T, n_e, n_v, pad, shift, cuda_device):
    import torch
    g = torch.Generator(device=cuda_device).manual_seed(T + n_e + n_v)
    ld = n_v + pad
    store = torch.randn(T * ld + shift, dtype=torch.float64, device=cuda_device, generator=g)
    V = store[shift:].view(T, ld)
    Mt = torch.randn(n_e, n_v, dtype=torch.float64, device=cuda_device, generator=g)
    out = torch.full((T, n_e), float("nan"), dtype=torch.float64, device=cuda_device)
    _lib.check(_lib.lib().phs_egm_contract_f64(T, n_v, n_e, _p(V), ld, _p(Mt), _p(out), None), "phs_egm_contract_f64")
    torch.cuda.synchronize()
    want = V[:, :n_v] @ Mt.T
    # both are FP64 sums of n_v products: n_v eps sum |v m| at most, and that is far
    # above what either order loses
    bound = 2 * n_v * 2.2e-16 * (V[:, :n_v].abs() @ Mt.abs().T)
    assert bool(((out - want).abs() <= bound).all())


@pytest.mark.parametrize("terms,n_e,tensor", [(6, 1, False), (6, 16, True), (6, 17, False), (9, 33, True)])
def test_leadfield_terms_and_chunks(terms, n_e, tensor, cuda_device):
    """Any CSR of gradient terms, more than six to a voxel among them."""
    import torch
    rng = np.random.default_rng(terms * 100 + n_e)
    n = 300
    xyz, exyz = rng.uniform(0, 20, (n, 3)), rng.uniform(0, 20, (n_e, 3))
    exyz[0] = xyz[0] + 0.1                                        # within the 1 mm clamp
    c, D0 = rng.uniform(0, 2, n), rng.normal(size=(n, 3, 3)) if tensor else None
    cnt = rng.integers(0, terms + 1, n)
    ptr = np.zeros(n + 1, np.int32)
    np.cumsum(cnt, out=ptr[1:])
    src = rng.integers(0, n, ptr[-1]).astype(np.int32)
    dirs = (rng.integers(1, 4, ptr[-1]) * rng.choice([-1, 1], ptr[-1])).astype(np.int8)
    d = lambda a: None if a is None else torch.as_tensor(np.ascontiguousarray(a), device=cuda_device)
    t = [d(a) for a in (xyz, exyz, c, D0, ptr, src, dirs)]
    Mt = torch.empty((n_e, n), dtype=torch.float64, device=cuda_device)
    q = lambda x: None if x is None else _p(x)
    _lib.check(_lib.lib().phs_egm_leadfield_f64(n, n_e, q(t[0]), q(t[1]), q(t[2]), q(t[3]), q(t[4]), q(t[5]), q(t[6]),
                                                1.25, _p(Mt), None), "phs_egm_leadfield_f64")
    torch.cuda.synchronize()
    want, mag = np.zeros((n_e, n)), np.zeros((n_e, n))
    for w in range(n):
        for k in range(ptr[w], ptr[w + 1]):
            v, a = src[k], abs(int(dirs[k])) - 1
            l = xyz[v] - exyz
            proj = l[:, a] if D0 is None else l @ D0[v][:, a]
            val = np.sign(dirs[k]) * c[v] * proj / np.maximum(np.linalg.norm(l, axis=1), 1.0) ** 3 * 1.25
            want[:, w] += val
            full = np.abs(l).sum(axis=1) * (1.0 if D0 is None else np.abs(D0[v]).max())
            mag[:, w] += c[v] * full / np.maximum(np.linalg.norm(l, axis=1), 1.0) ** 3 * 1.25
    # a term has some 20 roundings
    assert np.all(np.abs(Mt.cpu().numpy() - want) <= 40 * 2.2e-16 * mag)


@pytest.mark.parametrize("is64", [False, True])
@pytest.mark.parametrize("rows,cols,ld,rows_out,ld_out", [(1, 1, 1, 1, 1), (3, 63, 63, 128, 64), (5, 64, 67, 5, 66),
                                                          (2, 1023, 1024, 4, 1088), (7, 130, 131, 9, 131)])
def test_split_is_exact_by_element(rows, cols, ld, rows_out, ld_out, is64, cuda_device):
    import torch
    g = torch.Generator(device=cuda_device).manual_seed(rows * 1000 + cols)
    src = torch.randn((rows, ld), dtype=torch.float64, device=cuda_device, generator=g)
    src = src if is64 else src.float()
    hi = torch.full((rows_out, ld_out), 7, dtype=torch.uint16, device=cuda_device)
    lo = hi.clone()
    _lib.check(_lib.lib().phs_split_bf16(rows, cols, _p(src), ld, int(is64), _p(hi), _p(lo), rows_out, ld_out, None),
               "phs_split_bf16")
    torch.cuda.synchronize()
    want_hi = torch.zeros((rows_out, ld_out), dtype=torch.bfloat16, device=cuda_device)
    want_lo = want_hi.clone()
    x = src[:, :cols]
    want_hi[:rows, :cols] = x.float().bfloat16()
    want_lo[:rows, :cols] = (x.double() - want_hi[:rows, :cols].double()).float().bfloat16()
    assert torch.equal(hi.view(torch.bfloat16), want_hi) and torch.equal(lo.view(torch.bfloat16), want_lo)


@pytest.mark.parametrize("is64", [False, True])
@pytest.mark.parametrize("T,n_e", [(1, 5), (31, 1), (33, 31), (100, 33), (64, 600)])
def test_normalise(T, n_e, is64, cuda_device):
    import torch
    g = torch.Generator(device=cuda_device).manual_seed(T * 1000 + n_e)
    egm = torch.randn((T, n_e), dtype=torch.float64, device=cuda_device, generator=g)
    egm = egm if is64 else egm.float()
    want = egm.double()
    want = want / (want.max(0).values - want.min(0).values).mean()
    _lib.check(_lib.lib().phs_egm_normalize(T, n_e, _p(egm), int(is64), None), "phs_egm_normalize")
    torch.cuda.synchronize()
    if T == 1:                                   # no range to scale by: 1 / 0, as before
        assert not bool(torch.isfinite(egm).any())
        return
    # one product per value and a mean of n_e: a few eps of the type
    assert bool(((egm.double() - want).abs() <= (1e-14 if is64 else 3e-7) * want.abs()).all())


# pairs of CTAs (configuration 3) against single ones (1): the same products in
# the same order; T_pad an odd number of 128-row tiles falls back to single ones,
# n_e_pad 128 leaves half of a pair's columns empty, K_pad 64 is one stage
@pytest.mark.parametrize("T,E,K", [(200, 40, 64), (256, 256, 192), (100, 300, 1000), (500, 130, 9000),
                                   (1000, 600, 20000)])
def test_contraction_by_pairs_equals_single(T, E, K, cuda_device):
    import torch
    L = _lib.lib()
    up = lambda x, m: -(-x // m) * m
    Tp, Ep, Kp = up(T, 128), up(E, 128), up(K, 64)
    g = torch.Generator(device=cuda_device).manual_seed(T + E + K)
    pad = lambda r, c, rp: torch.nn.functional.pad(
        torch.randn((r, c), device=cuda_device, generator=g), (0, Kp - c, 0, rp - r)).bfloat16()
    vh, vl, mh, ml = pad(T, K, Tp), pad(T, K, Tp) * 2 ** -8, pad(E, K, Ep), pad(E, K, Ep) * 2 ** -8
    work = torch.empty(L.phs_egm_bf16x3_workspace(Tp, Ep, Kp), dtype=torch.uint8, device=cuda_device)
    out = []
    for cfg in (1, 3):
        o = torch.full((T, E), float("nan"), device=cuda_device)
        _lib.check(L.phs_egm_contract_bf16x3_cfg(T, E, Tp, Ep, Kp, _p(vh), _p(vl), _p(mh), _p(ml), _p(o), _p(work), cfg,
                                                 None), "phs_egm_contract_bf16x3_cfg")
        _lib.check(L.phs_egm_bf16x3_status(_p(work), None), "phs_egm_bf16x3_status")
        out.append(o)
    d = lambda t: t[:, :K].double()
    want = d(vh)[:T] @ d(mh)[:E].T + d(vh)[:T] @ d(ml)[:E].T + d(vl)[:T] @ d(mh)[:E].T
    # FP32 accumulation of 3 K products of sizes around 1: K eps of their magnitude
    bound = 3 * K * 6e-8 * (d(vh)[:T].abs() @ d(mh)[:E].abs().T)
    assert bool(((out[0].double() - want).abs() <= bound).all())
    assert torch.equal(out[0], out[1])


def test_contractions_and_normalisation_under_capture(cuda_device):
    """Captured in a graph after a first call outside (as the allocation-free form
    asks), replayed on new inputs; the workspaces of the others belong to the graph."""
    import torch
    L = _lib.lib()
    T, n_e, n = 130, 70, 3001
    g = torch.Generator(device=cuda_device).manual_seed(5)
    V = torch.randn((T, n), dtype=torch.float64, device=cuda_device, generator=g)
    Mt = torch.randn((n_e, n), dtype=torch.float64, device=cuda_device, generator=g)
    a, b = (torch.empty((T, n_e), dtype=torch.float64, device=cuda_device) for _ in range(2))

    def call():
        s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        _lib.check(L.phs_egm_contract_f64(T, n, n_e, _p(V), n, _p(Mt), _p(a), s), "phs_egm_contract_f64")
        _lib.check(L.phs_egm_contract_f64_noalloc(T, n, n_e, _p(V), n, _p(Mt), _p(b), s), "noalloc")
        _lib.check(L.phs_egm_normalize(T, n_e, _p(a), 1, s), "phs_egm_normalize")
        _lib.check(L.phs_egm_normalize(T, n_e, _p(b), 1, s), "phs_egm_normalize")

    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    V.copy_(torch.randn((T, n), dtype=torch.float64, device=cuda_device, generator=g))
    graph.replay()
    torch.cuda.synchronize()
    got = a.clone(), b.clone()
    call()
    torch.cuda.synchronize()
    assert torch.equal(got[0], a) and torch.equal(got[1], b)
    want = V @ Mt.T
    want = want / (want.max(0).values - want.min(0).values).mean()
    # n products a value, normalised: far within 1e-11 of values around 1
    assert float((a - want).abs().max()) < 1e-11 and float((b - want).abs().max()) < 1e-11
