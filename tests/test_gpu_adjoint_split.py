"""The adjoint contraction of one system, whose 64-row blocks go to four CTAs each."""
import ctypes

import numpy as np
import pytest
import torch

from mpdok_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [0, 1])
@pytest.mark.parametrize("n,dim,k", [(1, 1, 1), (15, 2, 2), (17, 3, 1), (63, 2, 3), (65, 1, 4), (255, 3, 4),
                                     (257, 2, 1), (530, 2, 5), (1000, 3, 2)])
def test_one_system_against_numpy(n, dim, k, kernel):
    from mpdok_gb300._device import ptr, stream_handle
    rng = np.random.default_rng(10 * n + k)
    C, X, L = rng.random((n, dim)), rng.standard_normal((k, n)), rng.standard_normal((k, n))
    eps = 3.0
    gam = eps * eps
    df = C[:, None, :] - C[None, :, :]
    r2 = (df ** 2).sum(-1)
    phi = np.exp(-gam * r2) if kernel == 0 else np.sqrt(1.0 + gam * r2)
    g, h = (-gam * phi, -r2 * phi) if kernel == 0 else (0.5 * gam / phi, 0.5 * r2 / phi)
    W = L.T @ X
    S = W + W.T
    T = (S * g)[:, :, None] * df
    ref_c, abs_c = -2.0 * T.sum(1), 2.0 * np.abs(T).sum(1)
    ref_e, abs_e = -2.0 * eps * (W * h).sum(), 2.0 * eps * np.abs(W * h).sum()
    ref_r, abs_r = -(L * X).sum(), np.abs(L * X).sum()
    lib = N.load()
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    c, x, l = dev(C), dev(X), dev(L)
    gc, ge, gr = torch.empty_like(c), torch.empty(1, dtype=torch.float64).cuda(), torch.empty(1, dtype=torch.float64).cuda()
    w = torch.empty(lib.mpdok_rbf_adjoint_workspace_size(n), dtype=torch.uint8, device="cuda")
    N.check(lib.mpdok_rbf_adjoint(ptr(c), n, dim, kernel, ctypes.c_double(eps), k, ptr(x), ptr(l), ptr(gc), ptr(ge),
                                  ptr(gr), ptr(w), w.numel(), stream_handle()))
    # sums of n (gradients of the centres) and n^2 terms, each with a handful of
    # roundings besides phi's few 2^-53; what cancels counts through |S| and |W|
    u = 2.0 ** -53
    mag = (np.abs(L).T @ np.abs(X) + np.abs(X).T @ np.abs(L))[:, :, None] * np.abs(g)[:, :, None] * np.abs(df)
    assert (np.abs(gc.cpu().numpy() - ref_c) <= 2 * (n + 40) * u * (2.0 * mag.sum(1) + abs_c) + 1e-300).all()
    mag_e = eps * ((np.abs(L).T @ np.abs(X) + np.abs(X).T @ np.abs(L)) * np.abs(h)).sum()
    assert abs(ge.item() - ref_e) <= 2 * (2 * n + 40) * u * (mag_e + abs_e) + 1e-300
    assert abs(gr.item() - ref_r) <= 2 * (n + k) * u * abs_r
