"""GPU tests of the kernels' size-dependent paths, at the sizes where a rule
switches and at the edges of tiles and windows, against the oracle.

Tolerances (relative L2, derived): the compared programs evaluate the same
sums in the same precision; double paths differ by a few roundings per term
(an exponent of E2^m amplifies one ulp of E2 at most 11 times, about 3e-15,
and the FFT adds log2(ng) 1e-16), so 1e-13.
"""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mods(native_built):
    from cunfft_adjoint_gb300 import cuna, nfft
    return cuna, nfft


@pytest.mark.parametrize("n,ng", [(1, 1 << 14), (777, 1 << 14), (40_001, 1 << 17), (70_000, 1 << 21)])
def test_compat_double_powers_and_factors(mods, oracle_lib, n, ng):
    """E2^m by running products (many and few tiles per SM) and the row
    pass's deconvolution factors between exps, with samples on both ends of
    the grid and on tile boundaries."""
    cuna, _ = mods
    rng = np.random.default_rng(n)
    x = rng.uniform(-0.5, 0.5, n)
    edge = np.array([-0.5, 0.5, np.nextafter(0.5, 0), (4096 - 0.5) / (ng - 1) - 0.5, 4096.5 / (ng - 1) - 0.5])
    x[:min(n, len(edge))] = edge[:min(n, len(edge))]
    y = rng.normal(0, 1, n)
    xd, yd = torch.as_tensor(x, device="cuda"), torch.as_tensor(y, device="cuda")
    fp = cuna.generate_filter_properties(xd, n, ng)
    f_hat = torch.zeros(ng, dtype=torch.complex128, device="cuda")
    cuna.cunfft_adjoint_raw(xd, yd, f_hat, n, ng, fp)
    assert rel_l2(f_hat.cpu().numpy(), oracle_lib.compat_adjoint(x, y, ng, "d")) < 1e-13
