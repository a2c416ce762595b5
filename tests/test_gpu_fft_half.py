"""The half-spectrum FFT Poisson solve on odd, ragged and long lengths, against numpy.fft restatements.

The x spectrum of a real right-hand side is kept up to Mx / 2.  That leans on the k-space factor being even,
which the reference's frequency rule (kernel_fft.cu:90-104) is not on odd axes: it takes (N - 1) / 2 as a negative
frequency, unlike numpy's fftfreq, so the periodic reference below restates it over the whole spectrum.  The grid
class takes multiples of 8 only, so these sizes go through the native entry, on a random density.
"""
import ctypes as C

import numpy as np
import pytest

import qmtools
from qmtools import _native as N
from qmtools import synthetic as syn
from oracle import poisson as op
from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = 2e-5   # FP32 transforms against FP64 numpy.fft, as for the even lengths


def _periodic(q, shape, h, org, coords, types, sigma, cutoff):
    f = np.fft.fftn(op.fft_rhs(q, shape, h, org, coords, types, sigma, cutoff))
    k = [np.where(np.arange(n) > n // 2 - 1, np.arange(n) - n, np.arange(n)) / (n * h / qmtools.ANG2BOR)
         for n in shape]
    k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
    k2[0, 0, 0] = 1.0
    f = -f / (4 * np.pi ** 2 * k2)
    f[0, 0, 0] = 0.0
    return np.fft.ifftn(f).real


def _solve(basis, shape, padded):
    import torch
    sm = syn.config_molecule("c0")
    mol = sm.molecule(basis, qmtools.Molecule)
    N.ensure_device()
    n = int(np.prod(shape))
    h = float(np.float32(0.5))
    org = [float(np.float32(c - s * h / 2)) for c, s in zip(np.asarray(sm.coords_bohr).mean(axis=0), shape)]
    q = torch.rand(n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(5)) * 1e-2
    v = torch.empty(n, device="cuda")
    N.call("qmt_fft_poisson", mol.handle, *shape, h, *org, 0.2, 6.0, int(padded), C.c_void_p(q.data_ptr()),
           C.c_void_p(v.data_ptr()), N.stream_handle())
    fn = op.hockney_poisson if padded else _periodic
    ref = fn(q.cpu().numpy(), shape, h, org, mol.coords, mol.types, 0.2, 6)
    return v.cpu().numpy().reshape(shape), ref


@pytest.mark.parametrize("shape", [(25, 27, 35), (21, 32, 24), (32, 21, 24), (32, 24, 21), (33, 26, 65),
                                   (50, 9, 70), (2, 24, 30), (3, 24, 25), (30, 2, 3)])
def test_periodic_odd_lengths(basis, shape):
    assert rel_l2(*_solve(basis, shape, False)) < TOL


@pytest.mark.parametrize("shape", [(37, 16, 22), (16, 37, 22), (22, 16, 37), (50, 12, 9), (12, 9, 54),
                                   (9, 45, 12), (2, 3, 2)])
def test_padded_ragged_lengths(basis, shape):
    """2 * 37 = 74 is padded to 75, an odd length; the rest mixes the radices 2, 3, 5 and 7."""
    assert rel_l2(*_solve(basis, shape, True)) < TOL


@pytest.mark.parametrize("shape", [(4, 6, 10), (11, 22, 13), (12, 14, 15), (49, 5, 81), (704, 4, 12), (12, 720, 4),
                                   (4, 12, 1715), (1875, 2, 12), (2, 2048, 17), (40, 36, 127)])
def test_periodic_line_plans(basis, shape):
    """One stage to five, every radix, 16 and 4 lines per block, remainders of lines, and lengths with other primes."""
    assert rel_l2(*_solve(basis, shape, False)) < TOL
