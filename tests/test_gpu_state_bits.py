"""The fused engine's states keep their bits from one version of its kernels to the next (GPU).

A run's last bits are part of what it returns: fp64 records of fp32 runs are compared between
versions at 1e-9, where another rounding anywhere in an fp32 step moves them by 1e-7 to 2e-6.
``golden/state_bits.json`` holds digests of states recorded with the kernels of commit e6eaa50
(one thread per pair in every 2D column pass, unpacked 3D sums); a kernel that rounds anything
else, or a compiler that fuses other products, changes them.

``python tests/test_gpu_state_bits.py OUT.json`` records the digests of the library in use.
"""

from __future__ import annotations

import hashlib
import json
import sys
from pathlib import Path

import numpy as np
import pytest

FUSED = "b200/fused-fft-graph"
GOLDEN = Path(__file__).resolve().parent / "golden" / "state_bits.json"
PHYSICS = dict(nu=1e-3, alpha=0.1, alpha_kmax=2.0, force_amp=0.2, force_klo=3, force_khi=5)


def _noise(rng, shape):
    """Complex numbers of 21-bit parts: with products and quotients of float64 only, the states
    below are the same on every machine."""
    return rng.integers(-2**20, 2**20, shape) / 2.0**20, rng.integers(-2**20, 2**20, shape) / 2.0**20


def _complex(re, im):
    out = np.empty(re.shape, np.complex128)
    out.real, out.imag = re, im
    return out


def _vorticity(torch, n, seed):
    """Spectral vorticity on the device: random modes below min(n/3, 128), steep spectrum."""
    m = min((n - 1) // 3, 128)
    k = np.concatenate([np.arange(m + 1), np.arange(-m, 0)]).astype(np.float64)
    k2 = k[:, None] ** 2 + np.arange(m + 1.0)[None, :] ** 2
    amp = float(n) * n / (8.0 + k2 * np.sqrt(k2) / 2.0)
    a = _complex(*(c * amp for c in _noise(np.random.default_rng(seed), k2.shape)))
    a[m + 1:, 0] = a[1:m + 1, 0][::-1].conj()  # ky = 0 of a real field is Hermitian
    a[0, 0] = 0.0
    out = torch.zeros((n, n // 2 + 1), dtype=torch.complex128, device="cuda")
    a = torch.from_numpy(a).cuda()
    out[: m + 1, : m + 1], out[n - m:, : m + 1] = a[: m + 1], a[m + 1:]
    return out


def _velocity(torch, n, seed):
    """Spectral velocity k x a on the device: random modes a below min(n/3, 16)."""
    m = min((n - 1) // 3, 16)
    k = np.concatenate([np.arange(m + 1), np.arange(-m, 0)]).astype(np.float64)
    kx, ky, kz = k[:, None, None], k[None, :, None], np.arange(1.0, m + 1.0)[None, None, :]
    k2 = kx * kx + ky * ky + kz * kz
    amp = float(n) ** 3 / 8.0 / (1.0 + k2 * k2)
    re, im = (c * amp for c in _noise(np.random.default_rng(seed), (3, 2 * m + 1, 2 * m + 1, m)))
    u = [_complex(ka * re[b] - kb * re[a], ka * im[b] - kb * im[a])
         for ka, kb, a, b in ((ky, kz, 1, 2), (kz, kx, 2, 0), (kx, ky, 0, 1))]
    out = torch.zeros((3, n, n, n // 2 + 1), dtype=torch.complex128, device="cuda")
    idx = torch.from_numpy(k.astype(np.int64) % n).cuda()  # kz >= 1: no Hermitian plane
    for c in range(3):
        plane = torch.zeros((2 * m + 1, n, n // 2 + 1), dtype=torch.complex128, device="cuda")
        plane[:, idx, 1: m + 1] = torch.from_numpy(u[c]).cuda()
        out[c, idx] = plane
    return out


def _digest(h, tensor):
    h.update(tensor.cpu().contiguous().numpy().tobytes())


def _batch(n, dtype, tile):
    """Members with states, steps and forcing of their own: the batched passes of one tile."""
    import torch

    from pyspectral_b200 import Config
    from pyspectral_b200.ensemble import Ensemble

    count = 16 if n <= 128 else 4
    ens = Ensemble([Config(n=n, dim=2, dtype=dtype, **PHYSICS)] * count, autotune=False, worklist=0)
    ens.classes[0].set_tile(tile)
    ens.set_states([_vorticity(torch, n, i).cpu().numpy() for i in range(count)])
    ens.set_forcing_amplitudes([0.1 + 0.01 * i for i in range(count)])
    for dt in (1e-4, 2e-4, 1e-3):
        ens.step([dt * (1 + 0.01 * i) for i in range(count)])
    h = hashlib.sha256()
    for i in range(count):
        _digest(h, ens.state_native(i))
    return h.hexdigest()[:16]


def _single(n, dim, dtype, form, streamed=True):
    import torch

    from pyspectral_b200 import Config
    from pyspectral_b200.registry import get
    from pyspectral_b200.solver import set_column_streaming

    prev = set_column_streaming(streamed)
    try:
        s = get(FUSED).make(Config(n=n, dim=dim, dtype=dtype, form=form, **PHYSICS))
        h = hashlib.sha256()
        for seed in range(4 if n <= 64 else 1):
            s.set_state((_vorticity if dim == 2 else _velocity)(torch, n, seed))
            for dt in (1e-4, 2e-4, 1e-3):
                s.step(dt)
            _digest(h, s.state_native())
            h.update(np.float64(s.diag.max_velocity_sum(s.state_native())).tobytes())
        return h.hexdigest()[:16]
    finally:
        set_column_streaming(prev)


CASES = {}
for _dtype in ("float32", "float64"):
    for _n in (16, 32, 64, 128, 256, 512, 1024):
        for _tile in (1, 2, 4):
            CASES[f"2d-{_n}-{_dtype}-tile{_tile}"] = (_batch, _n, _dtype, _tile)
    for _n in (2048, 4096):
        for _streamed in (True, False):
            CASES[f"2d-{_n}-{_dtype}-{'streamed' if _streamed else 'columns'}"] = (
                _single, _n, 2, _dtype, "basdevant", _streamed)
    for _n in (16, 32, 64, 128, 256):
        for _form in ("basdevant", "rotational"):
            CASES[f"3d-{_n}-{_dtype}-{_form}"] = (_single, _n, 3, _dtype, _form)


@pytest.mark.gpu
@pytest.mark.parametrize("name", CASES)
def test_states_keep_their_bits(name):
    fn, *args = CASES[name]
    assert fn(*args) == json.loads(GOLDEN.read_text())[name]


if __name__ == "__main__":
    Path(sys.argv[1]).write_text(
        json.dumps({k: fn(*args) for k, (fn, *args) in CASES.items()}, indent=1) + "\n")
