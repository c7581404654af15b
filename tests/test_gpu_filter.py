"""Gradient band-pass filter (reference bandpass_filter, FD2DGPU.cu:4125-4182) on the GPU against
the FP64 restatement of the reference's steps and against the reference's own cuFFT results."""
import numpy as np
import pytest

from ds2d_b200.api import bandpass_filter, bandpass_filter_device
from oracle import pyoracle as po
from tests.helpers import load, rel

pytestmark = pytest.mark.gpu

# FP64 transforms stored as FP32: the GPU's DFT products, numpy's FFT and cuFFT round the FP64
# intermediates differently, which reaches the FP32 results at the last-bit level only.
TOL = 1e-6


@pytest.mark.parametrize("nx,nz,z1,z2", [(1201, 401, 0, 80), (1201, 401, 20, 80), (81, 41, 3, 12),
                                         (64, 32, 0, 6)])
def test_bandpass_vs_oracle(cuda_device, nx, nz, z1, z2):
    rng = np.random.default_rng(nx + z1)
    pp = rng.standard_normal((nx, nz)).astype(np.float32)
    ps = rng.standard_normal((nx, nz)).astype(np.float32)
    fpp, fps = bandpass_filter(pp, ps, z1, z2)
    assert rel(fpp, po.bandpass(pp, z1, z2)) < TOL
    assert rel(fps, po.bandpass(ps, z1, z2)) < TOL
    assert np.array_equal(pp, pp)  # inputs untouched (copies are filtered)


def test_bandpass_device_in_place(cuda_device):
    import torch
    rng = np.random.default_rng(5)
    img = rng.standard_normal((121, 41)).astype(np.float32)
    d = torch.from_numpy(img).cuda()
    torch.cuda.synchronize()
    bandpass_filter_device(d.data_ptr(), 0, 121, 41, 0, 10)
    assert rel(d.cpu().numpy(), po.bandpass(img, 0, 10)) < TOL


def test_bandpass_vs_reference_golden(cuda_device):
    fx = load("bandpass.npz")
    assert fx is not None, "golden fixture bandpass.npz missing"
    for i, (nx, nz, z1, z2) in enumerate(fx["cases"]):
        fpp, fps = bandpass_filter(fx[f"in_pp{i}"], fx[f"in_ps{i}"], int(z1), int(z2))
        assert rel(fpp, fx[f"out_pp{i}"]) < TOL, (i, rel(fpp, fx[f"out_pp{i}"]))
        assert rel(fps, fx[f"out_ps{i}"]) < TOL, (i, rel(fps, fx[f"out_ps{i}"]))


def test_bandpass_rejects_bad_arguments(cuda_device):
    from ds2d_b200._lib import DS2DError
    with pytest.raises(DS2DError):
        bandpass_filter(np.zeros((8, 8), np.float32), np.zeros((8, 8), np.float32), 0, 0)


# Lengths around the powers of two that the chirp transforms pad to, the shortest, the longest of
# the in-memory transforms and one beyond them (dense products).
@pytest.mark.parametrize("nx,nz,z1,z2", [(2, 2, 0, 3), (3, 2, 1, 2), (5, 8, 0, 2), (32, 33, 2, 9),
                                         (33, 65, 0, 9), (4096, 3, 5, 60), (3, 4096, 0, 60),
                                         (2049, 17, 0, 40), (4097, 6, 0, 60)])
def test_bandpass_lengths(cuda_device, nx, nz, z1, z2):
    rng = np.random.default_rng(nx + nz)
    pp = rng.standard_normal((nx, nz)).astype(np.float32)
    ps = 1e-3 * rng.standard_normal((nx, nz)).astype(np.float32)
    fpp, fps = bandpass_filter(pp, ps, z1, z2)
    assert rel(fpp, po.bandpass(pp, z1, z2)) < TOL
    assert rel(fps, po.bandpass(ps, z1, z2)) < TOL


def test_bandpass_sizes_in_two_threads(cuda_device):
    """Calls on a large and a small image in two threads (ctypes releases the interpreter lock):
    both keep the results that they have alone."""
    import threading
    rng = np.random.default_rng(17)
    cases = [(1201, 401, 10, 60, 60), (60, 40, 3, 12, 600)]
    images = [rng.standard_normal((2, nx, nz)).astype(np.float32) for nx, nz, *_ in cases]
    alone = [bandpass_filter(*im, z1, z2) for im, (_, _, z1, z2, _) in zip(images, cases)]
    go, failed = threading.Barrier(2), []

    def work(k):
        _, _, z1, z2, calls = cases[k]
        go.wait()
        for _ in range(calls):
            try:
                got = bandpass_filter(*images[k], z1, z2)
            except Exception as e:  # noqa: BLE001 - reported by the assertion below
                failed.append((k, str(e)))
                return
            if not all(np.array_equal(a, b) for a, b in zip(got, alone[k])):
                failed.append((k, "another result"))
                return

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


@pytest.mark.parametrize("shift", [0, 5])
def test_bandpass_device_images_that_share_memory(cuda_device, shift):
    """One buffer as both images, and two overlapping ones: filtered one after the other, the
    second as the first left it."""
    import torch
    nx, nz = 24, 10
    base = np.random.default_rng(4).standard_normal(nx * nz + shift * nz).astype(np.float32)
    want = base.copy()
    for at in (0, shift * nz):
        want[at:at + nx * nz] = po.bandpass(want[at:at + nx * nz].reshape(nx, nz), 2, 5).ravel()
    d = torch.from_numpy(base).cuda()
    torch.cuda.synchronize()
    bandpass_filter_device(d.data_ptr(), d.data_ptr() + 4 * shift * nz, nx, nz, 2, 5)
    assert rel(d.cpu().numpy(), want) < TOL
