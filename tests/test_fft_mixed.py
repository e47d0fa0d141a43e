"""The mixed-radix image transforms (csrc/fft_mixed.cuh), built for the host with g++ and compared
with numpy's FFT in double: spectrum, low-pass and inverse of every shape family (radix pairs,
columns split in a pass of their own).  CPU only.

Tolerance: each output passes through 4 (spectrum) to 8 (low-pass) float DFT stages of at most
32 terms with a twiddle; 2^-24 times sqrt(stages x 5 roundings) times a peak factor of 4 over
the rms error is below 2e-6 of the largest value."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from test_fft_radix import CSRC, HERE, _cuda_include


def test_mixed_transforms_match_numpy(tmp_path):
    inc = _cuda_include()
    if shutil.which('g++') is None or inc is None:
        pytest.skip('g++ or the CUDA headers are missing')
    exe = str(tmp_path / 'fft_mixed_host')
    subprocess.run(['g++', '-std=c++17', '-O1', '-I', CSRC, '-I', inc,
                    os.path.join(HERE, 'native', 'fft_mixed_host.cpp'), '-o', exe], check=True)
    data = subprocess.run([exe], check=True, capture_output=True).stdout
    off, seen = 0, 0
    while off < len(data):
        N, r1 = np.frombuffer(data, np.int32, 2, off)
        off += 8
        Nh = N // 2 + 1

        def take(n):
            nonlocal off
            v = np.frombuffer(data, np.float32, n, off).astype(np.float64)
            off += 4 * n
            return v

        spec = take(2 * N * Nh).view(complex).reshape(N, Nh)
        low, back = take(N * N).reshape(N, N), take(N * N).reshape(N, N)
        r, c = np.meshgrid(np.arange(N), np.arange(N), indexing='ij')
        x = np.sin(0.37 * r + 0.011 * c * c) + 0.3 * np.cos(0.9 * c - 0.2 * r * c)
        x = (x.astype(np.float32).astype(np.float64) - 0.25) * 2
        F = np.fft.fft2(x)
        f = np.minimum(np.arange(N), N - np.arange(N))
        g = 1 / (1 + 0.01 * f[:, None] ** 2 + 0.02 * f[None, :] ** 2)
        for got, ref in ((spec, F[:, :Nh]), (low, np.fft.ifft2(F * g).real * N * N),
                         (back, x * N * N)):
            err = np.abs(got - ref).max() / np.abs(ref).max()
            assert err < 2e-6, (N, r1, err)
        seen += 1
    assert seen == 14
