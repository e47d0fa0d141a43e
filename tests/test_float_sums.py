"""The pair sums of the NLSA kernels (csrc/float_sums.cuh), built for the host with g++: every value
that a pair decides is the float of the FP64 sum, bit for bit, over CTFs, wide ranges, sums with
few bits (ties), cancellation, the ends of the float range, infinities and NaN.  CPU only."""
import os
import shutil
import subprocess

import pytest

from test_fft_radix import CSRC, HERE


def test_decided_pair_sums_round_as_fp64_does(tmp_path):
    if shutil.which('g++') is None:
        pytest.skip('g++ is missing')
    exe = str(tmp_path / 'float_sums_host')
    subprocess.run(['g++', '-std=c++17', '-O2', '-ffp-contract=off', '-frounding-math', '-I', CSRC,
                    os.path.join(HERE, 'native', 'float_sums_host.cpp'), '-o', exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    counts = {w[0]: [int(x) for x in w[1:]] for w in map(str.split, out.splitlines())}
    assert len(counts) == 9 + 5 * 7
    for name, (values, undecided, wrong, caught) in counts.items():
        assert values > 0 and wrong == 0, (name, counts[name])
    # the pair alone is wrong where a large term has left the window or terms cancel
    assert counts['large_leaves'][3] > 0 and counts['cancel_15'][3] > 0
    # ordinary CTFs hardly ever need FP64
    for name in ('ctf_c1', 'ctf_c20', 'ctf_c200'):
        assert counts[name][1] < 1e-3 * counts[name][0]
