"""Host-side logic of the reconstruction server that needs no GPU: the
argument key that decides which retired Rec a request may take over, and the
device-memory estimate admission uses."""
import types

import numpy as np

from holotomocupy_b200.serving import args_key, estimate_bytes, radon_slices
from holotomocupy_b200.synthetic import workload_args


def test_equal_arguments_share_a_key():
    assert args_key(workload_args(128, 224, 4)) == args_key(workload_args(128, 224, 4))
    hash(args_key(workload_args(128, 224, 4)))


def test_any_differing_argument_changes_the_key():
    base = workload_args(128, 224, 4)
    key = args_key(base)
    assert args_key(workload_args(256, 448, 4)) != key
    assert args_key(workload_args(128, 224, 3)) != key
    for name, value in (("distance", np.array([3e-3, 4e-3, 5e-3, 7e-3])), ("rho", [1, 0.05, 0.03]),
                        ("mask", 0.8), ("lam_prbfit", 1e-3)):
        other = types.SimpleNamespace(**vars(base))
        setattr(other, name, value)
        assert args_key(other) != key, name
    # a theta array with one angle moved
    other = types.SimpleNamespace(**vars(base))
    other.theta = base.theta.copy()
    other.theta[5] += 1e-6
    assert args_key(other) != key


def test_estimate_grows_with_the_problem():
    small, large = estimate_bytes(workload_args(128, 224, 4)), estimate_bytes(workload_args(256, 448, 4))
    assert 0 < small < large
    # n^4 work, n^3-and-more memory: a 512^3 x 900 x 4 reconstruction needs tens of GB
    assert 40e9 < estimate_bytes(workload_args(512, 900, 4)) < 120e9


def test_estimate_counts_the_radon_workspace_slices():
    """Slices are interleaved by 4, 8 or 16 at every size; from 1024^2 on a short
    remainder runs in the room of the others (tests/test_gpu_tomo.py compares
    these numbers with the memory a Tomo takes)."""
    assert [radon_slices(256, nz) for nz in (1, 4, 5, 8, 9, 16, 17, 24, 33)] == [4, 4, 8, 8, 16, 16, 32, 32, 48]
    assert [radon_slices(2048, nz) for nz in (1, 9, 16, 17, 20, 21, 31, 36, 37)] == [4, 16, 16, 16, 16, 32, 32, 32, 48]
    a, b = workload_args(128, 224, 4), workload_args(128, 224, 4)
    a.nzobj, b.nzobj = 16, 17
    a.nobj = b.nobj = 512
    one = 512 * 512 * 8 * 3 + 224 * 512 * 8 * 7   # one more slice of the arrays
    assert estimate_bytes(b) - estimate_bytes(a) > 1.09 * (one + 16 * (6 * 512 * 512 + 224 * 512) * 8)
