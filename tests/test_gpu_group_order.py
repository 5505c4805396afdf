"""The group kernels of a class give the same integrals to the last bits: all sum a target over its primitives
in their order and run one HRR recursion. On the 64-molecule l <= 3 workload an
element of the HRR is a difference of terms many orders larger, so that another order of either shows in K:
the HRR as a dense product moved single elements by 7e-10 of K's root mean square on this sample, and by 4e-8 on
sixteen times as many set quartets; partial sums of the primitives in four lanes moved elements of a
12-molecule cluster's K by 1.3e-10."""
import ctypes

import numpy as np
import pytest

from libgint_b200.workload import Api, Session, Workload

# What may differ is the order of K's own additions: up to N ~ 1e4 of them an element, each rounding by up to
# half a unit of the partial sum, which stays within some 30 root mean squares of K: sqrt(N) 1.1e-16 30 = 3e-13.
ORDER_TOL = 1e-12


PERIODIC64 = dict(name="periodic_l3", setq_stride=65536)
PERIODIC2 = dict(basis=3, n_mol=2, box_ang=5.0, periodic=1, n_img_1d=3, n_occ=16, setq_stride=61)
PERIODIC64_ROWS = dict(name="periodic_l3", setq_stride=16384)
CLUSTER12 = dict(basis=3, n_mol=12, box_ang=17.3, periodic=0, n_img_1d=1, n_occ=60, setq_stride=512)


def _largest_difference(engine_so, sample, classes):
    """Of K with the group kernel choice 0 and 1 for the given classes, over K's element or root mean square."""
    from libgint_b200.capi import load_engine
    lib, D = load_engine(), ctypes.POINTER(ctypes.c_double)
    sample = dict(sample)
    wl = Workload(sample.pop("name", None), **sample)
    s = Session(Api(engine_so), wl, max_mem_mb=40000)
    h = ctypes.c_void_p(s.h)
    lib.libgint_record(h, 2)
    s.build_K()
    lib.libgint_record(h, 0)
    P, K = wl.Pflat, []
    for variant in (0, 1):
        tune = (ctypes.c_int * 512)()
        for c in range(256):
            if classes((c >> 6) + (c >> 4 & 3) + (c >> 2 & 3) + (c & 3)):
                tune[2 * c + 1] = variant
        lib.libgint_set_tuning(h, tune)
        lib.libgint_set_P(h, P.ctypes.data_as(D), P.size)
        assert lib.libgint_replay(h) > 0
        K.append(np.zeros(P.size))
        lib.libgint_get_K(h, K[-1].ctypes.data_as(D))
    assert lib.libgint_last_error(h) == 0, lib.libgint_error_string(h)
    s.close()
    rms = np.sqrt(np.mean(K[1] ** 2))
    assert rms > 0
    return (np.abs(K[0] - K[1]) / np.maximum(np.abs(K[1]), rms)).max()


@pytest.mark.gpu
@pytest.mark.parametrize("sample", [PERIODIC64, PERIODIC2])
def test_one_block_per_group_equals_one_warp_per_row(engine_so, sample):
    assert _largest_difference(engine_so, sample, lambda L: L >= 4) <= ORDER_TOL


@pytest.mark.gpu
@pytest.mark.parametrize("sample", [CLUSTER12, PERIODIC64_ROWS])
def test_lanes_of_a_row_equal_one_warp_per_row(engine_so, sample):
    assert _largest_difference(engine_so, sample, lambda L: L <= 3) <= ORDER_TOL
