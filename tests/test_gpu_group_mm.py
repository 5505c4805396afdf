"""The block-per-group kernel (classes with la+lb+lc+ld >= 4) at the edges of its tiles: one
contraction row per group, nine, eighty-one (one more than a tile of eight, and many tiles), shells of
more primitives than one round of coefficients, one image pair and several to a group, against the oracle;
and two spin densities, against one after the other and, with f shells, against the oracle."""
import ctypes

import numpy as np
import pytest

from libgint_b200.workload import Api, Session, Workload
from test_gpu_parity import TOL, _compare, assert_fp64_parity

CLUSTER = dict(basis=3, periodic=0, n_img_1d=1, box_ang=12.0, n_occ=6)
CASES = {"one_row": dict(CLUSTER, n_mol=2, max_prm=1, max_ncontr=1, setq_stride=3),
         "many_rows_and_primitives": dict(CLUSTER, n_mol=1, max_prm=16, max_ncontr=4, setq_stride=5),
         "nine_rows": dict(CLUSTER, n_mol=2, max_prm=8, max_ncontr=3, setq_stride=97),
         "image_pairs": dict(basis=3, periodic=1, n_mol=1, box_ang=5.0, n_img_1d=3, n_occ=6, max_prm=3,
                             max_ncontr=2, setq_stride=11)}


@pytest.mark.gpu
@pytest.mark.parametrize("name", CASES)
def test_group_products_vs_oracle(engine_so, oracle_path, name):
    _compare(engine_so, oracle_path, Workload(None, **CASES[name]))


@pytest.mark.gpu
def test_two_spins_equal_one_at_a_time(engine_so):
    """The same terms in another order of atomic additions: within TOL of max|K|."""
    from libgint_b200.capi import load_engine
    lib, D = load_engine(), ctypes.POINTER(ctypes.c_double)
    wl = Workload("small_l2")
    s = Session(Api(engine_so), wl)
    h = ctypes.c_void_p(s.h)
    lib.libgint_record(h, 2)
    s.build_K()
    lib.libgint_record(h, 0)
    Pa = wl.Pflat
    Pb = np.random.default_rng(3).standard_normal(Pa.size) * np.abs(Pa).max()
    one = []
    for P in (Pa, Pb):
        lib.libgint_set_P(h, P.ctypes.data_as(D), P.size)
        assert lib.libgint_replay(h) > 0
        one.append(np.zeros(P.size))
        lib.libgint_get_K(h, one[-1].ctypes.data_as(D))
    two = [np.zeros(Pa.size), np.zeros(Pa.size)]
    lib.libgint_set_P_polarized(h, Pa.ctypes.data_as(D), Pb.ctypes.data_as(D), Pa.size)
    assert lib.libgint_replay(h) > 0
    lib.libgint_get_K_polarized(h, two[0].ctypes.data_as(D), two[1].ctypes.data_as(D))
    assert lib.libgint_last_error(h) == 0, lib.libgint_error_string(h)
    for a, b in zip(one, two):
        assert np.abs(a).max() > 0 and np.abs(a - b).max() <= TOL * np.abs(a).max()
    s.close()


@pytest.mark.gpu
def test_two_spins_with_f_shells_vs_oracle(engine_so, oracle_path):
    """The tile's height and its shared memory depend on the class, the room for P's elements on the spins; in
    (ff|ff) a tile is one row and a row's K update takes more rounds than one."""
    from libgint_b200.capi import load_engine
    lib, D = load_engine(), ctypes.POINTER(ctypes.c_double)
    wl = Workload(None, **dict(CLUSTER, n_mol=1, max_prm=4, max_ncontr=2))
    ls = wl.sets()[:, 1][wl.setq()[:, :4]]
    classes = set((ls @ np.array([64, 16, 4, 1])).tolist())
    assert {255, 127, 63, 170} <= classes          # (ff|ff), (pf|ff), (sf|ff), (dd|dd)
    s = Session(Api(engine_so), wl)
    h = ctypes.c_void_p(s.h)
    lib.libgint_record(h, 2)
    s.build_K()
    lib.libgint_record(h, 0)
    Pb = np.random.default_rng(3).standard_normal(wl.Pflat.size) * np.abs(wl.Pflat).max()
    K = [np.zeros(Pb.size), np.zeros(Pb.size)]
    lib.libgint_set_P_polarized(h, wl.Pflat.ctypes.data_as(D), Pb.ctypes.data_as(D), Pb.size)
    assert lib.libgint_replay(h) > 0
    lib.libgint_get_K_polarized(h, K[0].ctypes.data_as(D), K[1].ctypes.data_as(D))
    assert lib.libgint_last_error(h) == 0, lib.libgint_error_string(h)
    s.close()
    api = Api(oracle_path)
    for Ke, P in zip(K, (wl.Pflat, Pb)):
        ref = []
        for magnitudes in (0, 1):
            o = Session(api, wl)
            api.symbol("oracle_set_absmode", None, [ctypes.c_void_p, ctypes.c_int])(o.h, magnitudes)
            ref.append(o.build_K(P)[0])
            o.close()
        assert_fp64_parity(Ke, ref[0], ref[1], wl)
