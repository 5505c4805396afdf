"""A replay of small segments uses sixteen worker streams where the device has room for their buffers of
image-summed targets, and otherwise six, as a replay of large segments does: it does not fail for want of
the larger buffer."""
import ctypes

import numpy as np
import pytest

from libgint_b200.workload import Api, Session, Workload

CLUSTER = dict(basis=3, n_mol=12, box_ang=17.3, periodic=0, n_img_1d=1, n_occ=60, setq_stride=32)
TOL = 1e-12   # of max|K|: the same terms in another order of atomic additions


@pytest.mark.gpu
def test_replay_where_the_larger_buffer_does_not_fit(engine_so):
    import torch
    from libgint_b200.capi import load_engine
    lib, D = load_engine(), ctypes.POINTER(ctypes.c_double)
    wl = Workload(None, **CLUSTER)
    torch.cuda.empty_cache()

    def session():
        s = Session(Api(engine_so), wl, max_mem_mb=40000)
        h = ctypes.c_void_p(s.h)
        lib.libgint_record(h, 2)
        s.build_K()
        lib.libgint_record(h, 0)
        lib.libgint_set_P(h, wl.Pflat.ctypes.data_as(D), wl.Pflat.size)
        return s, h

    def replay(h):
        lib.libgint_set_P(h, wl.Pflat.ctypes.data_as(D), wl.Pflat.size)
        assert lib.libgint_replay(h) > 0, lib.libgint_error_string(h)
        K = np.zeros(wl.Pflat.size)
        lib.libgint_get_K(h, K.ctypes.data_as(D))
        assert lib.libgint_last_error(h) == 0, lib.libgint_error_string(h)
        return K

    s, h = session()
    free = torch.cuda.mem_get_info()[0]
    K0 = replay(h)
    took = free - torch.cuda.mem_get_info()[0]     # the buffer for all streams, and the graph
    s.close()
    s, h = session()
    free = torch.cuda.mem_get_info()[0]
    print(f"buffer {took / 2**20:.0f} MiB")
    assert took >= 128 << 20
    fill = torch.empty(free - int(0.85 * took), dtype=torch.uint8, device="cuda")
    for _ in range(2):                             # the second time the smaller buffer is there
        K = replay(h)
        assert np.abs(K - K0).max() <= TOL * np.abs(K0).max()
    del fill
    torch.cuda.empty_cache()
    s.close()
