"""Path costs and sweep features of different sizes from several threads at a time: no
call's shared memory depends on what another one has asked for."""
import ctypes as C
import threading

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)
CALLS = 1500


def _run_together(makes):
    """Each entry's calls in a thread and stream of its own; the first bad status of each."""
    bad = [None] * len(makes)

    def work(i):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            call = makes[i](stream.cuda_stream)
            for _ in range(CALLS):
                rc = call()
                if rc:
                    bad[i] = rc
                    break
        stream.synchronize()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(makes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return bad


def test_path_costs_of_several_horizons_at_a_time():
    from mbd_icenav_b200 import _abi
    lib = _abi.load_library()
    P = _abi.DemRolloutCostParams(x_origin=0.0, y_origin=0.0, resolution=1.0, rows=4, cols=4, oob_penalty=1.0,
                                  ship_length=0.0, ship_beam=0.0, goal_x=0.0, goal_y=0.0)
    P.action_scale[:] = [1.0, 1.0, 1.0]
    grid = torch.zeros((4, 4), device=DEV)

    def make(H):
        eta0, hist = torch.zeros((1, 3), device=DEV), torch.zeros((H, 1, 3), device=DEV)
        out = torch.zeros((1, 5), dtype=torch.float64, device=DEV)
        return lambda stream: lambda: lib.dem_rollout_costs(
            _abi.DEM_F32, 1, H, None, eta0.data_ptr(), hist.data_ptr(), None, grid.data_ptr(), C.byref(P), None, None,
            None, out.data_ptr(), stream)
    makes = [make(H) for H in (2000, 1400, 2000, 1400)]
    torch.cuda.synchronize()
    assert _run_together(makes) == [None] * 4


def test_sweep_features_of_several_windows_at_a_time():
    from mbd_icenav_b200 import _abi
    lib = _abi.load_library()

    def make(n):
        eta0, hist = torch.zeros((1, 3), device=DEV), torch.zeros((4, 1, 3), device=DEV)
        pos = torch.full((n, 2), 1e4, device=DEV)
        r, m = torch.ones(n, device=DEV), torch.ones(n, device=DEV)
        out = torch.zeros((1, 8), device=DEV)
        return lambda stream: lambda: lib.dem_rollout_sweep_features(
            _abi.DEM_F32, 1, 4, eta0.data_ptr(), hist.data_ptr(), n, pos.data_ptr(), r.data_ptr(), m.data_ptr(), 0, None,
            None, 30.0, 6.0, 0.5, out.data_ptr(), stream)
    makes = [make(n) for n in (65536, 50000, 65536, 50000)]
    torch.cuda.synchronize()
    assert _run_together(makes) == [None] * 4
