"""The order of the sweep features' sums: element e to sum e mod 256, the sums in a
binary tree (128 apart first), alike for every population.  The masses are chosen
such that an order shows in the float32 result: one is 2^60, another half a unit in the
last place of that (a tie, which rounds down), and a few are a half or a quarter of
the double's unit there and are lost when they meet the large sum one by one."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


def _ordered_sum(m):
    s = np.zeros(256)
    for e, x in enumerate(m):
        s[e % 256] += x
    while len(s) > 1:
        s = s[:len(s) // 2] + s[len(s) // 2:]
    return np.float32(s[0])


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("n", [3, 31, 290, 1000, 4999])
def test_sums_have_one_order_for_every_population(n, dtype):
    from mbd_icenav_b200 import _abi
    lib = _abi.load_library()
    code, dt = (_abi.DEM_F32, torch.float32) if dtype == "f32" else (_abi.DEM_F64, torch.float64)
    pos = torch.zeros((n, 2), dtype=dt, device=DEV)  # every element is hit at the first pose
    radii = torch.ones(n, dtype=dt, device=DEV)

    def features(mass, Q):
        eta0, hist = torch.zeros((Q, 3), dtype=dt, device=DEV), torch.zeros((2, Q, 3), dtype=dt, device=DEV)
        out = torch.full((Q, 8), float("nan"), device=DEV)
        assert lib.dem_rollout_sweep_features(code, Q, 2, eta0.data_ptr(), hist.data_ptr(), n, pos.data_ptr(),
                                              radii.data_ptr(), mass.data_ptr(), 0, None, None, 30.0, 6.0, 0.5,
                                              out.data_ptr(), None) == _abi.DEM_OK
        return out.cpu().numpy()
    tops = set()
    for seed in range(16):
        rng = np.random.default_rng(seed)
        m = np.zeros(n)
        # one lane's elements of every warp, as far as there are enough of them
        idx = 32 * rng.permutation(n // 32) + rng.integers(0, 2) if n >= 96 else rng.permutation(n)
        few = min(len(idx) - 2, 5)
        m[idx[0]], m[idx[1]] = 2.0 ** 60, 2.0 ** 36
        m[idx[2:2 + few]] = 2.0 ** rng.integers(5, 8, few)
        want = _ordered_sum(m)
        tops.add(float(want))
        mass = torch.as_tensor(m, dtype=dt, device=DEV)
        for Q in (1, 2371):
            got = features(mass, Q)
            assert (got[:, 0] == n).all()
            assert (got[:, 1] == want).all() and (got[:, 4] == want).all(), (seed, Q)
    assert len(tops) == 2 or n < 96  # both roundings occur
