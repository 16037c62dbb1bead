"""The frames in which every neighbour list is rebuilt (a handle's first, or one from
another state), with no, few and many active elements on the 12k-element field."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


@pytest.fixture(scope="module")
def scene():
    from mbd_icenav_b200 import rollouts, scene
    from mbd_icenav_b200.sim import build_sim_context
    from mbd_icenav_b200.state import build_initial_ice_state, build_initial_ship_state
    f = scene.make_medium_field(seed=2, n_frames=4)
    eta0 = rollouts.ice_edge_pose(f, gap=30.0)  # out of reach: what is active is chosen below

    def make():
        ctx = build_sim_context(f.polygons, f.centroids, f.bonds, eta0[:2], f.ship_length, f.ship_beam, 4, f.dt,
                                (0.0, 0.0), f.thicknesses, f.ship_props, parent_ids=f.parent_ids, verbose=False,
                                n_ice_steps=f.n_ice_steps, hull_local=f.hull_local, dilation=0.05,
                                dtype=torch.float32, device="cuda")
        ice = build_initial_ice_state(f.n, f.centroids, len(f.bonds), ctx.static.initial_floe_of.cpu().numpy(),
                                      dtype=torch.float32, device="cuda")
        ship = build_initial_ship_state(eta0[:2], float(eta0[2]), dtype=torch.float32, device="cuda")
        return ctx.frame_step, ice, ship
    rows = torch.as_tensor(np.tile(np.concatenate([eta0, eta0]), (3, 1)), dtype=torch.float32, device=DEV)
    return f.n, make, rows, torch.zeros((3, f.n, 2), dtype=torch.float32, device=DEV)


def test_lists_stand_after_the_first_frame_without_an_active_element(scene):
    n, make, rows, water = scene
    fs, ice, ship = make()
    ice, ship, _ = fs.scan_segment(ice, ship, rows[:1], water[:1])
    first = fs.info()
    assert first["rebuilt_lists_total"] == n and first["escaped_total"] == n
    fs.scan_segment(ice, ship, rows[1:], water[1:])
    later = fs.info()
    fs.close()
    assert not ice.elem_active.any()
    assert later["rebuilt_lists_total"] == n and later["escaped_total"] == n


# few; one below and at the count whose CTAs (four elements each) have 128 lists each; all
@pytest.mark.parametrize("active", [1, 4, "below", "at", "all"])
def test_first_frames_do_not_depend_on_the_split(scene, active):
    from mbd_icenav_b200 import _abi
    n, make, rows, water = scene
    at = 4 * -(-n // 128) - 3
    active = {"below": at - 1, "at": at, "all": n}.get(active, active)
    rng = np.random.default_rng(active)
    on = torch.as_tensor(rng.permutation(n) < active, device=DEV)
    vel = torch.as_tensor(rng.normal(0, 0.5, (n, 2)), dtype=torch.float32, device=DEV) * on[:, None]
    runs = []
    for split in (_abi.DEM_SPLIT_AUTO, _abi.DEM_SPLIT_THREAD):
        fs, ice, ship = make()
        fs.set_work_split(split, 0)
        ice = ice._replace(elem_active=on, velocities=vel)
        out = []
        for shift in (0.0, 40.0):  # the second call is from another state of the same handle
            st, sh, h = fs.scan_segment(ice._replace(positions=ice.positions + shift), ship, rows, water)
            out += list(st) + list(sh) + [x for x in h if x is not None]
        assert fs.info()["rebuilt_lists_total"] >= 2 * n
        fs.close()
        runs.append(out)
    for a, b in zip(*runs):
        assert torch.equal(a, b)
