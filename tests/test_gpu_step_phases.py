"""The entry points between and inside advection steps: the water removed at the
ground arrives with the call that removed it, a member of an FP64 batch is binned
after its step, and a particle pass takes the wind the grid holds at the call.

Tolerance: water removed is a sum of positive products, 1e-12 (the product's and
the reference's sums differ by their roundings only, some 1e-13 for the 300 SIPs
here)."""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _falling(seed=4, n_low=300):
    """A small state with SIPs just above the ground, falling."""
    from lacmopy_gb300 import synthetic
    st = synthetic.make_icmw_state(Nx=6, Nz=5, no_spcm=(6, 8), seed=seed, kernel_type="Long_Bott",
                                   r_tot=11E-3)
    rng = np.random.default_rng(seed)
    dx, dz = st["grid_steps"]
    sel = rng.permutation(st["xi"].size)[:n_low]
    st["pos"][1, sel] = rng.uniform(0.0, 1.5, n_low)
    st["cells"][1, sel] = np.floor(st["pos"][1, sel] / dz).astype(np.int64)
    st["rel_pos"][1, sel] = st["pos"][1, sel] / dz - st["cells"][1, sel]
    R = rng.uniform(100.0, 400.0, n_low)
    st["m_w"][sel] = 4.18879e3 * R ** 3
    st["xi"][sel] = rng.uniform(1e2, 1e4, n_low)
    st["vel"][1, sel] = -5.0
    return st


class Ledger:
    """water_removed against the SIPs that left since the last look."""

    def __init__(self, ds):
        self.ds = ds
        self.act = ds.cell.cpu().numpy() >= 0
        self.total = float(ds.water_removed.cpu()[0])

    def check(self, least):
        act = self.ds.cell.cpu().numpy() >= 0
        left = self.act & ~act
        self.act = act
        m_w, xi = self.ds.m_w.cpu().numpy(), self.ds.xi.cpu().numpy()
        self.total += math.fsum(m_w[left] * xi[left])
        assert np.count_nonzero(left) >= least
        np.testing.assert_allclose(self.ds.water_removed.cpu().numpy()[0], self.total, rtol=1e-12)


def _call(ds, name, *args):
    from lacmopy_gb300 import _lib
    from lacmopy_gb300.device import _ptr, _stream
    _lib.check(getattr(ds.lib, name)(ctypes.byref(ds.sips), ctypes.byref(ds.grid), *args,
                                     _ptr(ds.ws), ds.ws_bytes, _stream()), name)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_water_removed_by_the_particle_pass_alone(precision):
    from lacmopy_gb300 import DeviceState, _lib
    st = _falling()
    st["act_collisions"] = False
    ds = DeviceState(st, draws="philox", seed=3, precision=precision)
    water = Ledger(ds)
    prm = ctypes.byref(ds.params)
    for _ in range(2):
        _call(ds, "lacmo_particles_only", prm, 0.1, 0.1)
        _call(ds, "lacmo_bin")
        water.check(10)
    # whole steps of either precision afterwards neither lose nor repeat it
    for p in (_lib.PRECISION_MIXED, _lib.PRECISION_FP64):
        ds.params.precision = p
        ds.adv_step(1)
        water.check(0)


def test_water_removed_by_the_half_step_move():
    from lacmopy_gb300 import DeviceState
    ds = DeviceState(_falling(), draws="philox", seed=3)
    water = Ledger(ds)
    prm = ctypes.byref(ds.params)
    _call(ds, "lacmo_adv_step_begin", prm)
    water.check(10)
    _call(ds, "lacmo_adv_substep", prm, ds.params.dt_sub, 0)
    water.check(1)


def test_water_removed_by_a_batch_particle_pass():
    from lacmopy_gb300 import BatchState, _lib
    from lacmopy_gb300.device import _stream
    b = BatchState([_falling(4), _falling(5)], [3, 4], precision="fp64", draws="philox")
    water = [Ledger(m) for m in b.members]
    for _ in range(2):
        _lib.check(b.lib.lacmo_batch_particles_only(b.handle, ctypes.byref(b.params), _stream()),
                   "batch_particles_only")
        for w in water:
            w.check(10)
    b.adv_step(1)
    for w in water:
        w.check(0)


@pytest.mark.parametrize("graph", [False, True])
def test_members_of_an_fp64_batch_are_binned_after_a_step(graph):
    from lacmopy_gb300 import BatchState, DeviceState, _lib
    from lacmopy_gb300.device import _stream
    b = BatchState([_falling(4), _falling(5)], [3, 4], precision="fp64", draws="philox")
    b.adv_step(2, graph=graph)
    for m, seed in ((0, 4), (1, 5)):
        mb = b.members[m]
        ws, size = ctypes.c_void_p(), ctypes.c_size_t()
        _lib.check(b.lib.lacmo_batch_member_workspace(b.handle, m, ctypes.byref(ws),
                                                      ctypes.byref(size)), "member_workspace")
        _lib.check(b.lib.lacmo_update_grid_r_l(ctypes.byref(mb.sips), ctypes.byref(mb.grid), ws,
                                               size.value, _stream()), "update_grid_r_l")
        one = DeviceState(_falling(seed), draws="philox", seed=3 + m)
        one.adv_step(2)
        one.update_grid_r_l()
        r_l = one.snapshot()["grid_scalar_fields"][5]
        assert np.count_nonzero(r_l) == r_l.size
        assert np.array_equal(b.snapshot(m)["grid_scalar_fields"][5], r_l)


def _new_wind(ds, seed):
    """Another wind of the same size into the grid's own array."""
    v = ds.gvel.cpu().numpy()
    ds.gvel.copy_(ds.gvel.new_tensor(v[:, ::-1].copy() + 0.1 * seed))


@pytest.mark.parametrize("entry", ["particles_only", "substep", "batch"])
def test_wind_changed_before_a_particle_pass(entry):
    """Against a state that had the new wind from its start, bit for bit."""
    from lacmopy_gb300 import BatchState, DeviceState, _lib
    from lacmopy_gb300.device import _stream
    if entry == "batch":
        def make():
            return BatchState([_falling(4), _falling(5)], [3, 4], precision="fp64", draws="philox")

        def run(b):
            _lib.check(b.lib.lacmo_batch_particles_only(b.handle, ctypes.byref(b.params),
                                                        _stream()), "batch_particles_only")
        one, two = make(), make()
        for q, m in enumerate(two.members):
            _new_wind(m, q + 1)
        _lib.check(two.lib.lacmo_batch_prepare(two.handle, ctypes.byref(two.params), _stream()),
                   "batch_prepare")
        pairs = list(zip(one.members, two.members))
    else:
        def make():
            return DeviceState(_falling(), draws="philox", seed=3)

        def run(ds):
            prm = ctypes.byref(ds.params)
            if entry == "substep":
                _call(ds, "lacmo_adv_substep", prm, 0.1, 0)
            else:
                _call(ds, "lacmo_particles_only", prm, 0.1, 0.1)
        one, two = make(), make()
        _new_wind(two, 1)
        two.prepare()
        pairs = [(one, two)]
        if entry == "substep":
            for ds in (one, two):
                _call(ds, "lacmo_adv_step_begin", ctypes.byref(ds.params))
    for q, (m, _) in enumerate(pairs):
        _new_wind(m, q + 1)
    before = pairs[0][0].snapshot()["vel"]
    run(one)
    run(two)
    for m, ref in pairs:
        a, b = m.snapshot(), ref.snapshot()
        for k in ("vel", "pos", "m_w", "rel_pos", "cells"):
            assert np.array_equal(a[k], b[k]), k
    assert np.abs(pairs[0][0].snapshot()["vel"] - before).max() > 0.05
