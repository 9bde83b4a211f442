"""Drop-in replacements for collision/all_or_nothing.py and the box-model
collision driver, running the all-or-nothing step on the GPU.

Same names, arguments and in-place semantics as the reference; keyword-only
``draws`` selects the uniform draws ("numpy": NumPy's global generator with
the reference's count and order, "philox": device Philox with ``seed`` and
``step``, or an explicit array).  Collision decisions and multiplicity/mass
updates are bit-exact with the reference given the same draws (see the
kernel file k_collision.cu for how).
"""
import ctypes
import math

import numpy as np
import torch

from . import _lib
from .device import DeviceState, _ptr, _stream, to_device
from .integration import _minimal_state, _writeback


def _box_draws(draws, n):
    need = n * (n - 1) // 2
    if isinstance(draws, str):
        if draws == "numpy":
            return to_device(np.random.rand(need) if need else np.zeros(1))
        if draws == "philox":
            return None
        raise ValueError(f"unknown draw source {draws!r}")
    t = to_device(draws)
    if t.numel() < need:
        raise ValueError(f"need {need} draws, got {t.numel()}")
    return t


def collision_step_Golovin_np(xis, masses, dt_over_dV, no_cols, *, draws="numpy", seed=0,
                              step=0):
    """collision/all_or_nothing.py:109-185 (Golovin kernel, box model)."""
    lib = _lib.load()
    n = int(np.shape(xis)[0])
    x, m, nc = to_device(xis), to_device(masses), to_device(no_cols, torch.int64)
    r = _box_draws(draws, n)
    _lib.check(lib.lacmo_collision_step_golovin(_ptr(x), _ptr(m), n, float(dt_over_dV), _ptr(nc),
                                                _ptr(r), int(seed), int(step), _stream()),
               "collision_step_golovin")
    for dst, t in ((xis, x), (masses, m), (no_cols, nc)):
        _writeback(dst, t)


def collision_step_kernel_grid_m_np(xis, masses, dt_over_dV, kernel_grid, no_kernel_bins,
                                    m_kernel_low_log, bin_factor_m_log, no_cols, *,
                                    draws="numpy", seed=0, step=0):
    """collision/all_or_nothing.py:392-491 (kernel K(m1, m2) on a logarithmic
    mass grid, box model)."""
    lib = _lib.load()
    n = int(np.shape(xis)[0])
    x, m, nc = to_device(xis), to_device(masses), to_device(no_cols, torch.int64)
    K = to_device(kernel_grid)
    r = _box_draws(draws, n)
    _lib.check(lib.lacmo_collision_step_kernel_grid_m(
        _ptr(x), _ptr(m), n, float(dt_over_dV), _ptr(K), int(no_kernel_bins),
        float(m_kernel_low_log), float(bin_factor_m_log), _ptr(nc), _ptr(r), int(seed), int(step),
        _stream()), "collision_step_kernel_grid_m")
    for dst, t in ((xis, x), (masses, m), (no_cols, nc)):
        _writeback(dst, t)


def collision_step_Ecol_grid_R_np(xis, masses, radii, vel, mass_densities, dt_over_dV,
                                  E_col_grid, no_kernel_bins, R_kernel_low_log, bin_factor_R_log,
                                  no_cols, *, draws="numpy", seed=0, step=0):
    """collision/all_or_nothing.py:269-390 (E_col(R1,R2) table, box model)."""
    lib = _lib.load()
    n = int(np.shape(xis)[0])
    x, m, R = to_device(xis), to_device(masses), to_device(radii)
    v, rho, E = to_device(vel), to_device(mass_densities), to_device(E_col_grid)
    nc = to_device(no_cols, torch.int64)
    r = _box_draws(draws, n)
    _lib.check(lib.lacmo_collision_step_ecol_grid_r_box(
        _ptr(x), _ptr(m), _ptr(R), _ptr(v), _ptr(rho), n, float(dt_over_dV), _ptr(E),
        int(no_kernel_bins), float(R_kernel_low_log), float(bin_factor_R_log), _ptr(nc), _ptr(r),
        int(seed), int(step), _stream()), "collision_step_ecol_grid_r_box")
    for dst, t in ((xis, x), (masses, m), (radii, R), (no_cols, nc)):
        _writeback(dst, t)


def update_velocity_Beard(vel, R):
    """collision/kernel.py:193-210 (Beard terminal velocity), in place."""
    lib = _lib.load()
    v, r = to_device(vel), to_device(R)
    _lib.check(lib.lacmo_update_velocity_beard(_ptr(v), _ptr(r), v.numel(), _stream()),
               "update_velocity_beard")
    _writeback(vel, v)


def collision_step_Ecol_grid_R_all_cells_2D_multicomp_np(
        xis, m_w, m_s, vel, grid_temperature, cells, no_cells, dt_over_dV, E_col_grid,
        no_kernel_bins, R_kernel_low_log, bin_factor_R_log, no_cols, solute_type, *,
        draws="numpy", seed=0, col_step=None):
    """collision/all_or_nothing.py:754-846: one AON step in every grid cell.

    With ``draws="philox"`` or ``"thinned"`` consecutive calls with the same
    ``seed`` continue one stream of draws (lacmopy_gb300.integration);
    ``col_step`` pins the collision-step counter."""
    Nx, Nz = int(no_cells[0]), int(no_cells[1])
    n = int(np.shape(xis)[0])
    cells_np = np.asarray(cells)
    act = (cells_np[1] >= 0) & (cells_np[1] < Nz) & (cells_np[0] >= 0) & (cells_np[0] < Nx)
    gsf = np.zeros((10, Nx, Nz))
    gsf[0] = np.asarray(grid_temperature)
    st = _minimal_state(Nx, Nz, n, m_w=m_w, xi=xis, cells=np.where(act, cells_np, 0),
                        active_ids=act, gsf=gsf, m_s=m_s, vel=vel)
    st.update(dt_col_over_dV=dt_over_dV, E_col_grid=E_col_grid, no_kernel_bins=no_kernel_bins,
              R_kernel_low_log=R_kernel_low_log, bin_factor_R_log=bin_factor_R_log,
              solute_type=solute_type, no_cols=no_cols)
    mode = draws if isinstance(draws, str) else "philox"
    ds = DeviceState(st, draws=mode, seed=seed)
    philox = isinstance(draws, str) and draws in ("philox", "thinned")
    if philox:
        ds.continue_philox(col_step)
    ds.collision_step(None if isinstance(draws, str) else draws)
    if philox:
        ds.record_philox()
    torch.cuda.current_stream().synchronize()
    for dst, t in ((xis, ds.xi), (m_w, ds.m_w), (m_s, ds.m_s), (no_cols, ds.no_cols)):
        _writeback(dst, t)


def compute_radius_and_kernel_index(masses, mass_densities, R_kernel_low_log, bin_factor_R_log,
                                    no_kernel_bins):
    """Collision-path radius (microphysics.py:83-100) and kernel bin
    (collision/all_or_nothing.py:35-67), correctly rounded; returns (R, bin)."""
    lib = _lib.load()
    m, rho = to_device(masses), to_device(mass_densities)
    R = torch.empty_like(m)
    k = torch.empty(m.numel(), dtype=torch.int64, device=m.device)
    _lib.check(lib.lacmo_radius_and_bin(_ptr(m), _ptr(rho), m.numel(), float(R_kernel_low_log),
                                        float(bin_factor_R_log), int(no_kernel_bins), _ptr(R),
                                        _ptr(k), _stream()), "radius_and_bin")
    return R.cpu().numpy(), k.cpu().numpy()


class _Packed:
    """NumPy arrays (or tensors) side by side in one device buffer, filled by one
    copy from pinned memory.  Item 2 is of 64-bit integers, the others of
    doubles."""

    def __init__(self, arrays):
        self.size = [a.numel() if isinstance(a, torch.Tensor) else int(np.size(a)) for a in arrays]
        # 16-byte alignment of every item
        self.at = np.concatenate(([0], np.cumsum([(k + 1) // 2 * 2 for k in self.size]))).tolist()
        self.pin = torch.empty(self.at[-1], dtype=torch.float64, pin_memory=True)
        buf = torch.empty(self.at[-1], dtype=torch.float64, device="cuda")
        self.buf = buf
        self.dev = [buf[o:o + k] for o, k in zip(self.at, self.size)]
        self._np = self.pin.numpy()
        tensors = []
        for q, a in enumerate(arrays):
            dst = self.host(q)
            if isinstance(a, torch.Tensor):
                tensors.append((self.dev[q].view(torch.int64) if q == 2 else self.dev[q], a))
            elif q == 2:
                dst[:] = np.asarray(a).astype(np.int64, copy=False).reshape(-1)
            else:
                dst[:] = np.asarray(a).reshape(-1)
        buf.copy_(self.pin, non_blocking=True)
        for d, a in tensors:
            d.copy_(a.reshape(-1))

    def host(self, q):
        """Item q of the pinned copy."""
        v = self._np[self.at[q]:self.at[q] + self.size[q]]
        return v.view(np.int64) if q == 2 else v

    def fetch(self, items):
        """The first ``items`` items back to the pinned copy."""
        self.pin[:self.at[items]].copy_(self.buf[:self.at[items]], non_blocking=True)
        torch.cuda.current_stream().synchronize()

    def put_back(self, q, dst):
        if isinstance(dst, torch.Tensor):
            dst.copy_((self.dev[q].view(torch.int64) if q == 2 else self.dev[q]).reshape(dst.shape))
        else:
            np.copyto(dst, self.host(q).reshape(np.shape(dst)))


class _Snapshots:
    """Multiplicities and masses between steps, kept on the device and copied to
    the output arrays a few megabytes at a time."""

    def __init__(self, buf, n, rows, xis, masses):
        self.src, self.n, self.out = buf, n, (xis, masses)
        self.rows = max(1, min(rows, (1 << 20) // max(1, n)))
        self.dev = self.pin = None
        self.first = self.k = 0

    def take(self, row):
        if self.dev is None:
            self.dev = torch.empty((self.rows, 2, self.n), dtype=torch.float64, device="cuda")
            self.pin = torch.empty(self.dev.shape, dtype=torch.float64, pin_memory=True)
        if self.k == 0:
            self.first = row
        self.dev[self.k, 0].copy_(self.src.dev[0])
        self.dev[self.k, 1].copy_(self.src.dev[1])
        self.k += 1
        if self.k == self.rows:
            self.flush()

    def flush(self):
        if self.k:
            self.pin[:self.k].copy_(self.dev[:self.k], non_blocking=True)
            torch.cuda.current_stream().synchronize()
            p = self.pin.numpy()
            for out, c in zip(self.out, (0, 1)):
                out[self.first:self.first + self.k] = p[:self.k, c]
            self.k = 0


def simulate_collisions(SIP_quantities, kernel_quantities, kernel_name, kernel_method, dV, dt,
                        t_end, dt_save, no_cols, seed, save_dir=None, *, draws="numpy"):
    """Box-model time loop (collision/box_model.py:44-205) on the GPU.

    The state and its snapshots stay on the device between steps; the saved
    (xis, masses) snapshots and save times are returned (and written to ``save_dir`` with the
    reference's file names when it is given).  ``draws="numpy"`` seeds NumPy's
    global generator with ``seed`` like the reference; ``"philox"`` uses the
    device generator keyed by ``seed``.
    """
    lib = _lib.load()
    if draws == "numpy":
        np.random.seed(seed)
    # box_model.py:135-145 picks the step by kernel_name first, then loops by
    # kernel_method (:160-194); the Golovin kernel runs with any method but the
    # two tabulated ones
    if kernel_name == "Golovin" and kernel_method not in ("Ecol_grid_R", "kernel_grid_m"):
        method = "golovin"
        xis, masses = SIP_quantities
    elif kernel_method == "Ecol_grid_R":
        method = "ecol"
        xis, masses, radii, vel, mass_densities = SIP_quantities
        E_col_grid, no_kernel_bins, R_kernel_low_log, bin_factor_R_log = kernel_quantities
    elif kernel_method == "kernel_grid_m":
        method = "kgrid"
        xis, masses = SIP_quantities
        kernel_grid, no_kernel_bins, m_kernel_low_log, bin_factor_m_log = kernel_quantities
    else:
        raise ValueError(f"kernel_name {kernel_name!r} with kernel_method {kernel_method!r}")
    n = int(np.shape(xis)[0])
    no_steps = int(math.ceil(t_end / dt))
    no_saves = int(t_end / dt_save - 0.001) + 2
    dn_save = int(math.ceil(dt_save / dt))
    dt_over_dV = dt / dV
    # One copy in and one out: the arrays lie side by side, the ones that come
    # back first (separate copies of pageable memory, each waiting for the one
    # before, took 0.45 to 0.7 ms of a call)
    ins = [xis, masses, no_cols]
    if method == "ecol":
        ins += [radii, vel, mass_densities, E_col_grid]
    elif method == "kgrid":
        ins.append(kernel_grid)
    buf = _Packed(ins)
    x, m, nc = buf.dev[0], buf.dev[1], buf.dev[2].view(torch.int64)
    if method == "ecol":
        R, v, rho, E = buf.dev[3:]
    elif method == "kgrid":
        K = buf.dev[3]
    if x.numel() != n or any(t.numel() < n for t in ((m, R, v, rho) if method == "ecol" else (m,))):
        raise ValueError("SIP quantities of different lengths")
    xis_vs_time = np.zeros((no_saves, n))
    masses_vs_time = np.zeros((no_saves, n))
    save_times = np.zeros(no_saves)
    save_n = 0
    snaps = _Snapshots(buf, n, no_saves, xis_vs_time, masses_vs_time)
    s = _stream()
    for step_n in range(no_steps):
        if step_n % dn_save == 0:
            if step_n == 0 and not any(isinstance(a, torch.Tensor) for a in (xis, masses)):
                xis_vs_time[0], masses_vs_time[0] = buf.host(0), buf.host(1)
            else:
                snaps.take(save_n)
            save_times[save_n] = step_n * dt
            save_n += 1
        r = _box_draws(draws, n)
        if method == "golovin":
            _lib.check(lib.lacmo_collision_step_golovin(_ptr(x), _ptr(m), n, dt_over_dV, _ptr(nc),
                                                        _ptr(r), int(seed), step_n, s), "golovin")
        elif method == "kgrid":
            # no velocity update: the kernel table holds the whole K(m1, m2)
            _lib.check(lib.lacmo_collision_step_kernel_grid_m(
                _ptr(x), _ptr(m), n, dt_over_dV, _ptr(K), int(no_kernel_bins),
                float(m_kernel_low_log), float(bin_factor_m_log), _ptr(nc), _ptr(r), int(seed),
                step_n, s), "kernel_grid_m")
        else:
            _lib.check(lib.lacmo_collision_step_ecol_grid_r_box(
                _ptr(x), _ptr(m), _ptr(R), _ptr(v), _ptr(rho), n, dt_over_dV, _ptr(E),
                int(no_kernel_bins), float(R_kernel_low_log), float(bin_factor_R_log), _ptr(nc),
                _ptr(r), int(seed), step_n, s), "ecol_box")
            _lib.check(lib.lacmo_update_velocity_beard(_ptr(v), _ptr(R), n, s), "beard")
    snaps.flush()
    buf.fetch(5 if method == "ecol" else 3)
    xis_vs_time[save_n], masses_vs_time[save_n] = buf.host(0), buf.host(1)
    save_times[save_n] = no_steps * dt
    buf.put_back(0, xis)
    buf.put_back(1, masses)
    buf.put_back(2, no_cols)
    if method == "ecol":
        buf.put_back(3, radii)
        buf.put_back(4, vel)
    if save_dir is not None:
        np.save(save_dir + f"xis_vs_time_{seed}", xis_vs_time)
        np.save(save_dir + f"masses_vs_time_{seed}", masses_vs_time)
        np.save(save_dir + f"save_times_{seed}", save_times)
    return xis_vs_time, masses_vs_time, save_times
