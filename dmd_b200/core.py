"""SimulationConfig and Engine -- the drop-in for the reference's pybind module
``_dmd_core`` (python/dmd/core.cpp:97-430).

``SimulationConfig`` keeps the same attribute names, defaults
(src/sim/simulation_config.h:27-84) and numpy-array properties as the pybind
class.  ``Engine`` keeps the EngineWrapper surface (run, run_n, positions,
velocities, forces, potential_energy, current_step, current_time, box_size,
n_atoms; python/dmd/core.cpp:417-428) but holds all state on the GPU: run_n(k)
is ONE call into the C ABI that advances k steps on the device, and the
getters copy from device memory.

Backend options are keyword arguments (or DMD_PRECISION / DMD_PROFILE /
DMD_SKIN / DMD_DEVICE environment variables) because the strict config.json
schema admits no extra keys.
"""
from __future__ import annotations

import ctypes as C
import math
import os

import numpy as np

from . import _capi


class ThermostatConfig:
    """src/sim/simulation_config.h:11-16"""

    def __init__(self):
        self.type = "none"
        self.temperature = 300.0
        self.tau = 0.1
        self.frequency = 10.0


class BarostatConfig:
    """src/sim/simulation_config.h:18-23"""

    def __init__(self):
        self.type = "none"
        self.pressure = 1.0
        self.tau = 1.0
        self.compressibility = 4.5e-5


def _f64(a):
    return np.ascontiguousarray(np.asarray(a, dtype=np.float64).ravel())


def _i32(a):
    return np.ascontiguousarray(np.asarray(a, dtype=np.int32).ravel())


class SimulationConfig:
    """Same fields and defaults as the reference's SimulationConfig."""

    _F64 = ("masses", "charges", "pos_x", "pos_y", "pos_z", "vel_x", "vel_y", "vel_z",
            "lj_sigma", "lj_epsilon", "bond_k", "bond_r0", "angle_k_theta", "angle_theta0",
            "dihedral_k_phi", "dihedral_phi0", "improper_k_phi", "improper_phi0")
    _I32 = ("atom_types", "bond_i", "bond_j", "angle_i", "angle_j", "angle_k", "dihedral_i",
            "dihedral_j", "dihedral_k", "dihedral_l", "dihedral_periodicity", "improper_i",
            "improper_j", "improper_k", "improper_l")

    def __init__(self):
        object.__setattr__(self, "_arrays", {})
        self.dt = 0.002
        self.n_steps = 1000
        self.init_temperature = 300.0
        self.gen_vel = False
        self.seed = 42
        self.box_size = 3.0
        self.lj_cutoff = 1.2
        self.use_lj = False
        self.coulomb_type = "cutoff"
        self.coulomb_cutoff = 1.2
        self.pme_order = 4
        self.pme_grid_spacing = 0.12
        self.ewald_coeff = 0.34
        self.trajectory_path = "trajectory.h5"
        self.nstxout = 0
        self.nstvout = 0
        self.nstenergy = 10
        self.energy_path = "energy.h5"
        self.checkpoint_interval = 500
        self.checkpoint_path = "checkpoint.bin"
        self.thermostat = ThermostatConfig()
        self.barostat = BarostatConfig()
        self.constraint_type = "none"
        self.constraint_tolerance = 1e-6
        self.constraint_i = []
        self.constraint_j = []
        self.constraint_dist = []
        self.excl_i = []
        self.excl_j = []
        for k in self._F64:
            self._arrays[k] = np.zeros(0, np.float64)
        for k in self._I32:
            self._arrays[k] = np.zeros(0, np.int32)

    def __getattr__(self, name):
        arrays = object.__getattribute__(self, "_arrays")
        if name in arrays:
            return arrays[name]
        if name == "mass":
            return arrays["masses"]
        raise AttributeError(name)

    def __setattr__(self, name, value):
        if name == "mass":
            name = "masses"
        if name in self._F64:
            self._arrays[name] = _f64(value)
        elif name in self._I32:
            self._arrays[name] = _i32(value)
        else:
            object.__setattr__(self, name, value)

    @property
    def lj_n_types(self) -> int:
        """n_types = sqrt(len(lj_sigma)) as the pybind setter derives it (core.cpp:196-205)."""
        return int(math.isqrt(len(self._arrays["lj_sigma"]))) if len(self._arrays["lj_sigma"]) else 0


# PHYS Verlet skin (nm) unless DMD_SKIN or the caller sets one.  Measured on
# one B200 with the SPME chain beside the pair kernel: water 30k 0.1312 ms/step
# at 0.15 nm against 0.1363 at 0.10; the 256-replica LJ / decane batch 1.330
# ms/step against 1.360 (1.349 at 0.20).
DEFAULT_SKIN_NM = 0.15


def default_skin() -> float:
    return float(os.environ.get("DMD_SKIN", DEFAULT_SKIN_NM))


def _options(precision=None, profile=None, skin=None, device=None, rng_seed=None, nb_form=None):
    precision = precision or os.environ.get("DMD_PRECISION", "mixed")
    profile = profile or os.environ.get("DMD_PROFILE", "ref")
    if skin is None:
        skin = default_skin()
    if device is None:
        device = int(os.environ.get("DMD_DEVICE", "0"))
    if precision not in _capi.PRECISIONS:
        raise ValueError(f"precision must be one of {list(_capi.PRECISIONS)}")
    if profile not in _capi.PROFILES:
        raise ValueError(f"profile must be one of {list(_capi.PROFILES)}")
    o = _capi.dmdgpu_options()
    o.profile = _capi.PROFILES[profile]
    o.precision = _capi.PRECISIONS[precision]
    o.skin = float(skin)
    o.device = int(device)
    o.rng_seed = int(rng_seed if rng_seed is not None else 0x5EED)
    nb_form = nb_form or os.environ.get("DMD_NB_FORM", "auto")
    if nb_form not in _capi.NB_FORMS:
        raise ValueError(f"nb_form must be one of {list(_capi.NB_FORMS)}")
    o.nb_form = _capi.NB_FORMS[nb_form]
    return o


class DmdGpuError(RuntimeError):
    """A non-zero status from the C ABI (status code in ``.code``)."""

    def __init__(self, code, msg):
        super().__init__(f"[{_capi.ERR_NAMES.get(code, code)}] {msg}")
        self.code = code


class Engine:
    """GPU-resident SimulationEngine with the EngineWrapper interface."""

    def __init__(self, cfg: SimulationConfig, precision=None, profile=None, skin=None,
                 device=None, rng_seed=None, nb_form=None):
        self._lib = _capi.lib()
        self._desc = _capi.SystemDesc(cfg)
        self._opt = _options(precision, profile, skin, device, rng_seed, nb_form)
        h = C.c_void_p()
        rc = self._lib.dmdgpu_create(C.byref(self._desc.s), C.byref(self._opt), C.byref(h))
        if rc != 0:
            msg = self._lib.dmdgpu_last_error(h)
            if h:
                self._lib.dmdgpu_destroy(h)
            raise DmdGpuError(rc, (msg or b"dmdgpu_create failed").decode())
        self._h = h
        self._n = int(len(cfg.masses))
        self._box0 = float(cfg.box_size)
        self._n_steps = int(cfg.n_steps)
        self.precision = precision or os.environ.get("DMD_PRECISION", "mixed")
        self.profile = profile or os.environ.get("DMD_PROFILE", "ref")

    # -- lifecycle ---------------------------------------------------------
    def close(self):
        if getattr(self, "_h", None):
            self._lib.dmdgpu_destroy(self._h)
            self._h = None

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass

    def _check(self, rc):
        if rc != 0:
            raise DmdGpuError(rc, (self._lib.dmdgpu_last_error(self._h) or b"").decode())

    # -- EngineWrapper surface --------------------------------------------
    def run(self):
        self._check(self._lib.dmdgpu_run(self._h))

    def run_n(self, steps: int):
        self._check(self._lib.dmdgpu_step(self._h, int(steps)))

    def _state(self, which):
        rows = np.empty((self._n, 3))
        self._check(self._lib.dmdgpu_get_state_rows(self._h, which, _capi.dptr(rows)))
        return rows

    @property
    def positions(self):
        return self._state(0)

    @property
    def velocities(self):
        return self._state(1)

    @property
    def forces(self):
        return self._state(2)

    def scalars(self) -> _capi.dmdgpu_scalars:
        s = _capi.dmdgpu_scalars()
        self._check(self._lib.dmdgpu_get_scalars(self._h, C.byref(s)))
        return s

    @property
    def potential_energy(self) -> float:
        return self.scalars().potential_energy

    @property
    def current_step(self) -> int:
        return int(self.scalars().step)

    @property
    def current_time(self) -> float:
        return self.scalars().time

    @property
    def box_size(self) -> float:
        # EngineWrapper returns the construction box (python/dmd/core.cpp:23, :46)
        return self._box0

    @property
    def n_atoms(self) -> int:
        return self._n

    # -- extensions (device single-point API, state I/O, checkpoints) -----
    def energy_terms(self) -> dict:
        s = self.scalars()
        return {k: s.e_terms[i] for i, k in enumerate(_capi.E_TERMS)}

    def _set_state(self, which, rows):
        rows = np.asarray(rows, dtype=np.float64)
        if rows.shape == (self._n, 3):
            rows = np.ascontiguousarray(rows)
            self._check(self._lib.dmdgpu_set_state_rows(self._h, which, _capi.dptr(rows)))
            return
        x, y, z = (np.ascontiguousarray(rows[:, k]) for k in range(3))
        self._check(self._lib.dmdgpu_set_state(self._h, which, _capi.dptr(x), _capi.dptr(y), _capi.dptr(z)))

    def set_positions(self, pos):
        self._set_state(0, pos)

    def set_velocities(self, vel):
        self._set_state(1, vel)

    def compute_forces(self):
        """Single-point forces (N x 3) and energy terms at the current positions."""
        e = np.zeros(len(_capi.E_TERMS))
        self._check(self._lib.dmdgpu_compute_forces(self._h, None, None, None, _capi.dptr(e)))
        return self._state(2), dict(zip(_capi.E_TERMS, e))

    def component_compute(self, component: int, pos, box, forces=None, energy=0.0):
        """ForceComponent::compute: accumulate one component's forces/energy."""
        pos = np.asarray(pos, dtype=np.float64)
        x, y, z = (np.ascontiguousarray(pos[:, k]) for k in range(3))
        if forces is None:
            forces = np.zeros((self._n, 3))
        fx, fy, fz = (np.ascontiguousarray(forces[:, k]) for k in range(3))
        e = C.c_double(energy)
        self._check(self._lib.dmdgpu_component_compute(
            self._h, int(component), _capi.dptr(x), _capi.dptr(y), _capi.dptr(z), float(box),
            _capi.dptr(fx), _capi.dptr(fy), _capi.dptr(fz), C.byref(e)))
        return np.stack([fx, fy, fz], axis=1), e.value

    def pair_list(self):
        cnt = C.c_int64()
        self._check(self._lib.dmdgpu_pair_list(self._h, None, None, 0, C.byref(cnt)))
        pi = np.empty(cnt.value, np.int32)
        pj = np.empty(cnt.value, np.int32)
        self._check(self._lib.dmdgpu_pair_list(self._h, _capi.iptr(pi), _capi.iptr(pj), cnt.value,
                                               C.byref(cnt)))
        return pi, pj

    def save_checkpoint(self, path: str):
        self._check(self._lib.dmdgpu_save_checkpoint(self._h, path.encode()))

    def load_checkpoint(self, path: str):
        self._check(self._lib.dmdgpu_load_checkpoint(self._h, path.encode()))

    def kernel_launches(self) -> int:
        return int(self._lib.dmdgpu_kernel_launches(self._h))

    def stream(self) -> int:
        """cudaStream_t (as an integer) every launch of this engine is issued on."""
        return int(self._lib.dmdgpu_stream(self._h) or 0)

    def launch_info(self) -> dict:
        """The launch configuration of the device table (valid after a step):
        pair-kernel form, its blocks per SM, whether the minimum-image pair
        kernel runs, kernels per captured step."""
        info = _capi.dmdgpu_launch_info()
        self._check(self._lib.dmdgpu_get_launch_info(self._h, C.byref(info)))
        return _capi.launch_info_dict(info)

    def repack(self):
        """Rebuild the device table with the state carried over bit for bit (pair
        list rebuilt in the frame of its last build, forces evaluated again at
        the current positions): what a running slot of a Batch goes through when
        another slot is admitted or released.  The trajectory is unchanged."""
        self._check(self._lib.dmdgpu_repack(self._h))

    def set_frame_writer(self, interval: int, writer=None):
        """Export a frame every `interval` steps while run_n / run continue on
        the device (the reference's run_n writes H5MD frames at
        trajectory_interval, python/dmd/core.cpp:29-44).  `writer(frame)` gets a
        dict with step, time, box, positions and velocities (N x 3 copies); it
        is called from a CUDA host-callback thread, in step order, and must not
        call back into this engine.  `interval` <= 0 or writer None turns export
        off.  Frames still in flight when a run returns are delivered by
        flush_frames() (or close())."""
        if interval <= 0 or writer is None:
            self._frame_cb = None
            self._check(self._lib.dmdgpu_set_frame_writer(self._h, 0, _capi.FRAME_FN(), None))
            return

        def deliver(fp, _user):
            f = fp.contents
            n = f.n_atoms
            arr = lambda p: np.ctypeslib.as_array(p, shape=(n,)).copy()  # noqa: E731
            writer({"step": int(f.step), "time": float(f.time), "box": float(f.box),
                    "positions": np.stack([arr(f.x), arr(f.y), arr(f.z)], 1),
                    "velocities": np.stack([arr(f.vx), arr(f.vy), arr(f.vz)], 1)})

        self._frame_cb = _capi.FRAME_FN(deliver)  # kept alive while export is on
        self._check(self._lib.dmdgpu_set_frame_writer(self._h, int(interval), self._frame_cb, None))

    def flush_frames(self):
        """Wait until every exported frame has been handed to the writer."""
        self._check(self._lib.dmdgpu_flush_frames(self._h))

    def test_inject(self, what: str):
        """Test-only, host-side fault injection for the failure paths:
        "barrier_timeout" (the next list build's bounded grid-barrier waits run
        out) or "list_capacity" (the next list build overflows its capacity)."""
        code = {"barrier_timeout": 1, "list_capacity": 2}[what]
        self._check(self._lib.dmdgpu_test_inject(self._h, code))

    def step_timed(self, steps: int, l2_flush_bytes: int = 0) -> dict:
        """Advance `steps` steps as one CUDA graph with device timing of every step
        and of every non-bonded / PME launch (optional L2 flush between steps)."""
        t = _capi.dmdgpu_timing()
        self._check(self._lib.dmdgpu_step_timed(self._h, int(steps), int(l2_flush_bytes), C.byref(t)))
        return {k: getattr(t, k) for k, _ in t._fields_}
