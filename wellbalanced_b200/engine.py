"""Device state and step driver shared by `MHD2D` and `MHD3D`.

Holds the two state pools of the Heun step (the state U and the stage U1), the layout
of a hierarchy (`wellbalanced_b200.mesh.Layout`) uploaded to the device, and launches
through the C ABI:

* ``fill(pool)`` — patchwork's ``exchange_halos`` plus the boundary faces, level by
  level: interpolation from the level below, same-level copies, outflow / wall faces;
* ``restrict(pool, groups)`` — patchwork's ``restrict``;
* ``stage(...)`` — one fused RK stage over every tile;
* ``stable_dt()`` — the stable step on the device in one call (``rate()`` and
  ``finalize_dt()`` apart where ranks reduce between them);
* ``run_steps(...)`` — whole steps from a launch list put together once.

One step is the reference's ``step`` (``carafe/mhd.py:965-994``,
``carafe/mhd3d.py:726-754``): stage 1 into U1, restrict the potential, fill U1, stage 2
back into U with the Heun combine, reflux, restrict, fill. torch is used for device
memory and streams only; every numerical kernel is in ``libwb200.so``.
"""

from __future__ import annotations

import contextlib
import ctypes

import numpy as np
import torch

from wellbalanced_b200 import _lib
from wellbalanced_b200.mesh import Layout, _concat, number_faces, size_ops

_DTYPES = {32: torch.float32, 64: torch.float64, _lib.MATH32_STATE64: torch.float64}


def _ptr(t):
    return ctypes_ptr(t)


def ctypes_ptr(t):
    if t is None:
        return None
    return t.data_ptr()


def _device_bytes(array, device, dtype):
    """A uint8 device tensor holding a numpy structured array in the C layout ``dtype``
    (None if empty). NumPy may repack a padded structured dtype (``np.concatenate`` does),
    so the records are cast back to the exact layout the kernels read."""
    if array is None or array.size == 0:
        return None
    array = np.ascontiguousarray(np.asarray(array).astype(dtype, copy=False))
    if array.dtype != dtype or array.dtype.itemsize != dtype.itemsize:
        raise TypeError(f"op records of dtype {array.dtype} do not have the C layout {dtype}")
    return torch.from_numpy(array.view(np.uint8).reshape(-1).copy()).to(device)


#: instances up to which `wb_stable_dt` is one launch (kOneLaunchInstances of csrc/rate.cu)
_ONE_LAUNCH_INSTANCES = 256
#: the slots of cfl, eta and kappa among the arguments of `wb_stable_dt`
_DT_SLOTS = slice(15, 18)


class Engine:
    """Device pools + op lists of one hierarchy; the kernels' launch sequence."""

    def __init__(self, hierarchy, *, precision=32, walls=None, limiter=1, gamma=5.0 / 3.0, mean_field=(0.0, 0.0, 0.0),
                 instances=None, device="cuda", lx=32, stream=None, layout=None, suit_tile=False):
        precision = _lib.precision_code(precision)
        if not torch.cuda.is_available():
            raise RuntimeError("wellbalanced_b200 needs a CUDA device (there is no CPU path)")
        _lib.load()
        self.device = torch.device(device)
        self.precision = precision
        self.dtype = _DTYPES[precision]
        self.limiter = int(limiter)
        self.gamma = float(gamma)
        self.mean_field = tuple(float(b) for b in mean_field) + (0.0,) * (3 - len(mean_field))
        self.layout = layout if layout is not None else Layout(
            hierarchy, walls=walls, precision=precision, lx=lx, instances=instances, suit_tile=suit_tile)
        L = self.layout
        self.ndim = L.ndim
        #: finest level of the layout (the hierarchy's property walks every patch)
        self.max_level = int(L.max_level)
        self.state = torch.zeros(L.pool_size, dtype=self.dtype, device=self.device)
        self.stage_pool = torch.zeros(L.pool_size, dtype=self.dtype, device=self.device)
        self.patches = _device_bytes(L.rows, self.device, _lib.PATCH)
        self.tiles = _device_bytes(L.tiles, self.device, _lib.TILE)
        self.ntiles = int(L.tiles.size)
        self.chunk_patch = torch.from_numpy(L.chunk_patch).to(self.device)
        self.chunk_start = torch.from_numpy(L.chunk_start).to(self.device)
        self.nchunks = int(L.chunk_patch.size)
        self.inv_dx2_sum = torch.from_numpy(L.inv_dx2_sum).to(self.device)
        levels = np.ascontiguousarray(getattr(L, "inv_dx2_levels", L.inv_dx2_sum[:, None]), dtype=np.float64)
        #: levels of the per-(instance, level) diffusion limit
        self.nlevels = int(levels.shape[1])
        self.inv_dx2_levels = torch.from_numpy(levels.reshape(-1)).to(self.device)
        self.level_keys = torch.zeros(max(self.nlevels * L.ninstances, 1), dtype=torch.int64, device=self.device)
        #: reduce the smallest density per level (set by the solvers when a diffusion limit
        #: applies on a refined hierarchy: each level's own density and spacing decide)
        self.per_level_dt = False
        # op lists on the device, each cut for the op kernels by its size (`size_ops`)
        def upload(ops, dtype):
            ops = size_ops(ops) if np.asarray(ops).size else np.zeros(0, dtype)
            return _device_bytes(ops, self.device, dtype), int(ops.size)

        self.copy_phases = [
            (*upload(same, _lib.COPY_OP), [upload(b, _lib.COPY_OP) for b in bnd]) for same, bnd in L.copy_phases
        ]
        self.interp_levels = [upload(ops, _lib.INTERP_OP) for ops in L.interp_levels]
        self.restrict_levels = {
            level: {g: upload(ops, _lib.RESTRICT_OP) for g, ops in groups.items()}
            for level, groups in L.restrict_levels.items()
        }
        # the ops of every field group of a level in one list: the groups write different
        # fields of the coarse level and read only the fine one, so one launch runs them all
        self.restrict_merged = {}
        for level, groups in L.restrict_levels.items():
            if len(groups) > 1:
                ops = _concat(list(groups.values()), _lib.RESTRICT_OP)
                self.restrict_merged[level] = (frozenset(groups), *upload(ops, _lib.RESTRICT_OP))
        n = L.ninstances
        self.ninstances = n
        #: what the host reads after a step, in one copy (`read_status`): the bad-cell count,
        #: then every instance's time and dt by their bits
        self.status = torch.zeros(1 + 2 * n, dtype=torch.int64, device=self.device)
        self.dt = self.status[1 + n :].view(torch.float64)
        self.keys = torch.zeros(2 * n, dtype=torch.int64, device=self.device)
        #: scratch of `stable_dt`: a ticket and the identities of the keys (largest rate 0,
        #: smallest density +inf per instance and per level), as every launch leaves them
        identities = np.full(1 + 2 * n + n * self.nlevels, 0xFFF0000000000000, dtype=np.uint64)
        identities[0] = 0
        identities[1 : 1 + 2 * n : 2] = 0x8000000000000000
        self.dt_scratch = torch.from_numpy(identities.view(np.int64)).to(self.device)
        self.time = self.status[1 : 1 + n].view(torch.float64)
        self.end = torch.zeros(n, dtype=torch.float64, device=self.device)
        self.bad = self.status[:1]
        #: the 2D stage kernel's boundary-face fluxes (float64, allocated on first use): the
        #: register reads the fine faces there instead of recomputing them
        self.bflux = None
        self.staged_fluxes = True
        face_ops, self.nface_faces = number_faces(L.face_flux_ops)
        self.face_flux_ops = _device_bytes(face_ops, self.device, _lib.FACE_FLUX_OP)
        self.nface = int(L.face_flux_ops.size)
        self.reflux_ops = _device_bytes(L.reflux_ops, self.device, _lib.REFLUX_OP)
        self.nreflux = int(L.reflux_ops.size)
        counts = [int(ops.size) for ops in L.reflux_phases]
        starts = np.cumsum([0, *counts])[: len(counts)]
        #: (first op, op count) of each reflux phase in `reflux_ops`
        self.reflux_phases = [(int(a), c) for a, c in zip(starts, counts, strict=True) if c]
        self.register = torch.zeros(max(L.register_size, 1), dtype=torch.float64, device=self.device)
        self.stream = stream
        #: kernels launched by this engine (counted per C-ABI call)
        self.launches = 0
        #: optional list collecting (start, end) CUDA events around each stage kernel
        self.stage_events = None
        #: non-ideal terms, None for ideal MHD: 2D (eta, kappa_par, kappa_perp, gx, gy),
        #: 3D (eta, gx, gy, gz)
        self.physics = None
        #: a level's interpolation and same-level copies in one launch (`wb_fill_ops`)
        self.fused_fill = True
        #: run stage 1's flux-register kernel on a second stream, beside the restriction
        #: and halo fill of the stage pool (it reads U, which those do not write)
        self.overlap_fluxes = True
        self._flux_stream = None
        self._flux_events = None
        #: the launching stream's handle while a step issues its launches (looked up once)
        self._step_stream = None
        #: the list that launches are put into instead of being issued, and the launch lists
        #: kept by step (`run_steps`); any other attribute that is set drops them
        self._recording = None
        self._lists = {}
        #: run the reflux, restriction, halo-fill and stable-step phases between the stage
        #: kernels as op programs (`wb_run_program`, one launch each: six launches per
        #: refined step instead of 24). Off by default: on the B200 the separate launches
        #: finish the ~2300-patch Harris step in 0.38 ms against 0.51 ms for the programs,
        #: whose in-kernel phase waits cost more than the launch boundaries they replace
        self.use_programs = False
        self._programs = {}
        #: dt on the device belongs to the current state (set by `prime_dt` and each
        #: programmed step; cleared by every other launch or write that changes the state)
        self.dt_ready = False

    # low-level launches ----------------------------------------------------------------------
    #: attributes that launches read nothing from: setting them keeps the launch lists
    _COUNTERS = frozenset(("launches", "dt_ready", "_step_stream", "_recording", "_lists"))

    def __setattr__(self, name, value):
        object.__setattr__(self, name, value)
        # another setting or buffer: the lists are out of date
        if name not in Engine._COUNTERS and self.__dict__.get("_lists"):
            object.__setattr__(self, "_lists", {})
        if name == "physics" and value is not None:
            self._default_tiles()

    def _default_tiles(self):
        """The non-ideal kernels run on the default tile: a work list cut to a shape chosen by
        the grid's size (not one asked for) is cut again."""
        layout = self.layout
        if getattr(layout, "_suit_tile", False) and layout.tile is None and layout.tile_shape != layout.default_tile:
            layout._suit_tile = False
            layout.tile_shape = layout.default_tile
            layout._cut_tiles()
            self._ideal_tiles = self.tiles  # launches in flight on another stream may read it
            self.tiles = _device_bytes(layout.tiles, self.device, _lib.TILE)
            self.ntiles = int(layout.tiles.size)

    def _s(self):
        if self._step_stream is not None:
            return self._step_stream
        return self._main().cuda_stream

    def _launch(self, name, *args, stream=None):
        """One C-ABI call, `args` before the stream, on `stream` or the engine's; while a
        launch list is put together, an entry of it."""
        if self._recording is not None:
            self._recording.append((name, args, None if stream is None else stream.cuda_stream))
        else:
            _lib.call(name, *args, self._s() if stream is None else stream.cuda_stream)

    def _main(self):
        return self.stream if self.stream is not None else torch.cuda.current_stream(self.device)

    def fill(self, pool, levels=None):
        """Halos of every patch of `pool`, level by level (coarse first)."""
        for level in range(len(self.copy_phases)):
            if levels is None or level in levels:
                self._fill_level(pool, level)

    def _fill_level(self, pool, level):
        """Interpolation from the level below, same-level copies, boundary faces."""
        prec = self.precision
        same, nsame, boundary = self.copy_phases[level]
        interp, ninterp = self.interp_levels[level]
        if ninterp and nsame and self.fused_fill:
            # the layout's interpolation ops skip the points the copies write: one launch
            self._launch("wb_fill_ops", prec, pool.data_ptr(), self.patches.data_ptr(), interp.data_ptr(), ninterp,
                         same.data_ptr(), nsame)
            self.launches += 1
        else:
            if ninterp:
                self._launch("wb_interp_ops", prec, pool.data_ptr(), self.patches.data_ptr(), interp.data_ptr(),
                             ninterp)
                self.launches += 1
            if nsame:
                self._launch("wb_copy_ops", prec, pool.data_ptr(), self.patches.data_ptr(), same.data_ptr(), nsame)
                self.launches += 1
        for ops, nops in boundary:
            if nops:
                self._launch("wb_copy_ops", prec, pool.data_ptr(), self.patches.data_ptr(), ops.data_ptr(), nops)
                self.launches += 1

    def restrict(self, pool, groups):
        """Coarse values under finer patches from the fine ones (finest level first)."""
        key = frozenset(groups)
        for level in range(self.max_level, 0, -1):
            merged = self.restrict_merged.get(level)
            if merged is not None and merged[0] == key:
                ops, nops = merged[1], merged[2]
                if nops:
                    self._launch("wb_restrict_ops", self.precision, pool.data_ptr(), self.patches.data_ptr(),
                                 ops.data_ptr(), nops)
                    self.launches += 1
                continue
            for g in groups:
                self._restrict_level(pool, level, g)

    def _restrict_level(self, pool, level, g):
        ops, nops = self.restrict_levels[level][g]
        if nops:
            self._launch("wb_restrict_ops", self.precision, pool.data_ptr(), self.patches.data_ptr(), ops.data_ptr(),
                         nops)
            self.launches += 1

    def _uses_staged_fluxes(self):
        """Whether the register takes the fine faces from the 2D stage kernel's boundary-face
        output (ideal 2D refined hierarchies; the non-ideal terms and 3D recompute them)."""
        return self.staged_fluxes and self.ndim == 2 and self.nface > 0 and self.physics is None

    def _stage_bflux(self):
        if self.bflux is None:
            self.bflux = torch.zeros(max(int(self.layout.bflux_size), 1), dtype=torch.float64, device=self.device)
        return self.bflux

    def stage(self, src, base, dst, bflux=None):
        b = self.mean_field
        if self.ntiles == 0:
            return
        if bflux is None and self._uses_staged_fluxes():
            bflux = self._stage_bflux()
        timing = self.stage_events is not None
        if timing:
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record(torch.cuda.current_stream(self.device) if self.stream is None else self.stream)
        self.launches += 1
        if self.ndim == 2 and self.physics is not None:
            if tuple(self.layout.tile_shape) != tuple(self.layout.default_tile):
                raise ValueError("the non-ideal 2D stage kernel runs on the default tile shape")
            self._launch("wb_stage2d_physics", self.precision, src.data_ptr(),
                         None if base is None else base.data_ptr(), dst.data_ptr(), self.patches.data_ptr(),
                         self.tiles.data_ptr(), self.ntiles, self.dt.data_ptr(),
                         self.gamma, b[0], b[1], self.limiter, *self.physics, self.bad.data_ptr())
        elif self.ndim == 2:
            tx, ty = self.layout.tile_shape
            self._launch("wb_stage2d_tiled", self.precision, src.data_ptr(),
                         None if base is None else base.data_ptr(), dst.data_ptr(), self.patches.data_ptr(),
                         self.tiles.data_ptr(), self.ntiles, self.dt.data_ptr(),
                         self.gamma, b[0], b[1], self.limiter, tx, ty, self.bad.data_ptr(),
                         None if bflux is None else bflux.data_ptr())
        elif self.physics is not None:
            if tuple(self.layout.tile_shape) != tuple(self.layout.default_tile):
                raise ValueError("the non-ideal 3D stage kernel runs on the default tile shape")
            self._launch("wb_stage3d_physics", self.precision, src.data_ptr(),
                         None if base is None else base.data_ptr(), dst.data_ptr(), self.patches.data_ptr(),
                         self.tiles.data_ptr(), self.ntiles, self.dt.data_ptr(), self.gamma, b[0], b[1], b[2],
                         self.limiter, self.layout.march, *self.physics, self.bad.data_ptr())
        else:
            ty, tz = self.layout.tile_shape
            self._launch("wb_stage3d_tiled", self.precision, src.data_ptr(),
                         None if base is None else base.data_ptr(), dst.data_ptr(), self.patches.data_ptr(),
                         self.tiles.data_ptr(), self.ntiles, self.dt.data_ptr(),
                         self.gamma, b[0], b[1], b[2], self.limiter, self.layout.march, ty, tz, self.bad.data_ptr(),
                         None if bflux is None else bflux.data_ptr())
        if timing:
            end.record(torch.cuda.current_stream(self.device) if self.stream is None else self.stream)
            self.stage_events.append((start, end))

    def rate(self, pool=None):
        pool = self.state if pool is None else pool
        b = self.mean_field
        if self.per_level_dt:
            _lib.call("wb_rate_levels", self.precision, self.ndim, pool.data_ptr(), self.patches.data_ptr(),
                      self.layout.npatches, self.chunk_patch.data_ptr(), self.chunk_start.data_ptr(), self.nchunks,
                      b[0], b[1], b[2], self.gamma, self.keys.data_ptr(), self.ninstances,
                      self.level_keys.data_ptr(), self.nlevels, self._s())
        else:
            _lib.call("wb_rate", self.precision, self.ndim, pool.data_ptr(), self.patches.data_ptr(),
                      self.layout.npatches, self.chunk_patch.data_ptr(), self.chunk_start.data_ptr(), self.nchunks,
                      b[0], b[1], b[2], self.gamma, self.keys.data_ptr(), self.ninstances, self._s())
        self.launches += 2 if self.nchunks else 1

    def finalize_dt(self, cfl, eta=0.0, kappa=0.0, *, clip_to_end=False, advance=False):
        end = self.end.data_ptr() if clip_to_end else None
        if self.per_level_dt:
            _lib.call("wb_finalize_dt_levels", self.keys.data_ptr(), self.ninstances, float(cfl), float(eta),
                      float(kappa), self.gamma, self.level_keys.data_ptr(), self.inv_dx2_levels.data_ptr(),
                      self.nlevels, self.time.data_ptr(), end, self.dt.data_ptr(), int(advance), self._s())
        else:
            _lib.call("wb_finalize_dt", self.keys.data_ptr(), self.ninstances, float(cfl), float(eta), float(kappa),
                      self.gamma, self.inv_dx2_sum.data_ptr(), self.time.data_ptr(), end, self.dt.data_ptr(),
                      int(advance), self._s())
        self.launches += 1

    def stable_dt(self, cfl, eta=0.0, kappa=0.0, *, advance=False):
        """`rate` of the state and `finalize_dt` in one call, and in one launch up to
        `_ONE_LAUNCH_INSTANCES` (as for them, one stream at a time: the keys and the dt are the
        engine's own)."""
        b = self.mean_field
        levels = self.per_level_dt
        self._launch("wb_stable_dt", self.precision, self.ndim, self.state.data_ptr(), self.patches.data_ptr(),
                     self.chunk_patch.data_ptr(), self.chunk_start.data_ptr(), self.nchunks, b[0], b[1], b[2],
                     self.gamma, self.keys.data_ptr(), self.ninstances, self.level_keys.data_ptr() if levels else None,
                     self.nlevels if levels else 0, float(cfl), float(eta), float(kappa), self.inv_dx2_sum.data_ptr(),
                     self.inv_dx2_levels.data_ptr() if levels else None, self.time.data_ptr(), None, self.dt.data_ptr(),
                     int(advance), self.dt_scratch.data_ptr())
        self.launches += 1 if self.ninstances <= _ONE_LAUNCH_INSTANCES else 3 if self.nchunks else 2

    def read_status(self):
        """(bad cells, times, dts) on the host, once the launches so far are done: one copy."""
        host = self.status.cpu().numpy()
        n = self.ninstances
        return int(host[0]), host[1 : 1 + n].view(np.float64), host[1 + n :].view(np.float64)

    def rate_values(self):
        """(max rate, min density) per instance, on the host."""
        keys = self.keys.view(torch.int64).cpu().numpy().view(np.uint64).reshape(-1, 2)
        out = np.empty(keys.shape)
        for index, k in np.ndenumerate(keys):
            k = int(k)
            bits = (k & 0x7FFFFFFFFFFFFFFF) if k >> 63 else (~k & 0xFFFFFFFFFFFFFFFF)
            out[index] = np.frombuffer(np.uint64(bits).tobytes(), dtype=np.float64)[0]
        return out

    def face_fluxes(self, pool, stream=None):
        """Register += fine-mean minus coarse fluxes of every coarse-fine interface face
        (on `stream`, else the engine's stream). `pool` is the input of the stage just
        launched: with staged fluxes its fine faces are read from that stage's output."""
        if self.nface:
            b = self.mean_field
            if self.physics is not None:
                eta, kappa_par, kappa_perp = self.physics[:3] if self.ndim == 2 else (self.physics[0], 0.0, 0.0)
            if self.physics is not None and (eta or kappa_par or kappa_perp):
                self._launch("wb_face_flux_ops_physics", self.precision, pool.data_ptr(), self.patches.data_ptr(),
                             self.face_flux_ops.data_ptr(), self.nface, b[0], b[1], b[2], self.gamma, self.limiter, eta,
                             kappa_par, kappa_perp, self.register.data_ptr(), stream=stream)
            elif self._uses_staged_fluxes():
                # the fine faces as the stage kernel that read `pool` wrote them
                self._launch("wb_face_flux_ops_staged", self.precision, pool.data_ptr(), self.patches.data_ptr(),
                             self.face_flux_ops.data_ptr(), self.nface, self.nface_faces, b[0], b[1], b[2], self.gamma,
                             self.limiter, self._stage_bflux().data_ptr(), self.register.data_ptr(), stream=stream)
            else:
                self._launch("wb_face_flux_ops", self.precision, pool.data_ptr(), self.patches.data_ptr(),
                             self.face_flux_ops.data_ptr(), self.nface, b[0], b[1], b[2], self.gamma, self.limiter,
                             self.register.data_ptr(), stream=stream)
            self.launches += 1

    def reflux(self, pool):
        """Coarse cells beside fine patches take the register's correction (then cleared)."""
        size = _lib.REFLUX_OP.itemsize
        for start, count in self.reflux_phases:
            self._launch("wb_reflux_apply", self.precision, pool.data_ptr(), self.patches.data_ptr(),
                         self.reflux_ops.data_ptr() + start * size, count, self.register.data_ptr(),
                         self.dt.data_ptr())
            self.launches += 1

    def capture(self, step):
        """A CUDA graph of the launches `step()` issues. `step` runs once outside the graph
        first (lazy loading and launch attributes happen there, not in the recording)."""
        stream = torch.cuda.Stream(self.device)
        stream.wait_stream(torch.cuda.current_stream(self.device))
        with torch.cuda.stream(stream):
            step()
        torch.cuda.current_stream(self.device).wait_stream(stream)
        torch.cuda.synchronize(self.device)
        graph = torch.cuda.CUDAGraph()
        graph.tiles = self.tiles  # replayed with this work list, also where another replaces it
        with torch.cuda.graph(graph):
            step()
        torch.cuda.synchronize(self.device)
        return graph

    def heun_step(self, groups_potential, groups_all):
        """One Heun step with the dt already in self.dt (device), refluxed and restricted."""
        self.run_steps(1, groups_potential, groups_all)

    def run_steps(self, count, groups_potential, groups_all, dt_params=None, *, advance=True, clear_bad=False):
        """`count` Heun steps, each at the dt on the device or, with dt_params (cfl, eta, kappa),
        at the stable dt of its state (`stable_dt`; the time advanced by it unless not `advance`);
        with clear_bad the bad-cell count is zeroed before each. The launches of a step are put
        together once (`_lib.launch_list`) and issued by one native call for all steps; a rank
        of a partition, whose exchanges run between them, and timed stages issue them one by one."""
        self.dt_ready = False

        def launches():
            if dt_params is not None:
                self.stable_dt(*dt_params, advance=advance)
            self._heun_launches(groups_potential, groups_all)

        if type(self) is not Engine or self.stage_events is not None:
            with self.launching():
                for _ in range(count):
                    if clear_bad:
                        self.bad.zero_()
                    launches()
            return
        # the list holds the dt parameters in slots that are written when they change: one list
        # for every cfl a run takes
        key = (tuple(groups_potential), tuple(groups_all), dt_params is not None, advance, clear_bad)
        found = self._lists.get(key)
        if found is None:
            if self.max_level > 0 and self._uses_staged_fluxes():
                self._stage_bflux()  # allocated before the recording, not by it
            self._side_stream()
            before = self.launches
            self._recording = []
            try:
                if clear_bad:
                    self._launch("clear_bytes", self.bad.data_ptr(), 8)
                launches()
                rows = [k for k, (name, *_) in enumerate(self._recording) if name == "wb_stable_dt"]
                found = [_lib.launch_list(self._recording), self.launches - before, rows, dt_params]
            finally:
                self._recording = None
                self.launches = before
            self._lists[key] = found
        entries, kernels, rows, written = found
        if written != dt_params:
            entries["args"][rows, _DT_SLOTS] = np.array(dt_params, dtype=np.float64).view(np.int64)
            found[3] = dt_params
        _lib.call("wb_run_launches", entries.ctypes.data, int(entries.size), int(count), self._s())
        self.launches += kernels * count

    @contextlib.contextmanager
    def launching(self):
        """A run of launches on the engine's stream as it is now (its handle looked up once,
        not per launch)."""
        outer = self._step_stream
        if outer is None:
            self._step_stream = self._main().cuda_stream
        try:
            yield
        finally:
            self._step_stream = outer

    def _side_stream(self):
        """The flux register's own stream and its fork and join events (made on first use), or
        None where the register runs with the rest."""
        if not (self.overlap_fluxes and self.nface):
            return None
        if self._flux_stream is None:
            self._flux_stream = torch.cuda.Stream(self.device)
            self._flux_events = (torch.cuda.Event(), torch.cuda.Event())
            for event in self._flux_events:  # an event has its handle from its first record on
                event.record(self._flux_stream)
        return self._flux_stream

    def _order(self, event, first, then):
        """`then` waits for what `first` has issued so far (None: the engine's stream)."""
        if self._recording is not None:
            self._launch("record_event", event.cuda_event, stream=first)
            self._launch("wait_event", event.cuda_event, stream=then)
            return
        event.record(self._main() if first is None else first)
        (self._main() if then is None else then).wait_event(event)

    def _heun_launches(self, groups_potential, groups_all):
        U, U1 = self.state, self.stage_pool
        refined = self.max_level > 0
        self.stage(U, None, U1)
        # stage 1's register kernel beside the restriction and fill of U1 (small,
        # latency-bound launches that leave the SMs idle), not beside the stage kernel
        side = self._side_stream()
        if side is not None:
            forked, joined = self._flux_events
            self._order(forked, None, side)
        self.face_fluxes(U, side)
        if refined:
            self.restrict(U1, groups_potential)
        if not self.layout.wraps:  # else the stage has written U1's halo
            self.fill(U1)
        if side is not None:
            self._order(joined, side, None)  # stage 1's fluxes have read U before stage 2 writes it
        self.stage(U1, U, U)
        self.face_fluxes(U1)
        self.reflux(U)
        if refined:
            self.restrict(U, groups_all)
        if not self.layout.wraps:
            self.fill(U)

    # op programs ------------------------------------------------------------------------------
    def _fill_phases(self, pool):
        """Phases of the halo fill of every level of pool (0: the state, 1: the stage pool),
        as `fill` launches them."""
        phases = []
        for level in range(len(self.copy_phases)):
            same, nsame, boundary = self.copy_phases[level]
            interp, ninterp = self.interp_levels[level]
            # the interpolation ops are trimmed to the points no copy writes: one phase
            phases.append([s for s in (("interp", pool, interp, ninterp), ("copy", pool, same, nsame)) if s[3]])
            phases.extend([("copy", pool, ops, nops)] for ops, nops in boundary if nops)
        return phases

    def _restrict_phases(self, pool, groups):
        """Phases of the restriction of `groups` in pool, finest level first, as `restrict`
        launches them."""
        key = frozenset(groups)
        phases = []
        for level in range(self.max_level, 0, -1):
            merged = self.restrict_merged.get(level)
            if merged is not None and merged[0] == key:
                phases.append([("restrict", pool, merged[1], merged[2])] if merged[2] else [])
            else:
                phases.append([("restrict", pool, *self.restrict_levels[level][g]) for g in groups
                               if self.restrict_levels[level][g][1]])
        return phases

    def _program(self, phases, dt_params=None):
        """An op program (segment records, parameters, counters) from phases of segments
        (kind, pool, ops tensor or None, count[, aux tensor]); empty phases dropped."""
        phases = [p for p in phases if p]
        rows = []
        for k, phase in enumerate(phases):
            for seg in phase:
                kind, pool, ops, count = seg[:4]
                aux = seg[4] if len(seg) > 4 else None
                rows.append((_lib.SEGMENT_KINDS[kind], pool, k, int(count), 0, 0,
                             0 if ops is None else ops.data_ptr(), 0 if aux is None else aux.data_ptr()))
        if len(rows) > _lib.PROGRAM_MAX_SEGMENTS:
            raise ValueError(f"an op program of {len(rows)} segments (at most {_lib.PROGRAM_MAX_SEGMENTS})")
        segments = np.array(rows, dtype=_lib.PROGRAM_SEGMENT) if rows else np.zeros(0, _lib.PROGRAM_SEGMENT)
        params = _lib.ProgramParams()
        for a in range(3):
            params.b0[a] = self.mean_field[a]
        params.gamma = self.gamma
        params.ndim = self.ndim
        params.ninstances = self.ninstances
        params.nlevels = self.nlevels
        params.reg = self.register.data_ptr()
        params.dt = self.dt.data_ptr()
        params.time = self.time.data_ptr()
        params.keys = self.keys.data_ptr()
        params.inv_dx2_sum = self.inv_dx2_sum.data_ptr()
        params.inv_dx2_levels = self.inv_dx2_levels.data_ptr()
        if self.per_level_dt:
            params.level_keys = self.level_keys.data_ptr()
        if dt_params is not None:
            params.cfl, params.dt_eta, params.dt_kappa = dt_params
        counters = torch.zeros(3 + len(phases), dtype=torch.int32, device=self.device)
        return segments, params, counters

    def programs(self, groups_potential, groups_all, dt_params=None):
        """The two op programs of a step: after stage 1 the restriction of the stage pool's
        potential and its halo fill; after stage 2 the reflux, the state's restriction and
        halo fill and, with dt_params (cfl, eta, kappa), the time advanced by this step's
        dt first and the next step's dt from the new state last."""
        key = (tuple(groups_potential), tuple(groups_all), dt_params, self.per_level_dt)
        found = self._programs.get(key)
        if found is None:
            first = self._restrict_phases(1, groups_potential) + self._fill_phases(1)
            second = [[("advance_time", 0, None, 1), ("init_keys", 0, None, 1)]] if dt_params is not None else []
            size = _lib.REFLUX_OP.itemsize
            second += [[("reflux", 0, self.reflux_ops[start * size:], count)] for start, count in self.reflux_phases]
            second += self._restrict_phases(0, groups_all) + self._fill_phases(0)
            if dt_params is not None:
                if self.nchunks:
                    second.append([("rate", 0, self.chunk_patch, self.nchunks, self.chunk_start)])
                second.append([("finalize_dt", 0, None, 1)])
            found = (self._program(first), self._program(second, dt_params))
            self._programs[key] = found
        return found

    def run_program(self, program):
        segments, params, counters = program
        if segments.size == 0:
            return
        _lib.call("wb_run_program", self.precision, self.state.data_ptr(), self.stage_pool.data_ptr(),
                  self.patches.data_ptr(), segments.ctypes.data, int(segments.size), ctypes.addressof(params),
                  counters.data_ptr(), self._s())
        self.launches += 1

    def program_error(self):
        """The error bits the op programs have set since the last call (0: none); cleared."""
        bits = 0
        for pair in self._programs.values():
            for _, _, counters in pair:
                bits |= int(counters[2].item())
                counters[2].zero_()
        return bits

    def prime_dt(self, cfl, eta=0.0, kappa=0.0):
        """dt of the next programmed step from the current state (time not advanced)."""
        with self.launching():
            self.stable_dt(cfl, eta, kappa)
        self.dt_ready = True

    def programmed_step(self, groups_potential, groups_all, cfl, eta=0.0, kappa=0.0):
        """One Heun step through op programs at the dt on the device (`prime_dt` before the
        first, then each step leaves the next one): stage 1, the register's face fluxes
        (beside program 1), program 1, stage 2, face fluxes, program 2. Equal, bit for
        bit, to rate, finalize_dt(advance) and `heun_step` at the same dt."""
        first, second = self.programs(groups_potential, groups_all, (float(cfl), float(eta), float(kappa)))
        with self.launching():
            U, U1 = self.state, self.stage_pool
            self.stage(U, None, U1)
            side = self._side_stream()
            if side is not None:
                forked, joined = self._flux_events
                main = self._main()
                forked.record(main)
                side.wait_event(forked)
            self.face_fluxes(U, side)
            self.run_program(first)
            if side is not None:
                joined.record(side)
                main.wait_event(joined)  # stage 1's fluxes have read U before stage 2 writes it
            self.stage(U1, U, U)
            self.face_fluxes(U1)
            self.run_program(second)
        self.dt_ready = True  # the second program left the next step's dt

    # host views --------------------------------------------------------------------------------
    def view(self, pool, patch, field):
        return self.layout.patch_view(pool, patch, field)
