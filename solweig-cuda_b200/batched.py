"""Batched form: a whole day (or many days) per CUDA-graph replay.

All hours of a day are planned on the host first (FP64 solar geometry,
Perez luminance, patch weights, sun rays: ``engine.plan_day``), written into
pinned memory and replayed as one captured graph: the hour-record and ray
uploads, the state reset and the three kernels of every hour (``solweig_day``),
or the few launches of the whole day (:class:`ChosenDay`).  The graph is
captured once per scene, on its second day, and replays for any forcing of the
same length, because every kernel reads its hour record from device memory.
"""
from __future__ import annotations

import ctypes

import numpy as np
import torch

from . import _lib
from . import sun as _sun
from .engine import HourBuffers, device_ptr, outputs_struct, plan_day, stream_handle

__all__ = ["BatchedDay", "ChosenDay", "MultiDay", "TileBatch", "DayError"]

# Bits of the sticky error word (word 1 of the flag pair at the start of the
# work buffer): bit v is set when a day raised flag v.  Flags 1 (a tensor-core
# wait of the contraction timed out) and 3 (a sun ray stayed inside the raster
# for more than max(rows, cols) + 2 steps) leave invalid results; flag 2 (a
# window sweep's TMA wait timed out) does not (that tile walked from the raster).
_INVALID_BITS = (1 << 1) | (1 << 3)
_FLAG_TEXT = {1: "a tensor-core wait of the patch contraction timed out",
              2: "a sweep window's TMA wait timed out (results exact)",
              3: "a sun ray table stayed inside the raster longer than max(rows, cols) + 2 steps"}


class DayError(RuntimeError):
    """A batched day raised a device error flag that invalidates its results."""


def _error_words(work):
    """The flag pair at the start of a batched-day work buffer (int32 view)."""
    return work[:8].view(torch.int32)


def clear_day_errors(work):
    """Zero both words of the flag pair (the days never clear the sticky word)."""
    _error_words(work).zero_()


def check_day_errors(work, what="batched day"):
    """Raise DayError when a day run in `work` since the last clear raised a
    flag that invalidates results; returns the sticky bit set (synchronises)."""
    bits = int(_error_words(work)[1].item())
    if bits & _INVALID_BITS:
        raised = [v for v in _FLAG_TEXT if bits & (1 << v)]
        raise DayError(f"{what}: " + "; ".join(_FLAG_TEXT[v] for v in raised) + " - results invalid")
    return bits


class BatchedDay:
    """Run days of ``hours`` rows each through one captured graph."""

    def __init__(self, scene, latitude, longitude, site_altitude=3.0, utc=0.0, hours=24,
                 outputs=("tmrt", "utci"), use_graph=True):
        self.scene = scene
        self.latitude, self.longitude, self.site_altitude, self.utc = latitude, longitude, site_altitude, utc
        self.hours = hours
        dev = scene.device
        self.state = {k: torch.zeros(scene.shape, dtype=torch.float32, device=dev)
                      for k in _lib.STATE_FIELDS}
        self.scratch = torch.empty((_lib.SCRATCH_PLANES, scene.rows, scene.cols), dtype=torch.float32,
                                   device=dev)
        self.buffers = HourBuffers(scene, hours)
        self.layout_dev = scene.layout.device(dev)
        self.out_names = tuple(outputs)
        self.out = {k: torch.empty((hours,) + scene.shape, dtype=torch.float32, device=dev)
                    for k in self.out_names}
        self.use_graph = use_graph
        self.graph = None
        self.warm = False  # an eager day has run

    @property
    def launches_per_day(self):
        """Shadow, GVF and radiation kernel of every hour."""
        return 3 * self.hours

    def _state_struct(self):
        s = _lib.SolweigState()
        for k in _lib.STATE_FIELDS:
            setattr(s, k, self.state[k].data_ptr())
        return s

    def _sequence(self):
        """Uploads, state reset and the day's kernels, on the current stream."""
        self.buffers.upload(0, self.hours, self.buffers.kmax)
        for t in self.state.values():
            t.zero_()
        sc = self.scene
        base = outputs_struct(self.out, 0)
        stride = sc.pixels
        _lib.check(_lib.lib().solweig_day(
            ctypes.byref(sc.struct), device_ptr(self.layout_dev), self.buffers.ptr(), self.hours,
            ctypes.byref(self._state_struct()), ctypes.byref(base), stride, sc.gvf_host_ptr,
            sc.first_steps, sc.second_steps, device_ptr(self.scratch), stream_handle()),
            "solweig_day")

    def plan(self, met):
        met = np.asarray(met, dtype=np.float64)
        if len(met) != self.hours:
            raise ValueError(f"expected {self.hours} forcing rows, got {len(met)}")
        plan = plan_day(self.scene, met, self.latitude, self.longitude, self.site_altitude, self.utc)
        self.buffers.wait_free()
        self.buffers.put_plan(plan)
        self.last_plan = plan
        return plan

    @property
    def last_scalars(self):
        """HourScalars of the rows of the last day."""
        return [p[2] for p in self.last_plan]

    def run_day(self, met, outputs=None):
        """Plan the day on the host and run it; returns {name: [H, rows, cols]} views
        that stay valid until the next call.  The first day runs eagerly (a run of
        one day pays for no capture), the second captures the graph."""
        self.plan(met)
        if not self.use_graph or self.graph is None and not self.warm:
            self._sequence()
            self.warm = True
        else:
            if self.graph is None:
                torch.cuda.synchronize()
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g):
                    self._sequence()
                self.graph = g
            self.graph.replay()
        self.buffers.mark()
        names = self.out_names if outputs is None else outputs
        return {k: self.out[k] for k in names}


def day_launches(scene, config, sweep_parts=1):
    """Kernel launches of one batched day for this scene and launch shapes,
    with the sweep stage issued in ``sweep_parts`` hour ranges: per range the
    ray exits, the ceilings and the sweep; once the height dilation, for the
    ceilings or the raster sweep's plane of heights (and the tile maxima of the
    window sweep); then the GVF (the walk words where the scene has none for
    its step table, sample codes and the walk kernel, or the per-hour kernel),
    weights, two splits (sky and vegetation weights), tables, contraction and
    radiation."""
    s = scene.struct
    ceiling = int(not config.no_ceiling)
    window = int(config.sweep_window != 0 and scene.geo32 is not None and not s.has_water)
    height = scene.geo32 is not None and not window and scene.pixels <= _lib.PACKED_MAX_PIXELS
    walk = config.gvf_hours == 1 and scene.first_steps == 1 and 2 <= scene.second_steps <= 22 and not s.has_water
    statics = s.gvf_walks and s.gvf_nosh and s.gvf_table == _lib.lib().solweig_gvf_table_key(
        scene.gvf_host_ptr, scene.first_steps, scene.second_steps)
    gvf = (2 if statics else 3) if walk else 1
    return sweep_parts * (2 + ceiling) + int(ceiling or height) + window + gvf + 6


class ChosenDay(BatchedDay):
    """The batched form: every hour of a day in a few launches
    (``solweig_day_batched``: ray ceilings and shadow sweep, GVF over all hours,
    the BF16 tensor-core patch contraction, hour-looping radiation), captured
    as one CUDA graph with the upload of the hour records.

    Produces the all-direction planes (Tmrt, UTCI, Kdown, Kup, Ldown, Lup,
    Kside, Lside, shadow, Tg ...); the cardinal E/S/W/N planes are only made
    by the per-hour form."""

    CARDINAL = ("keast", "ksouth", "kwest", "knorth", "least", "lsouth", "lwest", "lnorth")

    def __init__(self, scene, latitude, longitude, site_altitude=3.0, utc=0.0, hours=24,
                 outputs=("tmrt", "utci"), use_graph=True, pipeline_hours=0):
        bad = [o for o in outputs if o in self.CARDINAL]
        if bad:
            raise ValueError(f"the batched form does not produce {bad}")
        super().__init__(scene, latitude, longitude, site_altitude, utc, hours, outputs, use_graph)
        self.scratch = None
        # pipeline_hours: an int or a sequence of range lengths (the last one
        # repeats) issues the sweep stage in ranges of hours with a graph each, 0
        # as a whole.  The day is planned before either: that takes 0.2 ms after
        # the sun positions, less than seven more sweep launches cost a small
        # raster, so ranges only bound the sweep stage's single launches.
        self.ranges = self._ranges(hours, pipeline_hours)
        self.part_graphs = None
        L = _lib.lib()
        self.work_bytes = int(L.solweig_day_batched_work_bytes(scene.rows, scene.cols, hours,
                                                               int(scene.struct.has_water)))
        if self.work_bytes <= 0:
            raise ValueError("bad batched-day shape")
        self.work = torch.empty(self.work_bytes, dtype=torch.uint8, device=scene.device)
        clear_day_errors(self.work)
        self.config = _lib.SolweigDayConfig.default()

    @staticmethod
    def _ranges(hours, pipeline_hours):
        if isinstance(pipeline_hours, int):
            if pipeline_hours <= 0:
                return None
            lengths = [pipeline_hours]
        else:
            lengths = [int(x) for x in pipeline_hours]
            if not lengths or min(lengths) <= 0:
                raise ValueError("pipeline_hours: range lengths must be positive")
        out, h, i = [], 0, 0
        while h < hours:
            n = lengths[min(i, len(lengths) - 1)]
            out.append((h, min(h + n, hours)))
            h, i = h + n, i + 1
        return out

    @property
    def launches_per_day(self):
        """Kernels of one day (``day_launches``)."""
        return day_launches(self.scene, self.config, len(self.ranges) if self.ranges else 1)

    def set_config(self, config):
        """Launch shapes (``SolweigDayConfig`` or a tuple of its fields); drops captured graphs."""
        if not isinstance(config, _lib.SolweigDayConfig):
            config = _lib.SolweigDayConfig(*config)
        self.config = config
        self.graph = None
        self.part_graphs = None
        self.warm = False

    def _part(self, part, h0=0, h1=0):
        """One part of the day on the current stream (``solweig_day_batched_part``):
        part 0 uploads the records and rays of hours [h0, h1) and sweeps them,
        part 1 runs the rest of the day."""
        if part == 0:
            self.buffers.upload(h0, h1 - h0, self.buffers.kmax)
        sc = self.scene
        base = outputs_struct(self.out, 0)
        _lib.check(_lib.lib().solweig_day_batched_part(
            ctypes.byref(sc.struct), device_ptr(self.layout_dev), self.buffers.ptr(), self.hours,
            ctypes.byref(_lib.SolweigState()), ctypes.byref(base), sc.pixels, sc.gvf_host_ptr,
            sc.first_steps, sc.second_steps, device_ptr(self.work), self.work_bytes,
            ctypes.byref(self.config), part, h0, h1, stream_handle()), "solweig_day_batched_part")

    def run_day(self, met, outputs=None):
        """Plan the day on the host and run it, in one graph or in the ranges of
        ``pipeline_hours``.  Returns {name: [H, rows, cols]} views that stay valid
        until the next call."""
        if self.ranges is None:
            return super().run_day(met, outputs)
        self.plan(met)
        if self.use_graph and self.part_graphs is None and self.warm:
            torch.cuda.synchronize()
            graphs = []
            for part in [(0, h0, h1) for h0, h1 in self.ranges] + [(1,)]:
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g):
                    self._part(*part)
                graphs.append(g)
            self.part_graphs = graphs
        if self.use_graph and self.part_graphs is not None:
            for g in self.part_graphs:
                g.replay()
        else:
            for h0, h1 in self.ranges:
                self._part(0, h0, h1)
            self._part(1)
            self.warm = True
        self.buffers.mark()
        names = self.out_names if outputs is None else outputs
        return {k: self.out[k] for k in names}

    def _sequence(self):
        # Each day starts from the reset state (src/series.py:425-436): the
        # batched kernel starts from zero state when no state planes are given,
        # and nothing needs the day's final state.
        self.buffers.upload(0, self.hours, self.buffers.kmax)
        sc = self.scene
        base = outputs_struct(self.out, 0)
        _lib.check(_lib.lib().solweig_day_batched_ex(
            ctypes.byref(sc.struct), device_ptr(self.layout_dev), self.buffers.ptr(), self.hours,
            ctypes.byref(_lib.SolweigState()), ctypes.byref(base), sc.pixels, sc.gvf_host_ptr,
            sc.first_steps, sc.second_steps, device_ptr(self.work), self.work_bytes,
            ctypes.byref(self.config), stream_handle()), "solweig_day_batched_ex")

    @staticmethod
    def stage_bytes(pixels, hours, day_hours):
        """Algorithmic HBM bytes of each stage of one day.

        shadow (with the ray ceilings): per daytime pixel-hour 4 B of the plane
        of heights and the pixel's own 16 B sample read, 8 B ceiling and window
        maximum written and read back, 8 B wall height + 1 B flags + 20 B
        float32 fields read, 16 B quad written (81 B); GVF (walk words): 16 B
        quad + 4 B emissivity read, a quarter of 4 B codes written and read
        back and of 72 B words read, 3 planes written (52 B) and the
        albedo-without-shadow plane once; tables: per-hour tables (negligible); contraction: 40 B
        of mask words per pixel read, 2 sums per pixel-hour written (8 B: sky
        plus transmitted vegetation, luminance and luminance*cos*omega);
        radiation: 109 B of per-pixel statics and 16 B of state per day, 20 B
        per daytime pixel-hour (3 GVF planes, 2 sums) and 8 B per pixel-hour
        written (Tmrt, UTCI)."""
        return {
            "day_shadow_kernel": pixels * day_hours * 81,
            "day_gvf_kernel": pixels * (52 * day_hours + 4),
            "day_tables_kernel": hours * 9680,
            "patch_gemm_kernel": pixels * (40 + 8 * hours),
            "day_radiation_kernel": pixels * (125 + 20 * day_hours + 8 * hours),
        }

    @staticmethod
    def gemm_flops(pixels, hours, patches):
        """Algorithmic FLOPs of the contraction: 2 x pixels x patches x 2 hour
        columns (luminance, luminance x cos x omega) x 2 masks (sky,
        vegetation); the BF16 hi/lo duplication is not counted."""
        return 2 * pixels * patches * (2 * hours) * 2

    STAGES = ("day_shadow_kernel", "day_gvf_kernel", "day_tables_kernel", "patch_gemm_kernel",
              "day_radiation_kernel")

    def profile_day(self, met):
        """Device time of each stage of one day, {stage: ms}, from CUDA events
        recorded on the launching stream between the stages."""
        self.plan(met)
        self.buffers.upload(0, self.hours, self.buffers.kmax)
        sc = self.scene
        base = outputs_struct(self.out, 0)
        ms = (ctypes.c_float * len(self.STAGES))()
        _lib.check(_lib.lib().solweig_day_batched_timed(
            ctypes.byref(sc.struct), device_ptr(self.layout_dev), self.buffers.ptr(), self.hours,
            ctypes.byref(_lib.SolweigState()), ctypes.byref(base), sc.pixels, sc.gvf_host_ptr,
            sc.first_steps, sc.second_steps, device_ptr(self.work), self.work_bytes,
            ctypes.byref(self.config), stream_handle(), ms), "solweig_day_batched_timed")
        self.buffers.mark()
        return dict(zip(self.STAGES, (float(x) for x in ms)))

    WORK_FIELDS = ("quads", "lup_first", "gvf", "nosh", "sums", "wf32", "bw", "tables", "error", "tilemax",
                   "total")

    def work_offsets(self):
        """{field: byte offset} of the work buffer (``solweig_day_batched_layout``)."""
        sc = self.scene
        off = (ctypes.c_int64 * 11)()
        _lib.check(_lib.lib().solweig_day_batched_layout(sc.rows, sc.cols, self.hours,
                                                         int(sc.struct.has_water), off),
                   "solweig_day_batched_layout")
        return dict(zip(self.WORK_FIELDS, (int(x) for x in off)))

    def quads(self):
        """The sweep's per-pixel GVF inputs of the last day as a [H, rows, cols, 4]
        float32 view: shadow, Lup excess, albedo and the ground (1) / sunlit-wall
        (2) bits as an int32 bit pattern (daytime hours only; night hours hold
        stale values)."""
        o = self.work_offsets()
        n = 16 * self.hours * self.scene.pixels
        return self.work[o["quads"]:o["quads"] + n].view(torch.float32).view(self.hours, self.scene.rows,
                                                                                 self.scene.cols, 4)

    def patch_sums(self):
        """The contraction's output of the last day as a [2H, pixels] view: row
        2h + 0 the luminance and 2h + 1 the luminance*cos*omega summed over the
        sky patches plus 0.03 x the same over the vegetation patches."""
        o = self.work_offsets()
        n = 2 * self.hours * self.scene.pixels
        return self.work[o["sums"]:o["sums"] + 4 * n].view(torch.float32).view(2 * self.hours, self.scene.pixels)

    def check_errors(self):
        """Raise DayError if any day run by this object left invalid results."""
        return check_day_errors(self.work, "batched day")

    def error_flag(self):
        """Device error flag of the last day (0 = ok, 1 = a tensor-core wait timed
        out, 2 = a sweep window's TMA wait timed out: that tile walked from the raster,
        3 = a sun ray stayed inside the raster for more than max(rows, cols) + 2 steps)."""
        flag = torch.zeros(1, dtype=torch.int32, device=self.scene.device)
        sc = self.scene
        _lib.check(_lib.lib().solweig_day_batched_error(
            device_ptr(self.work), sc.rows, sc.cols, self.hours, int(sc.struct.has_water),
            device_ptr(flag), stream_handle()), "solweig_day_batched_error")
        return int(flag.item())


class MultiDay:
    """``days`` consecutive days of ``hours`` rows each through ONE captured
    graph: every hour record and sun ray uploaded once, then per day the state
    reset (``src/series.py:425-436``) and the batched day
    (``solweig_day_batched_ex``).  Outputs [days * hours, rows, cols]."""

    def __init__(self, scene, latitude, longitude, site_altitude=3.0, utc=0.0, days=30, hours=24,
                 outputs=("tmrt", "utci"), config=None):
        self.scene = scene
        self.latitude, self.longitude, self.site_altitude, self.utc = latitude, longitude, site_altitude, utc
        self.days, self.hours = days, hours
        dev = scene.device
        self.state = {k: torch.zeros(scene.shape, dtype=torch.float32, device=dev)
                      for k in _lib.STATE_FIELDS}
        self.buffers = HourBuffers(scene, days * hours)
        self.layout_dev = scene.layout.device(dev)
        self.out_names = tuple(outputs)
        self.out = {k: torch.empty((days * hours,) + scene.shape, dtype=torch.float32, device=dev)
                    for k in self.out_names}
        self.work_bytes = int(_lib.lib().solweig_day_batched_work_bytes(scene.rows, scene.cols, hours,
                                                                        int(scene.struct.has_water)))
        self.work = torch.empty(self.work_bytes, dtype=torch.uint8, device=dev)
        clear_day_errors(self.work)
        self.config = config if config is not None else _lib.SolweigDayConfig.default()
        self.graph = None
        self.launches = day_launches(scene, self.config) * days

    def plan(self, met):
        met = np.asarray(met, dtype=np.float64)
        if len(met) != self.days * self.hours:
            raise ValueError(f"expected {self.days * self.hours} forcing rows, got {len(met)}")
        self.buffers.wait_free()
        H = self.hours
        for d in range(self.days):
            plan = plan_day(self.scene, met[d * H:(d + 1) * H], self.latitude, self.longitude,
                            self.site_altitude, self.utc)
            self.buffers.put_plan(plan, d * H)

    def _sequence(self):
        sc = self.scene
        L = _lib.lib()
        self.buffers.upload(0, self.days * self.hours, self.buffers.kmax)
        st = _lib.SolweigState()  # zero state at the start of every day
        hsize = self.buffers.hsize
        for d in range(self.days):
            base = outputs_struct(self.out, d * self.hours)
            hours_ptr = ctypes.c_void_p(self.buffers.h_dev.data_ptr() + d * self.hours * hsize)
            _lib.check(L.solweig_day_batched_ex(
                ctypes.byref(sc.struct), device_ptr(self.layout_dev), hours_ptr, self.hours,
                ctypes.byref(st), ctypes.byref(base), sc.pixels, sc.gvf_host_ptr, sc.first_steps,
                sc.second_steps, device_ptr(self.work), self.work_bytes, ctypes.byref(self.config),
                stream_handle()), "solweig_day_batched_ex")

    def capture(self):
        self._sequence()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            self._sequence()
        self.graph = g

    def replay(self):
        self.graph.replay()
        self.buffers.mark()
        return self.out

    def run(self, met):
        self.plan(met)
        if self.graph is None:
            self.capture()
        return self.replay()

    def check_errors(self):
        """Raise DayError if any day of any replay so far left invalid results."""
        return check_day_errors(self.work, "multi-day batch")


class TileBatch:
    """Independent tiles (own scene, latitude and forcing) for one day each,
    captured as ONE graph; a single work buffer sized for the largest tile is
    reused tile after tile on the stream.  Each tile may carry its own launch
    shapes (from :mod:`tune`)."""

    def __init__(self, scenes, latitudes, longitudes, site_altitude=3.0, utc=0.0, hours=24,
                 outputs=("tmrt", "utci"), configs=None):
        self.scenes = list(scenes)
        n = len(self.scenes)
        self.latitudes = list(latitudes)
        self.longitudes = list(longitudes)
        self.site_altitude, self.utc, self.hours = site_altitude, utc, hours
        dev = self.scenes[0].device
        L = _lib.lib()
        self.work_bytes = max(int(L.solweig_day_batched_work_bytes(s.rows, s.cols, hours,
                                                                   int(s.struct.has_water)))
                              for s in self.scenes)
        self.work = torch.empty(self.work_bytes, dtype=torch.uint8, device=dev)
        clear_day_errors(self.work)
        self.buffers = [HourBuffers(s, hours) for s in self.scenes]
        self.layouts = [s.layout.device(dev) for s in self.scenes]
        self.state = [{k: torch.zeros(s.shape, dtype=torch.float32, device=dev) for k in ("tgmap1", "tgout1")}
                      for s in self.scenes]
        self.out_names = tuple(outputs)
        self.out = [{k: torch.empty((hours,) + s.shape, dtype=torch.float32, device=dev) for k in outputs}
                    for s in self.scenes]
        self.configs = list(configs) if configs is not None else [_lib.SolweigDayConfig.default()] * n
        self.graph = None
        self.warm = False  # an eager day has run
        self.launches = sum(day_launches(s_, c) for s_, c in zip(self.scenes, self.configs))

    @property
    def pixels(self):
        return sum(s.pixels for s in self.scenes)

    def plan(self, mets):
        suns = []  # tiles of one case share their sun positions: (forcing times, lat, lon, SolarHours)
        for s, b, met, lat, lon in zip(self.scenes, self.buffers, mets, self.latitudes, self.longitudes):
            met = np.asarray(met, dtype=np.float64)
            if len(met) != self.hours:
                raise ValueError(f"expected {self.hours} forcing rows, got {len(met)}")
            for when, at, sol in suns:
                if at == (lat, lon) and np.array_equal(when, met[:, :4]):
                    break
            else:
                sol = _sun.metdata(met, lat, lon, self.site_altitude, self.utc)
                suns.append((met[:, :4], (lat, lon), sol))
            plan = plan_day(s, met, lat, lon, self.site_altitude, self.utc, sol)
            b.wait_free()
            b.put_plan(plan)

    def _sequence(self):
        L = _lib.lib()
        for s, b, lay, state, out, cfg in zip(self.scenes, self.buffers, self.layouts, self.state, self.out,
                                              self.configs):
            b.upload(0, self.hours, b.kmax)
            st = _lib.SolweigState()  # zero state at the start of the day
            base = outputs_struct(out, 0)
            _lib.check(L.solweig_day_batched_ex(
                ctypes.byref(s.struct), device_ptr(lay), b.ptr(), self.hours, ctypes.byref(st),
                ctypes.byref(base), s.pixels, s.gvf_host_ptr, s.first_steps, s.second_steps,
                device_ptr(self.work), self.work_bytes, ctypes.byref(cfg), stream_handle()),
                "solweig_day_batched_ex")

    def capture(self):
        if not self.warm:
            self._sequence()
            self.warm = True
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            self._sequence()
        self.graph = g

    def replay(self):
        self.graph.replay()
        for b in self.buffers:
            b.mark()
        return self.out

    def run(self, mets):
        """One day on every tile: eagerly the first time, then as one graph."""
        self.plan(mets)
        if self.graph is None and not self.warm:
            self._sequence()
            self.warm = True
            for b in self.buffers:
                b.mark()
            return self.out
        if self.graph is None:
            self.capture()
        return self.replay()

    def check_errors(self):
        """Raise DayError if any tile-day of any replay so far left invalid results."""
        return check_day_errors(self.work, "tile batch")
