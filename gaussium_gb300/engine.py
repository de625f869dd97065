"""Device-side ERI engine: shells and shell pairs in HBM, class-sorted quartet task lists,
and the launches of the sm_103a class kernels through the C ABI.

Layout in HBM (all owned by torch tensors):
  DeviceShells  per shell: centre[3] f64, l i32, prim_off i32, func_off i32, comp_scale[6] f64;
                per primitive: exponent f64, effective coefficient f64.
  PairSet       per shell pair a 48-byte PairRec (AB, primitive-pair range, shells, Schwarz
                bound); per primitive pair an 80-byte f64 record and a 48-byte f32 record
                (p, 1/2p, P, PA, Kp) -- see csrc/eri_common.cuh.
  tasks         write tasks (24 B: bra, ket, permutation code, output offset) or Fock
                tasks (8 B: bra, ket), grouped by angular-momentum class and sorted by
                primitive-quartet count, largest first (so a launch does not end on its
                longest blocks), equal primitive counts together (a warp's threads run
                the same loop trip counts).
"""
import ctypes
import functools

import numpy as np
import torch

from . import _lib
from .basis import COMPONENTS, ShellBasis

PAIR_ORDER = [(0, 0), (1, 0), (1, 1), (2, 0), (2, 1), (2, 2)]
PAIR_CLASS = {p: i for i, p in enumerate(PAIR_ORDER)}
NCART = np.array([1, 3, 6, 10])
PAIR_REC, PRIM64, PRIM32, WRITE_TASK = 48, 80, 48, 24
# Primitive pairs with alpha*beta/p |AB|^2 above this (Gaussian-product factor < 1e-24)
# are dropped by the pair builder when screening is on.
PRIM_SCREEN = 55.262
WRITE_TASK_DTYPE = np.dtype([("bra", "<i4"), ("ket", "<i4"), ("code", "<i4"), ("pad", "<i4"),
                             ("off", "<i8")])

# Quartets with many primitive quartets (after the pair screen) of a class that runs one
# thread per quartet run in the split form instead: one warp per quartet, its lanes taking
# the primitive quartets 32 at a time with the same straight-line code, then summing their
# contraction accumulators.  One thread walking them all would make the launch end on a
# few long-running warps.  "Many" is at least HEAVY_PRIM_QUARTETS and twice the class's
# accumulator count (the warp's final sum costs five additions per accumulator).
HEAVY_PRIM_QUARTETS = 32
# Quartets with at least COOP_PRIM_QUARTETS primitive quartets of a class that runs one
# warp per quartet run in the cooperative form: up to eight warps per quartet (as many as
# fit the shared memory), warp w taking primitive quartets w, w + warps, ..., the partial
# sums added in shared memory before one HRR.  The class's time would otherwise have a floor at its heaviest quartet,
# walked by one warp while the other warps of the launch have finished.
COOP_PRIM_QUARTETS = 128
THREAD_FORM, WARP_FORM, GROUPED_FORM, SPLIT_FORM, COOP_FORM, STACKED_FORM, CLUSTER_FORM = range(1, 8)
# (class, precision) pairs whose heavy quartets stay on the class's own form (set by the
# autotuner where that measured faster)
SPLIT_OFF = set()
# (class, precision): form, where the autotuner measured the launch plan (class_plan) faster than
# that form, the class's chosen one: unpartitioned calls follow the plan as long as the form stays
# chosen, mixed-precision builds the form (mixed_plan)
PLAN_ON = {}


@functools.lru_cache(maxsize=None)
def heavy_threshold(cls):
    """Primitive quartets from which a quartet of class ``cls`` is run in the split form."""
    la, lb, lc, ld = cls
    ne = sum((x + 1) * (x + 2) // 2 for x in range(la, la + lb + 1))
    nf = sum((x + 1) * (x + 2) // 2 for x in range(lc, lc + ld + 1))
    return max(HEAVY_PRIM_QUARTETS, 2 * ne * nf)

_pc_lut = np.full((3, 3), -1, dtype=np.int64)
for _i, (_a, _b) in enumerate(PAIR_ORDER):
    _pc_lut[_a, _b] = _i


def heavy_counts(cls, work_desc):
    """(split, cooperative): how many tasks of a segment whose primitive-quartet counts
    ``work_desc`` are sorted in descending order reach heavy_threshold(cls), and how many
    reach COOP_PRIM_QUARTETS -- both prefixes of the segment."""
    w = -np.asarray(work_desc, dtype=np.int64)
    return (int(np.searchsorted(w, -heavy_threshold(cls), side="right")),
            int(np.searchsorted(w, -COOP_PRIM_QUARTETS, side="right")))


def split_forms(cls, precision, heavy):
    """[(form, first, count)] for a class segment whose tasks are sorted by descending
    primitive-quartet count, with heavy = heavy_counts(cls, ...): the heavy prefix in the
    split form when the class runs one thread per quartet, in the cooperative form when it
    runs one warp per quartet, the rest in the class's form.  form 0 = the class's
    configured form; count None = to the end of the segment."""
    if (cls, precision) in SPLIT_OFF:
        return [(0, 0, None)]
    form = _lib.lib().gs_class_form(*cls, precision)
    if form == THREAD_FORM:
        h, hform = heavy[0], SPLIT_FORM
    elif form in (WARP_FORM, GROUPED_FORM, STACKED_FORM):
        h, hform = heavy[1], COOP_FORM
    else:
        h, hform = 0, 0
    if h <= 0:
        return [(0, 0, None)]
    return [(hform, 0, h), (form, h, None)]


# ---------------------------------------------------------------------- launch plans
# Times here are in slots of 64 cycles, what a warp-wide FP64 instruction holds its scheduler's
# pipe for (measured: the same for one warp as for four, so a scheduler has no more FP64
# throughput than one busy warp uses).
WORK_LEVELS = 18          # thresholds 1, 2, 4, ... 2^17 of a work profile
# quartets of fewer than 2^MANY_LEVEL primitive quartets share a warp's set-up, MANY_TASKS at
# most, in classes up to total angular momentum MANY_LMAX (csrc/eri_wide.cuh)
MANY_LEVEL, MANY_TASKS, MANY_LMAX = 4, 8, 6
# and as long as this many warps a scheduler remain: block writing brings up to 15 primitive
# quartets a quartet, the adjoint and Fock digestion of molecules one to five ((H2O)6/6-31G*
# gradient 10.4 ms with 4, 10.9 with 16; 300,000 random quartets' blocks 12.9 and 12.7)
MANY_WARPS = {"jk": 4, "write": 16}
COOP_LEVEL = COOP_PRIM_QUARTETS.bit_length() - 1     # one warp alone takes fewer than that
_LEVELS = 1 << np.arange(WORK_LEVELS, dtype=np.int64)
KEY_STEP = 1 << 57        # more than any quartet's primitive quartets; times 36 classes within int64
SEARCH_AT_ONCE = 1 << 20  # tasks
MIN_LATENCY = 600.0       # slots (20 us) below which a long quartet is not worth splitting
LATENCY_SHARE = 0.15      # of a call's whole work that one lane or warp may take alone
# and of a call's own work where it is for some of the classes only, in FP64: 21 classes of 300,000
# random quartets' blocks one by one 13.4 ms (1: 13.3, 4: 13.9, without: 18.4), of 2,000,000 71.2
# (69.9, 74.5, 86.7), Fock classes of (H2O)8 6.1 ms (6.7, 6.2, 6.2).  FP32's estimate of the work is
# too low for it (its kernels are not bound by their pipe).
ALONE_SHARE = 2.0


def work_profile(work_desc):
    """(sum, counts) of a segment's primitive-quartet counts, sorted in descending order:
    counts[k] tasks have at least 2^k."""
    w = -np.asarray(work_desc, dtype=np.int64)
    return -int(w.sum()), np.searchsorted(w, -_LEVELS, side="right").tolist()


def segment_profiles(cls_list, work_desc, bounds):
    """(heavy_counts, work_profile) of every segment [bounds[i], bounds[i+1]) of a device
    tensor of primitive-quartet counts, descending within each segment, in one transfer.  Up to
    SEARCH_AT_ONCE tasks one search finds every segment's thresholds: segment i's counts, negated
    and moved up by i times KEY_STEP, are one ascending list.  Longer lists go segment by segment,
    without copies of the whole (device planning of 4,096 quartets 2.4 ms, segment by segment 3.9;
    the task lists of (H2O)24 31.7 and, in one search, 36.5)."""
    dev = work_desc.device
    n = len(cls_list)
    if n == 0:
        return []
    first = np.asarray(bounds, dtype=np.int64)
    levels = np.array([[heavy_threshold(c), COOP_PRIM_QUARTETS, *_LEVELS.tolist()] for c in cls_list],
                      dtype=np.int64)
    step = np.arange(n, dtype=np.int64) * KEY_STEP
    w = work_desc[int(first[0]):int(first[-1])]
    if w.numel() > SEARCH_AT_ONCE:
        (query,) = upload(dev, -levels)
        parts = [work_desc[s:e] for s, e in zip(bounds[:-1], bounds[1:])]
        found = torch.stack([torch.searchsorted(-x, q, right=True) for x, q in zip(parts, query)])
        total = torch.stack([x.sum() for x in parts])
    else:
        at, length, query = upload(dev, first - first[0], np.diff(first), step[:, None] - levels)
        key = torch.repeat_interleave(torch.arange(n, device=dev) * KEY_STEP, length,
                                      output_size=w.numel()) - w
        found = torch.searchsorted(key, query, right=True) - at[:-1, None]
        upto = torch.cat([w.new_zeros(1), torch.cumsum(w, 0)])
        total = upto[at[1:]] - upto[at[:-1]]
    rows = torch.cat([total[:, None], found], 1).tolist()
    return [((r[1], r[2]), (r[0], r[3:])) for r in rows]


@functools.lru_cache(maxsize=None)
def class_sizes(cls):
    """(accumulators of the [e0|f0] set, integrals of a block)."""
    la, lb, lc, ld = cls
    ne = sum((x + 1) * (x + 2) // 2 for x in range(la, la + lb + 1))
    nf = sum((x + 1) * (x + 2) // 2 for x in range(lc, lc + ld + 1))
    return ne * nf, int(np.prod(NCART[list(cls)]))


@functools.lru_cache(maxsize=None)
def class_costs(cls, precision):
    """Slots per primitive quartet: of a lane in a full GPU, of a lone warp of the thread form
    (whose spills nothing hides), and of a warp of the warp forms.  The vertical recursion
    has about 11 operations per accumulator; the set-up and Boys function about 50."""
    n = class_sizes(cls)[0]
    if precision == 64:
        lane = 50 + 7.0 * n
        return lane, lane * min(3.0, 1.5 + n / 24), 10 + 0.3 * n
    return (100 + 12.0 * n) / 64, 30 + n * (0.5 if n <= 256 else 1.25), 10 + 0.1 * n


def total_slots(segments, profiles, precision, kind, schedulers):
    """Slots of a whole call on every scheduler of the GPU, all lanes busy."""
    t = 0.0
    for (cls, s, e), (work, _) in zip(segments, profiles):
        per = (40 + 6 * class_sizes(cls)[1]) if kind == "jk" else (10 + 3 * class_sizes(cls)[1])
        t += work * class_costs(cls, precision)[0] + (e - s) * per / (1 if precision == 64 else 30)
    return t / (32 * schedulers)


def class_plan(cls, precision, kind, n, profile, limit, built, schedulers=608):
    """[(form, first, count, latency)] for a class segment of n tasks sorted by descending
    primitive-quartet count w, when no form has been chosen for the class.  Tasks of a tier
    take at most ``limit`` slots in its form, so that no lane, warp or block walks its
    primitive quartets while the rest of the GPU has finished; ``latency`` is the tier's
    longest task's.  The lightest tier runs one thread per quartet where the class's
    accumulators allow it, else one warp per quartet (several quartets of few primitive
    quartets: form | per << 8); heavier ones a warp (thread code, or the warp forms), a block
    of eight warps, and a cluster of eight blocks per quartet.  Thresholds are powers of two
    (the profile's)."""
    nacc = class_sizes(cls)[0]
    lane, alone, warp = class_costs(cls, precision)
    has = lambda form: bool(built & (1 << (form - 1)))   # noqa: E731
    most = (496 if precision == 32 else 96 if cls[3] == 0 else 54) if kind == "jk" else \
        (96 if precision == 32 else 27)
    # (form, slots per primitive quartet, fixed slots, largest level), lightest tier first
    tiers = []
    if has(THREAD_FORM) and nacc <= most:
        tiers.append((THREAD_FORM, alone, 0.0, WORK_LEVELS))
        if nacc <= 27:
            tiers.append((SPLIT_FORM, alone / 32, 10.0 * nacc, WORK_LEVELS))
    if not tiers or nacc > 27:
        for form in ((GROUPED_FORM,) if nacc <= 96 else ()) + (STACKED_FORM, WARP_FORM):
            if has(form):
                if sum(cls) <= MANY_LMAX:
                    # several light quartets a warp, as long as enough warps remain
                    per = min(MANY_TASKS, n // (MANY_WARPS[kind] * schedulers))
                    if per > 1:
                        tiers.append((form | (per << 8), per * warp, 0.0, MANY_LEVEL))
                tiers.append((form, warp, 0.0, COOP_LEVEL))
                break
        if has(COOP_FORM):
            tiers.append((COOP_FORM, warp / 4, 0.0, WORK_LEVELS))
        if has(CLUSTER_FORM):
            tiers.append((CLUSTER_FORM, warp / 32, 0.0, WORK_LEVELS))
    if not tiers:
        return [(0, 0, n, 0.0)]
    counts = profile[1]
    top = max([k for k in range(WORK_LEVELS) if counts[k]], default=0)    # w < 2^(top+1)
    out, end = [], n
    for i, (form, slots, fixed, most) in enumerate(tiers):
        if i + 1 == len(tiers):
            k = WORK_LEVELS
        else:
            k = min(most, max(1, int(np.floor(np.log2(max(2.0, limit / slots))))))
        first = counts[k] if k < WORK_LEVELS else 0
        if first < end:
            out.append((form, first, end - first, fixed + slots * 2.0 ** min(k, top + 1)))
            end = first
    return out[::-1]


def launch_plan(engine_like, precision, kind, classes=None, share=1.0):
    """[(class, first task, count, form, latency)] of one call, longest latency first: the
    launches go to several streams, so the few long blocks run beside the rest.  Classes
    with a chosen form (gs_set_class_variant, the autotuner) follow split_forms, unless the
    autotuner left them to the plan (PLAN_ON)."""
    e = engine_like
    L = _lib.lib()
    key = (precision, kind)
    plans = e.__dict__.setdefault("_plans", {})
    if key not in plans:
        sch = 4 * torch.cuda.get_device_properties(e.tasks.device).multi_processor_count
        slots = {p: total_slots(e.segments, e.profiles, p, kind, sch) for p in (64, 32)}
        plans[key] = (slots, sch, {})
    slots, sch, cached = plans[key]
    limit = max(MIN_LATENCY, LATENCY_SHARE * share * slots[precision])
    if classes is not None and share == 1.0 and precision == 64:
        # a call for some classes alone: nothing runs beside their long tiers
        mine = [(seg, prof) for seg, prof in zip(e.segments, e.profiles) if seg[0] in classes]
        alone = total_slots(*zip(*mine), precision, kind, sch) if mine else 0.0
        limit = min(limit, max(MIN_LATENCY, ALONE_SHARE * alone))
    out = []
    for (cls, s, t), heavy, prof in zip(e.segments, e.heavy, e.profiles):
        if classes is not None and cls not in classes:
            continue
        variant = L.gs_class_variant(*cls, precision)
        if (variant or (cls, precision) in SPLIT_OFF) and PLAN_ON.get((cls, precision)) != variant:
            parts = [(form, first, (t - s - first) if count is None else count,
                      float("inf") if count is not None else 0.0)
                     for form, first, count in split_forms(cls, precision, heavy)]
        else:
            if (cls, limit) not in cached:
                cached[cls, limit] = class_plan(cls, precision, kind, t - s, prof, limit,
                                                L.gs_class_variants(*cls, precision), sch)
            parts = cached[cls, limit]
        out += [(cls, s + first, count, form, lat) for form, first, count, lat in parts if count > 0]
    return sorted(out, key=lambda x: -x[4])


def mixed_plan(engine_like, classes, mixed_cut):
    """(banded, tiers) of a mixed-precision build.  banded: [(class, first task, precision,
    form, count, lo, hi)], the heavy prefixes (mixed_prefix) of the classes whose form was
    chosen.  tiers: [(class, first task, count, form64, form32)], longest latency first, for
    one partitioned launch each: a class segment cut wherever either precision's plan
    (class_plan) changes its form.  Where the engine has a ``heavy_bound``, the quartets of the
    heavy prefix, which were banded with it before they were partitioned, keep that bound: the
    segment is cut there too, and their tiers' sixth entry is the bound's offset (24 molecules in
    one batch: 11.9 ms with it, 11.4 with the block bound, under which the Fock matrices' error
    against FP64 grew by 4 to 10 %)."""
    e = engine_like
    L = _lib.lib()
    bound = getattr(e, "heavy_bound", 0)
    banded, tiers = [], []
    for (cls, s, t), heavy in zip(e.segments, e.heavy):
        if classes is not None and cls not in classes:
            continue
        if any(L.gs_class_variant(*cls, p) or (cls, p) in SPLIT_OFF for p in (64, 32)):
            h, launches = mixed_prefix(cls, heavy, mixed_cut)
            banded += [(cls, s + first, p, form, n, lo, hi) for p, form, first, n, lo, hi in launches]
            if s + h < t:
                tiers.append((0.0, cls, s + h, t - s - h, 0, 0))
            continue
        plans = [launch_plan(e, p, "jk", [cls], 0.5) for p in (64, 32)]
        cuts = sorted({first for plan in plans for _, first, _, _, _ in plan} | {t} |
                      ({s + max(heavy)} if bound else set()))
        for x, y in zip(cuts[:-1], cuts[1:]):
            (f64, l64), (f32, l32) = [next((form, lat) for _, first, n, form, lat in plan
                                           if first <= x < first + n) for plan in plans]
            tiers.append((max(l64, l32), cls, x, y - x, f64, f32) +
                         ((bound,) if bound and x < s + max(heavy) else ()))
    tiers.sort(key=lambda x: -x[0])
    return banded, [x[1:] for x in tiers]


LAUNCH_DTYPE = np.dtype([("cls", "<i4", 4), ("form", "<i4"), ("form32", "<i4"), ("count", "<i4"),
                         ("bound", "<i4"), ("first", "<i8")])


def launch_records(launches):
    """[(class, first task, count, form, FP32 form)], or with a bound's offset as sixth entry, as
    the records of the list calls."""
    out = np.zeros(len(launches), dtype=LAUNCH_DTYPE)
    for r, (cls, first, count, form, form32, *bound) in zip(out, launches):
        r["cls"], r["first"], r["count"], r["form"], r["form32"] = cls, first, count, form, form32
        r["bound"] = bound[0] if bound else 0
    return out


def kept_plan(engine_like, key, build, *more):
    """``build()``, kept on the engine under ``key`` until a class's form is chosen anew (or
    ``more`` changes): task segments, profiles and the device are the engine's for good."""
    stamp = (_lib.lib().gs_class_variant_stamp(), frozenset(SPLIT_OFF), frozenset(PLAN_ON.items()),
             *more)
    kept = engine_like.__dict__.setdefault("_kept_plans", {})
    if key not in kept or kept[key][0] != stamp:
        kept[key] = (stamp, build())
    return kept[key][1]


def launch_list(engine_like, precision, kind, classes=None):
    """launch_plan as the records of a list call."""
    key = (precision, kind, None if classes is None else tuple(classes))
    return kept_plan(engine_like, key, lambda: launch_records(
        [(cls, first, n, form, 0) for cls, first, n, form, _ in
         launch_plan(engine_like, precision, kind, classes)]))


def mixed_list(engine_like, classes, mixed_cut):
    """mixed_plan with the tiers as the records of a list call."""
    key = ("mixed", None if classes is None else tuple(classes))

    def build():
        banded, tiers = mixed_plan(engine_like, classes, mixed_cut)
        return banded, launch_records(tiers)
    return kept_plan(engine_like, key, build, mixed_cut)


def mixed_prefix(cls, heavy, mixed_cut):
    """The heavy prefix of a class segment in a mixed-precision build, whose partitioned
    launch (gs_fock_jk_mixed) evaluates every quartet in the class's configured form.
    Returns (h, [(precision, form, first, count, prec_lo, prec_hi)]): tasks [0, h) run as
    banded launches -- FP64 for density-weighted bounds at or above ``mixed_cut``, FP32
    below, the same bands as the partition -- each precision's heavy tasks in its heavy
    form (split_forms) and the rest of the prefix in its configured form; the partitioned
    launch takes [h, end).  (0, []) when neither precision has a heavy form here."""
    parts = {p: split_forms(cls, p, heavy) for p in (64, 32)}
    h = max((pp[0][2] for pp in parts.values() if len(pp) > 1), default=0)
    if h == 0:
        return 0, []
    out = []
    for p, lo, hi in ((64, mixed_cut, float("inf")), (32, 0.0, mixed_cut)):
        pp = parts[p]
        c = pp[0][2] if len(pp) > 1 else 0
        if c > 0:
            out.append((p, pp[0][0], 0, c, lo, hi))
        if c < h:
            out.append((p, 0, c, h - c, lo, hi))
    return h, out


# Eight streams with the caller's, the hardware queues of a default context (CUDA_DEVICE_MAX_
# CONNECTIONS): 4,096 random cc-pVTZ-shaped quartets 831 us with four streams, 695 with six, 594
# with eight, 587 with twelve, which share queues; the unrestricted build of one (H2O)7 geometry
# 3.15, 3.06, 2.99, 2.99 ms (others take up to 4.4).
SIDE_STREAMS = 7
_SIDE = {}


class HeavyLane:
    """Side streams of a build, forked from the caller's stream before their first launch
    and joined back by ``join`` or at the end of a ``with``, also where a launch raised: the
    buffers of what runs on a side are free for others' use only behind it.  A build's launches go round the caller's stream and the
    sides (``lane``): the few long blocks of the heavy tiers then run beside the class
    launches instead of leaving most SMs idle while they finish, and one class's last
    partial wave overlaps the next class's first."""

    def __init__(self, device, stream=None):
        d = indexed_device(device)
        self.main = stream or torch.cuda.current_stream(d)
        if d not in _SIDE:
            _SIDE[d] = tuple(torch.cuda.Stream(device=d) for _ in range(SIDE_STREAMS))
        self.sides = _SIDE[d]
        self.forked = [False] * SIDE_STREAMS

    def stream(self, k=0):
        """Side stream k (as the C ABI takes it), forked on first use."""
        if not self.forked[k]:
            self.sides[k].wait_stream(self.main)
            self.forked[k] = True
        return _lib.stream(self.sides[k])

    def lane(self, i, lanes=SIDE_STREAMS + 1):
        """The stream of the i-th launch of a build over ``lanes`` streams.  The caller's
        stream comes last: a side forks behind whatever the caller's stream holds by then, and
        behind the longest launch of a build the others would wait for its few last blocks
        ((H2O)24 mixed 16.3 -> 15.0 ms, one batch of 24 molecules 14.6 -> 14.1)."""
        i %= lanes
        return _lib.stream(self.main) if i == lanes - 1 else self.stream(i)

    def streams(self, lanes=SIDE_STREAMS + 1):
        """(count, handles) of a list call's streams, which forks and joins them itself."""
        handles = [x.cuda_stream for x in self.sides[:lanes - 1]] + [self.main.cuda_stream]
        return lanes, (ctypes.c_void_p * lanes)(*handles)

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.join()

    def join(self):
        for k in range(SIDE_STREAMS):
            if self.forked[k]:
                self.main.wait_stream(self.sides[k])
                self.forked[k] = False


def check_record_sizes(lib=None):
    """The library's pair, primitive-pair and task record sizes (``gs_record_sizes``, a host
    call) must equal the layouts this module packs; raises GsError on a mismatch."""
    sizes = np.zeros(4, dtype=np.int32)
    _lib.check((lib or _lib.lib()).gs_record_sizes(sizes.ctypes.data), "gs_record_sizes")
    if tuple(int(x) for x in sizes) != (PAIR_REC, PRIM64, PRIM32, WRITE_TASK):
        raise _lib.GsError(f"record sizes mismatch: library {tuple(sizes)}, host "
                           f"{(PAIR_REC, PRIM64, PRIM32, WRITE_TASK)}")


def indexed_device(device):
    """The device with its index made explicit ('cuda' -> 'cuda:<current>'), so that a
    comparison with a tensor's device is exact."""
    d = torch.device(device)
    if d.type == "cuda" and d.index is None:
        d = torch.device("cuda", torch.cuda.current_device())
    return d


def _check_device_tensor(t, device, what, shape=None):
    """Tensors handed to a kernel must be float64 on the engine's CUDA device (a host
    pointer or a float32 buffer would be read as the wrong memory, a tensor on another
    GPU as another device's memory)."""
    if not isinstance(t, torch.Tensor) or not t.is_cuda or t.dtype != torch.float64:
        raise _lib.GsError(f"{what} must be a float64 CUDA tensor")
    if t.device != indexed_device(device):
        raise _lib.GsError(f"{what} is on {t.device}, the engine on {indexed_device(device)}")
    if shape is not None and tuple(t.shape) != tuple(shape):
        raise ValueError(f"{what} has shape {tuple(t.shape)}, expected {tuple(shape)}")
    if shape is None and not t.is_contiguous():
        raise ValueError(f"{what} must be contiguous")


PACK_BYTES = 1 << 20


def upload(device, *arrays):
    """numpy arrays as tensors on the device.  Small sets travel as one block, of which the
    tensors are views (a copy from pageable memory costs 10 us or more whatever its size)."""
    arrays = [np.ascontiguousarray(a) for a in arrays]
    offs, total = [], 0
    for a in arrays:
        offs.append(total)
        total += -(-a.nbytes // 256) * 256
    if len(arrays) < 2 or total > PACK_BYTES:
        return [torch.as_tensor(a).to(device) for a in arrays]
    block = np.zeros(total, dtype=np.uint8)
    for a, o in zip(arrays, offs):
        block[o:o + a.nbytes] = a.reshape(-1).view(np.uint8)
    dev = torch.from_numpy(block).to(device)
    typed, out = {}, []
    for a, o in zip(arrays, offs):
        if a.dtype not in typed:
            typed[a.dtype] = dev.view(torch.from_numpy(np.empty(0, a.dtype)).dtype)
        strides = [x // a.itemsize for x in a.strides]
        out.append(typed[a.dtype].as_strided(a.shape, strides, o // a.itemsize))
    return out


class DeviceShells:
    """A ShellBasis copied to the device."""

    def __init__(self, sb: ShellBasis, device="cuda"):
        self.host = sb
        self.device = indexed_device(device)

        # nprim: primitives per shell (device planning)
        (self.centre, self.l, self.prim_off, self.expo, self.coef, self.comp_scale, self.func_off,
         self.nprim) = upload(
            self.device, sb.centre.astype(np.float64, copy=False), sb.l.astype(np.int32, copy=False),
            sb.prim_off.astype(np.int32, copy=False), sb.expo.astype(np.float64, copy=False),
            sb.coef.astype(np.float64, copy=False), sb.comp_scale.astype(np.float64, copy=False),
            sb.func_off.astype(np.int32, copy=False), sb.nprim.astype(np.int64))
        self.nshell = sb.nshell
        self.nbf = sb.nbf


def pair_groups(sizes, lanes=32):
    """Start indices (and the end) of groups of consecutive shell pairs whose primitive
    pairs total at most ``lanes``: aligned runs of four pairs when they fit, else of two,
    else single pairs (vectorised; a pair with more primitive pairs is a group of its own)."""
    sizes = np.asarray(sizes, dtype=np.int64)
    n = len(sizes)
    if n == 0:
        return np.zeros(1, dtype=np.int32)
    m = -(-n // 4) * 4
    sz = np.zeros(m, dtype=np.int64)
    sz[:n] = sizes
    quad = np.repeat(sz.reshape(-1, 4).sum(1) <= lanes, 4)
    half = np.repeat(sz.reshape(-1, 2).sum(1) <= lanes, 2)
    r = np.tile(np.arange(4), m // 4)
    start = (r == 0) | ((r == 2) & ~quad) | ((r & 1).astype(bool) & ~quad & ~half)
    out = np.flatnonzero(start[:n]).astype(np.int32)
    return np.concatenate([out, np.array([n], dtype=np.int32)])


def pair_groups_device(sizes, lanes=32):
    """pair_groups on a device tensor of sizes (the same groups; int32 device tensor)."""
    dev = sizes.device
    n = sizes.numel()
    if n == 0:
        return torch.zeros(1, dtype=torch.int32, device=dev)
    m = -(-n // 4) * 4
    sz = torch.zeros(m, dtype=torch.int64, device=dev)
    sz[:n] = sizes
    quad = (sz.view(-1, 4).sum(1) <= lanes).repeat_interleave(4)
    half = (sz.view(-1, 2).sum(1) <= lanes).repeat_interleave(2)
    r = torch.arange(m, device=dev) % 4
    start = (r == 0) | ((r == 2) & ~quad) | (((r & 1) == 1) & ~quad & ~half)
    out = torch.nonzero(start[:n]).flatten().to(torch.int32)
    return torch.cat([out, torch.tensor([n], dtype=torch.int32, device=dev)])


def check_shell_indices(idx, nshell, what):
    """Shell indices handed to the kernels must lie in [0, nshell): a kernel trusts them."""
    idx = np.asarray(idx)
    if idx.size and (int(idx.min()) < 0 or int(idx.max()) >= nshell):
        raise ValueError(f"{what} hold a shell index outside [0, {nshell})")


class PairSet:
    """Shell pairs (la >= lb inside each pair) with their primitive-pair records."""

    def __init__(self, ds: DeviceShells, pair_shells, want32=True, stream=None, max_exp=0.0,
                 count=True):
        """``count=False``: leave the kept primitive pairs per pair on the device (``nprim`` then
        holds all of them)."""
        ps = np.ascontiguousarray(pair_shells, dtype=np.int32).reshape(-1, 2)
        sb = ds.host
        check_shell_indices(ps, sb.nshell, "shell pairs")
        if len(ps) and np.any(sb.l[ps[:, 0]] < sb.l[ps[:, 1]]):
            raise ValueError("pair shells must have l[first] >= l[second]")
        npp = sb.nprim[ps[:, 0]].astype(np.int64) * sb.nprim[ps[:, 1]]
        off = np.zeros(len(ps) + 1, dtype=np.int64)
        off[1:] = np.cumsum(npp)
        if off[-1] >= 2 ** 31:
            raise ValueError("too many primitive pairs for one PairSet")
        self.ds = ds
        self.n = len(ps)
        self.host_shells = ps
        self.nprim = npp
        self.la = sb.l[ps[:, 0]] if len(ps) else np.zeros(0, np.int32)
        self.lb = sb.l[ps[:, 1]] if len(ps) else np.zeros(0, np.int32)
        dev = ds.device
        # groups: consecutive pairs packed into warps of at most 32 primitive pairs (the build)
        self.shells, self.prim_start, self.groups = upload(dev, ps, off[:-1].astype(np.int32),
                                                           pair_groups(npp))
        self.rec = torch.empty(max(1, self.n) * PAIR_REC, dtype=torch.uint8, device=dev)
        total = max(1, int(off[-1]))
        self.p64 = torch.empty(total * PRIM64, dtype=torch.uint8, device=dev)
        self.p32 = torch.empty(total * PRIM32, dtype=torch.uint8, device=dev) if want32 else None
        self.nprim_pairs = int(off[-1])
        self.max_exp = max_exp
        self.ngroups = int(self.groups.numel()) - 1
        self.kept = torch.zeros(max(1, self.n), dtype=torch.int32, device=dev)
        self.build(stream)
        # primitive pairs kept per shell pair (the work per pair after screening)
        if count:
            self.nprim = self.kept[:self.n].cpu().numpy().astype(np.int64)

    def build(self, stream=None, want32=True):
        """(Re)compute the pair records (kernel K0) from the device shells; with
        ``want32=False`` only the FP64 records (enough for FP64-only evaluation)."""
        ds = self.ds
        L = _lib.lib()
        p32 = self.p32 if want32 else None
        _lib.check(L.gs_pairs_build(_lib.ptr(ds.centre), _lib.ptr(ds.l), _lib.ptr(ds.prim_off),
                                    _lib.ptr(ds.expo), _lib.ptr(ds.coef), self.n,
                                    _lib.ptr(self.shells), _lib.ptr(self.prim_start),
                                    _lib.ptr(self.rec), _lib.ptr(self.p64), _lib.ptr(p32),
                                    float(self.max_exp), _lib.ptr(self.kept), self.ngroups,
                                    _lib.ptr(self.groups), _lib.stream(stream)), "gs_pairs_build")

    def prims(self, precision):
        return self.p64 if precision == 64 else self.p32


class DevicePairSet(PairSet):
    """A PairSet planned on the device from a device tensor of shell pairs (m, 2) int32,
    l[first] >= l[second] (as canonical quartets give them): the same records, groups and
    kept counts; the host copies of the pair list and counts are made when first read."""

    def __init__(self, ds: DeviceShells, pair_shells, want32=True, stream=None, max_exp=0.0):
        dev = ds.device
        ps = pair_shells.to(device=dev, dtype=torch.int32).reshape(-1, 2).contiguous()
        m = ps.shape[0]
        npp = ds.nprim[ps[:, 0].long()] * ds.nprim[ps[:, 1].long()]
        off = torch.cumsum(npp, 0)
        total = int(off[-1]) if m else 0
        if total >= 2 ** 31:
            raise ValueError("too many primitive pairs for one PairSet")
        self.ds = ds
        self.n = m
        self.shells = ps
        self.prim_start = (off - npp).to(torch.int32)
        self.rec = torch.empty(max(1, m) * PAIR_REC, dtype=torch.uint8, device=dev)
        t = max(1, total)
        self.p64 = torch.empty(t * PRIM64, dtype=torch.uint8, device=dev)
        self.p32 = torch.empty(t * PRIM32, dtype=torch.uint8, device=dev) if want32 else None
        self.nprim_pairs = total
        self.max_exp = max_exp
        self.groups = pair_groups_device(npp, 32)
        self.ngroups = int(self.groups.numel()) - 1
        self.kept = torch.zeros(max(1, m), dtype=torch.int32, device=dev)
        self.build(stream)
        self.nprim_dev = self.kept[:m].long()

    def __getattr__(self, name):
        # host copies, made on first use
        if name == "host_shells":
            v = self.shells.cpu().numpy()
        elif name == "nprim":
            v = self.nprim_dev.cpu().numpy()
        elif name in ("la", "lb"):
            k = 0 if name == "la" else 1
            v = self.ds.host.l[self.shells[:, k].cpu().numpy()]
        else:
            raise AttributeError(name)
        setattr(self, name, v)
        return v


_DEVICE_LUTS = {}


def _device_luts(dev):
    """The canonicalisation and block-size tables on a device."""
    if dev not in _DEVICE_LUTS:
        pos, code, pcb, pck = _CANON_LUT
        _DEVICE_LUTS[dev] = {
            "pos": torch.as_tensor(np.asarray(pos, dtype=np.int64)).to(dev),
            "code": torch.as_tensor(np.asarray(code, dtype=np.int32)).to(dev),
            "cls": torch.as_tensor(np.asarray(pcb * 6 + pck, dtype=np.int64)).to(dev),
            "size": torch.as_tensor(np.asarray(_SIZE_LUT, dtype=np.int64)).to(dev),
        }
    return _DEVICE_LUTS[dev]


# ---------------------------------------------------------------------- shell-quartet blocks
def _canonicalize_rows(l4):
    """canonicalize, evaluated row by row from the rule (the table below is built from it)."""
    la, lb, lc, ld = l4[:, 0], l4[:, 1], l4[:, 2], l4[:, 3]
    s_ab = la < lb
    s_cd = lc < ld
    A = np.where(s_ab, 1, 0); B = 1 - A
    C = np.where(s_cd, 3, 2); Dd = 5 - C
    pc1 = _pc_lut[np.maximum(la, lb), np.minimum(la, lb)]
    pc2 = _pc_lut[np.maximum(lc, ld), np.minimum(lc, ld)]
    s_bk = pc2 > pc1
    code = np.where(s_bk, s_cd.astype(np.int32) | (s_ab.astype(np.int32) << 1) | 4,
                    s_ab.astype(np.int32) | (s_cd.astype(np.int32) << 1))
    pos = np.stack([np.where(s_bk, C, A), np.where(s_bk, Dd, B),
                    np.where(s_bk, A, C), np.where(s_bk, B, Dd)], axis=1)
    return pos, code.astype(np.int32), np.where(s_bk, pc2, pc1), np.where(s_bk, pc1, pc2)


# canonicalize's results and the block size for each of the 81 (la, lb, lc, ld) with l <= 2,
# indexed by ((la*3 + lb)*3 + lc)*3 + ld: a gather per quartet instead of a dozen
# elementwise passes over the batch
_L4_ALL = np.array([[a, b, c, d] for a in range(3) for b in range(3) for c in range(3)
                    for d in range(3)], dtype=np.int64)
_CANON_LUT = _canonicalize_rows(_L4_ALL)
_SIZE_LUT = np.prod(NCART[_L4_ALL], axis=1)


def _l4_index(l4):
    l4 = np.asarray(l4, dtype=np.int64)
    return ((l4[:, 0] * 3 + l4[:, 1]) * 3 + l4[:, 2]) * 3 + l4[:, 3]


def canonicalize(l4):
    """Per quartet of angular momenta (n,4): canonical order (bra pair class >= ket pair
    class, la >= lb, lc >= ld), the 3-bit permutation code, and index maps."""
    i = _l4_index(l4)
    pos, code, pcb, pck = _CANON_LUT
    return pos[i], code[i], pcb[i], pck[i]


class QuartetBatch:
    """A batch of shell quartets (n,4 shell indices, any order) evaluated into one flat f64
    buffer: quartet q's block occupies out[off[q] : off[q] + na*nb*nc*nd] in the caller's
    (a,b,c,d) order, row-major.  Host preparation sorts the quartets by class and
    primitive counts; ``run`` launches one kernel per class."""

    def __init__(self, ds: DeviceShells, quartets, want32=True, max_exp=0.0, plan="host"):
        """``plan="device"``: the same planning with torch on the device (quartets may be a
        host array or a device tensor); only the class histogram and heavy counts come back
        to the host, and the host copies of offsets and primitive counts are made when
        first read."""
        if plan == "device":
            self._plan_device(ds, quartets, want32, max_exp)
            return
        if plan != "host":
            raise ValueError(f"plan must be 'host' or 'device', not {plan!r}")
        q = np.ascontiguousarray(quartets, dtype=np.int64).reshape(-1, 4)
        sb = ds.host
        check_shell_indices(q, sb.nshell, "shell quartets")
        n = len(q)
        l4 = sb.l[q]
        li = _l4_index(l4)
        pos, code, pcb, pck = (x[li] for x in _CANON_LUT)
        qc = np.take_along_axis(q, pos, axis=1)          # canonical shells
        size = _SIZE_LUT[li]
        off = np.zeros(n + 1, dtype=np.int64)
        off[1:] = np.cumsum(size)
        self.n = n
        self.offsets = off
        self.total = int(off[-1])
        pairs = np.concatenate([qc[:, 0:2], qc[:, 2:4]], axis=0)
        self.pairs = PairSet(ds, pairs, want32=want32, max_exp=max_exp)
        self.full_prim_quartets = int(np.sum(sb.nprim[qc[:, 0]].astype(np.int64) * sb.nprim[qc[:, 1]] *
                                             sb.nprim[qc[:, 2]] * sb.nprim[qc[:, 3]]))
        nb = self.pairs.nprim[:n]
        nk = self.pairs.nprim[n:]
        cls = pcb * 6 + pck
        # within a class, most primitive quartets first (the longest blocks start first, so
        # the short ones fill the end of the launch), equal (K_bra, K_ket) kept together so
        # that the lanes of a warp run the same loop trip counts: one packed key (class,
        # then descending nb*nk, nb, nk) and a stable sort, the order of a lexsort on the four
        wb = int(nb.max()).bit_length() if n else 1
        wk = int(nk.max()).bit_length() if n else 1
        ww = int((nb * nk).max()).bit_length() if n else 1
        key = cls.astype(np.int64)
        key = (key << ww) | ((1 << ww) - 1 - nb * nk)
        key = (key << wb) | ((1 << wb) - 1 - nb)
        key = (key << wk) | ((1 << wk) - 1 - nk)
        wi = int(n).bit_length()
        if 6 + ww + wb + wk + wi <= 62:
            # the index as the last key field makes every key distinct: a plain value sort
            # gives the stable order (and is faster than a stable argsort)
            order = np.sort((key << wi) | np.arange(n, dtype=np.int64)) & ((1 << wi) - 1)
        else:
            order = np.argsort(key, kind="stable")
        tasks = np.zeros(n, dtype=WRITE_TASK_DTYPE)
        tasks["bra"] = order
        tasks["ket"] = order + n
        tasks["code"] = code[order]
        tasks["off"] = off[:-1][order]
        self.prim_quartets = int(np.sum(nb * nk))
        scls = cls[order]
        self.segments = []
        starts = np.flatnonzero(np.diff(np.concatenate([[-1], scls]))) if n else []
        bounds = list(starts) + [n]
        for s, e in zip(bounds[:-1], bounds[1:]):
            c = int(scls[s])
            (la, lb), (lc, ld) = PAIR_ORDER[c // 6], PAIR_ORDER[c % 6]
            self.segments.append(((la, lb, lc, ld), int(s), int(e)))
        self.tasks_host = tasks
        self.tasks = torch.as_tensor(tasks.view(np.uint8)).to(ds.device)
        self.ds = ds
        self.sorted_bra_nprim = nb[order]
        self.sorted_ket_nprim = nk[order]
        work = self.sorted_bra_nprim * self.sorted_ket_nprim
        self.heavy = [heavy_counts(cls, work[s:e]) for cls, s, e in self.segments]
        self.profiles = [work_profile(work[s:e]) for _, s, e in self.segments]

    def _plan_device(self, ds, quartets, want32, max_exp):
        dev = ds.device
        sb = ds.host
        q = torch.as_tensor(quartets).to(device=dev, dtype=torch.int64).reshape(-1, 4)
        n = q.shape[0]
        if n and (int(q.min()) < 0 or int(q.max()) >= sb.nshell):
            raise ValueError(f"shell quartets hold a shell index outside [0, {sb.nshell})")
        lut = _device_luts(dev)
        l4 = ds.l.long()[q]
        li = ((l4[:, 0] * 3 + l4[:, 1]) * 3 + l4[:, 2]) * 3 + l4[:, 3]
        qc = torch.gather(q, 1, lut["pos"][li])             # canonical shells
        off = torch.zeros(n + 1, dtype=torch.int64, device=dev)
        off[1:] = torch.cumsum(lut["size"][li], 0)
        self.n = n
        self._offsets_dev = off
        self.total = int(off[-1])
        self.pairs = DevicePairSet(ds, torch.cat([qc[:, 0:2], qc[:, 2:4]], 0), want32=want32,
                                   max_exp=max_exp)
        npr = ds.nprim
        self.full_prim_quartets = int((npr[qc[:, 0]] * npr[qc[:, 1]] * npr[qc[:, 2]] *
                                       npr[qc[:, 3]]).sum()) if n else 0
        nb = self.pairs.nprim_dev[:n]
        nk = self.pairs.nprim_dev[n:]
        w = nb * nk
        cls = lut["cls"][li]
        self.prim_quartets = int(w.sum()) if n else 0
        # the host form's order: class, then descending nb*nk, nb, nk; ties in input order
        wb = int(nb.max()).bit_length() if n else 1
        wk = int(nk.max()).bit_length() if n else 1
        ww = int(w.max()).bit_length() if n else 1
        key = (cls << ww) | ((1 << ww) - 1 - w)
        key = (key << wb) | ((1 << wb) - 1 - nb)
        key = (key << wk) | ((1 << wk) - 1 - nk)
        order = torch.sort(key, stable=True).indices
        tasks = torch.zeros((n, 6), dtype=torch.int32, device=dev)   # WRITE_TASK layout
        tasks[:, 0] = order.to(torch.int32)
        tasks[:, 1] = (order + n).to(torch.int32)
        tasks[:, 2] = lut["code"][li][order]
        tasks[:, 4:6] = off[:-1][order].contiguous().view(torch.int32).view(n, 2)
        self.tasks = tasks.view(torch.uint8).reshape(-1)
        self.ds = ds
        scls = cls[order]
        ws = w[order]
        nper = torch.bincount(scls, minlength=36).cpu().numpy()
        self.segments = []
        start = 0
        for c in range(36):
            if nper[c]:
                (la, lb), (lc, ld) = PAIR_ORDER[c // 6], PAIR_ORDER[c % 6]
                self.segments.append(((la, lb, lc, ld), start, start + int(nper[c])))
                start += int(nper[c])
        prof = segment_profiles([c for c, _, _ in self.segments], ws,
                                [s for _, s, _ in self.segments] + [n])
        self.heavy, self.profiles = [h for h, _ in prof], [p for _, p in prof]
        self._sorted_dev = (nb[order], nk[order])

    def __getattr__(self, name):
        # host copies of a device-planned batch, made on first use
        if name == "offsets" and "_offsets_dev" in self.__dict__:
            v = self._offsets_dev.cpu().numpy()
        elif name in ("sorted_bra_nprim", "sorted_ket_nprim") and "_sorted_dev" in self.__dict__:
            v = self._sorted_dev[0 if name == "sorted_bra_nprim" else 1].cpu().numpy()
        elif name == "tasks_host" and "_sorted_dev" in self.__dict__:
            v = self.tasks.cpu().numpy().view(WRITE_TASK_DTYPE)
        else:
            raise AttributeError(name)
        setattr(self, name, v)
        return v

    def class_counts(self):
        return {cls: e - s for cls, s, e in self.segments}

    def launch_count(self, precision=64, classes=None):
        """Kernel launches one ``run`` makes with the current kernel forms: one per class
        and tier of primitive work."""
        return len(launch_plan(self, precision, "write", classes))

    def run(self, out, precision=64, stream=None, classes=None):
        _check_device_tensor(out, self.ds.device, "output buffer")
        if out.numel() < self.total:
            raise ValueError(f"output buffer holds {out.numel()} doubles, the blocks need {self.total}")
        L = _lib.lib()
        plan = launch_list(self, precision, "write", classes)
        rc = L.gs_eri_blocks_list(len(plan), plan.ctypes.data, precision, _lib.ptr(self.pairs.rec),
                                  _lib.ptr(self.pairs.prims(precision)),
                                  _lib.ptr(self.ds.comp_scale), self.tasks.data_ptr(),
                                  _lib.ptr(out), *HeavyLane(self.ds.device, stream).streams())
        _lib.check(rc, "gs_eri_blocks_list")
        return out


RANGE_DTYPE = np.dtype([("first", "<i8"), ("base", "<i8"), ("bra", "<i4"), ("nbra", "<i4"),
                        ("ket", "<i4"), ("nket", "<i4"), ("size", "<i4"), ("pad", "<i4")])
MAX_RANGES = 1 << 15


def unique_pair_ranges(pair_class, nprim):
    """The unique quartets of pairs sorted by class and, in a class, by descending primitive
    count, as ranges (RANGE_DTYPE) of constant class and primitive-quartet count, each
    class segment by descending count: (ranges, counts w per range, segments), or None if
    they are too many (bases with hundreds of different contractions)."""
    key = pair_class.astype(np.int64) << 32 | (2 ** 31 - nprim.astype(np.int64))
    start = np.flatnonzero(np.diff(key, prepend=-1))
    end = np.append(start[1:], len(key))
    groups = [[] for _ in PAIR_ORDER]                  # per class: (first pair, pairs, nprim)
    for s, e in zip(start.tolist(), end.tolist()):
        groups[int(pair_class[s])].append((s, e - s, int(nprim[s])))
    if sum(len(g) for g in groups) ** 2 > 2 * MAX_RANGES:
        return None
    rows, work, segments = [], [], []
    first = base = 0
    for cb in range(len(PAIR_ORDER)):
        for ck in range(cb + 1):
            cls = PAIR_ORDER[cb] + PAIR_ORDER[ck]
            size = class_sizes(cls)[1]
            found = []
            for i, (b, nb, wb) in enumerate(groups[cb]):
                for j, (k, nk, wk) in enumerate(groups[ck]):
                    if cb != ck or j < i:
                        found.append((wb * wk, b, nb, k, nk, nb * nk))
                    elif j == i:
                        found.append((wb * wk, b, nb, 0, 0, nb * (nb + 1) // 2))
            begin = first
            for w, b, nb, k, nk, count in sorted(found, key=lambda x: -x[0]):
                rows.append((first, base, b, nb, k, nk, size, 0))
                work.append((w, count))
                first += count
                base += count * size
            if first > begin:
                segments.append((cls, begin, first))
    return np.array(rows, dtype=RANGE_DTYPE), work, segments


class TooManyRanges(ValueError):
    """A basis of so many different contractions that its unique quartets are no short list of
    ranges (UniqueQuartets)."""


class UniqueQuartets:
    """Blocks of every unique shell quartet of a basis, each in canonical shell order (bra
    pair class >= ket pair class, la >= lb), for the dense tensor: one record per shell pair,
    and tasks expanded on the device (``gs_product_tasks``) from a few ranges of pairs.
    Blocks go through QuartetBatch.run."""

    def __init__(self, ds: DeviceShells, want32=False):
        sb = ds.host
        i, j = np.tril_indices(sb.nshell)
        swap = sb.l[i] < sb.l[j]
        a, b = np.where(swap, j, i), np.where(swap, i, j)
        pc = _pc_lut[sb.l[a], sb.l[b]]
        npp = sb.nprim[a].astype(np.int64) * sb.nprim[b]
        order = np.lexsort((-npp, pc))                 # every primitive pair is kept (no screen)
        plan = unique_pair_ranges(pc[order], npp[order])
        if plan is None:
            raise TooManyRanges("too many ranges of equal primitive counts")
        ranges, work, self.segments = plan
        self.ds = ds
        self.pairs = PairSet(ds, np.stack([a, b], 1)[order], want32=want32, count=False)
        self.n = self.segments[-1][2] if self.segments else 0
        last = ranges[-1] if len(ranges) else None
        self.total = 0 if last is None else int(last["base"] + work[-1][1] * last["size"])
        at = 0
        self.heavy, self.profiles = [], []
        for cls, s, e in self.segments:
            mine = []
            while at < len(work) and ranges["first"][at] < e:
                mine.append(work[at])
                at += 1
            w, c = np.array(mine, dtype=np.int64).T    # w descending
            upto = np.concatenate([[0], np.cumsum(c)])
            ge = upto[np.searchsorted(-w, -np.concatenate(
                [[heavy_threshold(cls), COOP_PRIM_QUARTETS], _LEVELS]), side="right")].tolist()
            self.heavy.append((ge[0], ge[1]))
            self.profiles.append((int((w * c).sum()), ge[2:]))
        dev = ds.device
        r = torch.as_tensor(ranges.view(np.uint8)).to(dev)
        self.tasks = torch.empty(max(1, self.n) * WRITE_TASK, dtype=torch.uint8, device=dev)
        self.quartets = torch.empty((max(1, self.n), 4), dtype=torch.int32, device=dev)
        self.block_offsets = torch.empty(max(1, self.n), dtype=torch.int64, device=dev)
        _lib.check(_lib.lib().gs_product_tasks(self.n, len(ranges), _lib.ptr(r),
                                               _lib.ptr(self.pairs.shells), _lib.ptr(self.tasks),
                                               _lib.ptr(self.quartets),
                                               _lib.ptr(self.block_offsets), _lib.stream()),
                   "gs_product_tasks")

    run = QuartetBatch.run


def eri_blocks(sb: ShellBasis, quartets, precision=64, device="cuda"):
    """Convenience: blocks of the given shell quartets, returned as a host f64 array."""
    ds = DeviceShells(sb, device)
    batch = QuartetBatch(ds, quartets, want32=precision == 32)
    out = torch.zeros(max(1, batch.total), dtype=torch.float64, device=ds.device)
    batch.run(out, precision)
    return out[:batch.total].cpu().numpy(), batch.offsets


# ---------------------------------------------------------------------- Fock (J/K) engine
# streams of a mixed-precision build's partitioned launches; with eight (H2O)24 takes 14.93 ms,
# with six 14.95
MIXED_LANES = 6
# bytes of partition workspace above which a build takes fewer streams rather than more memory
MIXED_BYTES = 2 << 30


class MixedWorkspace:
    """The partition workspace of an engine: one region per stream of the partitioned launches,
    each as long as the stream's longest launch needs (16 bytes a task).  It is allocated once and
    never moves: its size follows from the task segments, which are the engine's for good, and not
    from the launch plan, which changes with the chosen forms, so that a captured graph's addresses
    stay the engine's.  The streams' longest launches are different tiers, so together they have at
    most the tasks of the MIXED_LANES longest segments."""

    def mixed_workspace(self, dev, tiers):
        """(address, bytes, streams) for the launch records ``tiers``."""
        L = _lib.lib()
        if getattr(self, "_ws", None) is None:
            need = [int(L.gs_fock_jk_mixed_workspace(n)) + 256 for n in
                    sorted((e - s for _, s, e in self.segments), reverse=True)[:MIXED_LANES] or [0]]
            size = max(need[0], min(sum(need) + MIXED_LANES * 512, MIXED_BYTES))
            self._ws = torch.empty(size, dtype=torch.uint8, device=dev)
        lanes = MIXED_LANES
        while lanes > 1 and L.gs_fock_jk_mixed_list_workspace(len(tiers), tiers.ctypes.data,
                                                              lanes) > self._ws.numel():
            lanes -= 1
        return self._ws.data_ptr(), self._ws.numel(), lanes


def task_keys(pairs, bra, ket):
    """Sort keys (descending) of Fock tasks: primitive-quartet count, the pairs' primitive
    counts, and the distance of the pairs (``gs_task_keys``).  A warp whose primitive quartets
    take both branches of the Boys function pays for both (FP64 (ps|ss) of (H2O)16: 24 of 32
    lanes active on average); which one a primitive quartet takes follows that distance."""
    keys = torch.empty_like(bra)
    _lib.check(_lib.lib().gs_task_keys(bra.numel(), _lib.ptr(bra), _lib.ptr(ket),
                                       _lib.ptr(pairs.kept), _lib.ptr(pairs.rec),
                                       _lib.ptr(pairs.p64), _lib.ptr(keys), _lib.stream()),
               "gs_task_keys")
    return keys


KEY_WORK = 4096 << 6          # a key over this is the primitive-quartet count


class JKEngine(MixedWorkspace):
    """Integral-direct Coulomb/exchange builder over all unique shell quartets of one
    basis, with Schwarz screening (task list built once per geometry) and optional
    density-weighted screening / precision selection per call."""

    def __init__(self, sb: ShellBasis, device="cuda", schwarz_thr=1e-12, want32=True,
                 max_exp=PRIM_SCREEN):
        self.sb = sb
        self.ds = ds = DeviceShells(sb, device)
        self.dev = ds.device
        ns = sb.nshell
        i, j = np.tril_indices(ns)                      # shell i >= shell j
        swap = sb.l[i] < sb.l[j]
        sa = np.where(swap, j, i)
        sbb = np.where(swap, i, j)
        self.pairs = PairSet(ds, np.stack([sa, sbb], axis=1), want32=want32, max_exp=max_exp)
        self.pair_class = _pc_lut[sb.l[sa], sb.l[sbb]]
        self.npairs = len(sa)
        self.schwarz_thr = schwarz_thr
        self.q = torch.zeros(self.npairs, dtype=torch.float64, device=self.dev)
        L = _lib.lib()
        for c, (la, lb) in enumerate(PAIR_ORDER):
            idx = np.flatnonzero(self.pair_class == c).astype(np.int32)
            if len(idx) == 0:
                continue
            it = torch.as_tensor(idx).to(self.dev)
            _lib.check(L.gs_schwarz(la, lb, _lib.ptr(self.pairs.rec), _lib.ptr(self.pairs.p64),
                                    _lib.ptr(ds.comp_scale), len(idx), _lib.ptr(it),
                                    _lib.ptr(self.q), self.npairs, _lib.stream()), "gs_schwarz")
        self._build_tasks()
        # function -> shell map for per-shell-block density maxima
        self.func_shell = torch.as_tensor(np.repeat(np.arange(ns), sb.nfunc)).to(self.dev)

    def _build_tasks(self):
        dev = self.dev
        q = self.q
        self.segments = []
        self.heavy = []           # heavy_counts of each segment
        self.profiles = []        # work_profile of each segment
        chunks, work = [], []
        ntot = 0
        thr = self.schwarz_thr
        pc = torch.as_tensor(self.pair_class).to(dev)
        for cb in range(len(PAIR_ORDER)):
            bra_ids = torch.nonzero(pc == cb).flatten()
            if bra_ids.numel() == 0:
                continue
            qb, ob = torch.sort(q[bra_ids], descending=True)
            bra_sorted = bra_ids[ob]
            for ck in range(cb + 1):
                ket_ids = torch.nonzero(pc == ck).flatten()
                if ket_ids.numel() == 0:
                    continue
                qk, ok = torch.sort(q[ket_ids], descending=True)
                ket_sorted = ket_ids[ok]
                # number of kets with qb*qk >= thr: prefix of the descending list
                need = torch.where(qb > 0, thr / qb, torch.full_like(qb, float("inf")))
                cnt = torch.searchsorted(-qk.contiguous(), -need.contiguous(), right=True)
                if cb == ck:
                    start = torch.arange(len(qb), device=dev)
                    cnt = torch.clamp(cnt - start, min=0)
                else:
                    start = torch.zeros(len(qb), dtype=torch.int64, device=dev)
                total = int(cnt.sum())
                if total == 0:
                    continue
                bra_pos = torch.repeat_interleave(torch.arange(len(qb), device=dev), cnt)
                first = torch.cumsum(cnt, 0) - cnt
                within = torch.arange(total, device=dev) - first[bra_pos]
                ket_pos = start[bra_pos] + within
                bra = bra_sorted[bra_pos]
                ket = ket_sorted[ket_pos]
                # most primitive quartets first (longest tasks start first), equal
                # (K_bra, K_ket) together, then by distance
                key, o = torch.sort(task_keys(self.pairs, bra, ket), descending=True, stable=True)
                t = torch.stack([bra[o], ket[o]], dim=1).to(torch.int32)
                (la, lb), (lc, ld) = PAIR_ORDER[cb], PAIR_ORDER[ck]
                self.segments.append(((la, lb, lc, ld), ntot, ntot + total))
                work.append(key // KEY_WORK)
                chunks.append(t)
                ntot += total
        self.tasks = torch.cat(chunks, 0).contiguous() if chunks else \
            torch.zeros((1, 2), dtype=torch.int32, device=dev)
        self.ntasks = ntot
        if chunks:
            prof = segment_profiles([c for c, _, _ in self.segments], torch.cat(work),
                                    [s for _, s, _ in self.segments] + [ntot])
            self.heavy, self.profiles = [h for h, _ in prof], [p for _, p in prof]

    def shell_dmax(self, mats):
        """max |P_ij| over each (shell, shell) block, over all given matrices."""
        ns = self.sb.nshell
        m = torch.stack([x.abs() for x in mats]).amax(0)
        fs = self.func_shell
        rows = torch.full((ns, m.shape[1]), 0.0, dtype=torch.float64, device=self.dev)
        rows.index_reduce_(0, fs, m, "amax", include_self=True)
        out = torch.full((ns, ns), 0.0, dtype=torch.float64, device=self.dev)
        out.index_reduce_(1, fs, rows, "amax", include_self=True)
        return out.contiguous()

    def jk(self, pj=None, pk=(), precision=64, screen_thr=0.0, mixed_cut=None, stream=None,
           classes=None):
        """J[pj] and K[pk_s] (symmetric densities, nbf x nbf f64 device tensors).

        precision 64 or 32 evaluates every task in that precision.  With ``mixed_cut``
        the quartets whose density-weighted bound is below it run in f32 and the rest in
        f64 (accumulation is always f64).  ``screen_thr`` > 0 additionally skips quartets
        whose density-weighted bound is below it."""
        n = self.sb.nbf
        dev = self.dev
        pk = list(pk)
        nk = len(pk)
        for d in ([pj] if pj is not None else []) + pk:
            _check_device_tensor(d, dev, "density matrix", (n, n))
        jbuf = torch.zeros((n, n), dtype=torch.float64, device=dev) if pj is not None else None
        kbuf = torch.zeros((max(nk, 1), n, n), dtype=torch.float64, device=dev) if nk else None
        pj_c = pj.contiguous() if pj is not None else None
        pk_c = torch.stack(pk).contiguous() if nk else None
        dmax, thr = None, 0.0
        if mixed_cut is not None or screen_thr > 0:
            mats = ([pj] if pj is not None else []) + pk
            dmax = self.shell_dmax(mats)
            thr = screen_thr if screen_thr > 0 else 1e-300
        L = _lib.lib()
        base = self.tasks.data_ptr()
        with HeavyLane(dev, stream) as lane:
            if mixed_cut is not None:
                banded, tiers = mixed_list(self, classes, mixed_cut)
                ws, size, lanes = self.mixed_workspace(dev, tiers)
                for i, (cls, first, prec, form, count, lo, hi) in enumerate(banded):
                    rc = L.gs_fock_jk(*cls, prec | (form << 8), _lib.ptr(self.pairs.rec),
                                      _lib.ptr(self.pairs.prims(prec)), _lib.ptr(self.ds.comp_scale),
                                      _lib.ptr(self.ds.func_off), self.sb.nshell, n, count,
                                      base + first * 8, _lib.ptr(pj_c), _lib.ptr(jbuf), nk,
                                      _lib.ptr(pk_c), _lib.ptr(kbuf), _lib.ptr(dmax), thr, lo, hi,
                                      lane.lane(i + 1))
                    _lib.check(rc, f"gs_fock_jk{cls}")
                rc = L.gs_fock_jk_mixed_list(
                    len(tiers), tiers.ctypes.data, _lib.ptr(self.pairs.rec), _lib.ptr(self.pairs.p64),
                    _lib.ptr(self.pairs.p32), _lib.ptr(self.ds.comp_scale), _lib.ptr(self.ds.func_off),
                    self.sb.nshell, n, base, _lib.ptr(pj_c), _lib.ptr(jbuf), nk, _lib.ptr(pk_c),
                    _lib.ptr(kbuf), _lib.ptr(dmax), thr, mixed_cut, ws, -size, *lane.streams(lanes))
                _lib.check(rc, "gs_fock_jk_mixed_list")
            else:
                plan = launch_list(self, precision, "jk", classes)
                rc = L.gs_fock_jk_list(
                    len(plan), plan.ctypes.data, precision, _lib.ptr(self.pairs.rec),
                    _lib.ptr(self.pairs.prims(precision)), _lib.ptr(self.ds.comp_scale),
                    _lib.ptr(self.ds.func_off), self.sb.nshell, n, base, _lib.ptr(pj_c),
                    _lib.ptr(jbuf), nk, _lib.ptr(pk_c), _lib.ptr(kbuf), _lib.ptr(dmax), thr, 0.0,
                    float("inf"), *lane.streams())
                _lib.check(rc, "gs_fock_jk_list")
        J = (jbuf + jbuf.T) if jbuf is not None else None
        K = [kbuf[s] + kbuf[s].T for s in range(nk)]
        return J, K
