"""The work that programs give this library, as timed cases.

A case is a program in the form cdvmh translates one to -- arrays, regions,
loops, reductions and actuality through the C dvmh_* ABI, called here by ctypes
-- with the CUDA handlers of the workload programs.  A state holds a program's
arrays; one pass runs `steps` of its time steps (SOR: sweeps) with the
reduction results read back after every step, as the programs do, and ends
with the queued loops launched.  The last kind of case is one training step of
the tuner's cost model.

Grids have walls held at fixed temperatures, so that a state can be stepped any
number of times: its field tends to the steady one between its walls' values.
`scale` is the size of the field: 1 for data in [0, 1), 100 for, say, degrees.
"""
import ctypes
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import __graft_entry__ as entry  # noqa: E402

_, gb = entry.package()

INT, LONG, PTR, STR = ctypes.c_int, ctypes.c_long, ctypes.c_void_p, ctypes.c_char_p
INTENT_IN, INTENT_INOUT = 1, 3
CUDA = 2
HOST_AND_CUDA = 3
RT_FLOAT, RT_DOUBLE = 3, 4
RF_SUM, RF_MAX, RF_MINLOC = 1, 3, 12
OMEGA, COEF = 1.5, 0.1


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # a small plate stepped interactively: one step and its eps, all latency
        {"name": "jac2d_130", "kind": "jacobi", "rank": 2, "n": 130, "steps": 1, "scale": 1.0, "mode": "batched"},
        # the 2-D program of the repository, 1024^2, eps read every step
        {"name": "jac2d_1024", "kind": "jacobi", "rank": 2, "n": 1024, "steps": 10, "scale": 1.0, "mode": "batched"},
        # a large odd plate in degrees, one launch per loop (the reference's execution model)
        {"name": "jac2d_4097_plain", "kind": "jacobi", "rank": 2, "n": 4097, "steps": 4, "scale": 100.0,
         "mode": "plain"},
        # a small odd cube: a coarse run before the fine one
        {"name": "jac3d_67", "kind": "jacobi", "rank": 3, "n": 67, "steps": 10, "scale": 1.0, "mode": "batched"},
        # an ordinary cube in degrees
        {"name": "jac3d_255_deg", "kind": "jacobi", "rank": 3, "n": 255, "steps": 10, "scale": 100.0,
         "mode": "batched"},
        # the headline: 512^3, data in [0, 1)
        {"name": "jac3d_512", "kind": "jacobi", "rank": 3, "n": 512, "steps": 10, "scale": 1.0, "mode": "batched"},
        # ACROSS sweeps (Gauss-Seidel with over-relaxation) of a small and of the repository's cube
        {"name": "sor3d_97", "kind": "sor", "n": 97, "steps": 2, "scale": 1.0, "mode": "batched"},
        {"name": "sor3d_384", "kind": "sor", "n": 384, "steps": 4, "scale": 1.0, "mode": "batched"},
        # uneven plates stepped together with a SUM and a MINLOC each: a few, and the repository's 256
        {"name": "heat_24", "kind": "heat", "count": 24, "lo": 64, "hi": 512, "steps": 4, "scale": 100.0,
         "mode": "batched"},
        {"name": "heat_256", "kind": "heat", "count": 256, "lo": 64, "hi": 2048, "steps": 20, "scale": 1.0,
         "mode": "batched"},
        # the reference's FP32 benchmark through handlers as cdvmh generates them (one point and one MAX slot a thread)
        {"name": "generated_f32_384", "kind": "generated", "rank": 3, "n": 384, "steps": 5, "scale": 100.0,
         "mode": "batched"},
        # one training step of the tuner's cost model on a batch of recorded timings
        {"name": "mlp_4096", "kind": "mlp", "rows": 4096},
    ]


def _between(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["jacobi", "jacobi", "jacobi", "sor", "heat", "generated", "mlp"])
    if kind == "mlp":
        return {"kind": kind, "rows": _between(rng, 64, 16384)}
    c = {"kind": kind, "steps": rng.choice([1, 2, 4, 8]), "scale": rng.choice([1.0, 1.0, 100.0])}
    if kind == "heat":
        lo = _between(rng, 16, 256)
        c.update(count=_between(rng, 2, 256), lo=lo, hi=_between(rng, 2 * lo, 2048), steps=rng.choice([1, 2, 4]))
    elif kind == "sor":
        c["n"] = _between(rng, 12, 384)
    else:
        c["rank"] = rng.choice([2, 3])
        c["n"] = _between(rng, 24, 6000) if c["rank"] == 2 else _between(rng, 12, 512 if kind == "jacobi" else 384)
    c["mode"] = rng.choice(["batched", "batched", "batched", "async", "plain"])
    return c


# ------------------------------------------------------------------ inputs

def _uniform(seed, *shape):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _field(seed, shape, scale):
    """A random interior between walls of one temperature each."""
    f = _uniform(seed, *shape)
    walls = (0.1 + 0.9 * _uniform(seed + 7919, 2 * len(shape))).tolist()
    for d in range(len(shape)):
        f.select(d, 0).fill_(walls[2 * d])
        f.select(d, shape[d] - 1).fill_(walls[2 * d + 1])
    return f * scale


def _sides(case):
    """The plates' sides: log-uniform between lo and hi, the same for every seed."""
    rng, ratio = random.Random(case["count"]), case["hi"] / case["lo"]
    return [max(8, int(case["lo"] * ratio ** rng.random())) for _ in range(case["count"])]


def _jacobi_inputs(case, seed, dtype):
    """A = the walls' values around zeros, B = a random interior between them."""
    b = _field(seed, (case["n"],) * case["rank"], case["scale"]).to(dtype)
    a = b.clone()
    a[(slice(1, -1),) * case["rank"]] = 0
    return a, b


# ------------------------------------------------------------------ programs on the dvmh_* ABI

def _abi(name, res, *args):
    f = gb.init()[name]
    f.restype, f.argtypes = res, args
    return f


def _handler(name):
    return ctypes.cast(getattr(gb.workloads(), name), PTR).value


class _Array:
    """A distributed array of the runtime, its data given from the device."""

    def __init__(self, data, like=None):
        self.shape, rank = tuple(data.shape), data.dim()
        single = data.dtype == torch.float32
        self.kind = "<f4" if single else "<f8"
        self.desc = (LONG * 64)()
        self.at = ctypes.addressof(self.desc)
        self.ref = PTR(self.at)
        sizes = [v for n in self.shape for v in (n, 1, 1)]
        _abi("dvmh_array_create_C", None, PTR, LONG, LONG, *[LONG] * (3 * rank))(
            self.at, rank, -RT_FLOAT if single else -RT_DOUBLE, *sizes)
        if like is None:
            block = _abi("dvmh_distribution_block_C", LONG, LONG)
            _abi("dvmh_distribute_C", None, PTR, LONG, *[LONG] * rank)(
                self.at, rank, *[block(d + 1) for d in range(rank)])
        else:
            _abi("dvmh_align_C", None, PTR, PTR, LONG, *[LONG] * rank)(
                self.at, like.at, rank, *[_linear()(d + 1, 1, 0) for d in range(rank)])
        self.base = _abi("dvmh_get_natural_base_C", PTR, LONG, PTR)
        host = (ctypes.c_float if single else ctypes.c_double) * data.numel()
        view = np.frombuffer(host.from_address(self.base(0, self.at)), dtype=self.kind).reshape(self.shape)
        torch.from_numpy(view).copy_(data)
        _abi("dvmh_actual_array2_", None, PTR)(self.at)
        self.views = {}

    def tensor(self):
        """The array's current device copy (the runtime's own buffer)."""
        p = self.base(1, self.at)
        if p not in self.views:
            hdr = (LONG * 16)()
            _abi("dvmh_fill_header_C", LONG, LONG, PTR, PTR, PTR, PTR)(1, p, self.at, ctypes.addressof(hdr), None)
            size = int(self.kind[2])
            strides = tuple(hdr[1 + d] * size for d in range(len(self.shape)))
            raw = type("DeviceArray", (), {"__cuda_array_interface__": {
                "shape": self.shape, "typestr": self.kind, "data": (p, False), "strides": strides, "version": 2}})()
            self.views[p] = torch.as_tensor(raw, device="cuda")
        return self.views[p]

    def free(self):
        self.views.clear()
        _abi("dvmh_array_free_C", None, PTR)(self.at)


class _Ref(LONG):
    """A reference the ABI hands out; as a subclass it comes back unconverted, ready for the next call."""


def _longs(*values):
    return tuple(LONG(v) for v in values)


def _linear():
    return _abi("dvmh_alignment_linear_C", LONG, LONG, LONG, LONG)


class _Program:
    """What the programs share: the ABI's entry points, and arguments made once (a compiled program's calls cost
    next to nothing, so these should cost little)."""

    def __init__(self, rank, mode):
        self.rank, self.arrays = rank, []
        abi = gb.init()

        def bare(name, res=None):
            f = abi[name]
            f.restype = res
            return f

        self.mode = INT(gb.MODES[mode])
        self.set_mode, self.flush = bare("dvmhgb_set_mode"), bare("dvmhgb_flush")
        self.actual, self.get_actual = bare("dvmh_actual_variable2_"), bare("dvmh_get_actual_variable2_")
        self.region, self.end = bare("dvmh_region_create_C", _Ref), bare("dvmh_region_end_C")
        self.use_array = bare("dvmh_region_register_array_C")
        self.use_scalar = bare("dvmh_region_register_scalar_C")
        self.start = bare("dvmh_region_execute_on_targets_C")
        self.loop_create, self.loop_map = bare("dvmh_loop_create_C", _Ref), bare("dvmh_loop_map_C")
        self.linear = bare("dvmh_alignment_linear_C", _Ref)
        self.axes = [_longs(d + 1, 1, 0) for d in range(rank)]
        self.reduction, self.across = bare("dvmh_loop_reduction_C"), bare("dvmh_loop_across_C")
        self.set_handler, self.set_block = bare("dvmh_loop_register_handler_C"), bare("dvmh_loop_set_cuda_block_C")
        self.handler_func, self.perform = bare("dvmh_handler_func_C", _Ref), bare("dvmh_loop_perform_C")
        self.renew = bare("dvmh_shadow_renew_C")
        self.zero, self.n_axes = LONG(0), LONG(rank)
        self.targets, self.on_cuda = LONG(HOST_AND_CUDA), _longs(CUDA, 0)

    def array(self, data, like=None):
        self.arrays.append(_Array(data, like))
        return self.arrays[-1]

    def scalar(self, address):
        """A variable of the program, just written on the host: whatever lived at its address is gone."""
        self.actual(PTR(address))
        return PTR(address)

    def loop(self, region, arr, interior):
        """A loop over the array's interior, mapped on it."""
        lp = self.loop_create(region, *interior)
        self.loop_map(lp, arr.ref, self.n_axes, *[self.linear(*a) for a in self.axes])
        return lp

    def run_loop(self, lp, call):
        self.set_handler(lp, *self.on_cuda, self.handler_func(*call))
        self.perform(lp)

    def __del__(self):
        for a in reversed(self.arrays):
            a.free()


def _call(handler, *params):
    """The arguments of dvmh_handler_func_C."""
    return (PTR(handler), LONG(len(params)), *params)


def _over(shape):
    """A loop's rank and bounds: the interior of an array."""
    return _longs(len(shape), *[v for n in shape for v in (1, n - 2, 1)])


class _Jacobi(_Program):
    """eps = max |B - A|, A = B; B = the mean of A's neighbours (jac2d.c, jac3d.c; in FP32: jacperf.c)."""

    def __init__(self, case, seed):
        rank, self.steps = case["rank"], case["steps"]
        super().__init__(rank, case["mode"])
        self.generated = case["kind"] == "generated"
        a, b = _jacobi_inputs(case, seed, torch.float32 if self.generated else torch.float64)
        self.A = self.array(a)
        self.B = self.array(b, self.A)
        A, B = self.A.ref, self.B.ref
        self.interior = _over(self.A.shape)
        self.eps = (ctypes.c_float if self.generated else ctypes.c_double)()
        eps = self.eps_ref = self.scalar(ctypes.addressof(self.eps))
        size = ctypes.sizeof(self.eps)
        self.use = [(LONG(INTENT_INOUT), A, b"A"), (LONG(INTENT_INOUT), B, b"B")]
        self.use_eps = (LONG(INTENT_INOUT), eps, LONG(size), b"eps")
        self.max_eps = (LONG(RF_MAX), eps, *_longs(RT_FLOAT if self.generated else RT_DOUBLE, 1), PTR(), LONG(0))
        name = ("loop_jacperf%d_" if self.generated else "loop_jac%dd_") % rank
        self.upd = _call(_handler(name + "upd_cuda"), A, B, eps)
        self.stn = _call(_handler(name + "stn_cuda"), A, B)
        self.block = _longs(*((32, 8, 1) if rank == 3 else (256, 1, 1)))

    def step(self):
        eps = self.eps_ref
        self.eps.value = 0
        self.actual(eps)
        r = self.region(self.zero)
        for u in self.use:
            self.use_array(r, *u)
        self.use_scalar(r, *self.use_eps)
        self.start(r, self.targets)
        lp = self.loop(r, self.A, self.interior)
        if self.generated:
            self.set_block(lp, *self.block)
        self.reduction(lp, *self.max_eps)
        self.run_loop(lp, self.upd)
        self.renew(self.A.ref, self.zero, self.zero)
        lp = self.loop(r, self.B, self.interior)
        if self.generated:
            self.set_block(lp, *self.block)
        self.run_loop(lp, self.stn)
        self.end(r)
        self.get_actual(eps)
        return self.eps.value

    def run(self):
        self.set_mode(self.mode)
        eps = [self.step() for _ in range(self.steps)]
        self.flush()
        return {"A": self.A.tensor(), "B": self.B.tensor(),
                "eps": np.array(eps, dtype=np.float32 if self.generated else np.float64)}


class _Sor(_Program):
    """SOR in place as an ACROSS loop, with the SUM of squared changes (sor3d.c)."""

    def __init__(self, case, seed):
        super().__init__(3, case["mode"])
        self.steps = case["steps"]
        self.A = self.array(_field(seed, (case["n"],) * 3, case["scale"]))
        A = self.A.ref
        self.interior = _over(self.A.shape)
        self.s, self.w = ctypes.c_double(), ctypes.c_double(OMEGA)
        s = self.s_ref = self.scalar(ctypes.addressof(self.s))
        w = self.scalar(ctypes.addressof(self.w))
        self.use = (LONG(INTENT_INOUT), A, b"A")
        self.use_s = (LONG(INTENT_INOUT), s, LONG(8), b"s")
        self.use_w = (LONG(INTENT_IN), w, LONG(8), b"w")
        self.depends = (LONG(0), A, *_longs(3, 1, 1, 1, 1, 1, 1))
        self.sum_s = (LONG(RF_SUM), s, *_longs(RT_DOUBLE, 1), PTR(), LONG(0))
        self.sweep = _call(_handler("loop_sor3d_cuda"), A, s, w)

    def step(self):
        self.s.value = 0
        self.actual(self.s_ref)
        r = self.region(self.zero)
        self.use_array(r, *self.use)
        self.use_scalar(r, *self.use_s)
        self.use_scalar(r, *self.use_w)
        self.start(r, self.targets)
        lp = self.loop(r, self.A, self.interior)
        self.across(lp, *self.depends)
        self.reduction(lp, *self.sum_s)
        self.run_loop(lp, self.sweep)
        self.end(r)
        self.get_actual(self.s_ref)
        return self.s.value

    def run(self):
        self.set_mode(self.mode)
        sums = [self.step() for _ in range(self.steps)]
        self.flush()
        return {"A": self.A.tensor(), "sums": np.array(sums)}


class _Heat(_Program):
    """An explicit heat step on many uneven plates, a SUM and a MINLOC each (heat.c)."""

    def __init__(self, case, seed):
        super().__init__(2, case["mode"])
        self.steps, self.done = case["steps"], 0
        cnt = case["count"]
        self.sums, self.mins = np.zeros(cnt), np.zeros(cnt)
        self.locs = np.zeros((cnt, 2), dtype=np.int32)
        self.coef = ctypes.c_double(COEF)
        self.results = [self.scalar(v.ctypes.data) for v in (self.sums, self.mins, self.locs)]
        coef = self.scalar(ctypes.addressof(self.coef))
        self.use = [(LONG(INTENT_INOUT), v, LONG(8 * cnt), name)
                    for v, name in zip(self.results, (b"sums", b"mins", b"locs"))]
        self.use.append((LONG(INTENT_IN), coef, LONG(8), b"coef"))
        self.intents = _longs(INTENT_IN, INTENT_INOUT)
        handler = _handler("loop_heat_cuda")
        self.U, self.V, self.loops = [], [], ([], [])
        for k, n in enumerate(_sides(case)):
            u = _field(seed + k, (n, n), case["scale"])
            v = u.clone()
            v[1:-1, 1:-1] = 0
            self.U.append(self.array(u))
            self.V.append(self.array(v, self.U[-1]))
            s, m, at = (PTR(v.value + 8 * k) for v in self.results)
            add = (LONG(RF_SUM), s, *_longs(RT_DOUBLE, 1), PTR(), LONG(0))
            least = (LONG(RF_MINLOC), m, *_longs(RT_DOUBLE, 1), at, LONG(8))
            for way, (a, b) in enumerate(((self.U[-1], self.V[-1]), (self.V[-1], self.U[-1]))):
                self.loops[way].append((a, b, _over((n, n)), add, least, _call(handler, a.ref, b.ref, s, m, at, coef)))
        cells = [a.shape[0] ** 2 for a in self.U]
        self.out = torch.empty(sum(cells), dtype=torch.float64, device="cuda")
        self.parts = [p.view(a.shape) for p, a in zip(self.out.split(cells), self.U)]
        self.stream = torch.cuda.ExternalStream(_abi("dvmhgb_stream", PTR)())

    def step(self):
        loops = self.loops[self.done % 2]
        self.sums[:] = 0
        self.mins[:] = 1e300
        self.locs[:] = -1
        for v in self.results:
            self.actual(v)
        r = self.region(self.zero)
        read, written = self.intents
        for a, b, *_ in loops:
            self.use_array(r, read, a.ref, b"src")
            self.use_array(r, written, b.ref, b"dst")
        for u in self.use:
            self.use_scalar(r, *u)
        self.start(r, self.targets)
        for a, b, interior, add, least, call in loops:
            self.renew(a.ref, self.zero, self.zero)
            lp = self.loop(r, b, interior)
            self.reduction(lp, *add)
            self.reduction(lp, *least)
            self.run_loop(lp, call)
        self.end(r)
        for v in self.results:
            self.get_actual(v)
        self.done += 1
        return self.sums.copy(), self.mins.copy(), self.locs.copy()

    def run(self):
        self.set_mode(self.mode)
        seen = [self.step() for _ in range(self.steps)]
        self.flush()
        with torch.cuda.stream(self.stream):  # the plates side by side
            for p, a in zip(self.parts, self.U if self.done % 2 == 0 else self.V):
                p.copy_(a.tensor())
        sums, mins, locs = (np.stack(v) for v in zip(*seen))
        return {"u": self.out, "sums": sums, "mins": mins, "locs": locs}


class _Mlp:
    """A training step of the cost model: loss and gradients, then Adam (tune.py)."""

    def __init__(self, case, seed):
        gb.init()
        self.n = case["rows"]
        self.rt = gb.runtime()
        nparams = _abi("dvmhgb_mlp_nparams", LONG)()
        nwork = _abi("dvmhgb_mlp_work_floats", LONG, LONG)(self.n)
        self.grad_call = _abi("dvmhgb_mlp_loss_grad", INT, PTR, PTR, PTR, LONG, PTR, PTR, PTR, PTR)
        self.adam_call = _abi("dvmhgb_mlp_adam", INT, PTR, PTR, PTR, PTR, LONG, ctypes.c_float, PTR)
        self.X, self.y, self.p = _mlp_inputs(self.n, seed)
        assert self.p.numel() == nparams
        self.g, self.m, self.v = (torch.zeros_like(self.p) for _ in range(3))
        self.loss = torch.zeros(1, device="cuda")
        self.work = torch.empty(nwork, device="cuda")
        self.step = 0

    def run(self):
        s = torch.cuda.current_stream().cuda_stream
        self.step += 1
        if self.grad_call(self.p.data_ptr(), self.X.data_ptr(), self.y.data_ptr(), self.n, self.g.data_ptr(),
                          self.loss.data_ptr(), self.work.data_ptr(), s):
            raise RuntimeError("dvmhgb_mlp_loss_grad refused its arguments")
        if self.adam_call(self.p.data_ptr(), self.g.data_ptr(), self.m.data_ptr(), self.v.data_ptr(), self.step, 1e-3,
                          s):
            raise RuntimeError("dvmhgb_mlp_adam refused its arguments")
        return {"loss": self.loss, "grad": self.g, "params": self.p, "m": self.m, "v": self.v}


_D, _H = 24, 128  # the cost model: 24 -> 128 -> 128 -> 1
_SPLIT = [_H * _D, _H, _H * _H, _H, _H, 1]


def _mlp_inputs(n, seed):
    """Normalised features, log-times that depend on them, and parameters some way into training."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    x = torch.randn(n, _D, generator=g, device="cuda")
    w = torch.randn(_D, generator=g, device="cuda") / _D ** 0.5
    y = x @ w + 0.1 * torch.randn(n, generator=g, device="cuda")
    scale = [(2.0 / _D) ** 0.5, 0.02, (2.0 / _H) ** 0.5, 0.02, (1.0 / _H) ** 0.5, 0.02]
    p = torch.cat([s * torch.randn(k, generator=g, device="cuda") for s, k in zip(scale, _SPLIT)])
    return x, y, p


_KINDS = {"jacobi": _Jacobi, "generated": _Jacobi, "sor": _Sor, "heat": _Heat, "mlp": _Mlp}


def prepare(case, seed):
    return _KINDS[case["kind"]](case, seed)


def run(state):
    return state.run()


# ------------------------------------------------------------------ what a pass cannot do without

def work(case):
    kind = case["kind"]
    if kind == "mlp":
        n = case["rows"]
        macs = _D * _H + _H * _H + _H
        # forward, weight gradients, and input gradients of the two upper layers; features, targets, p, m, v, g
        return {"bytes": 4 * (n * (_D + 1) + 8 * sum(_SPLIT)), "flops": 2 * n * (2 * macs + macs - _D * _H)}
    steps = case["steps"]
    if kind == "heat":
        cells = sum((n - 2) ** 2 for n in _sides(case)) * steps
        return {"bytes": 16 * cells, "flops": 8 * cells}
    rank, n = case.get("rank", 3), case["n"]
    cells, size = (n - 2) ** rank * steps, 4 if kind == "generated" else 8
    if kind == "sor":
        return {"bytes": 2 * size * cells, "flops": 11 * cells}
    return {"bytes": 4 * size * cells, "flops": (2 * rank + 2) * cells}  # A and B read and written


# ------------------------------------------------------------------ the same in 64 bits

def _exact_jacobi(case, seed):
    rank = case["rank"]
    a, b = (t.double() for t in _jacobi_inputs(case, seed, torch.float32 if case["kind"] == "generated" else
                                               torch.float64))
    n, inner = case["n"], (slice(1, -1),) * rank
    eps = []
    for _ in range(case["steps"]):
        eps.append(float((b[inner] - a[inner]).abs().max()))
        a[inner] = b[inner]
        total = None
        for d, lo in [(d, 0) for d in range(rank)] + [(d, 2) for d in reversed(range(rank))]:
            part = a[tuple(slice(lo, lo + n - 2) if x == d else slice(1, -1) for x in range(rank))]
            total = part.clone() if total is None else total.add_(part)
        b[inner] = total / (2 * rank)
    return {"A": a, "B": b, "eps": np.array(eps)}


def _exact_sor(case, seed):
    n = case["n"]
    a = _field(seed, (n,) * 3, case["scale"])
    flat, m = a.view(-1), n - 2
    r = torch.arange(m, device="cuda")
    plane = (r[:, None, None] + r[None, :, None] + r[None, None, :]).view(-1)
    counts = torch.bincount(plane).tolist()
    order = torch.argsort(plane)
    del plane
    k, j, i = order % m + 1, order // m % m + 1, order // (m * m) + 1
    order = (i * n + j) * n + k  # the interior's cells, hyperplane by hyperplane
    del i, j, k
    sums = []
    for _ in range(case["steps"]):
        s, at = torch.zeros((), dtype=torch.float64, device="cuda"), 0
        for c in counts:
            q = order[at:at + c]
            at += c
            old = flat[q]
            new = (1.0 - OMEGA) * old + OMEGA / 6.0 * (flat[q - n * n] + flat[q + n * n] + flat[q - n] + flat[q + n] +
                                                       flat[q - 1] + flat[q + 1])
            flat[q] = new
            s += (new - old).square().sum()
        sums.append(float(s))
    return {"A": a, "sums": np.array(sums)}


def _exact_heat(case, seed):
    us, sums, mins = [], [], []
    for k, n in enumerate(_sides(case)):
        u = _field(seed + k, (n, n), case["scale"])
        s, m = [], []
        for _ in range(case["steps"]):
            c = u[1:-1, 1:-1]
            new = c + COEF * (u[:-2, 1:-1] + u[2:, 1:-1] + u[1:-1, :-2] + u[1:-1, 2:] - 4.0 * c)
            u[1:-1, 1:-1] = new
            s.append(new.sum())
            m.append(new.min())
        us.append(u.view(-1))
        sums.append(torch.stack(s))
        mins.append(torch.stack(m))
    return {"u": torch.cat(us), "sums": torch.stack(sums, 1), "mins": torch.stack(mins, 1), "locs": None}


def _exact_mlp(case, seed):
    x, y, p = (t.double() for t in _mlp_inputs(case["rows"], seed))
    p.requires_grad_(True)
    w1, b1, w2, b2, w3, b3 = p.split(_SPLIT)
    h = torch.relu(x @ w1.view(_H, _D).t() + b1)
    h = torch.relu(h @ w2.view(_H, _H).t() + b2)
    loss = ((h @ w3 + b3 - y) ** 2).mean()
    g, = torch.autograd.grad(loss, p)
    c1, c2 = (1.0 - float(np.float32(b)) for b in (0.9, 0.999))  # Adam's constants are FP32 numbers
    m, v = c1 * g, c2 * g * g
    new = p.detach() - float(np.float32(1e-3)) * (m / c1) / ((v / c2).sqrt() + float(np.float32(1e-8)))
    return {"loss": loss.detach().view(1), "grad": g, "params": new, "m": m, "v": v}


def exact(case, seed):
    kind = case["kind"]
    if kind == "sor":
        return _exact_sor(case, seed)
    if kind == "heat":
        return _exact_heat(case, seed)
    return _exact_mlp(case, seed) if kind == "mlp" else _exact_jacobi(case, seed)
