"""The work this framework is used for, as cases that can be timed.

A case is one of its three ways to advance two-state shock decks:

chunk     one deck resident on the GPU (``Chunk``): ``step`` enqueues hydro
          steps, then the program reads the field summaries, the timesteps and,
          on the smaller grids, the state itself.
ensemble  many decks of drawn sizes advanced together (``Ensemble``), read by
          their per-deck summaries.
dropin    the reference's control flow over the drop-in C ABI (``DropIn``):
          one ABI call per reference kernel, dt returned to the host each step.

A pass continues the run of its state by ``steps`` hydro steps; FP64 and the
mixed FP32-storage policy both occur. Sizes are those of the tests, the
benchmark and the reference's decks (10x2x2, 32^3, 96^3, 512^3; ensembles of
24..128 and 16..48 cells per axis), and ragged ones between them.

``exact`` restates the hydro cycle in plain torch, in 64 bits, on whole arrays.
"""
import random

import numpy as np
import torch

import cloverleaf3d_ref_b200 as C

#: Far more steps than a program takes, so that no pass meets the decks' end.
END_STEP = {"chunk": 2_000_000, "ensemble": 20_000, "dropin": 2_000_000}

VELOCITIES = ("xvel0", "yvel0", "zvel0")


def listed():
    return [
        # the smallest deck, the reference's known-answer problem: all launches and latency
        dict(name="chunk_10x2x2", kind="chunk", nx=10, ny=2, nz=2, steps=75, mixed=False, fields=True),
        # a small development deck
        dict(name="chunk_32", kind="chunk", nx=32, ny=32, nz=32, steps=100, mixed=False, fields=True),
        # the size of the reference's clover.in
        dict(name="chunk_96", kind="chunk", nx=96, ny=96, nz=96, steps=100, mixed=False, fields=True),
        # an uneven grid whose rows and planes fill no tile
        dict(name="chunk_ragged", kind="chunk", nx=150, ny=61, nz=83, steps=60, mixed=False, fields=True),
        # the same of a larger grid, FP32 storage
        dict(name="chunk_ragged_mixed", kind="chunk", nx=203, ny=311, nz=118, steps=30, mixed=True, fields=False),
        # a medium production grid
        dict(name="chunk_256", kind="chunk", nx=256, ny=256, nz=256, steps=20, mixed=False, fields=False),
        # the headline grid, both policies
        dict(name="chunk_512", kind="chunk", nx=512, ny=512, nz=512, steps=20, mixed=False, fields=False),
        dict(name="chunk_512_mixed", kind="chunk", nx=512, ny=512, nz=512, steps=20, mixed=True, fields=False),
        # parameter studies: many decks at once, with the autotuner's schedules and with the default ones
        dict(name="ensemble_64", kind="ensemble", decks=64, lo=24, hi=128, steps=10, mixed=False, tuned=True),
        dict(name="ensemble_512_mixed", kind="ensemble", decks=512, lo=16, hi=48, steps=20, mixed=True, tuned=False),
        # the reference's own drivers relinked against the C ABI
        dict(name="dropin_96", kind="dropin", nx=96, ny=96, nz=96, steps=20),
        dict(name="dropin_208", kind="dropin", nx=208, ny=208, nz=208, steps=10),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    """A chunk (three in five), an ensemble or a drop-in run of drawn sizes."""
    u = rng.random()
    if u < 0.6:
        while True:
            n = [_log(rng, 2, 400) for _ in range(3)]
            cells = n[0] * n[1] * n[2]
            if 32 <= cells <= 48_000_000:
                break
        steps = max(10, min(100, 150_000_000 // cells))
        return dict(kind="chunk", nx=n[0], ny=n[1], nz=n[2], steps=steps, mixed=rng.random() < 0.4,
                    fields=cells <= 1_000_000)
    if u < 0.8:
        decks = _log(rng, 2, 48)
        lo = _log(rng, 8, 40)
        return dict(kind="ensemble", decks=decks, lo=lo, hi=lo + _log(rng, 4, 80),
                    steps=rng.randint(4, 12), mixed=rng.random() < 0.5, tuned=rng.random() < 0.5)
    while True:
        n = [_log(rng, 3, 240) for _ in range(3)]
        cells = n[0] * n[1] * n[2]
        if 64 <= cells <= 6_000_000:
            break
    return dict(kind="dropin", nx=n[0], ny=n[1], nz=n[2], steps=rng.randint(5, 20))


def _states(rng):
    """A light background and a denser, hotter cuboid in its corner."""
    u, v, w = (rng.uniform(1.0, 6.0) for _ in range(3))
    return [dict(density=rng.uniform(0.15, 0.3), energy=rng.uniform(0.5, 1.5)),
            dict(density=rng.uniform(0.7, 1.5), energy=rng.uniform(1.5, 3.0), geometry="cuboid",
                 xmin=0.0, xmax=u, ymin=0.0, ymax=v, zmin=0.0, zmax=w)]


def _decks(case, seed):
    """The values of the case's decks: [0,10]^3; cubic cells where an axis is much longer than another, as a bar of
    unit cells for grids a few cells thick."""
    rng = random.Random(seed)
    n = case["decks"] if case["kind"] == "ensemble" else 1
    out = []
    # the sizes belong to the case, the states to the seed
    sizes = random.Random(1000 * case["decks"] + case["lo"]) if case["kind"] == "ensemble" else None
    for _ in range(n):
        if sizes:
            nx, ny, nz = (sizes.randint(case["lo"], case["hi"]) for _ in range(3))
        else:
            nx, ny, nz = case["nx"], case["ny"], case["nz"]
        d = dict(x_cells=nx, y_cells=ny, z_cells=nz, xmin=0.0, ymin=0.0, zmin=0.0, xmax=10.0, ymax=10.0,
                 zmax=10.0, initial_timestep=0.04, max_timestep=0.04, timestep_rise=1.5,
                 end_step=END_STEP[case["kind"]], end_time=1.0e9, summary_frequency=10)
        least = min(nx, ny, nz)
        if case["kind"] != "ensemble" and (least < 8 or max(nx, ny, nz) > 3 * least):
            h = 1.0 if least < 8 else 10.0 / least
            d.update(xmax=nx * h, ymax=ny * h, zmax=nz * h)
        out.append(dict(d, states=_states(rng)))
    return out


def prepare(case, seed):
    """The decks set up on the GPU at step 0."""
    decks = [C.Deck.from_values(d["states"], **{k: v for k, v in d.items() if k != "states"})
             for d in _decks(case, seed)]
    state = {"case": case, "n": 0}
    if case["kind"] == "dropin":
        state["run"] = C.DropIn(decks[0])
        return state
    precision = C.PRECISION_MIXED if case["mixed"] else C.PRECISION_FP64
    if case["kind"] == "chunk":
        state["run"] = C.Chunk(decks[0], precision)
        return state
    state["run"] = C.Ensemble(decks, precision)
    if case["tuned"]:
        state["run"].autotune(1)
    return state


def run(state):
    """The run's next steps, and what its program reads of them."""
    case, r = state["case"], state["run"]
    if case["kind"] == "dropin":
        state["n"] += case["steps"]
        r.run(state["n"])
        return {"dt": r.dt_history(), "summaries": r.summaries()[0]}
    r.step(case["steps"])
    if case["kind"] == "ensemble":
        return {"summaries": np.stack([r.deck_summaries(d)[0] for d in range(len(r))])}
    out = {"dt": r.dt_history(), "summaries": r.summaries()[0]}
    if case["fields"]:
        out.update(_state(r))
    return out


def _state(r):
    """The state a program reads back; the velocity as one vector field, whose components can each be rounding alone."""
    return {"density0": r.field("density0"), "energy0": r.field("energy0"),
            "velocity0": np.stack([r.field(name) for name in VELOCITIES])}


def _cells(case):
    if case["kind"] == "ensemble":
        return sum(d["x_cells"] * d["y_cells"] * d["z_cells"] for d in _decks(case, 0))
    return case["nx"] * case["ny"] * case["nz"]


def work(case):
    """Per step, the state (density, energy, three velocities) once in and once out: calc_dt's minimum over the whole
    grid stands between any two steps. No flops are counted: a handful per byte, on no matrix unit."""
    per_cell = 2 * (8 + 4 * 4 if case.get("mixed") else 5 * 8)
    return {"bytes": per_cell * _cells(case) * case["steps"], "flops": 0}


def tolerance(case):
    """About four times, and more at single values next to a shock, what the path measures against exact(): 1e-14 in
    FP64 (sums in another order, grown over the steps), 1e-6 in the mixed policy (the stencils' FP32 roundings)."""
    if case.get("mixed"):
        return {"rel": 1.0e-5, "max": 5.0e-3}
    return {"rel": 1.0e-13, "max": 1.0e-10}


def exact(case, seed):
    """What run() returns, from a plain 64-bit torch restatement of the hydro cycle (None where it would take long)."""
    if case["kind"] == "ensemble" and case["decks"] > 80:
        return None
    runs = [_Hydro(d) for d in _decks(case, seed)]
    for h in runs:
        for _ in range(case["steps"]):
            h.step()
    if case["kind"] == "ensemble":
        return {"summaries": np.stack([h.summaries() for h in runs])}
    h = runs[0]
    if case["kind"] == "dropin":  # run() ends each call with a summary of its own
        h.summary()
        return {"dt": h.dts(), "summaries": h.summaries()}
    out = {"dt": h.dts(), "summaries": h.summaries()}
    if case["fields"]:
        out.update(_state(h))
    return out


class _Hydro:
    """The hydro cycle on one uniform mesh, arrays held as [z, y, x] with every index from -1."""

    G_SMALL, G_BIG = 1.0e-16, 1.0e21

    def __init__(self, d):
        self.d = d
        self.n = [d["x_cells"], d["y_cells"], d["z_cells"]]
        self.dx = [(d[a + "max"] - d[a + "min"]) / n for a, n in zip("xyz", self.n)]
        dx, dy, dz = self.dx
        self.vol, self.area = dx * dy * dz, [dy * dz, dx * dz, dx * dy]
        new = lambda: torch.zeros([n + 5 for n in reversed(self.n)], dtype=torch.float64, device="cuda")  # noqa: E731
        names = ["d0", "d1", "e0", "e1", "p", "q", "c", "pre", "post", "ef", "nf", "npost", "npre", "mom"]
        self.a = {k: new() for k in names + [f + str(i) for f in ("u", "v", "m") for i in range(3)] + ["w0", "w1", "w2"]}
        self.t = self.old = torch.tensor(d["initial_timestep"], dtype=torch.float64, device="cuda")
        self.steps, self.ax, self.dt_list, self.sums = 0, True, [], []
        self._generate()
        self.eos("d0", "e0")
        for f in ("d0", "e0", "p", "q", "d1", "e1"):
            self.halo_cell(f, 2)
        for k in range(3):
            self.halo_vel("u%d" % k, k, 2)
            self.halo_vel("w%d" % k, k, 2)
        self.summary()

    # u: velocities at time level 0, w: at level 1, v: volume fluxes, m: mass fluxes

    def s(self, name, lo, hi, off=(0, 0, 0)):
        """The view of a array over indices lo..hi (x, y, z), shifted by off."""
        a = self.a[name] if isinstance(name, str) else name
        return a[tuple(slice(lo[i] + off[i] + 1, hi[i] + off[i] + 2) for i in (2, 1, 0))]

    def _generate(self):
        d = self.d
        lo, hi = [-1] * 3, [n + 2 for n in self.n]
        for i, st in enumerate(d["states"]):
            if i == 0:
                self.s("d0", lo, hi).fill_(st["density"])
                self.s("e0", lo, hi).fill_(st["energy"])
                continue
            inside = None
            for k, a in enumerate("xyz"):
                j = torch.arange(-1, self.n[k] + 3, dtype=torch.float64, device="cuda")
                left, right = d[a + "min"] + self.dx[k] * (j - 1), d[a + "min"] + self.dx[k] * j
                b0, b1 = st[a + "min"] + self.dx[k] / 100.0, st[a + "max"] - self.dx[k] / 100.0
                one = ((right >= b0) & (left < b1)).reshape([-1 if q == 2 - k else 1 for q in range(3)])
                inside = one if inside is None else inside & one
            self.s("d0", lo, hi)[inside] = st["density"]
            self.s("e0", lo, hi)[inside] = st["energy"]

    # reflective faces, in the reference's order and extents
    def face(self, name, axis, high, depth, lo, hi, dst, src, sign):
        for m in range(1, depth + 1):
            to, of = (dst + m, src - m) if high else (1 - m, src + m)
            l1, h1, l2, h2 = list(lo), list(hi), list(lo), list(hi)
            l1[axis] = h1[axis] = to
            l2[axis] = h2[axis] = of
            self.s(name, l1, h1).copy_(sign * self.s(name, l2, h2))

    def halo_cell(self, name, d):
        lo, hi = [1 - d] * 3, [n + d for n in self.n]
        for k in (1, 0, 2):
            self.face(name, k, False, d, lo, hi, 0, 0, 1.0)
            self.face(name, k, True, d, lo, hi, self.n[k], self.n[k] + 1, 1.0)

    def halo_vel(self, name, comp, d):
        lo, hi = [1 - d] * 3, [n + 1 + d for n in self.n]
        for k in (1, 0, 2):
            sign = -1.0 if k == comp else 1.0
            self.face(name, k, False, d, lo, hi, 0, 1, sign)
            self.face(name, k, True, d, lo, hi, self.n[k] + 1, self.n[k] + 1, sign)

    def halo_flux(self, name, comp, d, volume):
        for k in (1, 0, 2):
            for high in (False, True):
                lo, hi = [1 - d] * 3, [n + d for n in self.n]
                # the faces along the flux's own axis reach one further, except an x or y flux on the z faces and
                # the volume flux z on the low y face
                if k != comp and not (k == 2 and comp < 2) and not (volume and comp == 2 and k == 1 and not high):
                    hi[comp] += 1
                n = self.n[k]
                if k == comp:
                    self.face(name, k, high, d, lo, hi, n + 1 if high else 0, n + 1 if high else 1, -1.0)
                else:
                    self.face(name, k, high, d, lo, hi, n if high else 0, n if high else 1, 1.0)

    def eos(self, den, ene):
        lo, hi = [1] * 3, self.n
        d, e = self.s(den, lo, hi), self.s(ene, lo, hi)
        v, p = 1.0 / d, (1.4 - 1.0) * d * e
        self.s("p", lo, hi).copy_(p)
        self.s("c", lo, hi).copy_(torch.sqrt(v * v * (p * ((1.4 - 1.0) * d) + d * p)))

    def corners(self, name, axis, side):
        """The sum of a node array over the four corners of each cell's low or high face of an axis."""
        lo, hi = [1] * 3, self.n
        total = 0.0
        others = [k for k in range(3) if k != axis]
        for b in (0, 1):
            for a in (0, 1):
                off = [0, 0, 0]
                off[axis], off[others[0]], off[others[1]] = side, a, b
                total = total + self.s(name, lo, hi, off)
        return total

    def viscosity_and_dt(self):
        lo, hi = [1] * 3, self.n
        diff = [[self.corners("u%d" % i, k, 1) - self.corners("u%d" % i, k, 0) for k in range(3)] for i in range(3)]
        div = sum(self.area[k] * diff[k][k] for k in range(3))
        g = []
        for k in range(3):
            off = [0, 0, 0]
            off[k] = 1
            g.append((self.s("p", lo, hi, off) - self.s("p", lo, hi, [-o for o in off])) / (2.0 * self.dx[k]))
        lim = sum(0.25 * diff[k][k] / self.dx[k] * g[k] * g[k] for k in range(3))
        for i, k in ((0, 1), (0, 2), (1, 2)):
            lim = lim + (0.25 * diff[i][k] / self.dx[k] + 0.25 * diff[k][i] / self.dx[i]) * g[i] * g[k]
        lim = lim / torch.clamp(sum(x * x for x in g), min=1.0e-16)
        g = [torch.copysign(torch.clamp(x.abs(), min=1.0e-16), x) for x in g]
        norm = torch.sqrt(sum(x * x for x in g))
        grad = torch.minimum(torch.minimum((self.dx[0] * norm / g[0]).abs(), (self.dx[1] * norm / g[1]).abs()),
                             (self.dx[2] * norm / g[2]).abs())
        d0 = self.s("d0", lo, hi)
        q = torch.where((lim > 0.0) | (div >= 0.0), torch.zeros_like(lim), 2.0 * d0 * grad * grad * lim * lim)
        self.s("q", lo, hi).copy_(q)
        del g, lim, grad, norm
        c = self.s("c", lo, hi)
        small = min(self.dx)
        dt = 0.75 / torch.clamp(torch.sqrt((c * c + 2.0 * q / d0) / (small * small)), min=self.G_SMALL)
        for k in range(3):
            x = torch.maximum(self.corners("u%d" % k, k, 0).abs(), self.corners("u%d" % k, k, 1).abs()) * self.area[k]
            dt = torch.minimum(dt, 0.5 * 4.0 * self.vol / torch.clamp(x, min=1.0e-5 * self.vol))
        dt = torch.minimum(dt, 0.5 * 4.0 * self.vol / torch.clamp(div.abs(), min=1.0e-5 * self.vol))
        return dt.min()

    def pdv(self, predict):
        lo, hi = [1] * 3, self.n
        second = "u" if predict else "w"
        f = [[self.area[k] * (self.corners("u%d" % k, k, sd) + self.corners(second + str(k), k, sd)) * 0.125 * self.t *
              (0.5 if predict else 1.0) for sd in (0, 1)] for k in range(3)]
        total = sum(x[1] - x[0] for x in f)
        d0 = self.s("d0", lo, hi)
        change = (self.s("p", lo, hi) + self.s("q", lo, hi)) / d0 * total / self.vol
        self.s("e1", lo, hi).copy_(self.s("e0", lo, hi) - change)
        self.s("d1", lo, hi).copy_(d0 * (self.vol / (self.vol + total)))

    def accelerate(self):
        lo, hi = [1] * 3, [n + 1 for n in self.n]
        at = lambda name, o: self.s(name, lo, hi, o)  # noqa: E731
        mass = sum(at("d0", (x, y, z)) for x in (-1, 0) for y in (-1, 0) for z in (-1, 0)) * self.vol * 0.125
        step = 0.25 * self.t / mass
        for k in range(3):
            others = [i for i in range(3) if i != k]
            total = 0.0
            for a in (0, -1):
                for b in (0, -1):
                    o = [0, 0, 0]
                    o[others[0]], o[others[1]] = a, b
                    below = list(o)
                    below[k] = -1
                    total = total + self.area[k] * ((at("p", o) - at("p", below)) + (at("q", o) - at("q", below)))
            self.s("w%d" % k, lo, hi).copy_(at("u%d" % k, (0, 0, 0)) - step * total)

    def flux_calc(self):
        for k in range(3):
            lo, hi = [1] * 3, list(self.n)
            hi[k] += 1
            others = [i for i in range(3) if i != k]
            total = 0.0
            for f in "uw":
                for a, b in ((0, 0), (1, 0), (0, 1), (1, 1)):
                    if k == 2 and f == "u" and (a, b) == (0, 1):
                        a, b = 1, 0  # flux_calc_kernel.f90:86 takes this node twice
                    o = [0, 0, 0]
                    o[others[0]], o[others[1]] = a, b
                    total = total + self.s(f + str(k), lo, hi, o)
            self.s("v%d" % k, lo, hi).copy_(0.125 * self.t * self.area[k] * total)

    def through(self, k, lo, hi):
        """The difference of the volume flux of an axis over each cell."""
        o = [0, 0, 0]
        o[k] = 1
        return self.s("v%d" % k, lo, hi, o) - self.s("v%d" % k, lo, hi)

    def along(self, name, k, lo, hi, i):
        o = [0, 0, 0]
        o[k] = i
        return self.s(name, lo, hi, o)

    def advec_cell(self, sweep, k):
        lo, hi = [-1] * 3, [n + 2 for n in self.n]
        if sweep == 1:
            add = (0, 1, 2)
        elif sweep == 2:
            add = (1, 2) if self.ax else (1, 0)
        else:
            add = (k,)
        self.s("pre", lo, hi).copy_(self.vol + sum(self.through(i, lo, hi) for i in add))
        lo, hi = [1] * 3, list(self.n)
        hi[k] += 2
        if k == 1:
            hi[2] += 2  # the y fluxes reach into the z halo
        at = lambda name, i: self.along(name, k, lo, hi, i)  # noqa: E731
        vf = at("v%d" % k, 0)
        pos = vf > 0.0

        def upwind(name):
            """Two beyond the face's low side, or the cell after its high one, which stops at the last halo cell."""
            high = at(name, 0).clone()
            last = [slice(None)] * 3
            last[2 - k] = slice(0, high.shape[2 - k] - 1)
            high[tuple(last)] = at(name, 1)[tuple(last)]
            return torch.where(pos, at(name, -2), high)

        def limited(name, sig, sig3, sig4):
            donor = torch.where(pos, at(name, -1), at(name, 0))
            du, dd = donor - upwind(name), torch.where(pos, at(name, 0), at(name, -1)) - donor
            one = torch.ones_like(dd)
            lim = (1.0 - sig) * torch.copysign(one, dd) * torch.minimum(
                torch.minimum(du.abs(), dd.abs()), (sig3 * du.abs() + sig4 * dd.abs()) / 6.0)
            return donor, torch.where(du * dd > 0.0, lim, torch.zeros_like(lim))

        pre = torch.where(pos, at("pre", -1), at("pre", 0))
        sig = vf.abs() / pre
        donor, lim = limited("d1", sig, 1.0 + sig, 2.0 - sig)
        mf = vf * (donor + lim)
        self.s("m%d" % k, lo, hi).copy_(mf)
        sigm = mf.abs() / (donor * pre)
        donor, lim = limited("e1", sigm, 1.0 + sig, 2.0 - sig)
        self.s("ef", lo, hi).copy_(mf * (donor + lim))
        del pre, sig, sigm, donor, lim, mf
        lo, hi = [1] * 3, list(self.n)
        mass = self.s("d1", lo, hi) * self.s("pre", lo, hi)
        after = mass + at_diff(self, "m%d" % k, k, lo, hi)
        ener = (self.s("e1", lo, hi) * mass + at_diff(self, "ef", k, lo, hi)) / after
        volume = self.s("pre", lo, hi) + at_diff(self, "v%d" % k, k, lo, hi)
        self.s("d1", lo, hi).copy_(after / volume)
        self.s("e1", lo, hi).copy_(ener)

    def advec_mom(self, sweep, k):
        lo, hi = [-1] * 3, [n + 2 for n in self.n]
        if sweep == 1:
            add = (1, 2) if k == 0 else (0, 1)
        elif sweep == 2:
            add = (2,) if self.ax else (0,)
        else:
            add = ()
        self.s("post", lo, hi).copy_(torch.full_like(self.s("post", lo, hi), self.vol) +
                                     sum(self.through(i, lo, hi) for i in add))
        others = [i for i in range(3) if i != k]
        lo, hi = [1] * 3, [n + 1 for n in self.n]
        lo[k], hi[k] = -1, self.n[k] + 2
        flux = 0.0
        for c in (0, 1):
            for a in (-1, 0):
                for b in (-1, 0):
                    o = [0, 0, 0]
                    o[k], o[others[0]], o[others[1]] = c, a, b
                    flux = flux + self.s("m%d" % k, lo, hi, o)
        self.s("nf", lo, hi).copy_(0.125 * flux)
        lo[k] = 0
        mass = 0.0
        for z in (-1, 0):
            for y in (-1, 0):
                for x in (-1, 0):
                    mass = mass + self.s("d1", lo, hi, (x, y, z)) * self.s("post", lo, hi, (x, y, z))
        self.s("npost", lo, hi).copy_(0.125 * mass)
        self.s("npre", lo, hi).copy_(0.125 * mass + at_diff(self, "nf", k, lo, hi, -1))
        del flux, mass
        hi[k] = self.n[k] + 1
        at = lambda name, i: self.along(name, k, lo, hi, i)  # noqa: E731
        nf = at("nf", 0)
        neg = nf < 0.0
        sig = nf.abs() / torch.where(neg, at("npre", 1), at("npre", 0))
        inner = [1] * 3, [n + 1 for n in self.n]
        for i in range(3):
            name = "w%d" % i
            donor = torch.where(neg, at(name, 1), at(name, 0))
            du = donor - torch.where(neg, at(name, 2), at(name, -1))
            dd = torch.where(neg, at(name, 0), at(name, 1)) - donor
            w = self.dx[k]
            lim = torch.minimum(torch.minimum(
                w * ((2.0 - sig) * dd.abs() / w + (1.0 + sig) * du.abs() / w) / 6.0, du.abs()), dd.abs())
            lim = torch.where(du * dd > 0.0, torch.where(dd <= 0.0, -lim, lim), torch.zeros_like(lim))
            self.s("mom", lo, hi).copy_((donor + (1.0 - sig) * lim) * nf)
            change = at_diff(self, "mom", k, *inner, -1)
            self.s(name, *inner).copy_((self.s(name, *inner) * self.s("npre", *inner) - change) / self.s("npost", *inner))

    def step(self):
        self.eos("d0", "e0")
        for f in ("p", "e0", "d0"):
            self.halo_cell(f, 1)
        for k in (0, 1):
            self.halo_vel("u%d" % k, k, 1)
        least = self.viscosity_and_dt()
        self.halo_cell("q", 1)
        self.t = torch.minimum(torch.minimum(torch.clamp(least, max=self.G_BIG), self.old * self.d["timestep_rise"]),
                               torch.full_like(least, self.d["max_timestep"]))
        self.old = self.t
        self.dt_list.append(self.t)
        self.pdv(True)
        self.eos("d1", "e1")
        self.halo_cell("p", 1)
        lo, hi = [1] * 3, self.n
        for a, b in (("d1", "d0"), ("e1", "e0")):
            self.s(a, lo, hi).copy_(self.s(b, lo, hi))
        self.accelerate()
        self.pdv(False)
        self.flux_calc()
        for sweep, k in ((1, 0 if self.ax else 2), (2, 1), (3, 2 if self.ax else 0)):
            if sweep < 3:
                self.halo_cell("e1", 2)
                self.halo_cell("d1", 2)
                for i in range(3):
                    self.halo_flux("v%d" % i, i, 2, True)
            self.advec_cell(sweep, k)
            self.halo_cell("d1", 2)
            self.halo_cell("e1", 2)
            for i in range(3):
                self.halo_vel("w%d" % i, i, 2)
                self.halo_flux("m%d" % i, i, 2, False)
            self.advec_mom(sweep, k)
        for a, b in (("d0", "d1"), ("e0", "e1")):
            self.s(a, lo, hi).copy_(self.s(b, lo, hi))
        for i in range(3):
            self.s("u%d" % i, lo, [n + 1 for n in hi]).copy_(self.s("w%d" % i, lo, [n + 1 for n in hi]))
        self.ax = not self.ax
        self.steps += 1
        if self.steps % self.d["summary_frequency"] == 0:
            self.summary()

    def summary(self):
        self.eos("d0", "e0")
        lo, hi = [1] * 3, self.n
        v2 = 0.0
        for i in range(3):
            for x in (0, 1):
                for y in (0, 1):
                    for z in (0, 1):
                        v2 = v2 + 0.125 * self.s("u%d" % i, lo, hi, (x, y, z)) ** 2
        mass = self.vol * self.s("d0", lo, hi)
        cells = self.n[0] * self.n[1] * self.n[2]
        self.sums.append(torch.stack([torch.full_like(mass.sum(), self.vol * cells), mass.sum(),
                                      (mass * self.s("e0", lo, hi)).sum(), (mass * 0.5 * v2).sum(),
                                      (self.vol * self.s("p", lo, hi)).sum()]))

    def dts(self):
        return torch.stack(self.dt_list).cpu().numpy()

    def summaries(self):
        return torch.stack(self.sums).cpu().numpy()

    def field(self, name):
        """A field as Fortran orders it, in the shape the reference declares."""
        a = self.a[{"density0": "d0", "energy0": "e0", "xvel0": "u0", "yvel0": "u1", "zvel0": "u2"}[name]]
        a = a.permute(2, 1, 0)
        return (a if name[1:] == "vel0" else a[:-1, :-1, :-1]).cpu().numpy()


def at_diff(h, name, k, lo, hi, back=1):
    """A face or node array's inflow less its outflow along an axis; back=-1: over the interval before each node,
    as the value there less the one before it."""
    if back == 1:
        return h.along(name, k, lo, hi, 0) - h.along(name, k, lo, hi, 1)
    return h.along(name, k, lo, hi, 0) - h.along(name, k, lo, hi, -1)
