"""Performance cases of the channel-flow engine: what its users run, over the range they run it.

Five ways in, all through the package's public calls:
  step     Instance.step_graph: RK3 time steps of one resident flow, as a long run takes them
  driver   the loop of the drop-in chanfast / channel drivers: CFL number, one step, its log row
  restart  four fields from (pinned) host arrays in the restart layout, steps, four fields back
  batch    Batch.run: an ensemble of flows of different sizes, one launch per stage
  serve    serve(): requests admitted, advanced together and retired, each result read as it retires
Grids run from 64 x 64 x 64 to 512 x 512 x 384 (x, y, wall-normal z), second and fourth order, the
z-implicit ("chanfast") and the fully implicit ("channel") scheme, power-of-two, even and odd sizes,
with and without buoyancy and a moving frame.  Everything is FP64.

A pass advances the state by whole time steps from wherever it stands and returns the interior of
u, v, w, c and p: the physical fields (a restart file holds the same points).  The wall ghost rows
around them are recomputed from these at the start of every substep and are not part of the result.
"""
import importlib
import math

import numpy as np
import torch

cf = importlib.import_module("ubiquitous-spoon_b200")

DEV = "cuda"
GZ = 3                    # wall-normal ghost rows of the engine's fields
AMP, C_AMP = 0.1, 0.01    # amplitude of the seeded perturbation (of 1.5 U_b) and of the scalar noise
# grids of the 64-flow ensemble and of the serving trace (bench.py)
ENSEMBLE_GRIDS = [(64, 64, 64), (96, 96, 64), (128, 128, 96), (192, 192, 128)]
SERVE_GRIDS = ENSEMBLE_GRIDS + [(256, 256, 192)]
# transform sizes the engine takes (factors 2, 3 and 5)
SIZES = sorted(2 ** a * 3 ** b * 5 ** c for a in range(10) for b in range(6) for c in range(4)
               if 48 <= 2 ** a * 3 ** b * 5 ** c <= 512)


# ------------------------------------------------------------------------------------------ cases
def flow(name, kind, order, nx, ny, nz, steps, scheme="chanfast", re=10000.0, dt=5e-4, lx=2 * math.pi, ly=math.pi,
         betg=0.0, uframe=0.0):
    return dict(name=name, kind=kind, scheme=scheme, order=order, nx=nx, ny=ny, nz=nz, steps=steps, re=re, dt=dt,
                lx=lx, ly=ly, betg=betg, uframe=uframe)


def many(name, kind, members, mix, steps, quantum=2):
    return dict(name=name, kind=kind, members=members, mix=mix, steps=steps, quantum=quantum)


def listed():
    return [
        # the reference's own CPU-sized case: every kernel is a few microseconds, launches and latency count
        flow("step2_64", "step", 2, 64, 64, 64, 2, re=2800.0, dt=1e-3, lx=4 * math.pi, ly=4 * math.pi / 3),
        # sizes nothing is tuned for: odd ny, no power of two, buoyancy and a moving frame on
        flow("step4_ragged", "step", 4, 90, 75, 53, 2, re=5000.0, dt=1e-3, betg=0.1, uframe=0.4),
        # one member of the ensemble on its own
        flow("step2_192", "step", 2, 192, 192, 128, 2, re=7000.0, dt=1e-3, lx=4 * math.pi, ly=4 * math.pi / 3),
        # the mid-size production run: fourth order with a scalar
        flow("step4_256", "step", 4, 256, 256, 192, 2),
        # the large production run that the benchmark quotes
        flow("step4_512", "step", 4, 512, 512, 384, 2, re=20000.0, dt=2.5e-4),
        # the fully implicit scheme, small (second order) and mid size (fourth order)
        flow("channel2_64", "step", 2, 64, 64, 64, 2, scheme="channel", re=2800.0, dt=1e-3, lx=4 * math.pi,
             ly=4 * math.pi / 3),
        flow("channel4_256", "step", 4, 256, 256, 192, 2, scheme="channel"),
        # the drop-in driver's loop: a CFL number and a log row read back for every step
        flow("driver4_128", "driver", 4, 128, 128, 96, 1, re=5000.0, dt=1e-3),
        # a restart: fields in from the host, a few steps, fields out
        flow("restart4_192", "restart", 4, 192, 160, 128, 2, re=7000.0),
        # a quarter of the 64-flow ensemble, second order
        many("ensemble2", "batch", 12, 0, 2),
        # a burst of requests, orders 2 and 4 mixed, served two steps a round
        many("serve_burst", "serve", 8, 3, 2),
    ]


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "channel", "driver", "restart", "batch", "serve"])
    if kind == "batch":
        return dict(kind="batch", members=rng.randint(4, 12), mix=rng.randrange(1, 1 << 20), steps=2, quantum=2)
    if kind == "serve":
        return dict(kind="serve", members=rng.randint(3, 8), mix=rng.randrange(1, 1 << 20), steps=rng.randint(1, 2),
                    quantum=rng.choice([1, 2, 4]))
    big = 512 if kind == "step" else 256

    def size():   # half of them powers of two, the others spread over the logarithm
        if rng.random() < 0.5:
            return rng.choice([n for n in (64, 128, 256, 512) if n <= big])
        want = math.exp(rng.uniform(math.log(48), math.log(big)))
        return min((n for n in SIZES if n <= big), key=lambda n: abs(math.log(n / want)))
    nx, ny = size(), size()
    if kind == "channel":
        nx = rng.choice([64, 128, 256])
    nz = int(round(math.exp(rng.uniform(math.log(24), math.log(384 if kind == "step" else 192)))))
    return dict(kind="step" if kind == "channel" else kind, scheme="channel" if kind == "channel" else "chanfast",
                order=rng.choice([2, 4]), nx=nx, ny=ny, nz=nz, steps=1 if kind == "driver" else 2,
                re=round(math.exp(rng.uniform(math.log(2800), math.log(20000)))), dt=2.5e-4,
                lx=2 * math.pi, ly=math.pi, betg=rng.choice([0.0, 0.0, 0.2]), uframe=rng.choice([0.0, 0.0, 0.5]))


def config(case):
    return cf.Config.make(case["order"], case["nx"], case["ny"], case["nz"], case["lx"], case["ly"], 2.0, case["dt"],
                          1.0 / case["re"], prandtl=0.71, setuframe=case["uframe"], betg_x=case["betg"],
                          scheme=case["scheme"])


def members_of(case):
    """The flows of a batch or serve case: grids, Reynolds numbers, (serve) orders and step counts from its mix."""
    rng = np.random.default_rng(case["mix"])
    grids = ENSEMBLE_GRIDS if case["kind"] == "batch" else SERVE_GRIDS
    out = []
    for m in range(case["members"]):
        nx, ny, nz = grids[int(rng.integers(len(grids)))]
        re, order = float(rng.uniform(2800.0, 10000.0)), int(rng.choice([2, 4]))
        steps = case["steps"] if case["kind"] == "batch" else case["steps"] * int(rng.integers(1, 4))
        out.append(flow("m%d" % m, "step", 2 if case["kind"] == "batch" else order, nx, ny, nz, steps, re=re, dt=1e-3,
                        lx=4 * math.pi, ly=4 * math.pi / 3))
    return out


# -------------------------------------------------------------------------------- state and pass
class DeviceField:
    """A device field of an instance as CUDA array interface; keeps the instance alive."""

    def __init__(self, inst, name, shape):
        ptr, _ = inst.device_field(name)
        self.inst = inst
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f8", data=(ptr, False), version=3)


def field_views(inst, case):
    shape = (case["nz"] + 2 * GZ, case["nx"], case["ny"])
    return {f: torch.as_tensor(DeviceField(inst, f, shape), device=DEV)[GZ:GZ + case["nz"]] for f in "uvwcp"}


def new_flow(case, seed):
    inst = cf.Instance(config(case))
    inst.init_fields(seed, AMP, C_AMP)
    return inst


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        flows = members_of(case)
        insts = [new_flow(m, seed + 1000 * q) for q, m in enumerate(flows)]
        return dict(kind=kind, steps=case["steps"], batch=cf.Batch(insts),
                    out=[field_views(i, m) for i, m in zip(insts, flows)])
    if kind == "serve":
        reqs = [dict(cfg=config(m), seed=seed + 1000 * q, amp=AMP, c_amp=C_AMP, nsteps=m["steps"], arrival_s=0.0)
                for q, m in enumerate(members_of(case))]
        # page-locked buffers for the results, kept by the server
        back = [{f: torch.empty(r["cfg"].interior_shape(), dtype=torch.float64, pin_memory=True).numpy() for f in "uvwc"}
                for r in reqs]
        return dict(kind=kind, requests=reqs, quantum=case["quantum"], back=back)
    inst = new_flow(case, seed)
    state = dict(kind=kind, steps=case["steps"], dt=case["dt"], inst=inst, out=field_views(inst, case))
    if kind == "restart":
        shape = inst.cfg.interior_shape()
        host = {f: torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy() for f in "uvwc"}
        back = {f: torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy() for f in "uvwc"}
        for f in "uvwc":
            inst.get_field(f, cf.LAYOUT_INTERIOR, out=host[f])
        state.update(host=host, back=back)
    return state


def run(state):
    kind = state["kind"]
    if kind == "step":
        state["inst"].step_graph(state["steps"])
        return state["out"]
    if kind == "batch":
        state["batch"].run(state["steps"])
        return state["out"]
    if kind == "driver":
        inst, cfl, rows = state["inst"], [], []
        for _ in range(state["steps"]):
            cfl.append(inst.cfl(state["dt"]))
            inst.step(3)
            rows.append(inst.log(1)[0])
        return dict(state["out"], cfl=cfl, log=rows)
    if kind == "restart":
        inst = state["inst"]
        for f in "uvwc":
            inst.set_field(f, state["host"][f], cf.LAYOUT_INTERIOR)
        inst.step_graph(state["steps"])
        for f in "uvwc":
            inst.get_field(f, cf.LAYOUT_INTERIOR, out=state["back"][f])
        return state["back"]
    back = state["back"]

    def done(index, view):
        for f in "uvwc":
            view.get_field(f, cf.LAYOUT_INTERIOR, out=back[index][f])

    res = cf.serve(state["requests"], 150e9, max_active=64, quantum=state["quantum"], on_done=done)
    if any(r["status"] for r in res):
        raise RuntimeError("a served request failed: %s" % [r["status"] for r in res])
    return back


def work(case):
    if case["kind"] in ("batch", "serve"):
        ws = [work(m) for m in members_of(case)]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    pts = case["nx"] * case["ny"] * case["nz"]
    sub = 3 * case["steps"]
    # a substep reads u, v, w, c and the four previous right-hand sides and writes u, v, w, c, p and the four new
    # ones; what its two global solves move in between is not counted
    moved = sub * pts * 17 * 8.0 + (8 * 8.0 * pts if case["kind"] == "restart" else 0.0)
    # right-hand sides, line solves and projection, and a 2-D real transform there and back (four more each way
    # for the fully implicit scheme)
    ffts = 1 if case["scheme"] == "chanfast" else 5
    ops = (520.0 if case["order"] == 4 else 300.0) + ffts * 5.0 * math.log2(case["nx"] * case["ny"])
    return {"bytes": moved, "flops": sub * pts * ops}


def tolerance(case):
    # FP64 throughout, but p is the inverse Laplacian of div(u*) / dt: rounding of u* by 1e-16 shows in p as up to
    # 8e-12 against the 64-bit statement below on these grids, and as 1.1e-10 after 100 steps of the fully implicit
    # scheme between two correct transforms, through which its u* passes
    return {"rel": 1e-10 if case.get("scheme") == "channel" else 4e-11}


# ------------------------------------------------------------------------- the same in plain torch
A1, A2, B1, B2 = 1.125, -0.125 / 3.0, 1.125 / 2.0, -0.125 / 2.0     # fourth-order difference, interpolation
ALP, BET = (29 / 96, -3 / 40, 1 / 6), (37 / 160, 5 / 24, 1 / 6)    # implicit RK3 weights (old, new)
GAM, ZET = (8 / 15, 5 / 12, 3 / 4), (0.0, -17 / 60, -5 / 12)       # explicit RK3 weights (new, previous)


def at_x(a, d):
    return torch.roll(a, -d, 1)


def at_y(a, d):
    return torch.roll(a, -d, 2)


class Plain:
    """One flow in 64-bit torch, fields [z, x, y] with GZ ghost rows; every solve by general elimination."""

    def __init__(self, case):
        self.c, self.o = case, case["order"]
        nz, self.n2 = case["nz"], case["nz"] + 2 * GZ
        self.k0, self.k1 = GZ, GZ + nz
        self.dx, self.dy = case["lx"] / case["nx"], case["ly"] / case["ny"]
        dz = [0.0] * self.n2
        for k in range(nz):
            dz[k + GZ] = math.cos(math.pi * k / nz) - math.cos(math.pi * (k + 1) / nz)
        for k in range(GZ):
            dz[k] = dz[2 * GZ - 1 - k]
            dz[self.n2 - 1 - k] = dz[self.n2 - 2 * GZ + k]
        self.dz = dz
        self.dzt = torch.tensor(dz, dtype=torch.float64, device=DEV)
        self.dzh = torch.cat([0.5 * (self.dzt[1:] + self.dzt[:-1]), self.dzt[:1]])   # z distance of cells k, k+1
        self.nu = 1.0 / case["re"]
        uf = case["uframe"]
        self.bc = dict(u=(-uf, -uf), v=(0.0, 0.0), c=(-0.5, 0.5), w=(0.0, 0.0))
        self.target = dict(u=1.0 - uf, c=0.0)
        self.g = {f: 0.0 for f in "uvwc"}
        self.s = 0
        self.lam = self.wavenumbers()

    def rows(self, v):
        return v.reshape(-1, 1, 1)

    # ---- wall ghost rows (in place)
    def walls(self, q, f, lo, hi, neumann=False):
        dz, n2, o = self.dz, self.n2, self.o
        if f == "w":
            for b, sgn, bc in ((GZ - 1, 1, lo), (n2 - GZ - 1, -1, hi)):
                q[b] = bc
                if o == 4:
                    near, far = (dz[b], dz[b + 1]) if sgn > 0 else (dz[b + 1], dz[b])   # ghost side, flow side
                    x0, x1 = q[b + sgn], q[b + 2 * sgn]
                    g2 = 2.0 * bc - x0
                    q[b - sgn] = g2
                    q[b - 2 * sgn] = ((-A1 / near + A2 / far) * g2 + (A1 / near + A1 / far) * bc
                                      + (A2 / near - A1 / far) * x0 - A2 / far * x1) * near / A2
            return
        for b, sgn, bc in ((GZ - 1, 1, lo), (n2 - GZ, -1, hi)):
            x0, x1, x2 = q[b + sgn], q[b + 2 * sgn], q[b + 3 * sgn]
            if o == 2:
                q[b] = x0 if neumann else 2.0 * bc - x0
                continue
            h = lambda a: 0.5 * (dz[b + sgn * a] + dz[b + sgn * (a + 1)])  # noqa: E731
            em, e0, ep = h(-1), h(0), h(1)
            g1 = x0.clone()
            g2 = x1.clone() if neumann else (bc - 0.5 * (A1 + 2 * A2) * (g1 + x0)) / (0.5 * A2) - x1
            q[b], q[b - sgn] = g1, g2
            q[b - 2 * sgn] = ((-A1 / em + 2 * A2 / e0) * g2 + (A1 / em + 2 * A1 / e0 - A2 / ep) * g1
                              + (A2 / em - 2 * A1 / e0 - A1 / ep) * x0 + (-2 * A2 / e0 + A1 / ep) * x1
                              + A2 / ep * x2) * em / A2

    # ---- z second difference on the interior rows (of a face field for w)
    def lapz(self, q, f):
        k0, k1 = self.k0, self.k1 - (f == "w")
        inner, outer = (self.dzt, self.dzh) if f == "w" else (self.dzh, self.dzt)
        off = 1 if f == "w" else 0
        h = lambda a: inner[k0 + a + off:k1 + a + off].reshape([-1] + [1] * (q.dim() - 1))  # noqa: E731
        Z = lambda a: q[k0 + a:k1 + a]  # noqa: E731
        vol = outer[k0:k1].reshape([-1] + [1] * (q.dim() - 1))
        if self.o == 2:
            return ((Z(1) - Z(0)) / h(0) - (Z(0) - Z(-1)) / h(-1)) / vol
        D = lambda a: (A1 * (Z(a + 1) - Z(a)) + A2 * (Z(a + 2) - Z(a - 1))) / h(a)  # noqa: E731
        return (A1 * (D(0) - D(-1)) + A2 * (D(1) - D(-2))) / vol

    def lapxy(self, q):
        out = 0.0
        for at, d in ((at_x, self.dx), (at_y, self.dy)):
            if self.o == 2:
                out = out + (at(q, 1) - 2.0 * q + at(q, -1)) / (d * d)
            else:
                g = A1 * (at(q, 1) - q) + A2 * (at(q, 2) - at(q, -1))
                out = out + (A1 * (g - at(g, -1)) + A2 * (at(g, 1) - at(g, -2))) / (d * d)
        return out

    def wavenumbers(self):
        def lam(n, d):
            t = 2.0 * math.pi * torch.arange(n, dtype=torch.float64, device=DEV) / n
            if self.o == 2:
                return (2 - 2 * torch.cos(t)) / (d * d)
            return ((2 * A2 * A2 + 2 * A1 * A1) + (4 * A1 * A2 - 2 * A1 * A1) * torch.cos(t)
                    - 4 * A1 * A2 * torch.cos(2 * t) - 2 * A2 * A2 * torch.cos(3 * t)) / (d * d)
        nx, ny = self.c["nx"], self.c["ny"]
        return (lam(nx, self.dx)[:nx // 2 + 1, None] + lam(ny, self.dy)[None]).reshape(-1)

    def fwd(self, a):
        return torch.fft.rfftn(a, dim=(2, 1), norm="forward").reshape(a.shape[0], -1)

    def bwd(self, a):
        nx, ny = self.c["nx"], self.c["ny"]
        return torch.fft.irfftn(a.reshape(a.shape[0], nx // 2 + 1, ny), s=(ny, nx), dim=(2, 1), norm="forward")

    # ---- column operators as matrices: z second difference with homogeneous walls, and its ghost rows
    def column(self, f, neumann=False, mean=False):
        n = self.k1 - self.k0 - (f == "w")
        E = torch.zeros(self.n2, n, dtype=torch.float64, device=DEV)
        E[self.k0:self.k0 + n] = torch.eye(n, dtype=torch.float64, device=DEV)
        if mean:      # Dirichlet at the bottom, Neumann at the top
            top = E.clone()
            self.walls(top, f, 0.0, 0.0, True)
            self.walls(E, f, 0.0, 0.0, False)
            E[self.k1:] = top[self.k1:]
        else:
            self.walls(E, f, 0.0, 0.0, neumann)
        return self.lapz(E, f), E

    @staticmethod
    def band_solve(A, shift, rhs):
        """(A + shift_c I) x_c = rhs_c for every column c: A banded (three each side), elimination in order."""
        n, band = A.shape[0], A.cpu()
        U, x, work = [], rhs.clone(), {}
        for i in range(n):
            for j in range(max(0, i - 3), min(n, i + 4)):
                work[i, j] = band[i, j].item() + (shift if i == j else 0.0)
        for i in range(n):
            piv = work[i, i]
            for r in range(i + 1, min(n, i + 4)):
                m = work[r, i] / piv
                for j in range(i + 1, min(n, i + 4)):
                    work[r, j] = work[r, j] - m * work[i, j]
                x[r] -= m * x[i]
            U.append([work[i, j] for j in range(i, min(n, i + 4))])
            for j in range(max(0, i - 3), i):
                work.pop((i, j), None)
        for i in range(n - 1, -1, -1):
            for q, u in enumerate(U[i][1:]):
                x[i] -= u * x[i + 1 + q]
            x[i] /= U[i][0]
        return x

    def pressure(self, F, dt):
        """p (with ghost rows) of (u, v, w), and the projected field."""
        u, v, w = F["u"], F["v"], F["w"]
        k0, k1 = self.k0, self.k1
        if self.o == 2:
            d = ((u - at_x(u, -1)) / self.dx + (v - at_y(v, -1)) / self.dy)[k0:k1]
            d = d + (w[k0:k1] - w[k0 - 1:k1 - 1]) / self.rows(self.dzt[k0:k1])
        else:
            D = lambda a, at: A1 * (a - at(a, -1)) + A2 * (at(a, 1) - at(a, -2))  # noqa: E731
            w = w.clone()
            w[k0 - 2] = 2 * w[k0 - 1] - w[k0]
            w[k1] = 2 * w[k1 - 1] - w[k1 - 2]
            d = (D(u, at_x) / self.dx + D(v, at_y) / self.dy)[k0:k1]
            d = d + (A1 * (w[k0:k1] - w[k0 - 1:k1 - 1]) + A2 * (w[k0 + 1:k1 + 1] - w[k0 - 2:k1 - 2])) \
                / self.rows(self.dzt[k0:k1])
        h = self.fwd(d) / dt
        A, E = self.column("p", True)
        Am, Em = self.column("p", mean=True)
        shift = -self.lam.clone()
        shift[0] = -1.0   # the mean mode has its own closure, below
        x = self.band_solve(A, shift, h)
        ph = (E.to(x.dtype) @ x)
        ph[:, 0] = (Em @ torch.linalg.solve(Am, h[:, 0].real)).to(x.dtype)
        p = self.bwd(ph)
        G = lambda at: (at(p, 1) - p) if self.o == 2 else A1 * (at(p, 1) - p) + A2 * (at(p, 2) - at(p, -1))  # noqa: E731
        F["u"][k0:k1] -= (G(at_x) * (dt / self.dx))[k0:k1]
        F["v"][k0:k1] -= (G(at_y) * (dt / self.dy))[k0:k1]
        a, b = k0 - 1, k1
        gz = p[a + 1:b + 1] - p[a:b]
        if self.o == 4:
            gz = A1 * gz + A2 * (p[a + 2:b + 2] - p[a - 1:b - 1])
        F["w"][a:b] -= gz * dt / self.rows(self.dzh[a:b])
        return p

    # ---- advection
    def flux(self, q, m, at):
        """Difference over a cell of the flux m q, m on the faces at +1/2 (periodic direction)."""
        d = m * 0.5 * (q + at(q, 1))
        d = d - at(d, -1)
        if self.o == 2:
            return d
        e = at(m, 1) * 0.5 * (q + at(q, 3))
        return A1 * d + A2 * (e - at(e, -3))

    def half(self, a, at):
        return 0.5 * (a + at(a, 1)) if self.o == 2 else B1 * (a + at(a, 1)) + B2 * (at(a, -1) + at(a, 2))

    def half_z(self, a):
        """z interpolation to the faces k+1/2 of rows 1 .. n2-3 (the others stay zero)."""
        out = torch.zeros_like(a)
        n = a.shape[0]
        if self.o == 2:
            out[:n - 1] = 0.5 * (a[:n - 1] + a[1:])
        else:
            out[1:n - 2] = B1 * (a[1:n - 2] + a[2:n - 1]) + B2 * (a[:n - 3] + a[3:])
        return out

    def flux_z(self, q, m, f):
        k0, k1 = self.k0, self.k1 - (f == "w")
        Q, M = (lambda a: q[k0 + a:k1 + a]), (lambda a: m[k0 + a:k1 + a])
        zp, zm = M(0) * 0.5 * (Q(0) + Q(1)), M(-1) * 0.5 * (Q(0) + Q(-1))
        if self.o == 2:
            return zp - zm
        p3, m3 = M(1) * 0.5 * (Q(0) + Q(3)), M(-2) * 0.5 * (Q(0) + Q(-3))
        if f != "w":
            wall = lambda a, s: 0.5 * A2 * (q[a - s] + q[a + 2 * s]) + 0.5 * (A1 + 2 * A2) * (q[a] + q[a + s])  # noqa: E731
            b, t = k0 - 1, k1
            qb, qt = wall(b, 1), wall(t, -1)
            zp[-1], zm[0] = m[t - 1] * qt, m[b] * qb
            p3[-1] = -m[t - 2] * 0.5 * (q[t - 3] + q[t]) + 2 * m[t - 1] * qt
            p3[-2] = m[t - 1] * qt
            m3[0] = -m[b + 1] * 0.5 * (q[b + 3] + q[b]) + 2 * m[b] * qb
            m3[1] = m[b] * qb
        return A1 * (zp - zm) + A2 * (p3 - m3)

    def explicit(self, F):
        """Explicit right-hand sides of u, v, w, c on their interior rows."""
        k0, k1, dx, dy = self.k0, self.k1, self.dx, self.dy
        u, v, c = F["u"], F["v"], F["c"]
        w = F["w"].clone()
        if self.o == 4:
            for b, s in ((k0 - 1, 1), (k1 - 1, -1)):
                w[b - s] = 2 * w[b] - w[b + s]
                w[b - 2 * s] = 2 * w[b] - w[b + 2 * s]
        W = dict(u=u, v=v, w=w, c=c)
        mu, mv, mw = u * self.rows(dy * self.dzt), v * self.rows(dx * self.dzt), w * (dx * dy)
        out = {}
        for f, half in (("u", lambda a: self.half(a, at_x)), ("v", lambda a: self.half(a, at_y)), ("w", self.half_z)):
            q, ke = W[f], k1 - (f == "w")
            vol = dx * dy * self.rows((self.dzh if f == "w" else self.dzt)[k0:ke])
            r = (self.flux(q, half(mu), at_x) + self.flux(q, half(mv), at_y))[k0:ke] + self.flux_z(q, half(mw), f)
            out[f] = -r / vol

        def quick(m, c0, c1, cm, c2):
            return m * (0.5 * (c0 + c1) - 0.125 * torch.where(m > 0, c1 - 2 * c0 + cm, c2 - 2 * c1 + c0))
        fx = quick(mu, c, at_x(c, 1), at_x(c, -1), at_x(c, 2))
        fy = quick(mv, c, at_y(c, 1), at_y(c, -1), at_y(c, 2))
        r = (fx - at_x(fx, -1) + fy - at_y(fy, -1))[k0:k1]
        a, b = k0 - 1, k1
        fz = quick(mw[a:b], c[a:b], c[a + 1:b + 1], c[a - 1:b - 1], c[a + 2:b + 2])
        out["c"] = -(r + fz[1:] - fz[:-1]) / (dx * dy * self.rows(self.dzt[k0:k1]))
        out["u"] = out["u"] + self.c["betg"] * self.half(c, at_x)[k0:k1]
        if self.c["scheme"] == "chanfast":
            for f in "uvwc":
                q = W[f][k0:k1 - (f == "w")]
                out[f] = out[f] + self.diffusivity(f) * self.lapxy(q)
        return out

    def diffusivity(self, f):
        return self.nu / 0.71 if f == "c" else self.nu

    # ---- one substep
    def substep(self, F):
        s, dt, k0 = self.s % 3, self.c["dt"], self.k0
        for f in "uvwc":
            self.walls(F[f], f, *self.bc[f])
        new = self.explicit(F)
        for f in "uvwc":
            k1 = self.k1 - (f == "w")
            q, nu = F[f], self.diffusivity(f)
            edge = torch.zeros(self.n2, 1, 1, dtype=torch.float64, device=DEV)
            self.walls(edge, f, *self.bc[f])
            lap = self.lapz(q, f)
            if self.c["scheme"] == "channel":
                lap = lap + self.lapxy(q[k0:k1])
            h = q[k0:k1] + ALP[s] * dt * nu * lap + dt * (GAM[s] * new[f] + ZET[s] * self.g[f]) \
                + BET[s] * dt * nu * self.lapz(edge, f)
            L, E = self.column(f)
            n = k1 - k0
            A = torch.eye(n, dtype=torch.float64, device=DEV) - BET[s] * dt * nu * L
            if self.c["scheme"] == "channel":
                q[k0:k1] = self.bwd(self.band_solve(A, BET[s] * dt * nu * self.lam, self.fwd(h)))
            else:
                q[k0:k1] = torch.linalg.solve(A, h.reshape(n, -1)).reshape(h.shape)
            self.walls(q, f, *self.bc[f])
            if f in self.target:      # constant flow rate, constant scalar mean
                G = E @ torch.linalg.solve(A, torch.full((n,), GAM[s] * dt, dtype=torch.float64, device=DEV))
                mean = lambda a: float((a[k0:k1] * self.dzt[k0:k1]).sum() / self.dzt[k0:k1].sum())  # noqa: E731
                m = (self.target[f] - mean(q.mean((1, 2)))) / mean(G)
                q += self.rows(G) * m
                new[f] = new[f] + m
        p = self.pressure(F, (ALP[s] + BET[s]) * dt)
        self.g = new
        self.s += 1
        return p

    # ---- the seeded initial state: laminar profile, SplitMix64 noise, projected
    def initial(self, seed):
        nx, ny, nz = (self.c[k] for k in ("nx", "ny", "nz"))
        wrap = lambda v: (v + (1 << 63)) % (1 << 64) - (1 << 63)  # noqa: E731
        shr = lambda z, b: (z >> b) & ((1 << (64 - b)) - 1)  # noqa: E731
        idx = torch.arange(nx * ny * nz, dtype=torch.int64, device=DEV)

        def noise(q):
            z = (idx | wrap((seed * 4 + q) << 40)) + wrap(0x9E3779B97F4A7C15)
            z = (z ^ shr(z, 30)) * wrap(0xBF58476D1CE4E5B9)
            z = (z ^ shr(z, 27)) * wrap(0x94D049BB133111EB)
            z = z ^ shr(z, 31)
            return (shr(z, 11).double() * 2.0 ** -53 * 2.0 - 1.0).reshape(nx, ny, nz).permute(2, 0, 1)
        F = {f: torch.zeros(self.n2, nx, ny, dtype=torch.float64, device=DEV) for f in "uvwc"}
        edges = torch.cumsum(self.dzt[self.k0:self.k1], 0)
        z = self.rows(edges - 0.5 * self.dzt[self.k0:self.k1])
        I = slice(self.k0, self.k1)
        F["u"][I] = 1.5 * (1 - (z - 1) ** 2) + AMP * 1.5 * noise(0)
        F["v"][I] = AMP * 1.5 * noise(1)
        F["w"][I] = AMP * 1.5 * noise(2)
        F["w"][self.k1 - 1] = 0.0
        F["c"][I] = -0.5 + z / 2 + C_AMP * noise(3)
        self.pressure(F, 1.0)
        return F


def exact(case, seed):
    if case["kind"] in ("batch", "serve"):
        out, spent = [], 0.0
        for q, m in enumerate(members_of(case)):
            spent += m["steps"] * (1.0 + m["nz"] / 100.0)   # about a second for every twenty
            if spent > 120.0:
                out.append({f: None for f in ("uvwc" if case["kind"] == "serve" else "uvwcp")})
                continue
            one = exact(m, seed + 1000 * q)
            out.append({f: one[f].permute(1, 2, 0) for f in "uvwc"} if case["kind"] == "serve" else one)
        return out
    flow_ = Plain(case)
    F = flow_.initial(seed)
    I, p, cfl = slice(flow_.k0, flow_.k1), None, []
    for n in range(3 * case["steps"]):
        if n % 3 == 0:
            cfl.append(float(max((F["u"][I].abs() / flow_.dx).max(), (F["v"][I].abs() / flow_.dy).max(),
                                 (F["w"][I].abs() / flow_.rows(flow_.dzh[I])).max())) * case["dt"])
        p = flow_.substep(F)
    out = {f: F[f][I] for f in "uvwc"}
    if case["kind"] == "restart":
        return {f: a.permute(1, 2, 0) for f, a in out.items()}
    out["p"] = p[I]
    if case["kind"] == "driver":
        out.update(cfl=cfl, log=[None] * case["steps"])
    return out
