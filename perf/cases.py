"""The propagations this framework is timed on, each through a public entry point.

Every case is a plain dict; ``kind`` says which call it stands for:

* ``single``  one drop-in MDPROP / LDPROP call (a Fortran host's call for one
  symmetry block and energy: plan, preparation and propagation in one call);
* ``rotor``   a batch of (JTOT, parity, energy) propagations of the atom +
  linear rotor system in one plan, as a MOLSCAT run over total angular momenta
  makes them;
* ``dense``   a plan over dense systems of given channel counts (mid-size
  close-coupling blocks of asymmetric tops, spin-resolved diatoms, the large
  blocks of N in the hundreds), several energies each;
* ``fields``  a magnetic-field sweep of the alkali-pair block (BOUND / FIELD):
  outward and inward MDPROP at every field and the matching counts;
* ``ldma``    MAPROP for many energies of one system;
* ``serve``   single solves of mixed size submitted at once to the server.

``prop`` is the propagator, ``via`` the entry point of a plan: "device" (device
Y in and out), "host" (host Y in and out) or "smatrix" (host Y in, S out).
"""
from __future__ import annotations

import math
from dataclasses import replace
from functools import lru_cache

import numpy as np
import torch

from molscat_b200 import alkali
from molscat_b200 import systems as S
from molscat_b200.ldma import LDMAPlan
from molscat_b200.propagators import Plan, Segment, propagate
from molscat_b200.serving import Server


def listed():
    return [
        # the smallest call: JTOT = 0, N = 6, a coarse grid; launch and set-up latency
        {"name": "single_ldj_n6", "kind": "single", "prop": "LDJ", "jtot": 0, "block": 1, "nstep": 400},
        # the reference's ordinary call: one N = 30 block over the full 4000-step grid
        {"name": "single_ldmd_n30", "kind": "single", "prop": "LDMD", "jtot": 10, "block": 1, "nstep": 4000},
        # a MOLSCAT scattering run: N 6-36, every 10th JTOT, both parities, host Y in and S out
        {"name": "rotor_ldmd_smatrix", "kind": "rotor", "prop": "LDMD", "via": "smatrix", "jmax": 80, "jstep": 10,
         "energies": 128, "nstep": 800},
        # the same run with Johnson's propagator
        {"name": "rotor_ldj_smatrix", "kind": "rotor", "prop": "LDJ", "via": "smatrix", "jmax": 16, "jstep": 4,
         "energies": 192, "nstep": 300},
        # and with the symplectic propagator (MA5)
        {"name": "rotor_ldmg5_smatrix", "kind": "rotor", "prop": "LDMG5", "via": "smatrix", "jmax": 12, "jstep": 3,
         "energies": 160, "nstep": 100},
        # blocks of 41-64 channels, ragged
        {"name": "dense_n45_60", "kind": "dense", "prop": "LDMD", "via": "device", "ns": "45,52,60", "energies": 400,
         "nstep": 40},
        # blocks of 65-200 channels in one plan, through to S matrices
        {"name": "dense_n72_199", "kind": "dense", "prop": "LDMD", "via": "smatrix", "ns": "72,90,128,199",
         "energies": 48, "nstep": 40},
        # mid-size blocks with Johnson's propagator
        {"name": "dense_ldj_n50_120", "kind": "dense", "prop": "LDJ", "via": "device", "ns": "50,85,120",
         "energies": 96, "nstep": 40},
        # BOUND / FIELD: the alkali-pair block (N = 106) over fields, out + in, with the matching counts
        {"name": "fields_n106", "kind": "fields", "fields": 148, "nout": 450, "nin": 600},
        # large blocks: an ordinary one and the largest
        {"name": "large_ldmd_n500", "kind": "dense", "prop": "LDMD", "via": "device", "ns": "500", "energies": 48,
         "nstep": 12},
        {"name": "large_ldj_n1000", "kind": "dense", "prop": "LDJ", "via": "device", "ns": "1000", "energies": 24,
         "nstep": 3},
        # MAPROP over an energy grid of one N = 30 block
        {"name": "ldma_n30", "kind": "ldma", "jtot": 10, "block": 1, "energies": 200, "nstep": 150},
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["single", "rotor", "rotor", "dense", "dense", "large", "fields", "ldma", "serve"])
    if kind == "single":
        return {"kind": "single", "prop": rng.choice(["LDMD", "LDJ"]), "jtot": rng.randint(0, 40),
                "block": rng.choice([1, 2]), "nstep": logint(400, 4000)}
    if kind == "rotor":
        prop = rng.choice(["LDMD", "LDJ", "LDMG4", "LDMG5"])
        return {"kind": "rotor", "prop": prop, "via": "smatrix",
                "jmax": rng.randint(10, 80), "jstep": rng.randint(7, 20), "energies": logint(16, 128),
                "nstep": logint(100, 500) // (3 if prop.startswith("LDMG") else 1)}
    if kind == "dense":
        ns = sorted(rng.randint(41, 200) for _ in range(rng.randint(1, 3)))
        return {"kind": "dense", "prop": rng.choice(["LDMD", "LDMD", "LDJ"]), "via": rng.choice(["device", "host", "smatrix"]),
                "ns": ",".join(str(n) for n in ns), "energies": logint(8, 64), "nstep": logint(16, 40)}
    if kind == "large":
        n = logint(201, 1000)
        return {"kind": "dense", "prop": rng.choice(["LDMD", "LDMD", "LDJ"]), "via": "device", "ns": str(n),
                "energies": rng.randint(8, 24), "nstep": rng.randint(2, 4)}
    if kind == "fields":
        return {"kind": "fields", "fields": rng.randint(40, 148), "nout": rng.randint(200, 450), "nin": rng.randint(200, 500)}
    if kind == "ldma":
        return {"kind": "ldma", "jtot": rng.randint(0, 30), "block": rng.choice([1, 2]), "energies": logint(16, 200),
                "nstep": logint(40, 150)}
    return {"kind": "serve", "prop": rng.choice(["LDMD", "LDJ"]), "nmin": 8, "nmax": rng.randint(30, 128),
            "systems": rng.randint(3, 6), "requests": logint(16, 96), "nstep": logint(16, 40)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _rotor(rng):
    """The atom + rotor system with its well depth drawn within a few percent."""
    s = S.rotor_system()
    s.epsil *= float(rng.uniform(0.97, 1.03))
    return s


def _rotor_segment(s, nstep, kind):
    rmin, rmax = S.ROTOR_RMIN_A / s.rm, S.ROTOR_RMAX_A / s.rm
    if kind.startswith("LDMG"):
        nham = len(s.lam)
        dr = (rmax - rmin) / 4000 * 4  # sectors four LDMD steps wide, from RMIN on
        return Segment.build(rmin, dr, nstep, s.pvec, nham, kind=kind)
    return Segment.build(rmin, (rmax - rmin) / max(nstep, 400), nstep, s.pvec, len(s.lam))


@lru_cache(maxsize=None)
def _rotor_coupling(jtot, block):
    return S.rotor_system().coupling(jtot, block)


@lru_cache(maxsize=2)
def _sweep(nout, nin):
    """The alkali-pair sweep 15 GHz below the lowest threshold (bound states)."""
    return replace(alkali.config4_sweep(nout=nout, nin=nin), energy_mhz=-15000.0)


def _dense_slice(n, nstep, rng):
    """nstep steps of the dense system's 3000-step grid, from the repulsive
    wall towards the well.  The couplings and radial terms come from the seed,
    the thresholds from N (so that the open channels do not change with it)."""
    c, seg, _, _ = S.synthetic_system(n, 3000, seed=int(rng.integers(1 << 30)))
    c.eint = np.sort(np.random.default_rng(n).uniform(0.0, 60.0, n))
    k0 = int(rng.integers(5, 25))
    sub = Segment(nstep, seg.dr, seg.rtab[2 * k0:2 * (k0 + nstep) + 1].copy(), seg.ptab[2 * k0:2 * (k0 + nstep) + 1].copy())
    return c, sub


def _wkb(c, seg, ereds):
    """Diagonal WKB starts (sqrt(W_ii) where locally closed, 0 where open)."""
    n = c.n
    ix = np.arange(n) * (np.arange(n) + 1) // 2 + np.arange(n)
    w = c.vl.reshape(-1, c.nvlblk)[ix, :c.nham] @ seg.ptab[0, :c.nham]
    w = w + min(1.0 / seg.rtab[0] ** 2, 1.0e16) * c.cent + c.eint
    return [np.diag(np.sqrt(np.maximum(w - e, 0.0))) for e in ereds]


def _problem(case, seed):
    """(prop, systems, segments, job system, job energy, job Y0) of a case."""
    rng = np.random.default_rng([int(seed), 77])
    kind = case["kind"]
    systems, segs, jsys, jered, y0s = [], [], [], [], []

    def add(c, seg, ereds):
        s = len(systems)
        systems.append(c)
        segs.append(seg)
        jsys.extend([s] * len(ereds))
        jered.extend(float(e) for e in ereds)
        y0s.extend(_wkb(c, seg, ereds))

    if kind in ("single", "rotor", "ldma"):
        sysm = _rotor(rng)
        prop = case.get("prop", "LDMD")
        seg = _rotor_segment(sysm, case["nstep"], prop)
        if kind == "single":
            ecm = rng.uniform(100.0, 480.0, size=1)
        else:  # the thresholds do not depend on the seed, nor do these: S keeps its shape
            ecm = S.batched_energies(case["energies"], seed=7)
        blocks = [(case["jtot"], case["block"])] if kind != "rotor" else [
            (jt, b) for jt in range(0, case["jmax"] + 1, case["jstep"]) for b in (1, 2) if sysm.channels(jt, b)]
        if kind != "rotor" and not sysm.channels(*blocks[0]):
            blocks = [(blocks[0][0], 3 - blocks[0][1])]
        for jt, b in blocks:
            add(_rotor_coupling(jt, b), seg, ecm * sysm.cm2ru)
    elif kind == "dense":
        prop = case["prop"]
        for n in (int(x) for x in case["ns"].split(",")):
            c, seg = _dense_slice(n, case["nstep"], rng)
            add(c, seg, 25.0 + 0.4 * np.arange(case["energies"]))
    elif kind == "serve":
        prop = case["prop"]
        for n in np.geomspace(case["nmin"], case["nmax"], case["systems"]).astype(int):
            c, seg = _dense_slice(int(n), case["nstep"], rng)
            add(c, seg, 25.0 + rng.uniform(0.0, 10.0, -(-case["requests"] // case["systems"])))
    else:  # fields
        prop = "LDMD"
        sw = _sweep(case["nout"], case["nin"])
        fields = float(rng.uniform(0.0, 50.0)) + np.linspace(0.0, 950.0, case["fields"])
        for seg in (sw.seg_out, sw.seg_in):
            for f in fields:
                add(sw.coupling_at(float(f)), seg, [sw.ered_at(float(f))])
    return prop, systems, segs, np.array(jsys, dtype=np.int32), np.array(jered), y0s


def prepare(case, seed):
    prop, systems, segs, jsys, jered, y0s = _problem(case, seed)
    st = {"kind": case["kind"], "prop": prop}
    if case["kind"] == "single":
        return dict(st, c=systems[0], seg=segs[0], ered=jered[0], y0=y0s[0])
    if case["kind"] == "ldma":
        return dict(st, plan=LDMAPlan(systems[0], segs[0]), y0s=y0s, jered=jered)
    if case["kind"] == "serve":
        srv = Server(prop, hbm_budget=8 << 30, streams=4, max_batch=1024, max_systems=len(systems))
        ids = [srv.add_system(c, g) for c, g in zip(systems, segs)]
        order = np.random.default_rng(int(seed)).permutation(len(jered))
        return dict(st, srv=srv, reqs=[(ids[jsys[k]], float(jered[k]), y0s[k]) for k in order])
    plan = Plan(prop, systems, segs, jsys, jered)
    y = plan.pack(y0s)
    st.update(plan=plan, y=y, via=case.get("via", "host"))
    if st["via"] == "device":
        st["y0"] = torch.from_numpy(y).cuda()
        st["yd"] = torch.empty_like(st["y0"])
        st["ints"] = torch.zeros(3, plan.njobs, dtype=torch.int32, device="cuda")
    if case["kind"] == "fields":
        nf = case["fields"]
        st["pairs"] = [(k, nf + k) for k in range(nf)]
    return st


def run(st):
    kind = st["kind"]
    if kind == "single":
        y, nodes = propagate(st["prop"], st["c"], st["seg"], st["ered"], st["y0"])
        return {"y": y, "nodes": nodes}
    if kind == "ldma":
        ys, nodes, status = st["plan"].run_host(st["y0s"], st["jered"])
        return {"y": np.stack(ys), "nodes": nodes, "status": status}
    if kind == "serve":
        srv = st["srv"]
        reqs = [srv.submit(*r) for r in st["reqs"]]
        ys = [r.wait() for r in reqs]
        nodes = np.array([r.nodes for r in reqs])
        for r in reqs:
            srv.release(r)
        return {"y": np.concatenate([y.ravel(order="F") for y in ys]), "nodes": nodes}
    plan = st["plan"]
    if st["via"] == "device":
        st["yd"].copy_(st["y0"])
        i = st["ints"]
        plan.run_device(st["yd"].data_ptr(), i[0].data_ptr(), i[1].data_ptr(), i[2].data_ptr(),
                        torch.cuda.current_stream().cuda_stream)
        return {"y": st["yd"], "nodes": i[0], "status": i[1]}
    if st["via"] == "smatrix":
        sr, si, nodes, status, _ = plan.run_host_smatrix(st["y"])
        return {"sr": sr, "si": si, "nodes": nodes, "status": status}
    y, nodes, status, _ = plan.run_host(st["y"])
    out = {"y": y, "nodes": nodes, "status": status}
    if kind == "fields":
        out["counts"] = plan.match_counts(st["pairs"])
    return out


def work(case):
    """Bytes: VL, the P rows, Y in and the results out, once each.  Flops: N^3
    an inversion, 2 NHAM N(N+1) / 2 terms a coupling sum (the reference's
    counts); MAPROP's basis change is 4 N^3 more."""
    prop, systems, segs, jsys, _, y0s = _problem(case, 0)
    ninv = {"LDMD": 2, "LDJ": 3, "LDMG4": 4, "LDMG5": 6}[prop]
    nsum = {"LDMD": 1, "LDJ": 2, "LDMG4": 5, "LDMG5": 6}[prop]
    flops = bytes_ = 0.0
    seen = set()
    for c, g in zip(systems, segs):
        key = (id(c.vl), id(g.ptab))
        if key in seen:
            continue
        seen.add(key)
        bytes_ += 8.0 * (c.vl.size + g.ptab.size)
        if prop == "LDMD" and case["kind"] != "ldma":
            flops += (c.n ** 3 + c.nham * c.n * (c.n + 1.0)) * g.nstep
    for s in jsys:
        n, nh, ns = systems[s].n, systems[s].nham, segs[s].nstep
        bytes_ += 16.0 * n * n
        if case["kind"] == "ldma":
            flops += 5.0 * n ** 3 * ns
        else:
            flops += (ninv * n ** 3 + nsum * nh * n * (n + 1.0)) * ns
    if case["kind"] == "ldma":
        bytes_ += 16.0 * systems[0].n ** 2 * segs[0].nstep
    return {"bytes": bytes_, "flops": flops}


# ---------------------------------------------------------------------------
# the same results in 64 bits from torch alone
# ---------------------------------------------------------------------------
_MG = {
    "LDMG4": (4, [0.20517766154229, 0.40302128160421, -0.12092087633891, 0.51272193319241, 0.0],
              [0.061758858135626, 0.33897802655364, 0.61479130717558, -0.14054801465937, 0.12501982279453]),
    "LDMG5": (6, [0.33983962583911, -0.088601336903027, 0.58585647682596, -0.60303935653649, 0.32358079655470,
                  0.44236379421975],
              [0.11939002928757, 0.69892737038248, -0.17131235827160, 0.40126950225135, 0.010705081848236,
               -0.058979625498031]),
}


class _Batch:
    """Jobs padded to one size NP: a padding channel is uncoupled, W = 1."""

    def __init__(self, systems, segs, jsys, jered, y0s):
        self.dev = torch.device("cuda")
        self.np_ = max(c.n for c in systems)
        self.segs = segs
        np_, nsys = self.np_, len(systems)
        nh = max(c.nham for c in systems)
        vl = np.zeros((nsys, nh, np_, np_))
        self.diag = np.zeros((nsys, np_))
        self.cent = np.zeros((nsys, np_))
        self.mask = np.zeros((nsys, np_))
        uniq = {}
        self.vid = []
        for s, c in enumerate(systems):
            n = c.n
            if id(c.vl) not in uniq:
                uniq[id(c.vl)] = len(uniq)
                v = c.vl.reshape(-1, c.nvlblk)[:n * (n + 1) // 2, :c.nham]
                col = np.repeat(np.arange(n), np.arange(1, n + 1))
                row = np.arange(n * (n + 1) // 2) - col * (col + 1) // 2
                vl[uniq[id(c.vl)], :c.nham, row, col] = v
                vl[uniq[id(c.vl)], :c.nham, col, row] = v
            self.vid.append(uniq[id(c.vl)])
            self.diag[s, :n] = c.eint[:n]
            self.diag[s, n:] = 1.0
            self.cent[s, :n] = c.cent[:n]
            self.mask[s, :n] = 1.0
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=self.dev)  # noqa: E731
        self.vl = t(vl[:len(uniq)])
        js = torch.as_tensor(np.asarray(jsys), dtype=torch.long, device=self.dev)
        self.js = js
        self.jv = torch.as_tensor(np.asarray(self.vid), dtype=torch.long, device=self.dev)[js]
        self.jmask = t(self.mask)[js]
        self.jdiag = t(self.diag)[js] - t(jered)[:, None] * self.jmask
        self.jcent = t(self.cent)[js]
        y = np.zeros((len(y0s), np_, np_))
        for j, y0 in enumerate(y0s):
            n = y0.shape[0]
            y[j, :n, :n] = y0
            y[j, range(n, np_), range(n, np_)] = 1.0
        self.y = t(y)

    def sums(self, ir):
        """The coupling sums of every distinct VL at row ir of the tables."""
        p = torch.as_tensor(self.segs[0].ptab[ir], dtype=torch.float64, device=self.dev)
        if len(self.segs) > 1 and self.segs[0].ptab is not self.segs[-1].ptab:
            first = {}
            for s, v in enumerate(self.vid):
                first.setdefault(v, s)
            p = torch.as_tensor(np.stack([self.segs[first[v]].ptab[ir] for v in range(len(first))]),
                                dtype=torch.float64, device=self.dev)
            return torch.einsum("vhij,vh->vij", self.vl, p)
        return torch.einsum("vhij,h->vij", self.vl, p)

    def w(self, ir):
        r = float(self.segs[0].rtab[ir])
        if len(self.segs) > 1 and self.segs[0].rtab is not self.segs[-1].rtab:
            r = torch.as_tensor([float(g.rtab[ir]) for g in self.segs], dtype=torch.float64, device=self.dev)[self.js][:, None]
        w = self.sums(ir)[self.jv]
        d = torch.diagonal(w, dim1=1, dim2=2)
        d += self.jdiag + self.jcent / (r * r)
        return w


def _inv(a):
    return torch.linalg.inv(a)


def _sym(a):
    return 0.5 * (a + a.transpose(1, 2))


def _ldmd(b):
    seg = b.segs[0]
    h = seg.dr / 2.0
    d1, eye = h * h / 3.0, torch.eye(b.np_, dtype=torch.float64, device=b.dev)
    y = h * b.y + d1 * b.w(0)
    for k in range(1, seg.nstep + 1):
        s = b.sums(2 * k - 1)
        off = s - torch.diag_embed(torch.diagonal(s, dim1=1, dim2=2))
        q = (_inv(eye / 8 - (h * h / 48) * off) - 8 * eye)[b.jv]
        wr = torch.diagonal(b.w(2 * k - 1), dim1=1, dim2=2)
        arg = 0.5 * h * wr.abs().sqrt()
        tn, th = torch.tan(arg), torch.tanh(arg)
        y14 = torch.where(wr < 0, arg / tn - arg * tn, arg / th + arg * th)
        y23 = torch.where(wr < 0, arg / tn + arg * tn, arg / th - arg * th)
        y14b = torch.diag_embed(y14 - d1 * wr)
        yy = y23[:, :, None] * y23[:, None, :]
        y = q + 2 * torch.diag_embed(y14) - yy * _inv(_sym(y + y14b))
        y = (d1 if k == seg.nstep else 2 * d1) * b.w(2 * k) + y14b - yy * _inv(_sym(y))
    return y / h


def _ldj(b):
    seg = b.segs[0]
    h = seg.dr / 2.0
    d1, eye = h * h / 3.0, torch.eye(b.np_, dtype=torch.float64, device=b.dev)
    z = h * b.y + d1 * b.w(0) + eye
    for k in range(1, seg.nstep + 1):
        z = _inv(eye / 8 - (d1 / 16) * b.w(2 * k - 1)) - _inv(_sym(z)) - 6 * eye
        z = (d1 if k == seg.nstep else 2 * d1) * b.w(2 * k) + 2 * eye - _inv(_sym(z))
    return (z - eye) / h


def _ldmg(b, prop):
    stride, aa, bb = _MG[prop]
    seg, eye, y = b.segs[0], torch.eye(b.np_, dtype=torch.float64, device=b.dev), b.y
    for s in range(seg.nstep):
        for k, (ak, bk) in enumerate(zip(aa, bb)):
            y = y + bk * seg.dr * b.w(s * stride + k)
            if ak != 0.0:
                y = (eye - _inv(_sym(eye + ak * seg.dr * y))) / (ak * seg.dr)
    return y


def _bessel(l, x):
    """x j_l, (x j_l)', x y_l, (x y_l)' and d/dx ln(x k_l) for arrays l, x."""
    lmax = int(l.max())
    ym, y = np.sin(x) / x, -np.cos(x) / x
    km, kc = 1.0 / x, 1.0 / x
    ylm, yl, klm, kl = (np.zeros_like(x) for _ in range(4))
    with np.errstate(over="ignore", invalid="ignore"):
        for m in range(lmax + 1):
            hit = l == m
            ylm[hit], yl[hit], klm[hit], kl[hit] = ym[hit], y[hit], km[hit], kc[hit]
            ym, y = y, (2 * m + 1) / x * y - ym
            km, kc = kc, km + (2 * m + 1) / x * kc
    # j_l: Miller's downward recurrence, normalised by the larger of j_0 and j_1
    top = int(max(lmax, x.max())) + 60
    fp, f = np.zeros_like(x), np.full_like(x, 1e-280)
    jl, jlm, f1 = np.zeros_like(x), np.zeros_like(x), np.zeros_like(x)
    for m in range(top, 0, -1):
        fm = (2 * m + 1) / x * f - fp
        hit = l == m
        jl[hit], jlm[hit] = f[hit], fm[hit]
        if m == 1:
            f1 = f.copy()
        fp, f = f, fm
        big = np.abs(f) > 1e200
        for a in (fp, f, jl, jlm, f1):
            a[big] *= 1e-200
    jl[l == 0] = f[l == 0]
    j0, j1 = np.sin(x) / x, np.sin(x) / x ** 2 - np.cos(x) / x
    sc = np.where(np.abs(j0) > np.abs(j1), j0 / f, j1 / np.where(f1 == 0.0, 1.0, f1))
    jl, jlm = jl * sc, jlm * sc
    jlm[l == 0] = (np.cos(x) / x)[l == 0]
    return x * jl, x * jlm - l * jl, x * yl, x * ylm - l * yl, -klm / kl - l / x


def _smatrices(y, systems, segs, jsys, jered):
    """SR and SI of every job, NOPEN x NOPEN column-major, job after job."""
    sr, si = [], []
    for j, s in enumerate(jsys):
        c = systems[s]
        n, r = c.n, float(segs[s].rtab[-1])
        if segs[s].kind != "LD":
            r = float(segs[s].rtab[0]) + segs[s].nstep * segs[s].dr
        nb = np.argsort(c.eint[:n], kind="stable")
        dif = jered[j] - c.eint[:n][nb]
        no = int((dif > 0).sum())
        if no == 0:
            continue
        l = np.rint(np.sqrt(c.cent[:n][nb] + 0.25) - 0.5).astype(int)
        w = np.sqrt(np.abs(dif))
        uj, ujp, un, unp, kd = _bessel(l, w * r)
        op = dif > 0
        sn, snp = np.where(op, un / np.sqrt(w), 1.0), np.where(op, unp * np.sqrt(w), kd * w)
        sj, sjp = (uj / np.sqrt(w))[:no], (ujp * np.sqrt(w))[:no]
        yy = y[j][nb][:, nb]
        k = np.linalg.solve(yy * sn - np.diag(snp), yy[:, :no] * sj - np.eye(n)[:, :no] * sjp)[:no]
        k = 0.5 * (k + k.T)
        m = np.linalg.inv(0.5 * (np.eye(no) + k @ k))
        sr.append((m - np.eye(no)).ravel(order="F"))
        si.append((m @ k).ravel(order="F"))
    return (np.concatenate(sr) if sr else np.zeros(1)), (np.concatenate(si) if si else np.zeros(1))


def _ldma(c, seg, y0s, jered):
    b = _Batch([c], [seg], np.zeros(1, dtype=int), np.zeros(1), [y0s[0]])
    dev = b.dev
    e = torch.as_tensor(jered, dtype=torch.float64, device=dev)
    y = torch.as_tensor(np.stack(y0s), dtype=torch.float64, device=dev)
    cr, dr = seg.dr / 6.0, seg.dr
    for k in range(seg.nstep):
        w0, w1, w2 = (b.w(2 * k + i)[0] for i in range(3))
        ev, u = torch.linalg.eigh(w1)
        y = _sym(u.T @ (y + (w0 - w1) * cr) @ u)
        wr = ev[None, :] - e[:, None]
        fl = 0.5 * wr.abs().sqrt()
        tn, th = torch.tan(fl * dr), torch.tanh(fl * dr)
        y1 = torch.where(wr < 0, fl / tn - fl * tn, fl / th + fl * th)
        y2 = torch.where(wr < 0, fl / tn + fl * tn, fl / th - fl * th)
        y = torch.diag_embed(y1) - y2[:, :, None] * y2[:, None, :] * _inv(y + torch.diag_embed(y1))
        y = u @ y @ u.T + (w2 - w1) * cr
    return y


def exact(case, seed):
    prop, systems, segs, jsys, jered, y0s = _problem(case, seed)
    if case["kind"] == "ldma":
        return {"y": _ldma(systems[0], segs[0], y0s, jered).cpu().numpy(), "nodes": None, "status": None}
    ys = [None] * len(jsys)
    # one padded batch for each run of segments of the same length and step
    groups = {}
    for j, s in enumerate(jsys):
        big = systems[s].n > 64
        groups.setdefault((segs[s].nstep, segs[s].dr, systems[s].n if big else 0), []).append(j)
    for js in groups.values():
        used = sorted({int(jsys[j]) for j in js})
        at = {s: i for i, s in enumerate(used)}
        b = _Batch([systems[s] for s in used], [segs[s] for s in used], [at[int(jsys[j])] for j in js],
                   [jered[j] for j in js], [y0s[j] for j in js])
        y = _ldmd(b) if prop == "LDMD" else _ldj(b) if prop == "LDJ" else _ldmg(b, prop)
        y = _sym(y).cpu().numpy()
        for i, j in enumerate(js):
            n = systems[jsys[j]].n
            ys[j] = y[i][:n, :n]
    if case["kind"] == "single":
        return {"y": ys[0], "nodes": None}
    if case["kind"] == "serve":
        order = np.random.default_rng(int(seed)).permutation(len(jered))
        return {"y": np.concatenate([ys[k].ravel(order="F") for k in order]), "nodes": None}
    if case.get("via") == "smatrix":
        sr, si = _smatrices(ys, systems, segs, jsys, jered)
        return {"sr": sr, "si": si, "nodes": None, "status": None}
    out = {"y": np.concatenate([y.ravel(order="F") for y in ys]), "nodes": None, "status": None}
    if case["kind"] == "fields":
        out["counts"] = None
    return out
