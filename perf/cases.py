"""The work that users of this framework have it do, as cases that can be timed.

A case is a dict of plain values.  Its "kind" is the entry point:

  modelling  gpu.Solver.modelling: inject the sources, solve, extract the
             receiver data, on a solver that the program keeps (complex64
             cycles with FP64 refinement unless "precision" says fp64)
  fields     gpu.Solver.solve on device buffers: E and H of given right-hand
             sides over a mesh of the caller's own
  forward    gpu.Fg.forward: the modelling of a survey from the padded model,
             with the homogenization and the solver's set-up in every pass
  gradient   gpu.Fg.eval: misfit, gradient and pseudo-Hessian of a survey
             (forward and adjoint solves, set-up in every pass)
  learned    gpu.Solver.learned_apply: one application of the learned
             correction to complex64 iterates

Models come from libemmi_mgfd_gb300.workloads, seeded.
"""
import dataclasses
import math

import numpy as np
import torch

from libemmi_mgfd_gb300 import gpu as G
from libemmi_mgfd_gb300 import host
from libemmi_mgfd_gb300 import workloads as W

MU0 = 4e-7 * math.pi


def _case(name, kind, model, n, shots, freqs, **more):
    c = dict(name=name, kind=kind, model=model, n1=n[0], n2=n[1], n3=n[2], shots=shots, freqs=freqs,
             precision="mixed", tol=1e-8, skip_post=0)
    c.update(more)
    return c


def listed():
    return [
        # one shot on the smallest mesh in use (the layered parity model): latency
        _case("shot_16", "modelling", "layered", (16, 16, 16), 1, "1"),
        # one rotated and tilted source, six channels, an anisotropic model, a ragged mesh
        _case("shot_aniso_ragged", "modelling", "aniso", (24, 20, 40), 1, "0.5"),
        # the layered forward configuration: what a rank of the reference runs for its shot
        _case("shot_64", "modelling", "layered", (64, 64, 64), 1, "1"),
        # a few shots at two frequencies on a ragged mesh
        _case("shots_ragged", "modelling", "lognormal", (80, 56, 72), 3, "0.25,1"),
        # VTI sediment under a rough sea floor, shots x frequencies over shared operators
        _case("survey_vti_96", "modelling", "vti", (96, 96, 96), 10, "0.25,0.75"),
        # the benchmark's batch: 25 shots at 128^3 with the benchmark's cycle
        _case("survey_128", "modelling", "lognormal", (128, 128, 128), 25, "1", skip_post=3),
        # the reference's arithmetic, one small solve and a batch
        _case("fields_fp64_16", "fields", "own", (16, 16, 16), 1, "1", precision="fp64", tol=1e-10),
        _case("fields_fp64_64", "fields", "own", (64, 56, 48), 2, "0.5,1", precision="fp64", tol=1e-10),
        # modelling a survey at a new model, and one objective evaluation of an inversion
        _case("forward_64", "forward", "lognormal", (64, 64, 64), 8, "1", skip_post=3),
        _case("gradient_64", "gradient", "reservoir", (64, 64, 64), 4, "0.25,0.5,1", tol=1e-9),
        # the learned correction as every corrected cycle applies it
        _case("learned_96", "learned", "lognormal", (96, 96, 96), 8, "1"),
    ]


# meshes that the semi-coarsening takes down to a few cells: an odd number up
# to nine times a power of two
_N_SMALL = (16, 20, 24, 28, 32, 36, 40)
_N_SURVEY = (32, 36, 40, 48, 56, 64, 72, 80, 96, 112, 128)
_N_DEPTH = (64, 72, 80, 96, 112, 128)


def draw(rng):
    def size(choice, lo=0):
        return choice[min(len(choice) - 1, int(lo + rng.random() * (len(choice) - lo)))]

    kind = rng.choice(["small", "small", "survey", "survey", "survey", "fields", "fields", "forward",
                       "gradient", "learned"])
    tol = 1e-8
    if kind == "small":
        return _unnamed("modelling", rng.choice(["layered", "aniso"]), [size(_N_SMALL) for _ in range(3)], 1,
                        "%.3g" % math.exp(rng.uniform(math.log(0.3), math.log(2.0))), tol=tol)
    n = [size(_N_SURVEY), size(_N_SURVEY), size(_N_DEPTH)]
    if kind == "fields":
        n = [size(_N_SMALL), size(_N_SMALL), size(_N_SMALL)] if rng.random() < 0.5 else [
            size(_N_SURVEY[:7]), size(_N_SURVEY[:7]), size(_N_SURVEY[:7])]
        return _unnamed("fields", "own", n, 1 + int(3 * rng.random()), rng.choice(["1", "0.5,1", "0.25"]),
                        precision="fp64", tol=1e-10)
    if kind == "learned":
        return _unnamed("learned", "lognormal", n, max(1, int(math.exp(rng.uniform(0, math.log(12))))), "1")
    # cells x right-hand sides spread over their logarithm, up to the benchmark's batch
    most = 25 * 128 ** 3 if kind == "survey" else 4e6
    freqs = rng.choice(["1", "0.25,0.75", "0.5,1"])
    if kind in ("forward", "gradient"):
        n = [size(_N_SURVEY[:7]), size(_N_SURVEY[:7]), size(_N_DEPTH[:3])]
    cells = n[0] * n[1] * n[2] * len(freqs.split(","))
    shots = max(1, min(25, int(math.exp(rng.uniform(math.log(cells), math.log(most))) / cells))) if cells < most else 1
    if kind == "survey":
        model = rng.choice(["lognormal", "lognormal", "vti", "layered"])
        return _unnamed("modelling", model, n, 1 if model == "layered" else shots, freqs,
                        skip_post=rng.choice([0, 3]), tol=tol)
    if kind == "forward":
        return _unnamed("forward", "lognormal", n, shots, freqs, skip_post=rng.choice([0, 3]), tol=tol)
    return _unnamed("gradient", "reservoir", n, min(shots, 6), freqs, tol=1e-9)


def _unnamed(*a, **k):
    c = _case(None, *a, **k)
    del c["name"]
    return c


# ---------------------------------------------------------------- inputs
def _survey(case, seed):
    """The seeded survey of a case; the resistivities, and the sources where
    the family leaves them free, come from the seed."""
    n = (case["n1"], case["n2"], case["n3"])
    rng = np.random.default_rng(seed)
    kind = case["model"]
    if kind == "layered":
        s = W.config1(n[2]) if n[2] >= 64 else W.tiny_layered(n)
        rho = s.rho11.copy()
        for v in np.unique(rho)[1:]:
            rho[s.rho11 == v] = v * float(rng.uniform(0.7, 1.4))
        s = dataclasses.replace(s, rho11=rho, rho22=rho.copy(), rho33=rho.copy())
    elif kind == "aniso":
        s = W.tiny_aniso(n, seed=seed)
    elif kind == "vti":
        s = W.config2(n[2], seed=seed)
    elif kind == "reservoir":
        s = W.config4(n[2], true_model=False)
        rho = s.rho11.copy()
        below = rho > W.RHO_WATER
        rho[below] = (10.0 ** (0.05 * rng.standard_normal(int(below.sum())))).astype(np.float32)
        s = dataclasses.replace(s, rho11=rho, rho22=rho.copy(), rho33=rho.copy())
    else:
        s = W.config3(n[2], seed=seed)
    k = case["shots"]
    pick = np.sort(rng.permutation(len(s.sources))[:k]) if k < len(s.sources) else np.arange(len(s.sources))
    return dataclasses.replace(s, n=n, sources=s.sources[pick], freqs=[float(f) for f in case["freqs"].split(",")],
                               pairs=W.all_pairs(len(pick), len(s.receivers)))


def _options(case):
    return G.Options(precision=G.PREC_FP64 if case["precision"] == "fp64" else G.PREC_MIXED, tol=case["tol"],
                     ncycle=100, skip_post=case["skip_post"])


def _radians(p):
    p = np.asarray(p, np.float32).copy()
    p[:, 3:] = np.deg2rad(p[:, 3:])
    return p


def _solver(case, s):
    """A solver of every shot and frequency of a survey, its cells
    homogenized on the device."""
    m = host.Model.from_survey(s)
    padded = m.padded()
    axes = [m.axes(*padded[:3], float(p[0]), float(p[1]), float(p[2])) for p in s.sources]
    k, nf = len(axes), len(s.freqs)
    cells = torch.empty((k, 4, int(np.prod(s.n))), dtype=torch.float32, device="cuda")
    G.homogenize_batch(padded, axes, s.n, cells.data_ptr())
    sv = G.Solver(s.n, *[np.stack([a[x] for a in axes]) for x in ("x1", "x2", "x3")], cells.data_ptr(),
                  np.tile(2 * np.pi * np.asarray(s.freqs), k).astype(np.float32),
                  op=np.repeat(np.arange(k, dtype=np.int32), nf), options=_options(case),
                  rho_water=np.float32(m.rho_water()))
    return sv, np.repeat(_radians(s.sources), nf, axis=0), _radians(s.receivers)


def _own_problem(case, seed):
    """A caller's own mesh: cells growing away from a source 50 m above the
    sea floor, air, 1000 m of water and rough sediment; one operator a
    "shot", a right-hand side for each frequency.  float32 numpy arrays as
    gpu.Solver takes them, and the complex128 right-hand sides."""
    rng = np.random.default_rng(seed)
    n, k = (case["n1"], case["n2"], case["n3"]), case["shots"]
    freqs = [float(f) for f in case["freqs"].split(",")]
    S1 = (n[2] + 1, n[1] + 1, n[0] + 1)
    X, cells, b, omega = [[], [], []], [], [], []
    for _ in range(k):
        x = []
        for e, (h0, far) in enumerate(((200.0, 20e3), (200.0, 20e3), (100.0, 15e3))):
            half = n[e] // 2
            lo, hi = 1.0, 4.0  # h0 (q + .. + q^half) = far
            for _ in range(60):
                q = 0.5 * (lo + hi)
                lo, hi = (q, hi) if h0 * sum(q ** i for i in range(half)) < far else (lo, q)
            up = np.cumsum(h0 * lo ** np.arange(n[e] - half) * rng.uniform(0.97, 1.03, n[e] - half))
            dn = np.cumsum(h0 * lo ** np.arange(half) * rng.uniform(0.97, 1.03, half))
            x.append(np.concatenate([-dn[::-1], [0.0], up]).astype(np.float32) + np.float32(950.0 if e == 2 else 0.0))
        zc = 0.5 * (x[2][1:] + x[2][:-1]).astype(np.float64)
        sig = 10.0 ** (0.3 * rng.standard_normal((n[2], n[1], n[0])))
        sig[zc < 1000.0] = 1.0 / W.RHO_WATER
        sig[zc < 0.0] = 1e-8
        cells.append(np.stack([sig, sig, np.where(zc[:, None, None] > 1000.0, 0.5 * sig, sig),
                               np.ones_like(sig)]).astype(np.float32))
        for f in freqs:
            om = np.float32(2 * np.pi * f)
            j = np.zeros((3,) + S1, np.complex128)
            i1, i2, i3 = (v // 2 for v in n)
            j[0, i3, i2, i1] = 1.0  # a unit x current on the edge at the source
            b.append((1j * float(om) * MU0 * j).reshape(-1) / (200.0 * 200.0 * 100.0))
            omega.append(om)
        for e in range(3):
            X[e].append(x[e])
    return n, [np.stack(v) for v in X], np.stack(cells), np.array(omega, np.float32), np.stack(b)


def _dipole_data(s):
    """Observed data of a whole-space dipole (0.5 S/m), [shot, channel,
    frequency, receiver] complex64: data of the survey's own magnitude."""
    d = s.receivers[None, :, :3].astype(np.float64) - s.sources[:, None, :3]
    d[..., 2] += 60.0
    r = np.sqrt((d ** 2).sum(-1))
    out = np.zeros((len(s.sources), len(s.chrec), len(s.freqs), len(s.receivers)), np.complex128)
    for f, fr in enumerate(s.freqs):
        kr = (1 - 1j) * np.sqrt(np.pi * fr * MU0 * 0.5) * r
        e = np.exp(-kr) / (4 * np.pi * 0.5 * r ** 3)
        h = np.exp(-kr) * (1 + kr) / (4 * np.pi * r ** 3)
        v = {"Ex": e * (d[..., 0] ** 2 / r ** 2 * (kr ** 2 + 3 * kr + 3) - (kr ** 2 + kr + 1)),
             "Ey": e * (d[..., 0] * d[..., 1] / r ** 2 * (kr ** 2 + 3 * kr + 3)),
             "Hx": 0.01 * h * r, "Hy": h * d[..., 2]}
        for c, name in enumerate(s.chrec):
            out[:, c, f] = v[name]
    return out.astype(np.complex64)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fields":
        n, X, cells, omega, b = _own_problem(case, seed)
        nf = len(omega) // case["shots"]
        sv = G.Solver(n, *X, cells, omega, op=np.repeat(np.arange(case["shots"], dtype=np.int32), nf),
                      options=_options(case))
        b = torch.from_numpy(b).cuda()
        return dict(kind=kind, solver=sv, b=b, x=torch.empty_like(b), h=torch.empty_like(b))
    s = _survey(case, seed)
    if kind in ("forward", "gradient"):
        m = host.Model.from_survey(s)
        if kind == "forward":
            return dict(kind=kind, model=m, fg=G.Fg(m, s, options=_options(case)))
        dobs = _dipole_data(s)
        delta = (0.03 * np.abs(dobs) + 1e-15).astype(np.float32)
        return dict(kind=kind, model=m, fg=G.Fg(m, s, dobs, delta, s.bathy, options=_options(case)))
    sv, src, rec = _solver(case, s)
    if kind == "learned":
        rng = np.random.default_rng(seed + 1)
        w = (0.03 * rng.standard_normal((2, 27, 8, 8))).astype(np.float32)
        w[0, :, 6:, :] = 0.0
        sv.set_learned(w.reshape(-1))
        gen = torch.Generator(device="cuda").manual_seed(seed)
        f, u = (torch.view_as_complex(torch.randn((sv.nrhs, 3 * sv.nslots, 2), generator=gen, device="cuda"))
                * _unknown(s.n, "cuda").reshape(-1) for _ in range(2))
        # a residual and an iterate of a cycle: f of the size of A u
        return dict(kind=kind, solver=sv, f=f * 1e-3, u=u)
    return dict(kind=kind, solver=sv, src=src, rec=rec, chsrc=s.chsrc, chrec=s.chrec)


def run(state):
    kind = state["kind"]
    if kind == "modelling":
        return state["solver"].modelling(state["src"], state["rec"], state["chsrc"], state["chrec"])[0]
    if kind == "fields":
        state["solver"].solve(state["b"].data_ptr(), device=True, x_out=state["x"].data_ptr(),
                              h_out=state["h"].data_ptr())
        return {"x": state["x"], "h": state["h"]}
    if kind == "forward":
        return state["fg"].forward(state["model"])[0]
    if kind == "gradient":
        fcost, grad, phess, dcal, rmse, _ = state["fg"].eval(state["model"])
        return {"fcost": fcost, "grad": grad, "phess": phess, "dcal": dcal, "rmse": rmse}
    u = state["u"].clone()
    state["solver"].learned_apply(state["f"], u)
    return u


def work(case):
    """A solve cannot do with less than reading the iterate, the right-hand
    side and three conductivities and writing the iterate once for each of
    the two line directions that a cycle relaxes, about one cycle for a digit;
    60 operations an edge equation.  The learned correction reads f, u and
    the conductivities and writes u, two 27-tap convolutions of 8 channels."""
    slots = (case["n1"] + 1) * (case["n2"] + 1) * (case["n3"] + 1) * case["shots"] * len(case["freqs"].split(","))
    c = 16 if case["precision"] == "fp64" else 8
    if case["kind"] == "learned":
        return {"bytes": slots * (9 * 8 + 12), "flops": slots * 2.0 * 2 * 27 * 64}
    cycles = round(-math.log10(case["tol"])) * (2 if case["kind"] == "gradient" else 1)
    return {"bytes": slots * (9 * c + 12) * 2.0 * cycles, "flops": slots * 3 * 60 * 2.0 * cycles}


# ---------------------------------------------------------------- 64 bits
def _stagger(x):
    ds = torch.empty_like(x)
    ds[:-1] = x[1:] - x[:-1]
    xs = x + 0.5 * ds
    xs[-1] = x[-1] + 0.5 * ds[-2]
    ds[-1] = xs[-1] - x[-1]
    d = torch.empty_like(x)
    d[1:] = xs[1:] - xs[:-1]
    d[0] = xs[0] - x[0]
    return ds, d


def _unknown(n, device):
    """[3, n3+1, n2+1, n1+1]: the edges inside the domain."""
    m = torch.zeros((3, n[2] + 1, n[1] + 1, n[0] + 1), dtype=torch.bool, device=device)
    m[0, 1:-1, 1:-1, :-1] = m[1, 1:-1, :-1, 1:-1] = m[2, :-1, 1:-1, 1:-1] = True
    return m


def _matrix(n, x, cells, omega):
    """Rows, columns and values of the finite-integration curl-curl operator
    with unit permeability over all edge slots (identity outside the
    unknowns): curl^T diag(face weights) curl - i omega mu0 diag(sigma V)."""
    x = [torch.as_tensor(v, dtype=torch.float64, device="cuda") for v in x]
    ds = [_stagger(v)[0] for v in x]
    N = (n[2] + 1, n[1] + 1, n[0] + 1)
    S = N[0] * N[1] * N[2]
    ax = {0: 2, 1: 1, 2: 0}  # direction -> tensor axis
    slot = torch.arange(S, device="cuda").reshape(N)
    vol = ds[2][:-1, None, None] * ds[1][None, :-1, None] * ds[0][None, None, :-1]
    sv = torch.as_tensor(np.asarray(cells[:3], np.float64), device="cuda") * vol
    unk = _unknown(n, "cuda").reshape(-1)
    rows, cols, vals = [], [], []
    for c in range(3):  # face of normal c: E_p, E_q around it, p = c+1, q = c+2
        p, q = (c + 1) % 3, (c + 2) % 3
        sl = [slice(None)] * 3
        sl[ax[p]] = sl[ax[q]] = slice(0, -1)
        sl[ax[c]] = slice(1, -1)
        s0 = slot[tuple(sl)]
        step = [1, N[2], N[2] * N[1]]
        shape = [1, 1, 1]
        shape[ax[p]], hp = -1, [1, 1, 1]
        dp = ds[p][:-1].reshape(shape)
        hp[ax[q]] = -1
        dq = ds[q][:-1].reshape(hp)
        hc = [1, 1, 1]
        hc[ax[c]] = -1
        # half of the volumes of the two cells that share the face
        w = 0.5 * (ds[c][:-2] + ds[c][1:-1]).reshape(hc) * dp * dq
        # curl E . n = (E_q(+p) - E_q) / dp - (E_p(+q) - E_p) / dq
        e = [(q * S + s0 + step[p], 1 / dp), (q * S + s0, -1 / dp), (p * S + s0 + step[q], -1 / dq), (p * S + s0, 1 / dq)]
        for r, a in e:
            for k, b in e:
                v = (w * a * b).expand(s0.shape).reshape(-1)
                rows.append(r.reshape(-1))
                cols.append(k.reshape(-1))
                vals.append(v.to(torch.complex128))
        # a quarter of the four cells around an edge along c
        box = torch.zeros(N, dtype=torch.float64, device="cuda")
        inner = [slice(None)] * 3
        inner[ax[c]] = slice(0, -1)
        inner[ax[p]] = inner[ax[q]] = slice(1, -1)
        acc = 0
        for i in (0, 1):
            for j in (0, 1):
                t = [slice(None)] * 3
                t[ax[p]] = slice(i, n[p] - 1 + i)
                t[ax[q]] = slice(j, n[q] - 1 + j)
                acc = acc + sv[c][tuple(t)]
        box[tuple(inner)] = 0.25 * acc
        rows.append(c * S + slot.reshape(-1))
        cols.append(c * S + slot.reshape(-1))
        vals.append(-1j * omega * MU0 * box.reshape(-1))
    r, k, v = torch.cat(rows), torch.cat(cols), torch.cat(vals)
    keep = unk[r] & unk[k]
    return r[keep], k[keep], v[keep], unk


def exact(case, seed):
    n = (case["n1"], case["n2"], case["n3"])
    if case["kind"] == "fields":
        if 3 * n[0] * n[1] * n[2] > 16000:
            return None
        n, X, cells, omega, b = _own_problem(case, seed)
        nf, xs, hs = len(omega) // case["shots"], [], []
        for r in range(len(omega)):
            o = r // nf
            x = [X[e][o] for e in range(3)]
            i, j, v, unk = _matrix(n, x, cells[o], float(omega[r]))
            at = torch.cumsum(unk, 0) - 1
            A = torch.zeros((int(unk.sum()),) * 2, dtype=torch.complex128, device="cuda")
            A.index_put_((at[i], at[j]), v, accumulate=True)
            ds, d = zip(*(_stagger(torch.as_tensor(t, dtype=torch.float64, device="cuda")) for t in x))
            dual = torch.stack([(ds if c == 2 else d)[2][:, None, None] * (ds if c == 1 else d)[1][None, :, None]
                                * (ds if c == 0 else d)[0][None, None, :] for c in range(3)]).reshape(-1)
            f = torch.as_tensor(b[r], device="cuda") * dual
            E = torch.zeros(unk.shape, dtype=torch.complex128, device="cuda")
            E[unk] = torch.linalg.solve(A, f[unk])
            # the residual once more: 64 bits of the matrix's own scale
            res = f[unk] - A @ E[unk]
            E[unk] += torch.linalg.solve(A, res)
            del A
            E = E.reshape(3, n[2] + 1, n[1] + 1, n[0] + 1)
            H = torch.zeros_like(E)
            ax = {0: 2, 1: 1, 2: 0}
            for c in range(3):
                p, q = (c + 1) % 3, (c + 2) % 3
                core = (slice(0, -1),) * 3

                def diff(F, e):
                    w = [1, 1, 1]
                    w[ax[e]] = -1
                    return (torch.roll(F, -1, ax[e])[core] - F[core]) / ds[e][:-1].reshape(w)
                H[(c,) + core] = (diff(E[q], p) - diff(E[p], q)) / (1j * float(omega[r]) * MU0)
            xs.append(E.reshape(-1))
            hs.append(H.reshape(-1))
        return {"x": torch.stack(xs), "h": torch.stack(hs)}
    return None
