"""Workloads of the library as its users call it: orbitals at the electrons of
a set of walkers, through the public entry points.

A case names a molecule (`nuclei`, `basis`, `mos`, `cube` side in bohr, all
cartesian Gaussian, built by qmckl_b200.gen with the distributions of the
repository's benchmark molecules), a number of `points` (electrons of the
walkers, placed around the nuclei; any count, not only whole walkers), the
arithmetic `form` (fp64: the parity form and the library's default at full
precision; mixed: the tensor-core form) and the `call`:

  mo_vgl      qmckl_b200_mo_vgl_device: one Monte Carlo step's orbitals with
              gradients and Laplacians, coordinates and results on the GPU
  mo_value    qmckl_b200_mo_value_device: values only (ratios of trial moves)
  ao_vgl      qmckl_b200_ao_vgl_device: the AOs themselves
  ao_hessian  qmckl_b200_ao_hessian_device: AO second derivatives (forces)
  host        qmckl_set_electron_coord + qmckl_get_mo_basis_mo_vgl: a step
              through the reference's own host interface, numpy in and out
  grad        qmckl_b200.torch_ops.mo_vgl and its backward pass: orbitals and
              the gradients of L = sum(W * mo_vgl) with respect to points,
              nuclei and MO coefficients (wave-function optimisation)
  batch       qmckl_b200_batch_mo_vgl_device: many molecules in one launch
"""
import functools
import math
import os

import numpy as np
import torch

from qmckl_b200 import gen
from qmckl_b200 import qmckl as pq
from qmckl_b200 import torch_ops
from qmckl_b200.system import make_context

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PRECISION = 53                                  # the library's default


def _case(name, call, form, nuclei, basis, mos, cube, points, systems=1):
    return {"name": name, "call": call, "form": form, "nuclei": nuclei, "basis": basis, "mos": mos, "cube": cube,
            "points": points, "systems": systems}


def listed():
    return [
        # one walker of a small molecule, the smallest call of a step-by-step code
        _case("one_walker_fp64", "mo_vgl", "fp64", 10, "dz", 90, 8.0, 30),
        # the reference's test molecule (CHBrClF: 263 AOs, 224 MOs) with its two
        # walkers through the host interface, the drop-in use
        _case("chbrclf_host", "host", "fp64", 5, "chbrclf", 224, 0.0, 136),
        # 64 walkers of the small molecule: a short vectorised step
        _case("small_mixed", "mo_vgl", "mixed", 10, "dz", 90, 8.0, 1920),
        # 128 walkers of the mid-size molecule in the default form
        _case("mid_fp64", "mo_vgl", "fp64", 80, "tz", 160, 20.0, 40704),
        # the benchmark step: 512 walkers of the mid-size molecule
        _case("mid_mixed", "mo_vgl", "mixed", 80, "tz", 160, 20.0, 162816),
        # the large molecule: 5,000 AOs, 350 MOs, 256 walkers
        _case("large_mixed", "mo_vgl", "mixed", 200, "tz", 350, 32.0, 179200),
        # values only on an odd number of points and of MOs (a trial-move sweep)
        _case("value_odd_fp64", "mo_value", "fp64", 33, "tz", 101, 14.3, 9973),
        # the AOs of the mid-size molecule, 101 walkers
        _case("ao_mid_fp64", "ao_vgl", "fp64", 80, "tz", 160, 20.0, 32118),
        # second derivatives of the AOs for a force evaluation
        _case("hessian_fp64", "ao_hessian", "fp64", 40, "tz", 80, 15.9, 5087),
        # orbital optimisation: forward and backward, 64 walkers, default form
        _case("grad_fp64", "grad", "fp64", 80, "tz", 160, 20.0, 20352),
        # the same with 128 walkers on the tensor cores
        _case("grad_mixed", "grad", "mixed", 80, "tz", 160, 20.0, 40704),
        # 24 molecules of uneven size in one launch
        _case("batch_mixed", "batch", "mixed", 80, "both", 0, 0.0, 9600, 24),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["mo_vgl", "mo_vgl", "mo_vgl", "mo_value", "ao_vgl", "ao_hessian", "host", "grad", "batch"])
    form = rng.choice(["fp64", "mixed"])
    if call == "batch":
        return {"call": call, "form": "mixed", "nuclei": _log_int(rng, 8, 80), "basis": "both", "mos": 0, "cube": 0.0,
                "points": _log_int(rng, 40, 9600), "systems": _log_int(rng, 2, 24)}
    nuclei = _log_int(rng, 5, 200)
    basis = rng.choice(["dz", "tz", "tz"]) if nuclei > 24 else rng.choice(["dz", "tz", "hl"])
    cube = round(8.0 * (nuclei / 10.0) ** (1.0 / 3.0) * rng.uniform(1.0, 1.25), 2)
    mos = _log_int(rng, max(4, nuclei), max(8, min(400, 4 * nuclei)))
    most = {"mo_vgl": 160000, "mo_value": 160000, "ao_vgl": 32000, "ao_hessian": 5000, "host": 4000,
            "grad": 40000}[call]
    if call in ("ao_vgl", "ao_hessian", "grad") or form == "fp64":
        most = int(most * min(1.0, 80.0 / nuclei))
    if call in ("mo_vgl", "mo_value") and form == "fp64":
        most = most // 4
    return {"call": call, "form": form, "nuclei": nuclei, "basis": basis, "mos": mos, "cube": cube,
            "points": _log_int(rng, 30, most), "systems": 1}


def _charges(rng, n):
    heavy = n - n // 2
    return list(rng.choice([6.0, 7.0, 8.0], size=heavy)) + [1.0] * (n - heavy)


def _system(nuclei, basis, mos, cube, points, seed, mol_seed=None):
    """One molecule and its points [P][3]; everything from the seed (the molecule from mol_seed where given)."""
    rng = np.random.default_rng([20260000, seed if mol_seed is None else mol_seed])
    if basis == "chbrclf":                      # fixed molecule, the walkers' electrons drawn around it
        d = gen.chbrclf(os.path.join(ROOT, "tests", "golden", "chbrclf.npz"))
        z = np.asarray(d["charge"], dtype=np.float64).reshape(-1)
        xyz = np.asarray(d["nucl_coord"], dtype=np.float64).reshape(3, -1).T
        own = rng.choice(z.size, size=points, p=z / z.sum())
        return d, xyz[own] + rng.standard_normal((points, 3))
    charges = _charges(rng, nuclei)
    xyz = gen.place_nuclei(rng, nuclei, cube)
    shapes = None
    if basis == "hl":
        shapes = [gen.SHAPES["hl_a"] if z == 6.0 else (gen.SHAPES["hl_b"] if z == 8.0 else gen.SHAPES["tz_heavy"])
                  if z > 1.0 else gen.SHAPES["tz_h"] for z in charges]
    heavy, h = ("tz_heavy", "tz_h") if basis != "dz" else ("dz_heavy", "dz_h")
    d = gen.build_system(rng, charges, xyz, gen.SHAPES[heavy], gen.SHAPES[h], mos, 1, elec_num=2, shapes=shapes)
    z = np.asarray(charges)
    if mol_seed is not None:
        rng = np.random.default_rng([20260001, seed, mol_seed])
    own = rng.choice(nuclei, size=points, p=z / z.sum())
    return d, xyz[own] + rng.standard_normal((points, 3))


def _systems(case, seed):
    if case["call"] != "batch":
        return [_system(case["nuclei"], case["basis"], case["mos"], case["cube"], case["points"], seed)]
    # a batch keeps its molecules from step to step: they and the walker counts
    # follow from the case, the electrons from the seed
    rng = np.random.default_rng([20260002, case["nuclei"], case["points"]])
    out = []
    for s in range(case["systems"]):
        nn = int(rng.integers(5, case["nuclei"] + 1))
        basis = "tz" if rng.integers(0, 2) else "dz"
        out.append(_system(nn, basis, 2 * nn, 8.0 * (nn / 10.0) ** (1.0 / 3.0),
                           int(rng.integers(30, case["points"] + 1)), seed, s + 1))
    return out


class State:
    """The context (or batch) and buffers of one case; destroys them with itself."""

    def __init__(self):
        self.ctxs, self.batch = [], None

    def __del__(self):
        torch.cuda.synchronize()
        if self.batch is not None:
            pq.b200_batch_destroy(self.batch)
        for c in self.ctxs:
            torch_ops.forget(c)
            pq.context_destroy(c)


def _outputs(case, d, P):
    A, M = int(d["ao_num"]), int(d["mo_num"])
    return {"mo_vgl": (P, 5, M), "mo_value": (P, M), "ao_vgl": (P, 5, A), "ao_hessian": (3, P, 4, A)}[case["call"]]


def prepare(case, seed):
    st = State()
    st.case = case
    form = pq.FORM_FP64 if case["form"] == "fp64" else pq.FORM_MIXED
    systems = _systems(case, seed)
    call = case["call"]
    for d, _ in systems:
        st.ctxs.append(make_context(d, points=False, form=form))
    if call == "batch":
        P = [x.shape[0] for _, x in systems]
        st.batch = pq.b200_batch_create(st.ctxs, P)
        co, oo, (ct, ot) = pq.b200_batch_layout(st.batch, len(P))
        coord = np.zeros(ct)
        for s, (_, x) in enumerate(systems):
            coord[co[s]:co[s] + 3 * P[s]] = np.ascontiguousarray(x.T).reshape(-1)
        st.coord = torch.from_numpy(coord).cuda()
        st.out = torch.empty(ot, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        return st
    d, x = systems[0]
    st.ctx = st.ctxs[0]
    st.P = x.shape[0]
    if call == "host":
        # (up, down) electrons of one walker that holds all the points
        pq.set_electron_num(st.ctx, st.P - st.P // 2, st.P // 2)
        st.x = np.ascontiguousarray(x).reshape(-1)
        st.size = st.P * 5 * int(d["mo_num"])
        return st
    st.coord = torch.from_numpy(np.ascontiguousarray(x.T)).cuda()
    if call == "grad":
        g = torch.Generator("cuda").manual_seed(seed)
        st.coord.requires_grad_()
        st.nucl = torch_ops.nucl_coord_tensor(d).requires_grad_()
        st.coef = torch.from_numpy(np.ascontiguousarray(d["mo_coef"])).cuda().requires_grad_()
        st.weight = torch.randn((st.P, 5, int(d["mo_num"])), dtype=torch.float64, device="cuda", generator=g)
    else:
        pq.b200_set_stream(st.ctx, torch.cuda.current_stream().cuda_stream)
        st.out = torch.empty(_outputs(case, d, st.P), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    return st


_DEVICE = {"mo_vgl": pq.b200_mo_vgl_device, "mo_value": pq.b200_mo_value_device, "ao_vgl": pq.b200_ao_vgl_device,
           "ao_hessian": pq.b200_ao_hessian_device}


def run(st):
    call = st.case["call"]
    if call == "host":
        pq.set_electron_coord(st.ctx, "N", 1, st.x)
        return pq.get_mo_basis_mo_vgl(st.ctx, st.size)
    if call == "batch":
        pq.b200_batch_mo_vgl_device(st.batch, st.coord.data_ptr(), st.out.data_ptr())
        return st.out
    if call == "grad":
        mo = torch_ops.mo_vgl(st.ctx, st.coord, st.nucl, st.coef)
        g = torch.autograd.grad(mo, [st.coord, st.nucl, st.coef], grad_outputs=st.weight)
        return {"mo": mo.detach(), "points": g[0], "nuclei": g[1], "coefficients": g[2]}
    _DEVICE[call](st.ctx, st.P, st.coord.data_ptr(), st.out.data_ptr())
    return st.out


# ---------------------------------------------------------------- work

def _shells(d):
    """nucleus and smallest exponent of every shell, and its AO count."""
    nuc = np.repeat(np.arange(int(d["nucl_num"])), np.asarray(d["nucleus_shell_num"]))
    amin = np.array([np.min(d["exponent"][i:i + n]) for i, n in zip(d["shell_prim_index"], d["shell_prim_num"])])
    l = np.asarray(d["shell_ang_mom"])
    return nuc, amin, (l + 1) * (l + 2) // 2


@functools.lru_cache(maxsize=None)
def _sample(key):
    """(AOs, MOs, AOs that reach a point on average, points) of each molecule of a case, over sampled points."""
    case = dict(key)
    few = dict(case, points=min(case["points"], 2000))
    out = []
    for d, x in _systems(case if case["call"] == "batch" else few, 0):
        P = x.shape[0] if case["call"] == "batch" else case["points"]
        nuc, amin, na = _shells(d)
        x = x[:200]
        xyz = np.asarray(d["nucl_coord"], dtype=np.float64).reshape(3, -1).T
        r2 = ((x[:, None, :] - xyz[None]) ** 2).sum(-1)[:, nuc]
        live = float(((r2 * amin <= (PRECISION - 1) * math.log(2.0)) * na).sum(1).mean())
        out.append((int(d["ao_num"]), int(d["mo_num"]), live, P, int(d["nucl_num"])))
    return out


def work(case):
    """Inputs read once, outputs written once, and the multiply-adds of the AOs that are not exact zeros."""
    case = {k: v for k, v in case.items() if k != "name"}
    nbytes = flops = 0.0
    for A, M, live, P, N in _sample(tuple(sorted(case.items()))):
        call = case["call"]
        coord, coef = 24.0 * P, 8.0 * A * M
        if call == "mo_value":
            nbytes += coord + coef + 8.0 * P * M
            flops += 2.0 * P * live * M
        elif call == "ao_vgl":
            nbytes += coord + 40.0 * P * A
            flops += 40.0 * P * live
        elif call == "ao_hessian":
            nbytes += coord + 96.0 * P * A
            flops += 100.0 * P * live
        elif call == "grad":
            nbytes += 2 * coord + 2 * coef + 80.0 * P * M + 48.0 * N
            flops += 30.0 * P * live * M
        else:
            nbytes += coord + coef + 40.0 * P * M
            flops += 10.0 * P * live * M
    return {"bytes": nbytes, "flops": flops}


# --------------------------------------------------------------- exact

def _powers(x, n):
    """x^n and its first three derivatives, per AO: x [p][A], n [A]."""
    out = []
    for k in range(4):
        c = torch.ones_like(n)
        for i in range(k):
            c = c * (n - i)
        out.append(c * x ** torch.clamp(n - k, min=0).double())
    return out


def _basis(d, dev):
    """Index tensors of the basis: per AO its shell, powers and factor; per primitive its shell and nucleus."""
    nuc, _, na = _shells(d)
    l = np.asarray(d["shell_ang_mom"])
    sh, abc = [], []
    for s, ls in enumerate(l):
        for a in range(int(ls), -1, -1):
            for b in range(int(ls) - a, -1, -1):
                sh.append(s)
                abc.append((a, b, int(ls) - a - b))
    pn = np.asarray(d["shell_prim_num"])
    pi = np.concatenate([np.arange(i, i + n) for i, n in zip(d["shell_prim_index"], pn)])
    psh = np.repeat(np.arange(l.size), pn)
    c = np.asarray(d["coefficient"]) * np.asarray(d["prim_factor"])
    t = lambda v: torch.as_tensor(np.ascontiguousarray(v), device=dev)  # noqa: E731
    W = torch.zeros((pi.size, l.size), dtype=torch.float64, device=dev)
    W[torch.arange(pi.size, device=dev), t(psh)] = t(c[pi] * np.asarray(d["shell_factor"])[psh])
    return {"sh": t(np.array(sh)), "abc": t(np.array(abc)), "f": t(d["ao_factor"]).double(), "nuc": t(nuc),
            "pnuc": t(nuc[psh]), "a": t(np.asarray(d["exponent"])[pi]).double(), "W": W,
            "cut": math.log(2.0) * (PRECISION - 1)}


def _ao(b, x, R, order):
    """AOs at points x [p][3], nuclei R [N][3]: [p][5][A] (order 2), or the Hessian rows [3][p][4][A] (order 3)."""
    v = x[:, None, :] - R[None]
    r2 = (v * v).sum(-1)
    ar2 = r2[:, b["pnuc"]] * b["a"]
    e = torch.where(ar2 > b["cut"], torch.zeros_like(ar2), torch.exp(-ar2))
    s = r2[:, b["nuc"]]
    S = [(e * b["a"] ** k) @ b["W"] for k in range(4 if order == 3 else 2)]
    lap = (e * b["a"] * (4.0 * ar2 - 6.0)) @ b["W"]
    sh = b["sh"]
    R0, R1 = S[0][:, sh], -S[1][:, sh]                       # R(s) and dR/ds, s = r^2
    lapR = lap[:, sh]
    va = [v[:, b["nuc"]][:, sh, c] for c in range(3)]
    X, Y, Z = (_powers(va[c], b["abc"][:, c]) for c in range(3))
    P = X[0] * Y[0] * Z[0]
    Pd = [X[1] * Y[0] * Z[0], X[0] * Y[1] * Z[0], X[0] * Y[0] * Z[1]]
    Rd = [2.0 * va[c] * R1 for c in range(3)]
    lapP = X[2] * Y[0] * Z[0] + X[0] * Y[2] * Z[0] + X[0] * Y[0] * Z[2]
    f = b["f"]
    if order == 2:
        rows = [P * R0] + [Pd[c] * R0 + P * Rd[c] for c in range(3)]
        rows.append(P * lapR + lapP * R0 + 2.0 * sum(Pd[c] * Rd[c] for c in range(3)))
        return torch.stack(rows, 1) * f
    R2 = S[2][:, sh]
    k3 = ((e * b["a"] ** 2 * (20.0 - 8.0 * ar2)) @ b["W"])[:, sh]   # grad lap R = v (20 R'' + 8 s R''')
    q = [X, Y, Z]

    def mono(i, j, k):
        return q[0][i] * q[1][j] * q[2][k]

    unit = [(1, 0, 0), (0, 1, 0), (0, 0, 1)]

    def at(*dirs):
        return mono(*[sum(unit[c][k] for c in dirs) for k in range(3)])

    out = []
    for i in range(3):
        rows = []
        t = 0.0
        for j in range(3):
            Rdd = 4.0 * va[i] * va[j] * R2 + (2.0 * R1 if i == j else 0.0)
            Pdd = at(i, j)
            rows.append(Pdd * R0 + Pd[i] * Rd[j] + Pd[j] * Rd[i] + P * Rdd)
            t = t + Pdd * Rd[j] + Pd[j] * Rdd
        dlapP = sum(at(i, j, j) for j in range(3))
        rows.append(dlapP * R0 + lapP * Rd[i] + 2.0 * t + Pd[i] * lapR + P * va[i] * k3)
        out.append(torch.stack(rows, 1) * f)
    return torch.stack(out, 0)


def exact(case, seed):
    """The same outputs in 64-bit torch, from the definitions."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    call = case["call"]
    if call == "grad" and case["points"] * case["nuclei"] > 6_000_000:
        return None
    outs = []
    for d, x in _systems(case, seed):
        b = _basis(d, dev)
        R = torch.as_tensor(np.asarray(d["nucl_coord"], dtype=np.float64).reshape(3, -1).T.copy(), device=dev)
        C = torch.as_tensor(np.ascontiguousarray(d["mo_coef"]), device=dev)
        x = torch.as_tensor(x, device=dev)
        A = int(d["ao_num"])
        step = max(16, min(4096, int(2.0e7 / (A * (6 if call == "grad" else 1)))))
        if call == "grad":
            g = torch.Generator(dev).manual_seed(seed)
            W = torch.randn((x.shape[0], 5, C.shape[0]), dtype=torch.float64, device=dev, generator=g)
            R.requires_grad_()
            C.requires_grad_()
            mo, gx, gR, gC = [], [], torch.zeros_like(R), torch.zeros_like(C)
            for p in range(0, x.shape[0], step):
                xp = x[p:p + step].clone().requires_grad_()
                m = _ao(b, xp, R, 2) @ C.T
                a = torch.autograd.grad(m, [xp, R, C], grad_outputs=W[p:p + step])
                mo.append(m.detach())
                gx.append(a[0])
                gR += a[1]
                gC += a[2]
            return {"mo": torch.cat(mo), "points": torch.cat(gx).T.contiguous(), "nuclei": gR, "coefficients": gC}
        parts = []
        for p in range(0, x.shape[0], step):
            ao = _ao(b, x[p:p + step], R, 3 if call == "ao_hessian" else 2)
            if call == "mo_value":
                ao = ao[:, 0] @ C.T
            elif call not in ("ao_vgl", "ao_hessian"):
                ao = ao @ C.T
            parts.append(ao)
        outs.append(torch.cat(parts, 1 if call == "ao_hessian" else 0))
    if call == "batch":
        return torch.cat([o.reshape(-1) for o in outs])
    return outs[0].reshape(-1).cpu().numpy() if call == "host" else outs[0]
