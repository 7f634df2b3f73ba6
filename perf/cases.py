"""The work that a user of this framework has it do, as cases that can be timed.

Kinds of case:

``frames2d``   whole nonlinear transient analyses of 2D RC frames through ``runtime.Analysis``:
               create, run the record, read the histories back
``frames3d``   the same for 3D RC frames with rigid-diaphragm floors (a band that fits shared memory
               for the small ones, a band in global memory for the tall ones)
``sections``   a batch of independent fiber sections taken through a loading cycle
``band``       one band factor-solve on a caller's device buffers
``mlp_train``  an epoch of training of the learned predictor's network
``mlp_infer``  the trained network applied to a table of node features

A case is a dict of plain values; ``prepare`` makes what a program holds before the call from the
case and a seed, ``run`` is one pass, ``work`` counts the bytes and operations that the pass cannot
do without, ``exact`` gives the 64-bit value where there is one.
"""
from __future__ import annotations

import copy
import functools
import math

import numpy as np
import torch

from strut_b200 import _abi as A
from strut_b200 import model as M
from strut_b200 import runtime
from strut_b200 import workloads as W


def listed():
    return [
        # the plain method on one small frame, the first thing a user runs: launches and the
        # latency of one Newton iteration
        _f2("frame2d_3x3", frames=1, stories=3, bays=3, steps=200),
        # one tall frame: the longest band and the largest single 2D system of the batched set
        _f2("frame2d_12x5", frames=1, stories=12, bays=5, steps=100),
        # displacement-based elements with P-Delta on a few frames
        _f2("frames2d_disp_8", frames=8, stories=0, bays=0, steps=100, element="dispBeamColumn2d", geom="PDelta"),
        # a suite of records on uneven frames, an ordinary batch
        _f2("frames2d_32", frames=32, stories=0, bays=0, steps=100),
        # the batched set the benchmark runs (256 uneven frames), a window of its steps
        _f2("frames2d_256", frames=256, stories=0, bays=0, steps=60),
        # 32 bidirectional records on a 4-story 3D diaphragm frame (the evaluation set of the
        # learned predictor), a window of its steps
        _f3("frames3d_32", frames=32, stories=4, bays=3, steps=40, fibers=148),
        # a tall 3D frame whose band lives in global memory, a window of its steps
        _f3("frame3d_tall", frames=1, stories=12, bays=4, steps=12, fibers=208),
        # a few sections through a loading cycle (moment-curvature work)
        {"name": "sections_300", "kind": "sections", "n": 300, "points": 8, "commit": True, "beam": False},
        # as many sections as the batched set has fibers: the streaming form of the fiber update
        {"name": "sections_78385", "kind": "sections", "n": 78385, "points": 8, "commit": True, "beam": False},
        # the band solve of a caller that keeps its own Newton loop: a 2D frame's system
        {"name": "band_216", "kind": "band", "n": 216, "bw": 20, "spd": False},
        # an epoch of the 2D predictor's training in the benchmark's minibatches
        {"name": "mlp_train_200k", "kind": "mlp_train", "n": 200_000, "n_in": 29, "n_out": 3, "batch": 8192},
        # features of a 3D set's nodes through the trained network
        {"name": "mlp_infer_100k", "kind": "mlp_infer", "n": 100_001, "n_in": 41, "n_out": 6},
    ]


def _f2(name, frames, stories, bays, steps, element="forceBeamColumn2d", geom="Linear"):
    """2D frames; stories / bays 0: uneven, drawn per frame from 3..12 and 2..5."""
    return {"name": name, "kind": "frames2d", "frames": frames, "stories": stories, "bays": bays, "steps": steps,
            "element": element, "geom": geom}


def _f3(name, frames, stories, bays, steps, fibers):
    return {"name": name, "kind": "frames3d", "frames": frames, "stories": stories, "bays": bays, "steps": steps,
            "fibers": fibers}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["one2d", "batch2d", "disp2d", "batch3d", "tall3d", "sections", "band", "mlp_train",
                       "mlp_infer"])
    if kind == "one2d":
        c = _f2("", 1, rng.randint(3, 12), rng.randint(2, 5), rng.randint(40, 120))
    elif kind == "batch2d":
        n = _log(rng, 4, 256)
        c = _f2("", n, 0, 0, max(24, min(100, 60 * 256 // n // 4)) - rng.randint(0, 12))
    elif kind == "disp2d":
        c = _f2("", _log(rng, 1, 48), 0, 0, rng.randint(40, 100), "dispBeamColumn2d",
                rng.choice(["PDelta", "Linear"]))
    elif kind == "batch3d":
        c = _f3("", _log(rng, 1, 32), rng.randint(2, 4), rng.randint(2, 3), rng.randint(16, 40), 148)
    elif kind == "tall3d":
        c = _f3("", 1, rng.randint(8, 12), rng.randint(3, 4), rng.randint(6, 12), 208)
    elif kind == "sections":
        c = {"name": "", "kind": "sections", "n": _log(rng, 1, 78385), "points": rng.randint(4, 8),
             "commit": rng.random() < 0.75, "beam": rng.random() < 0.5}
    elif kind == "band":
        n = _log(rng, 24, 512)
        bw = rng.randint(4, 25)
        c = {"name": "", "kind": "band", "n": n, "bw": min(bw, n - 1), "spd": rng.random() < 0.4}
    else:
        n_in, n_out = rng.choice([(29, 3), (41, 6)])
        if kind == "mlp_train":
            c = {"name": "", "kind": kind, "n": _log(rng, 2_000, 200_000), "n_in": n_in, "n_out": n_out,
                 "batch": rng.choice([4096, 8192])}
            c["batch"] = min(c["batch"], c["n"])
        else:
            c = {"name": "", "kind": kind, "n": _log(rng, 500, 100_001), "n_in": n_in, "n_out": n_out}
    del c["name"]
    return c


def prepare(case, seed):
    return _KINDS[case["kind"]][0](case, seed)


def run(state):
    return state["run"](state)


def work(case):
    return _KINDS[case["kind"]][1](case)


def exact(case, seed):
    f = _KINDS[case["kind"]][2]
    return f(case, seed) if f else None


# ---- transient analyses ------------------------------------------------------------------------
#
# What a program holds: the models (Strut's JSON schema, loaded).  A pass is the whole analysis:
# create the handle, run the record, read back the histories of every node displacement, of the
# first element's forces and the Newton iterations.  The result is an iterate that a convergence
# test accepted after a path-dependent history, so there is no 64-bit value to hold it against.


@functools.lru_cache(maxsize=64)
def _frame2d(stories, bays, element, geom):
    case = W.rc_frame_case(stories=stories, bays=bays, steps=1, element=element, geom=geom, record=np.zeros(2))
    nodes = [n["id"] for n in case["nodes"] if "constraints" not in n]
    case["recorders"][0]["nodes"] = nodes
    return case


@functools.lru_cache(maxsize=16)
def _frame3d(stories, bays, fibers):
    if fibers == 208:
        case = W.tall_frame3d_case(stories=stories, bays=bays, steps=1)
    else:
        case = W.rc_frame3d_case(stories=stories, bays_x=bays, bays_y=bays, dt=0.005, steps=1, diaphragm=True,
                                 bidirectional=True)
    nodes = [n["id"] for n in case["nodes"] if "constraints" not in n]
    case["recorders"][0]["nodes"] = nodes
    return case


def _with_records(base, records, dt, steps):
    """The case with its ground motions and its number of steps."""
    case = dict(base)
    case["time_series"] = [{"type": "Path", "tag": k + 1, "dt": dt, "values": [float(v) for v in r]}
                           for k, r in enumerate(records)]
    case["analysis"] = dict(copy.deepcopy(base["analysis"]), steps=steps, dt=dt)
    return case


def _prepare_frames(case, seed):
    steps, models = case["steps"], []
    sizes = np.random.default_rng(1000)
    rng = np.random.default_rng(seed)
    for k in range(case["frames"]):
        wg, pga = float(rng.uniform(8.0, 25.0)), float(rng.uniform(0.2, 0.6))
        rec = int(rng.integers(1 << 30))
        if case["kind"] == "frames2d":
            st, ba = int(sizes.integers(3, 13)), int(sizes.integers(2, 6))
            dt = 0.01
            base = _frame2d(case["stories"] or st, case["bays"] or ba, case["element"], case["geom"])
        else:
            dt = 0.005
            base = _frame3d(case["stories"], case["bays"], case["fibers"])
        # strong shaking soon after the start, so that the window holds cracking and yielding
        recs = [W.kanai_tajimi_record(rec + d, steps + 1, dt, wg=wg, pga_g=pga, rise=0.2)
                for d in range(len(base["time_series"]))]
        models.append(M.Model(_with_records(base, recs, dt, steps)))
    return {"run": _run_frames, "models": models, "steps": steps}


def _run_frames(s):
    with runtime.Analysis(s["models"]) as an:
        an.run(s["steps"], check=False)
        disp, ef, iters = an.history_all()
        return {"disp": disp, "ef": ef, "iters": iters, "status": an.instance_status()}


def _work_frames(case):
    # per step: at least two Newton iterations (the test looks at an increment), each reading every
    # fiber's committed history (Concrete02 40 B, Steel02 84 B) and factoring the band, and one
    # commit that reads and writes it; about 60 operations per fiber evaluation
    two_d = case["kind"] == "frames2d"
    sizes = np.random.default_rng(1000)
    byte = flop = 0.0
    for _ in range(case["frames"]):
        st, ba = int(sizes.integers(3, 13)), int(sizes.integers(2, 6))
        if two_d:
            st, ba = case["stories"] or st, case["bays"] or ba
            elements, n, bw = st * (ba + 1) + st * ba, 3 * st * (ba + 1), 3 * (ba + 2)
            c2, s2 = 140, 8
        else:
            st, ba = case["stories"], case["bays"]
            col = (ba + 1) ** 2
            elements, n = st * (col + 2 * ba * (ba + 1)), st * (3 * col + 3)
            bw = 3 * col + 8
            c2, s2 = case["fibers"] - 8, 8
        fibers = 5.0 * elements
        byte += case["steps"] * fibers * (2 * (40 * c2 + 84 * s2) + 80 * c2 + 168 * s2)
        flop += case["steps"] * (3 * 60.0 * fibers * (c2 + s2) + 2 * 2.0 * n * bw * bw)
    return {"bytes": byte, "flops": flop}


# ---- fiber sections ----------------------------------------------------------------------------


def _section(beam):
    return W.rc_section(1, 0.4, 0.6) if beam else W.rc_section(1, 0.5, 0.5)


def _cycle(case, seed):
    """Strains of the loading cycle: points x n x (eps0, kappa), on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n, k = case["n"], case["points"]
    ph = torch.rand((1, n), generator=g, device="cuda", dtype=torch.float64) * (2.0 * math.pi)
    amp = 2.0e-3 + 6.0e-3 * torch.rand((1, n), generator=g, device="cuda", dtype=torch.float64)
    t = torch.arange(k, device="cuda", dtype=torch.float64)[:, None] * (2.0 * math.pi / k)
    ek = torch.empty((k, n, 2), dtype=torch.float64, device="cuda")
    ek[:, :, 0] = -3.0e-4 + 2.0e-4 * torch.sin(t + ph)
    ek[:, :, 1] = amp * torch.sin(t + 2.0 * ph)
    return ek


def _prepare_sections(case, seed):
    mats = [{"id": 1, "type": "Concrete02", "params": dict(W.CORE)},
            {"id": 2, "type": "Concrete02", "params": dict(W.COVER)},
            {"id": 3, "type": "Steel02", "params": dict(W.STEEL)}]
    m, nm, f, nf = M.section_fibers(_section(case["beam"]), mats)
    ek = _cycle(case, seed)
    resp = torch.empty((case["points"], case["n"], 5), dtype=torch.float64, device="cuda")
    return {"run": _run_sections, "batch": runtime.SectionBatch(m, nm, f, nf, case["n"]), "ek": ek, "resp": resp,
            "commit": case["commit"]}


def _run_sections(s):
    stream = torch.cuda.current_stream().cuda_stream
    for k in range(s["ek"].shape[0]):
        s["batch"].eval(s["ek"][k].data_ptr(), s["resp"][k].data_ptr(), commit=s["commit"], stream=stream)
    return s["resp"]


def _work_sections(case):
    per = 140 * (80 if case["commit"] else 40) + 8 * (168 if case["commit"] else 84) + 56
    return {"bytes": float(case["points"]) * case["n"] * per, "flops": 60.0 * case["points"] * case["n"] * 148}


def _exact_sections(case, seed):
    """The cycle in plain torch, 64 bits: Concrete02 and Steel02 fibers from their virgin state."""
    ek = _cycle(case, seed)
    b, h = (0.4, 0.6) if case["beam"] else (0.5, 0.5)
    c, h2 = W.COVER_T, 0.5 * h
    dy = 2.0 * (h2 - c) / 10
    fib = [(-(h2 - c) + (i + 0.5) * dy, dy * 2.0 * (0.5 * b - c) / 10, 0) for i in range(10) for _ in range(10)]
    fib += [(s * (h2 - 0.5 * c), c * b / 20, 1) for s in (1.0, -1.0) for _ in range(20)]
    fib += [(s * (h2 - c), W.BAR_AREA, 2) for s in (1.0, -1.0) for _ in range(4)]
    ybar = sum(y * a for y, a, _ in fib) / sum(a for _, a, _ in fib)
    out = []
    for part in torch.split(ek, 4096, dim=1):
        states, rows = {}, []
        for p in part:
            e0, ka = p[:, 0:1], p[:, 1:2]
            s = [0.0] * 5
            for m, mat in enumerate((W.CORE, W.COVER, W.STEEL)):
                y = torch.tensor([q[0] - ybar for q in fib if q[2] == m], device="cuda", dtype=torch.float64)
                a = torch.tensor([q[1] for q in fib if q[2] == m], device="cuda", dtype=torch.float64)
                f = _steel02 if m == 2 else _concrete02
                sig, tan, new = f(mat, states.get(m), e0 - y * ka)
                if case["commit"]:
                    states[m] = new
                fs, ks = sig * a, tan * a
                for i, v in enumerate((fs, -fs * y, ks, -ks * y, ks * y * y)):
                    s[i] = s[i] + v.sum(1)
            rows.append(torch.stack(s, 1))
        out.append(torch.stack(rows))
    return torch.cat(out, 1)


def _concrete02(m, st, eps):
    """Yassin's concrete with linear tension softening (Concrete02)."""
    fc, e0, fcu, eu, rat, ft, ets = (m[k] for k in ("fpc", "epsc0", "fpcu", "epscu", "rat", "ft", "Ets"))
    z = torch.zeros_like(eps)
    ec0 = 2.0 * fc / e0
    if st is None:
        st = (z, z, z + ec0, z, z)
    cep, csig, ctan, ecmin, dept = st

    def compr(e):
        r = e / e0
        soft = (fcu - fc) / (eu - e0)
        sig = torch.where(e >= e0, fc * r * (2.0 - r), torch.where(e > eu, soft * (e - e0) + fc, z + fcu))
        return sig, torch.where(e >= e0, ec0 * (1.0 - r), torch.where(e > eu, z + soft, z + 1.0e-10))

    def tens(e):
        e1, e2 = ft / ec0, ft * (1.0 / ets + 1.0 / ec0)
        sig = torch.where(e <= e1, e * ec0, torch.where(e <= e2, ft - ets * (e - e1), z))
        return sig, torch.where(e <= e1, z + ec0, torch.where(e <= e2, z - ets, z + 1.0e-10))

    epsr = (fcu - rat * ec0 * eu) / (ec0 * (1.0 - rat))
    sigmm, _ = compr(ecmin)
    er = (sigmm - ec0 * epsr) / (ecmin - epsr)
    ept = ecmin - sigmm / er
    sicn, _ = tens(dept)
    etn = torch.where(dept != 0.0, sicn / torch.where(dept != 0.0, dept, z + 1.0), z + ec0)
    lo, hi = sigmm + er * (eps - ecmin), 0.5 * er * (eps - ept)
    s, e = csig + ec0 * (eps - cep), z + ec0
    s, e = torch.where(s <= lo, lo, s), torch.where(s <= lo, er, e)
    s, e = torch.where(s >= hi, hi, s), torch.where(s >= hi, 0.5 * er, e)
    ts, te = tens(eps - ept)
    tail = eps > ept + dept
    s = torch.where(eps <= ept, s, torch.where(tail, ts, etn * (eps - ept)))
    e = torch.where(eps <= ept, e, torch.where(tail, te, etn))
    cs, ct = compr(eps)
    env, same = eps < ecmin, (eps - cep).abs() < 2.220446049250313e-16
    s = torch.where(same, csig, torch.where(env, cs, s))
    e = torch.where(same, ctan, torch.where(env, ct, e))
    return s, e, (eps, s, e, torch.where(env & ~same, eps, ecmin),
                  torch.where(tail & ~env & ~same, eps - ept, dept))


def _steel02(m, st, eps):
    """Giuffre-Menegotto-Pinto steel without isotropic hardening (a1 = a3 = 0): Steel02."""
    fy, es, b, r0, c1, c2 = (m[k] for k in ("Fy", "E0", "b", "R0", "cR1", "cR2"))
    z = torch.zeros_like(eps)
    ey, esh = fy / es, b * es
    if st is None:
        st = (z, z, z + es, z + ey, z - ey, z, z, z, z, z, z)  # kon 0: no loading branch yet
    cep, csig, ctan, emax, emin, epl, es0, ss0, er, sr, kon = st
    de = eps - cep
    virgin = kon == 0
    still = virgin & (de.abs() < 2.220446049250313e-15)
    up = (de > 0.0) | ((de == 0.0) & (kon == 1))
    sg = torch.where(up, z + 1.0, z - 1.0)
    turn = ~virgin & (((kon == 2) & up) | ((kon == 1) & ~up))
    er, sr = torch.where(turn, cep, er), torch.where(turn, csig, sr)
    emin = torch.where(turn & up, torch.minimum(emin, cep), emin)
    emax = torch.where(turn & ~up, torch.maximum(emax, cep), emax)
    es0 = torch.where(virgin, sg * ey, torch.where(turn, (sg * fy - sg * esh * ey - sr + es * er) / (es - esh), es0))
    ss0 = torch.where(virgin, sg * fy, torch.where(turn, sg * fy + esh * (es0 - sg * ey), ss0))
    epl = torch.where(virgin, sg * ey, torch.where(turn, torch.where(up, emax, emin), epl))
    xi = ((epl - es0) / ey).abs()
    r = r0 * (1.0 - c1 * xi / (c2 + xi))
    x = (eps - er) / (es0 - er)
    d1 = 1.0 + x.abs() ** r
    d2 = d1 ** (1.0 / r)
    s = (b * x + (1.0 - b) * x / d2) * (ss0 - sr) + sr
    e = (b + (1.0 - b) / (d1 * d2)) * (ss0 - sr) / (es0 - er)
    s, e = torch.where(still, z, s), torch.where(still, z + es, e)
    kon = torch.where(still, kon, torch.where(up, z + 1.0, z + 2.0))
    return s, e, (eps, s, e, emax, emin, epl, es0, ss0, er, sr, kon)


# ---- band factor-solve -------------------------------------------------------------------------


def _band_system(case, seed):
    """Dense symmetric positive definite band matrix (an effective stiffness) and right-hand side."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n, bw = case["n"], case["bw"]
    k = torch.randn((n, n), generator=g, device="cuda", dtype=torch.float64)
    i = torch.arange(n, device="cuda")
    k = torch.where((i[:, None] - i[None, :]).abs() <= bw, k + k.T, torch.zeros_like(k))
    k = k + torch.diag(k.abs().sum(1) * (1.0 + 0.5 * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)))
    return 1.0e6 * k, torch.randn(n, generator=g, device="cuda", dtype=torch.float64)


def _prepare_band(case, seed):
    k, rhs = _band_system(case, seed)
    n, bw = case["n"], case["bw"]
    i = torch.arange(n, device="cuda")[:, None]
    o = torch.arange(bw + 1 if case["spd"] else 2 * bw + 1, device="cuda")[None, :]
    j = i - o if case["spd"] else i + o - bw
    ok = (j >= 0) & (j < n)
    band = torch.where(ok, k[i, j.clamp(0, n - 1)], torch.zeros((), device="cuda", dtype=torch.float64)).contiguous()
    return {"run": _run_band, "band": band, "rhs": rhs, "x": torch.empty_like(rhs), "n": n, "bw": bw,
            "status": torch.zeros(1, dtype=torch.int32, device="cuda"),
            "system": A.SYSTEM_BAND_SPD if case["spd"] else A.SYSTEM_BAND_GENERAL}


def _run_band(s):
    rc = runtime.lib().strut_gpu_band_solve_noalloc(
        s["band"].data_ptr(), s["n"], s["bw"], s["system"], s["rhs"].data_ptr(), s["x"].data_ptr(),
        s["status"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    if rc != A.STRUT_OK:
        raise RuntimeError(f"band solve: {A.STATUS_NAMES.get(rc, rc)}")
    return [s["x"], s["status"]]


def _work_band(case):
    n, bw = case["n"], case["bw"]
    width = bw + 1 if case["spd"] else 2 * bw + 1
    return {"bytes": 8.0 * n * (width + 2), "flops": 2.0 * n * bw * bw * (0.5 if case["spd"] else 1.0) + 4.0 * n * bw}


def _exact_band(case, seed):
    k, rhs = _band_system(case, seed)
    return [torch.linalg.solve(k, rhs), None]


# ---- the learned predictor's network -----------------------------------------------------------

_H = 128


def _mlp_data(case, seed):
    """Parameters (Glorot scaled) and feature / target tables, host arrays as the library takes."""
    rng = np.random.default_rng(seed)
    n_in, n_out, n = case["n_in"], case["n_out"], case["n"]

    def glorot(a, b):
        return (rng.standard_normal((a, b)) * math.sqrt(2.0 / (a + b))).astype(np.float32)

    p = {"W1": glorot(n_in, _H), "b1": 0.1 * rng.standard_normal(_H).astype(np.float32),
         "W2": glorot(_H, _H), "b2": 0.1 * rng.standard_normal(_H).astype(np.float32),
         "W3": glorot(_H, n_out), "b3": 0.1 * rng.standard_normal(n_out).astype(np.float32)}
    x = rng.standard_normal((n, n_in), dtype=np.float32)
    w = rng.standard_normal((n_in, n_out), dtype=np.float32) / np.float32(math.sqrt(n_in))
    return p, x, np.tanh(x @ w).astype(np.float32)


def _prepare_mlp(case, seed):
    p, x, t = _mlp_data(case, seed)
    net = runtime.Mlp(case["n_in"], case["n_out"])
    net.set_params(p)
    train = case["kind"] == "mlp_train"
    return {"run": _run_train if train else _run_infer, "net": net, "p": p, "x": x, "t": t,
            "batch": case.get("batch", 0)}


def _run_train(s):
    s["net"].set_params(s["p"])  # from the initial parameters, the optimiser's moments cleared
    loss = s["net"].train(s["x"], s["t"], epochs=1, batch=s["batch"], lr=1.0e-3, seed=11)
    return [loss, s["net"].get_params()]


def _run_infer(s):
    return s["net"].forward(s["x"])


def _mlp_flops(case):
    return 2.0 * case["n"] * (case["n_in"] * _H + _H * _H + _H * case["n_out"])


def _work_train(case):
    return {"bytes": 4.0 * case["n"] * (case["n_in"] + case["n_out"]), "flops": 3.0 * _mlp_flops(case)}


def _work_infer(case):
    return {"bytes": 4.0 * case["n"] * (case["n_in"] + case["n_out"]), "flops": _mlp_flops(case)}


def _net64(p, x):
    gelu = functools.partial(torch.nn.functional.gelu, approximate="tanh")
    return gelu(gelu(x @ p["W1"] + p["b1"]) @ p["W2"] + p["b2"]) @ p["W3"] + p["b3"]


def _exact_infer(case, seed):
    p, x, _t = _mlp_data(case, seed)
    return _net64({k: torch.from_numpy(v).cuda().double() for k, v in p.items()}, torch.from_numpy(x).cuda().double())


def _exact_train(case, seed):
    """Adam in 64 bits over the same minibatches (the order is the documented seeded shuffle)."""
    p, x, t = _mlp_data(case, seed)
    p = {k: torch.from_numpy(v).cuda().double().requires_grad_() for k, v in p.items()}
    x, t = torch.from_numpy(x).cuda().double(), torch.from_numpy(t).cuda().double()
    n, mask = case["n"], (1 << 64) - 1
    st = (11 * 6364136223846793005 + 1442695040888963407) & mask
    perm = list(range(n))
    for i in range(n - 1, 0, -1):
        st = (st * 6364136223846793005 + 1442695040888963407) & mask
        j = (st >> 33) % (i + 1)
        perm[i], perm[j] = perm[j], perm[i]
    perm = torch.tensor(perm, device="cuda")
    opt = torch.optim.Adam(p.values(), lr=1.0e-3, betas=(0.9, 0.999), eps=1.0e-8)
    se = 0.0
    for b0 in range(0, n, case["batch"]):
        at = perm[b0:b0 + case["batch"]]
        err = _net64(p, x[at]) - t[at]
        opt.zero_grad()
        err.square().mean().backward()
        opt.step()
        se += float(err.detach().square().sum())
    return [se / (n * case["n_out"]), {k: v.detach() for k, v in p.items()}]


_KINDS = {
    "frames2d": (_prepare_frames, _work_frames, None),
    "frames3d": (_prepare_frames, _work_frames, None),
    "sections": (_prepare_sections, _work_sections, _exact_sections),
    "band": (_prepare_band, _work_band, _exact_band),
    "mlp_train": (_prepare_mlp, _work_train, _exact_train),
    "mlp_infer": (_prepare_mlp, _work_infer, _exact_infer),
}
