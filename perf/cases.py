"""What a user of this framework has it do, as cases that can be timed.

The cases follow the two modes a road design is valued in (the fixed-traffic
MTE population simulation and the controlled-traffic ROV), one road per call
and a whole GA generation at a time, and what stands beside them: the species
model of one road, the sensitivities of a valuation, and the surrogates that
screen a generation.  Every case goes through the public Python entry points
with host arrays, as a GA does, and returns everything the call returns.

Single-road cases take migration models made here (patches scattered over a
square grid, a 5-cell exponential migration range, 30% mortality a road
crossing - the shapes that the species models of `synth` have), so that
`exact` can restate them in 64 bits; the generation cases take a scene and
random roads and build their species models inside the call.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from transportoptimiser_gb300 import mlp
from transportoptimiser_gb300 import simulate_gpu as sg
from transportoptimiser_gb300 import synth
from transportoptimiser_gb300 import surrogate_ga as sga
from transportoptimiser_gb300.adjoint import FrozenPolicy, theta_from_problem
from transportoptimiser_gb300.generation import Generation, pack_segments

YEARS = 50
FLOWS = (0.0, 0.5, 1.0)                     # traffic of the three controls
HAZARD = -math.log(0.7)                     # per crossing at full flow


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one road, one species, 64 x 64 cells: the plain MTE call, the smallest valuation a user makes
        dict(name="mte_one_road", kind="mte", species=1, patches=40, side=64, paths=2000, sem=0),
        # the same call for a tight confidence bound on the end population (a final design)
        dict(name="mte_many_paths", kind="mte", species=2, patches=115, side=128, paths=40000, sem=1),
        # the species model of one road on a 200 x 200 region map, all matrices returned
        dict(name="species_model", kind="species", side=200, tile=30, res=10, points=36, sem=1),
        # the ROV of one road, 2 species, with the policy and the values of every path
        dict(name="rov_one_road", kind="rov", species=2, patches=115, side=128, paths=10000, bins=16,
             sem=1, algo=4, surfaces=False),
        # the ROV as the reference defines it (one species, its semantics), regression surfaces returned
        dict(name="rov_reference", kind="rov", species=1, patches=115, side=128, paths=2000, bins=16,
             sem=0, algo=4, surfaces=True),
        # the ROV by re-simulated paths (the reference's other algorithm), ragged sizes
        dict(name="rov_resimulated", kind="rov", species=2, patches=61, side=96, paths=1999, bins=11,
             sem=1, algo=6, surfaces=False),
        # the ROV of a small generation whose species models the caller already has
        dict(name="rov_batch", kind="rov_batch", roads=24, species=2, patches=115, side=128, paths=768,
             bins=16),
        # a GA generation valued by the MTE alone, as the GA loop calls it
        dict(name="generation_mte", kind="generation", roads=256, paths=64, rov_paths=0, bins=0, graph=False),
        # a GA generation valued in both modes at the path counts of a 1% Monte Carlo error
        dict(name="generation_both", kind="generation", roads=256, paths=64, rov_paths=768, bins=8, graph=True),
        # sensitivities of a valuation: outputs and the whole Jacobian (forward, then one backward per output)
        dict(name="adjoint", kind="adjoint", species=2, patches=115, side=128, paths=10000),
        # training the learned surrogate on pairs that the simulator made
        dict(name="mlp_train", kind="mlp", rows=20000, epochs=4, batch=512),
        # the reference's surrogate of the ROV value over initial animals at risk and unit use
        dict(name="surrogate_rov", kind="surrogate", samples=1000, dims=3, bins=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mte", "species", "rov", "rov", "rov_batch", "generation", "generation",
                       "adjoint", "mlp", "surrogate"])
    if kind == "mte":
        n = _log(rng, 5, 340)
        return dict(kind=kind, species=rng.randint(1, 3), patches=n, side=_side(n),
                    paths=_log(rng, 64, 40000), sem=rng.randint(0, 1))
    if kind == "species":
        res = rng.randint(4, 10)
        return dict(kind=kind, side=rng.choice([64, 96, 128, 160, 200]), tile=rng.randint(10, 32), res=res,
                    points=rng.randint(8, 64), sem=rng.randint(0, 1))
    if kind == "rov":
        sem = rng.choice([0, 1, 1, 1])
        algo = 6 if sem == 1 and rng.random() < 0.25 else 4
        n = _log(rng, 20, 130 if algo == 6 else 340)
        S = 1 if sem == 0 else rng.randint(1, 2 if algo == 6 else 3)
        bins = rng.randint(5, 8 if S == 3 else 16)
        return dict(kind=kind, species=S, patches=n, side=_side(n),
                    paths=_log(rng, 256, 2500 if algo == 6 else 10000),
                    bins=bins, sem=sem, algo=algo, surfaces=rng.random() < 0.3)
    if kind == "rov_batch":
        n = _log(rng, 30, 200)
        return dict(kind=kind, roads=_log(rng, 2, 24), species=2, patches=n, side=_side(n),
                    paths=_log(rng, 128, 1500), bins=rng.randint(5, 16))
    if kind == "generation":
        both = rng.random() < 0.6
        return dict(kind=kind, roads=_log(rng, 4, 160 if both else 256), paths=_log(rng, 32, 256),
                    rov_paths=_log(rng, 200, 1100) if both else 0, bins=rng.randint(5, 8) if both else 0,
                    graph=both or rng.random() < 0.3)
    if kind == "adjoint":
        n = _log(rng, 20, 130)
        return dict(kind=kind, species=rng.randint(1, 2), patches=n, side=_side(n), paths=_log(rng, 500, 10000))
    if kind == "mlp":
        return dict(kind=kind, rows=_log(rng, 500, 20000), epochs=rng.randint(1, 4),
                    batch=rng.choice([128, 250, 512, 1024]))
    d = rng.randint(2, 4)
    return dict(kind="surrogate", samples=_log(rng, 500, 2000), dims=d, bins={2: 40, 3: 16, 4: 8}[d])


def _side(patches):
    """Grid side on which that many patches lie as densely as on the region maps."""
    return int(max(24, round(128 * math.sqrt(patches / 115.0))))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _rng(seed):
    return np.random.default_rng([20110, int(seed) & 0x7FFFFFFF])


def _crossings(p, segs):
    """[N][N] segments of a road that the line between two patches crosses."""
    d1 = p[None, :, :] - p[:, None, :]
    out = np.zeros(d1.shape[:2], np.int32)
    for x3, y3, x4, y4 in segs:
        x43, y43 = x4 - x3, y4 - y3
        y13, x13 = (p[:, 1] - y3)[:, None], (p[:, 0] - x3)[:, None]
        den = y43 * d1[..., 0] - x43 * d1[..., 1]
        with np.errstate(divide="ignore", invalid="ignore"):
            ua = (x43 * y13 - y43 * x13) / den
            ub = (d1[..., 0] * y13 - d1[..., 1] * x13) / den
        out += (ua >= 0) & (ua <= 1) & (ub >= 0) & (ub <= 1)
    out = np.maximum(np.triu(out, 1), np.triu(out, 1).T)
    return out


def _model(rng, n, side):
    """Migration model of one species along one road: patches, capacities,
    crossings and the float matrices of every control, destination-major."""
    p = rng.uniform(0, side, (n, 2))
    cells = rng.integers(4, 101, n).astype(np.float64)
    m = max(8, min(64, side // 4))
    pts = np.column_stack([np.sort(rng.uniform(0, side, m)), rng.uniform(0, side, m)])
    cross = _crossings(p, np.column_stack([pts[:-1], pts[1:]]))
    dist = np.hypot(p[:, None, 0] - p[None, :, 0], p[:, None, 1] - p[None, :, 1])
    w = cells[None, :] * np.exp(rng.choice([0.0, -0.3, -0.6], n))[None, :] * np.exp(-0.2 * dist)
    w[dist > math.log(20.0) / 0.2] = 0.0
    trans = w / w.sum(1, keepdims=True)
    mmm = np.stack([(trans * np.exp(-HAZARD * f * cross)).T for f in FLOWS]).astype(np.float32)
    mmm[mmm <= 1e-5] = 0.0
    return dict(N=n, init_pops=(25 * cells).astype(np.float32), caps=(50 * cells).astype(np.float32),
                mmm=np.ascontiguousarray(mmm), crossings=cross)


def _models(case, seed, roads=1):
    rng = _rng(seed)
    return [[_model(rng, case["patches"] - 3 * (s % 2) if case["patches"] > 8 else case["patches"], case["side"])
             for s in range(case["species"])] for _ in range(roads)]


def _params(noise):
    # growth now / mean / sd, threshold, reversion, jump size, jump probability, local variability
    return np.array([0.05, 0.05, noise, 0.0, 0.5, 0.0, 0.0, 0.4], np.float32)


def _rov_problem(models, paths, bins, sem, algo, seed, road=0):
    unc = []
    for sigma, theta in ((0.1, 0.2), (0.2, 0.35), (0.3, 0.5)):
        unc += [1.0, 1.0, sigma, theta, 0.0, 0.0]
    return dict(n_paths=paths, n_years=YEARS, dim_res=bins, dt=1.0, rrr=7.0, unit_cost=0.5, unit_revenue=1.2,
                seed=int(seed), road=road, sem=sem, algo=algo,
                species=[dict(N=m["N"], params=_params(0.05), init_pops=m["init_pops"], caps=m["caps"],
                              mmm=m["mmm"]) for m in models],
                flows=np.asarray(FLOWS, np.float32) * 100.0, uncert=np.asarray(unc, np.float32),
                fuel_costs=np.array([0.3], np.float32), fuel_idx=np.array([0], np.int32),
                ore_content=np.array([0.8], np.float32), ore_sd=np.array([0.05], np.float32),
                demand_idx=2 if sem == 1 else -1)


def _species_scene(case, seed):
    # the region and the road are the case's, so that every seed has as many
    # patches; the animals on the map and the species' preferences are the seed's
    rng = _rng(case["side"] * 1000 + case["points"])
    W, types = case["side"], [synth.PRIMARY, synth.MARGINAL, synth.OTHER, 5, synth.CLEAR]
    base = synth.habitat_map(W, W, case["tile"], [0.35, 0.25, 0.15, 0.15, 0.1], types, rng)
    sp = synth.default_species(3, np.asarray(FLOWS), types[:4], threshold=0.0)
    road = synth.random_road(W, W, case["points"], rng)
    scene = synth.Scene(W=W, H=W, res=case["res"], base_map=base, species=[sp], n_controls=3,
                        flows=np.asarray(FLOWS), seed=seed)
    hab, rng = scene.hab_map(road), _rng(seed)
    for h in sp.habitats[:-1]:
        h.pref_mean = float(-rng.integers(0, 10) / 10.0)
    animals = np.where(np.isin(hab, types[:4]), rng.integers(5, 46, W * W), 0).astype(np.float64)
    return scene, sp, road, hab, animals


def _mlp_data(case, seed):
    rng = _rng(seed)
    x = rng.standard_normal((case["rows"], mlp.IN)).astype(np.float32)
    a = rng.standard_normal((mlp.IN, mlp.OUT)) / 4.0
    t = np.tanh(x @ a) + 0.1 * np.sin(2 * x[:, :mlp.OUT]) + 0.02 * rng.standard_normal((case["rows"], mlp.OUT))
    return x, t.astype(np.float32)


def _mlp_params(seed):
    rng = _rng(seed + 1)
    u = lambda n, fan: rng.uniform(-math.sqrt(6.0 / fan), math.sqrt(6.0 / fan), n)
    h, i, o = mlp.HID, mlp.IN, mlp.OUT
    return np.concatenate([u(h * i, i), np.zeros(h), u(h * h, h), np.zeros(h), 0.5 * u(o * h, h),
                           np.zeros(o)]).astype(np.float32)


def _surrogate_data(case, seed):
    rng = _rng(seed)
    n, d = case["samples"], case["dims"]
    pred = rng.uniform(0.05, 0.6, (d, n)).astype(np.float32).astype(np.float64)
    v = -40.0 * (1.2 - pred.sum(0) / d) ** 2 + 6.0 * np.sin(4.0 * pred[0]) + 0.5 * rng.standard_normal(n) - 12.0
    sd = np.abs(3.0 + 2.0 * pred[-1] + 0.2 * rng.standard_normal(n))
    return pred, v.astype(np.float32).astype(np.float64), sd.astype(np.float32).astype(np.float64)


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case, kind=kind)
    if kind == "mte":
        st["models"] = _models(case, seed)[0]
        st["params"] = [_params(0.02)] * case["species"]
        st["seed"] = int(seed)
    elif kind == "species":
        scene, sp, road, hab, animals = _species_scene(case, seed)
        st["args"] = (hab, animals, scene.W, scene.H, scene.res, sp.habitats, road.colmajor(),
                      road.G, sp.hazard, sp.lambda_mean)
    elif kind == "rov":
        st["problem"] = _rov_problem(_models(case, seed)[0], case["paths"], case["bins"], case["sem"],
                                     case["algo"], seed)
    elif kind == "rov_batch":
        st["problems"] = [_rov_problem(m, case["paths"], case["bins"], 1, 4, seed, r)
                          for r, m in enumerate(_models(case, seed, case["roads"]))]
    elif kind == "generation":
        scene = synth.generation(int(seed) & 0xFFFF, n_roads=0)
        roads = sga.random_roads(scene, case["roads"], _rng(seed))
        gen = Generation(scene, max_roads=case["roads"], max_patches=512)
        if case["rov_paths"]:
            tiny = [dict(N=1, init_pops=np.ones(1, np.float32), caps=np.ones(1, np.float32),
                         mmm=np.zeros((3, 1, 1), np.float32))] * len(scene.species)
            gen.set_rov(_rov_problem(tiny, case["rov_paths"], case["bins"], 1, 4, seed))
        st["gen"], st["packed"] = gen, pack_segments(roads)
        st["opts"] = gen.opts(case["paths"], YEARS, seed=int(seed), sem=1, graph=case["graph"])
    elif kind == "adjoint":
        models = _models(case, seed)[0]
        pr = _rov_problem(models, case["paths"], 8, 1, 4, seed)
        ctl = _rng(seed + 1).integers(0, 3, (YEARS, case["paths"])).astype(np.int32)
        hz = np.asarray(FLOWS) * HAZARD
        st["policy"] = FrozenPolicy(pr, ctl, [m["crossings"] for m in models], hz)
        st["theta"] = theta_from_problem(pr, hz)
    elif kind == "mlp":
        st["params"] = _mlp_params(seed)
        st["x"], st["t"] = _mlp_data(case, seed)
    else:
        st["data"] = _surrogate_data(case, seed)
    return st


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "mte":
        end, stats = sg.simulateMTECUDA(state["models"], state["params"], case["paths"], YEARS,
                                        seed=state["seed"], sem=case["sem"])
        return dict(end_pops=end, stats=stats)
    if kind == "species":
        out = sg.createSpeciesModel(*state["args"], sem=case["sem"], max_patches=1024)
        return out
    if kind == "rov":
        want = ("cond_exp", "opt_cont", "unit_profits", "adj_pops") + (("regression",) if case["surfaces"] else ())
        return sg.simulateROVCUDA(state["problem"], want=want)
    if kind == "rov_batch":
        outs = sg.simulateROVCUDA_batch(state["problems"], want=("cond_exp", "opt_cont"))
        return {k: np.stack([o[k] for o in outs]) for k in ("cond_exp", "opt_cont", "stats", "value_se", "n_best")}
    if kind == "generation":
        return state["gen"].evaluate_segments(state["packed"], state["opts"])
    if kind == "adjoint":
        out, jac = state["policy"].jacobian(state["theta"])
        return dict(outputs=out, jacobian=jac)
    if kind == "mlp":
        p, curve = mlp.train_raw(state["params"], state["x"], state["t"], epochs=case["epochs"],
                                 batch=case["batch"], lr=2e-3, seed=3)
        return dict(params=p, loss=curve)
    pred, v, sd = state["data"]
    mean, s = sg.buildSurrogateROVCUDA(pred, v, sd, case["bins"], sem=1)
    return dict(mean=mean, sd=s)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
_NORMAL = 30          # operations of one standard normal (its share of a Box-Muller pair)
_GROW = 8             # logistic growth of one patch


def _nnz(n):
    return n * min(n, 6)        # a patch and its neighbours within the migration range


def work(case):
    kind = case["kind"]
    f4, f8 = 4, 8
    if kind == "mte":
        S, N, P = case["species"], case["patches"], case["paths"]
        flops = S * P * YEARS * (2 * _nnz(N) + N * (_GROW + _NORMAL))
        return dict(bytes=S * (N * N * f4 + 2 * N * f4 + P * f8), flops=flops)
    if kind == "species":
        W, N = case["side"], 4 * case["res"] ** 2
        G = case["points"]
        return dict(bytes=W * W * (4 + 8) + G * 32 + N * N * (4 + 8 + 3 * 8 + 3 * 4), flops=N * N * 8 + _nnz(N) * G * 10)
    if kind in ("rov", "rov_batch", "generation"):
        if kind == "generation":
            S, N, R, P = 3, 280, case["roads"], case["rov_paths"]
        else:
            S, N, R, P = case["species"], case["patches"], case.get("roads", 1), case["paths"]
        C, d = len(FLOWS), S + 1
        nnz = 7 * N if kind == "generation" else _nnz(N)
        flops = bytes_ = 0
        if P:
            algo6 = case.get("algo") == 6
            sims = 1 + (YEARS / 2 if algo6 else 0)
            forward = R * S * P * YEARS * (2 * C * nnz + N * (_GROW + _NORMAL)) * sims
            # the fitted grid queries of a year: no more than the grid, nor than the corners the paths read
            Q = case["bins"] ** d
            q = C * (Q if case.get("surfaces") or case.get("sem") == 0 or algo6 else min(Q, 0.25 * Q + P))
            n = P / C
            k = (3 if algo6 else 10) * (math.log(max(n, 4)) + 1)
            per = 3 * d * n ** 0.5 * k ** 0.5 + k * ((d + 1) * (d + 4) + 20) + (d + 1) ** 3 / 3
            flops += forward + R * YEARS * q * per
            bytes_ += R * P * YEARS * (f8 + 4) if kind != "generation" else 0
            if kind == "rov":
                bytes_ += P * YEARS * f8 * (1 + S)
                bytes_ += YEARS * C * (case["bins"] * d + 2 * Q) * f8 if case["surfaces"] else 0
        if kind == "generation":
            flops += R * S * case["paths"] * YEARS * (2 * nnz + N * (_GROW + _NORMAL))
            flops += R * S * (N * N * 8 + nnz * 35 * 10 + 4 * 200 * 200)
            bytes_ += R * (35 * 32 + S * 24 * f8) + S * 200 * 200 * 8
        else:
            bytes_ += R * S * (C * N * N * f4 + 2 * N * f4)
        return dict(bytes=int(bytes_), flops=int(flops))
    if kind == "adjoint":
        S, N, P = case["species"], case["patches"], case["paths"]
        one = S * P * YEARS * (2 * _nnz(N) + N * (_GROW + _NORMAL))
        # forward, then per species output a recomputed forward and a reverse sweep twice as dear
        return dict(bytes=S * 3 * N * N * 8 + P * YEARS * 4, flops=int(one * 4))
    if kind == "mlp":
        n = mlp.NPARAM
        return dict(bytes=case["rows"] * 19 * f4 * case["epochs"] + 2 * n * f4, flops=6 * n * case["rows"] * case["epochs"])
    n, d, R = case["samples"], case["dims"], case["bins"]
    k = 25 + 0.02 * n
    return dict(bytes=(d + 2) * n * f8 + 2 * (R * d + R ** d) * f8,
                flops=int(R ** d * (3 * d * n + 2 * k * ((d + 1) * (d + 4) + 20))))


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch and numpy
# ---------------------------------------------------------------------------
_M32 = 0xFFFFFFFF
_GROWTH, _SP_BROWN, _SP_JUMPSIZE, _CONTROL, _EX_BROWN, _ORE = 1, 2, 3, 5, 6, 9


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _mul_hi_lo(a, b):
    lo16, hi16 = a * (b & 0xFFFF), a * (b >> 16)
    return (hi16 + (lo16 >> 16)) >> 16, (lo16 + ((hi16 & 0xFFFF) << 16)) & _M32


def _philox(seed, stream, road, path, year, group):
    """Philox4x32-10 words of (group, year, path, stream | road << 8)."""
    c0, c1, c2 = torch.broadcast_tensors(group, year, path)
    c3 = torch.full_like(c0, (stream | (road << 8)) & _M32)
    k0, k1 = seed & _M32, (seed >> 32) & _M32
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
        h0, l0 = _mul_hi_lo(0xD2511F53, c0)
        h1, l1 = _mul_hi_lo(0xCD9E8D57, c2)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
    return c0, c1, c2, c3


def _box_muller(a, b):
    u = ((a >> 8).float() + 0.5) * 2.0 ** -24
    rad = torch.sqrt(-2.0 * torch.log(u.double()))
    ang = (b >> 8).double() * (2.0 * math.pi * 2.0 ** -24)
    return rad * torch.cos(ang), rad * torch.sin(ang)


def _normals(words):
    a, b = _box_muller(words[0], words[1])
    c, d = _box_muller(words[2], words[3])
    return torch.stack([a, b, c, d], -1)


def _i(v):
    return torch.as_tensor(v, dtype=torch.int64, device=_dev())


def _normal1(seed, stream, road, path, year, lane):
    return _normals(_philox(seed, stream, road, path, _i(year), _i(lane >> 2)))[..., lane & 3]


def _growth_z(seed, road, path, year, s, n):
    n4 = (n + 3) // 4
    groups = _i((s * 4 * n4) >> 2) + torch.arange(n4, device=_dev())
    z = _normals(_philox(seed, _GROWTH, road, path[:, None], _i(year), groups[None, :]))
    return z.reshape(path.numel(), 4 * n4)[:, :n]


def _f64(a):
    return torch.as_tensor(np.asarray(a), dtype=torch.float64, device=_dev())


def _exact_mte(case, seed):
    P, cols, stats = case["paths"], [], []
    path = torch.arange(P, device=_dev())
    prm = [float(x) for x in _params(0.02)]
    for s, m in enumerate(_models(case, seed)[0]):
        M, cap, init = _f64(m["mmm"][-1]).T.contiguous(), _f64(m["caps"]), _f64(m["init_pops"])
        x = init.expand(P, -1).clone()
        g = torch.full((P,), prm[0], dtype=torch.float64, device=_dev())
        for t in range(YEARS):
            g = g + prm[4] * (prm[1] - g) + g * _normal1(seed, _SP_BROWN, 0, path, t, s) * prm[2]
            mig = x @ M
            gr = g[:, None] * (1.0 + prm[7] * _growth_z(seed, 0, path, t, s, m["N"]))
            x = mig * (1.0 + gr * (cap - mig) / cap)
        e = (mig if case["sem"] == 0 else x).sum(1).cpu().numpy()
        it = float(init.sum())
        cols.append(e)
        stats.append(dict(mean=float(e.mean()), sd=float(e.std()), se=float(e.std(ddof=1) / math.sqrt(P)),
                          p_below=float((e < 0.2 * it).mean()), init_total=it))
    return dict(end_pops=np.stack(cols, 1), stats=stats)


def _processes(pr, path):
    """[Y + 1][P] of each exogenous process, and the ore grade of every year."""
    U = []
    unc = np.asarray(pr["uncert"], np.float64).reshape(-1, 6)
    for u, (cur, mean, sd, rev, _, _) in enumerate(unc):
        x = [torch.full((path.numel(),), cur, dtype=torch.float64, device=_dev())]
        for t in range(YEARS):
            z = _normal1(pr["seed"], _EX_BROWN, pr["road"], path, t, u)
            x.append(x[-1] + rev * (mean - x[-1]) + x[-1] * z * sd)
        U.append(torch.stack(x))
    f = path[None, :] * YEARS + torch.arange(YEARS, device=_dev())[:, None]
    z = _normals(_philox(pr["seed"], _ORE, pr["road"], f >> 2, _i(0), _i(0)))
    ore = float(pr["ore_content"][0]) + float(pr["ore_sd"][0]) * z.gather(-1, (f & 3)[..., None])[..., 0]
    return U, ore


def _profit(pr, U, ore, t):
    base = pr["unit_cost"] + float(pr["fuel_costs"][0]) * U[0][t] - pr["unit_revenue"] * ore[t] * U[1][t]
    return base * U[pr["demand_idx"]][t]


def _exact_rov(case, seed):
    """The path states of the valuation; the decisions and what follows from
    them hang on exact ties of a regression Monte Carlo and have no such value."""
    pr = _rov_problem(_models(case, seed)[0], case["paths"], case["bins"], case["sem"], case["algo"], seed)
    P = pr["n_paths"]
    path = torch.arange(P, device=_dev())
    prm = [float(x) for x in _params(0.05)]
    prof = None
    if case["sem"] == 1:
        U, ore = _processes(pr, path)
        prof = torch.zeros((YEARS, P), dtype=torch.float64, device=_dev())
        for t in range(1, YEARS):
            prof[t] = _profit(pr, U, ore, t)
        prof = prof.cpu().numpy().reshape(-1)
    S = len(pr["species"])
    adj = torch.zeros((YEARS, S, P), dtype=torch.float64, device=_dev())
    for s, m in enumerate(pr["species"]):
        M = [_f64(c).T.contiguous() for c in m["mmm"]]
        cap = _f64(m["caps"])
        x = _f64(m["init_pops"]).expand(P, -1).clone()
        g = torch.full((P,), prm[0], dtype=torch.float64, device=_dev())
        for t in range(YEARS):
            u = _philox(seed, _CONTROL, 0, path, _i(t), _i(0))[0]
            ctl = ((u >> 8).float() * 2.0 ** -24 * 3.0).int().clamp(max=2)
            g = g + prm[4] * (prm[1] - g) + g * _normal1(seed, _SP_BROWN, 0, path, t, s) * prm[2]
            migs = [x @ A for A in M]
            if t:
                adj[t, s] = migs[-1].sum(1)
            mig = torch.where((ctl == 0)[:, None], migs[0], torch.where((ctl == 1)[:, None], migs[1], migs[2]))
            z = _growth_z(seed, 0, path, t, s, m["N"])
            if case["sem"] == 0:
                x = mig * (1.0 + (g[:, None] + prm[7] * z) * (cap - mig) / cap / 100.0)
            else:
                x = (mig * (1.0 + g[:, None] * (1.0 + prm[7] * z) * (cap - mig) / cap)).clamp(min=0.0)
    out = dict(cond_exp=None, opt_cont=None, unit_profits=prof, adj_pops=adj.cpu().numpy().reshape(-1),
               stats=None, value_se=None, n_best=None)
    if case["surfaces"]:
        out["regression"] = None
    return out


def _exact_adjoint(case, seed):
    models = _models(case, seed)[0]
    pr = _rov_problem(models, case["paths"], 8, 1, 4, seed)
    P, S, C = case["paths"], len(models), len(FLOWS)
    unc = np.asarray(pr["uncert"], np.float64).reshape(-1, 6)
    ctl = _i(_rng(seed + 1).integers(0, 3, (YEARS, P)))
    base_h = [float(np.float32(f * HAZARD)) for f in FLOWS]
    prm = [float(x) for x in _params(0.05)]
    nU = len(unc)
    theta = np.concatenate([unc[:, 3], unc[:, 2], [prm[1]] * S, [prm[7]] * S, base_h])
    path = torch.arange(P, device=_dev())
    out, jac = np.zeros(1 + S), np.zeros((1 + S, theta.size))
    flows = _f64(pr["flows"])
    # the present value: the processes by their parameters, path by path
    th = _f64(theta).requires_grad_(True)
    X = [torch.full((P,), float(unc[u, 0]), dtype=torch.float64, device=_dev()) for u in range(nU)]
    f = path[None, :] * YEARS + torch.arange(YEARS, device=_dev())[:, None]
    z = _normals(_philox(seed, _ORE, 0, f >> 2, _i(0), _i(0)))
    ore = float(pr["ore_content"][0]) + float(pr["ore_sd"][0]) * z.gather(-1, (f & 3)[..., None])[..., 0]
    pv, disc = 0.0, 1.0
    for t in range(YEARS):
        base = pr["unit_cost"] + float(pr["fuel_costs"][0]) * X[0] - pr["unit_revenue"] * ore[t] * X[1]
        pv = pv + disc * flows[ctl[t]] * base * X[2]
        X = [X[u] + th[u] * (float(unc[u, 1]) - X[u]) + X[u] * th[nU + u] *
             _normal1(seed, _EX_BROWN, 0, path, t, u) for u in range(nU)]
        disc /= 1.07
    v = pv.mean()
    out[0] = float(v.detach())
    jac[0] = torch.autograd.grad(v, th)[0].cpu().numpy()
    # the end populations, in blocks of paths
    for s, m in enumerate(models):
        cap = _f64(m["caps"])
        base, X0 = [_f64(c) for c in m["mmm"]], _f64(m["init_pops"])
        cr = _f64(m["crossings"].T)
        for p0 in range(0, P, 2500):
            th = _f64(theta).requires_grad_(True)
            pp = path[p0:p0 + 2500]
            M = [(base[c] * torch.exp(-cr * (th[2 * nU + 2 * S + c] - base_h[c]))).T for c in range(C)]
            x = X0.expand(pp.numel(), -1)
            g = torch.full((pp.numel(),), prm[0], dtype=torch.float64, device=_dev())
            for t in range(YEARS):
                g = g + prm[4] * (th[2 * nU + s] - g) + g * _normal1(seed, _SP_BROWN, 0, pp, t, s) * prm[2]
                c = ctl[t, p0:p0 + 2500][:, None]
                mig = torch.where(c == 0, x @ M[0], torch.where(c == 1, x @ M[1], x @ M[2]))
                gr = g[:, None] * (1.0 + th[2 * nU + S + s] * _growth_z(seed, 0, pp, t, s, m["N"]))
                x = (mig * (1.0 + gr * (cap - mig) / cap)).clamp(min=0.0)
            v = x.sum() / P
            out[1 + s] += float(v.detach())
            jac[1 + s] += torch.autograd.grad(v, th)[0].cpu().numpy()
    return dict(outputs=out, jacobian=jac)


def _exact_mlp(case, seed):
    x, t = (_f64(a) for a in _mlp_data(case, seed))
    h, i, o = mlp.HID, mlp.IN, mlp.OUT
    p = _f64(_mlp_params(seed))
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    n, batch, state, step, curve = case["rows"], min(case["batch"], case["rows"]), 3, 0, []
    for _ in range(case["epochs"]):
        rows = np.arange(n)
        for j in range(n - 1, 0, -1):                      # seeded shuffle (splitmix64)
            state = (state + 0x9E3779B97F4A7C15) & 0xFFFFFFFFFFFFFFFF
            w = ((state ^ (state >> 30)) * 0xBF58476D1CE4E5B9) & 0xFFFFFFFFFFFFFFFF
            w = ((w ^ (w >> 27)) * 0x94D049BB133111EB) & 0xFFFFFFFFFFFFFFFF
            k = (w ^ (w >> 31)) % (j + 1)
            rows[j], rows[k] = rows[k], rows[j]
        rows, total = _i(rows), 0.0
        for s0 in range(0, n, batch):
            r = rows[s0:s0 + batch]
            q = p.clone().requires_grad_(True)
            a, b, c, d, e, f = torch.split(q, [h * i, h, h * h, h, o * h, o])
            y = torch.relu(x[r] @ a.view(h, i).T + b)
            y = torch.relu(y @ c.view(h, h).T + d) @ e.view(o, h).T + f
            loss = ((y - t[r]) ** 2).sum()
            total = total + loss.detach()
            grad = torch.autograd.grad(loss / (o * r.numel()), q)[0]
            step += 1
            m, v = 0.9 * m + 0.1 * grad, 0.999 * v + 0.001 * grad * grad
            p = p - 2e-3 * (m / (1 - 0.9 ** step)) / (torch.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
        curve.append(float(total) / (o * n))
    return dict(params=p.cpu().numpy(), loss=np.asarray(curve))


def _exact_surrogate(case, seed):
    pred, v, sd = _surrogate_data(case, seed)
    d, n = pred.shape
    R = case["bins"]
    k = (5 if n < 50 else int(5 + 5 * math.ceil((n - 50) // 50)) if n < 100 else
         int(math.ceil(10 + 15 * math.ceil((n - 100) // 400))) if n < 500 else int(25 + math.ceil((n - 500) * 0.02)))
    lo, hi = pred.min(1), pred.max(1)
    axes = lo[:, None] + np.arange(R)[None, :] * ((hi - lo) / (R - 1))[:, None]
    grid = np.stack(np.meshgrid(*axes, indexing="ij"), -1).reshape(-1, d)
    X = _f64(((pred - lo[:, None]) / (hi - lo)[:, None]).T)
    Q = _f64((grid - lo) / (hi - lo))
    D = torch.cdist(Q, X, compute_mode="donot_use_mm_for_euclid_dist")
    dist, ind = torch.topk(D, min(k, n), dim=1, largest=False)
    w = torch.exp(-0.5 * (dist / dist[:, -1:]) ** 2)
    A = torch.cat([torch.ones_like(dist)[..., None], X[ind] - Q[:, None, :]], -1)
    lhs = (A * w[..., None]).transpose(1, 2) @ A
    out = []
    for y, clip in ((v, True), (sd, False)):
        rhs = (A * w[..., None]).transpose(1, 2) @ _f64(y)[ind][..., None]
        f = torch.linalg.solve(lhs, rhs)[:, 0, 0]
        f = f.clamp(max=0.0) if clip else f
        out.append(np.concatenate([axes.reshape(-1), f.cpu().numpy()]))
    return dict(mean=out[0], sd=out[1])


def _regions(grid):
    """The smallest cell index of each cell's 4-connected region of one code."""
    lab = np.arange(grid.size).reshape(grid.shape)
    same = [grid[1:] == grid[:-1], grid[:, 1:] == grid[:, :-1]]
    while True:
        new = lab.copy()
        new[1:] = np.where(same[0], np.minimum(new[1:], new[:-1]), new[1:])
        new[:-1] = np.where(same[0], np.minimum(new[1:], new[:-1]), new[:-1])
        new[:, 1:] = np.where(same[1], np.minimum(new[:, 1:], new[:, :-1]), new[:, 1:])
        new[:, :-1] = np.where(same[1], np.minimum(new[:, 1:], new[:, :-1]), new[:, :-1])
        if np.array_equal(new, lab):
            return lab
        lab = new


def _exact_species(case, seed):
    """Patches, migration and survival of the species model.  Patches are the
    regions of one habitat type within a coarse block, blocks row by row."""
    if case["sem"] != 1:
        return None
    _, sp, road, hab, animals = _species_scene(case, seed)
    W, res = case["side"], case["res"]
    grid, animals = hab.reshape(W, W), animals.reshape(W, W)   # [y][x]
    lab = _regions(grid)
    nb = res if W % res == 0 else res + 1
    step = (W - 1) // res
    rows = []
    for h, spec in enumerate(sp.habitats):
        if spec.type in (synth.CLEAR, synth.ROAD):
            continue
        for by in range(nb):
            for bx in range(nb):
                y0, x0 = by * step, bx * step
                ys = slice(y0, y0 + step if (by + 1) * step <= W else W)
                xs = slice(x0, x0 + step if (bx + 1) * step <= W else W)
                block = np.where(grid[ys, xs] == spec.type, lab[ys, xs], -1)
                for r in np.unique(block[block >= 0]):
                    yy, xx = np.nonzero(block == r)
                    rows.append((len(yy), len(yy) * spec.max_pop, animals[ys, xs][yy, xx].sum(), xx.mean() + x0,
                                 yy.mean() + y0, h))
    a = np.asarray(rows, np.float64)
    area, cx, cy, typ = a[:, 0], a[:, 3], a[:, 4], a[:, 5].astype(int)
    lam = sp.lambda_mean
    dist = np.hypot(cx[:, None] - cx[None, :], cy[:, None] - cy[None, :])
    w = (area * lam * np.exp([sp.habitats[t].pref_mean for t in typ]))[None, :] * np.exp(-lam * dist)
    near = dist <= math.log(20.0) / lam
    w[~near] = 0.0
    trans = w / w.sum(1, keepdims=True)
    cross = np.where(near, _crossings(np.stack([cx, cy], 1), road.segments), 0)
    surv = np.exp(-cross[None] * np.asarray(sp.hazard)[:, None, None])
    mmm = np.stack([(trans * s).T for s in surv])
    mmm[mmm <= 1e-5] = 0.0
    pop = a[:, 2]
    iar = 1.0 - np.array([(pop * (trans * s).sum(1)).sum() / pop.sum() for s in surv])
    return dict(area=area, cap=a[:, 1], pop=pop, cx=cx, cy=cy, type=None, N=None, n_transitions=None,
                crossings=None, trans=trans, surv=surv, mmm=mmm, init_pops=pop, caps=a[:, 1], iar=iar)


def exact(case, seed):
    fn = dict(mte=_exact_mte, rov=_exact_rov, adjoint=_exact_adjoint, mlp=_exact_mlp,
              surrogate=_exact_surrogate, species=_exact_species).get(case["kind"])
    return fn(case, seed) if fn else None
