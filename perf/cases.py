"""The work that a user of the integrator has it do, as cases that can be timed and checked.

A case names a call path (``op``), its sizes and its options; :func:`prepare` makes what a program
holds before the call, :func:`run` makes one pass through the public entry points, and
:func:`exact` gives the same outputs in 64 bits from plain torch (phase space, matrix elements,
CTEQ5L, flow and random numbers restated here).  The physics configuration is the library's
default one (13 TeV, pT_hat > 20 GeV, all five processes).
"""
import math

import numpy as np
import torch

import cupythia_b200 as cp

PRODUCTION_ITERATION = 1000     # counter iteration of the production passes
TRAIN_LR = 8e-3
ADAPT_LR = 0.2
RECORD_BYTES = 64


# ------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest adaptations: pilot runs of a few thousand points, where launches, the
        # grid refinement and the threshold's quantile count and the integrand hardly does
        {"name": "integrate_small", "op": "integrate", "n_iter": 5, "n_points": 4099, "bins": 50},
        # an ordinary adaptation (the stage driver's size), an odd number of points
        {"name": "integrate_ordinary", "op": "integrate", "n_iter": 10, "n_points": 1000003, "bins": 50},
        # the benchmark's adaptation: 10 x 2^24 points
        {"name": "integrate_full", "op": "integrate", "n_iter": 10, "n_points": 1 << 24, "bins": 50},
        # a small unweighted sample (the unweighting stage's default size), classic grid
        {"name": "produce_small", "op": "produce", "form": "plain", "n_points": 50021, "bins": 50},
        # the benchmark's production pass: 2^27 points through the trained flow
        {"name": "produce_flow", "op": "produce", "form": "flow", "n_points": 1 << 27, "bins": 50},
        # a sample with its 7-point scale-variation weights, an odd number of points
        {"name": "produce_scale", "op": "produce", "form": "scale", "n_points": 6000011, "bins": 50},
        # records of the flow form into pinned host memory, chunk by chunk (the end-to-end call)
        {"name": "host_flow", "op": "host", "form": "flow", "n_points": 1 << 24, "chunk": 1 << 21, "bins": 50},
        # half of the benchmark's training plan: 100 steps of 65,536 points on the third moment
        {"name": "train", "op": "train", "steps": 100, "batch": 65536, "moment": 3.0, "bins": 50},
        # sensitivities of sigma and Var to alpha_s, the scale factor, the pT cut and every edge
        {"name": "sensitivities", "op": "adjoint", "n_points": 1 << 20, "bins": 50},
        # the benchmark's variance-gradient adaptation of the grid (edge gradients only)
        {"name": "adapt_grid", "op": "adapt", "steps": 12, "n_points": 1 << 22, "moment": 2.0, "bins": 50},
        # records handed to the downstream stages' device event record, with scale variations
        {"name": "hand_off", "op": "hand_off", "n_events": 1000003, "n_var": 7, "bins": 50},
        # the partonic g g -> g g stage at the reference program's size: 2^20 threads x 1000 draws
        {"name": "partonic", "op": "partonic", "rng": "splitmix", "threads": 1 << 20, "draws": 1000},
    ]


def _size(rng, lo, hi, multiple=1):
    """Log-uniform size in [lo, hi], odd half of the time (or a multiple of `multiple`)."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if multiple > 1:
        return max(lo, n // multiple * multiple)
    return min(hi, n | 1 if rng.random() < 0.5 else n)


def draw(rng):
    op = rng.choice(["integrate", "integrate", "produce", "produce", "host", "train", "adjoint", "adapt",
                     "hand_off", "partonic"])
    bins = rng.choice([50, 50, 32, 77, 128])
    if op == "integrate":
        return {"op": op, "n_iter": rng.randint(2, 10), "n_points": _size(rng, 1 << 11, 1 << 24), "bins": bins}
    if op == "produce":
        form = rng.choice(["plain", "flow", "scale"])
        return {"op": op, "form": form, "n_points": _size(rng, 1 << 13, 1 << (23 if form == "scale" else 26)),
                "bins": bins}
    if op == "host":
        return {"op": op, "form": rng.choice(["plain", "flow"]), "n_points": _size(rng, 1 << 17, 1 << 25),
                "chunk": rng.choice([1 << 19, 1 << 20, 1 << 21, 1 << 22]), "bins": bins}
    if op == "train":
        return {"op": op, "steps": rng.choice([5, 10, 20, 50, 100]), "batch": _size(rng, 4096, 65536, 32),
                "moment": rng.choice([2.0, 3.0, 4.0]), "bins": bins}
    if op == "adjoint":
        return {"op": op, "n_points": _size(rng, 1 << 14, 1 << 21), "bins": bins}
    if op == "adapt":
        return {"op": op, "steps": rng.randint(3, 12), "n_points": _size(rng, 1 << 15, 1 << 22),
                "moment": rng.choice([2.0, 4.0]), "bins": bins}
    if op == "hand_off":
        return {"op": op, "n_events": _size(rng, 10000, 2000000), "n_var": rng.choice([1, 7]), "bins": bins}
    if rng.random() < 0.5:
        return {"op": op, "rng": "philox", "threads": _size(rng, 1 << 16, 1 << 28), "draws": 1}
    return {"op": op, "rng": "splitmix", "threads": _size(rng, 1 << 10, 1 << 20), "draws": rng.randint(100, 1000)}


# ------------------------------------------------------------------------------ the program
def _integrator(case, seed):
    return cp.Integrator(seed=1 + int(seed), n_bins=case.get("bins", 50))


def _adapted(case, seed):
    """A handle as a program has it before production: adapted grid, for the flow form gradient
    steps and a flow trained on the third and fourth moment, and the 99.9% threshold.  The flow is
    trained once, with the default key, and then serves samples of any key."""
    it = _integrator(case, seed)
    if case.get("form") == "flow":
        with cp.Integrator(n_bins=case["bins"]) as tr:
            tr.integrate(10, 1 << 20, alpha=1.5, skip=3)
            tr.adjoint_parameter_tangents(False)
            tr.adapt_gradient(12, 1 << 19, lr=ADAPT_LR, iteration0=200)
            tr.flow_init(7)
            for moment in (3.0, 4.0):
                tr.flow_objective(moment)
                tr.flow_train(100, 65536, lr=TRAIN_LR)
            it.grid = tr.grid
            it.flow_init(7)
            it.flow_params = tr.flow_params
        it.flow_enable(True)
    else:
        it.integrate(10, 1 << 20, alpha=1.5, skip=3)
    it.iteration(1 << 22, 300, alpha=0.0)
    return it, it.weight_quantile(0.999)


def _room(case):
    """Records a program keeps room for; a pass leaves the rows beyond its accepted events alone."""
    return int((0.66 if case["form"] == "flow" else 0.3) * case["n_points"]) + 4096


def prepare(case, seed):
    op = case["op"]
    st = {"case": case, "seed": int(seed)}
    if op == "produce":
        st["it"], st["wmax"] = _adapted(case, seed)
        st["records"] = torch.zeros((_room(case), RECORD_BYTES), dtype=torch.uint8, device="cuda")
        if case["form"] == "scale":
            st["ratios"] = torch.zeros((_room(case), 6), dtype=torch.float32, device="cuda")
    elif op == "host":
        st["it"], st["wmax"] = _adapted(case, seed)
        st["records"] = torch.zeros((_room(case), RECORD_BYTES), dtype=torch.uint8).pin_memory()
    elif op in ("train", "adjoint", "adapt"):
        it = st["it"] = _integrator(case, seed)
        it.integrate(10, 1 << 20, alpha=1.5, skip=3)
        st["grid"] = it.grid
    elif op == "hand_off":
        it = st["it"] = _adapted(case, seed)[0]
        n = case["n_events"]
        points = 8 * n + 4096
        room = torch.empty((4 * n + 4096, RECORD_BYTES), dtype=torch.uint8, device="cuda")
        if case["n_var"] > 1:
            rec, ratios, _ = it.unweight_scale_weights(points, iteration=PRODUCTION_ITERATION, records=room)
            st["ratios"] = ratios[:n].clone()
        else:
            rec, _ = it.unweight(points, iteration=PRODUCTION_ITERATION, records=room)
            st["ratios"] = None
        st["records"] = rec[:n].clone()
        st["events"] = it.to_device_events(st["records"], n_var=case["n_var"], scale_ratios=st["ratios"])
    elif op == "integrate":
        st["it"] = _integrator(case, seed)
    else:
        st["it"] = cp.Integrator()
    return st


_INT_STATS = ("n_points", "n_accepted", "n_overweight", "n_bad")


def run(st):
    case, it = st["case"], st["it"]
    op = case["op"]
    if op == "integrate":
        it.reset_grid()
        per, comb = it.integrate(case["n_iter"], case["n_points"], alpha=1.5, skip=case["n_iter"] // 3)
        return {"per_iteration": np.array([[r["sigma"], r["sigma_err"], r["w_max"], r["eta"]] for r in per]),
                "combined": comb, "threshold": it.weight_quantile(0.999), "grid": it.grid}
    if op == "produce" and case["form"] == "scale":
        _, ratios, stats = it.unweight_scale_weights(case["n_points"], iteration=PRODUCTION_ITERATION,
                                                     records=st["records"])
        st["ratios"][:ratios.shape[0]].copy_(ratios)   # the sample's own weight table
        return {"records": st["records"], "ratios": st["ratios"], "stats": stats}
    if op == "produce":
        _, stats = it.unweight(case["n_points"], iteration=PRODUCTION_ITERATION, records=st["records"])
        return {"records": st["records"], "stats": stats}
    if op == "host":
        stats = it.generate_host(case["n_points"], st["records"], iteration=PRODUCTION_ITERATION, chunk=case["chunk"])
        return {"records": st["records"], "stats": stats}
    if op == "train":
        it.flow_init(7)
        it.flow_objective(case["moment"])
        loss = it.flow_train(case["steps"], case["batch"], lr=TRAIN_LR)
        return {"loss": loss, "params": it.flow_params}
    if op == "adjoint":
        g = it.adjoint(case["n_points"], iteration=PRODUCTION_ITERATION)
        return {k: g[k] for k in g if k != "params"}
    if op == "adapt":
        it.grid = st["grid"]
        it.adjoint_parameter_tangents(False)
        it.gradient_objective(case["moment"])
        hist = it.adapt_gradient(case["steps"], case["n_points"], lr=ADAPT_LR, iteration0=200)
        return {"rel_var": np.array([h["rel_var"] for h in hist]), "sigma": np.array([h["sigma"] for h in hist]),
                "lr": np.array([h["lr"] for h in hist]), "grid": it.grid}
    if op == "hand_off":
        return it.to_device_events(st["records"], n_var=case["n_var"], scale_ratios=st["ratios"], events=st["events"])
    if case["rng"] == "philox":
        return it.partonic_integrate(case["threads"], seed=42 + st["seed"])
    return it.partonic_splitmix(case["threads"], case["draws"], seed=0xABCDEF01 + st["seed"])


# ------------------------------------------------------------------------------ what a pass needs
INTEGRAND_OPS = 795 + 72        # FP32 and special-function operations of one point's integrand
FLOW_FLOPS = 35072              # BF16 operations of one point's four couplings
ETA = {"plain": 0.21, "scale": 0.21, "flow": 0.55}   # accepted events per point


def work(case):
    op = case["op"]
    if op == "integrate":
        return {"bytes": 8 * 4 * case["bins"], "flops": case["n_iter"] * case["n_points"] * INTEGRAND_OPS}
    if op in ("produce", "host"):
        n, ev = case["n_points"], ETA[case["form"]] * case["n_points"]
        flops = n * INTEGRAND_OPS
        nbytes = ev * RECORD_BYTES
        if case["form"] == "flow":
            flops += n * FLOW_FLOPS
        if case["form"] == "scale":
            flops += 2 * ev * INTEGRAND_OPS
            nbytes += ev * 24
        return {"bytes": nbytes, "flops": flops}
    if op == "train":
        # forward, backward to the inputs and weight gradients; the integrand with its derivatives
        return {"bytes": 4 * 23072 * 4, "flops": case["steps"] * case["batch"] * (3 * FLOW_FLOPS + 4 * INTEGRAND_OPS)}
    if op == "adjoint":
        return {"bytes": 8 * 6 * case["bins"], "flops": case["n_points"] * 7 * INTEGRAND_OPS}
    if op == "adapt":
        return {"bytes": 8 * 3 * case["bins"], "flops": case["steps"] * case["n_points"] * 4 * INTEGRAND_OPS}
    if op == "hand_off":
        per = RECORD_BYTES + 4 * (5 * 8 + 8 * 4) + 4 + 8 + 3 * 8 + 2 * 4 + 1 + 8 * case["n_var"]
        return {"bytes": case["n_events"] * (per + (24 if case["n_var"] > 1 else 0)), "flops": 0}
    return {"bytes": 64, "flops": 27 * case["threads"] * case["draws"]}


# ------------------------------------------------------------------------------ 64-bit values
# CTEQ5L parametrisation (Lai et al., Eur.Phys.J. C12 (2000) 375): [parametrisation][coefficient][power]
_QMIN = [0., 0., 0., 0., 0., 0., 1.3, 4.5]
_ALPHA = [0.2987216, 0.3407552, 0.4491863, 0.2457668, 0.5293999, 0.3713141, 0.03712017, 0.004952010]
_UT1 = [4.971265, 2.612618, -0.4656819, 3.862583, 0.1895615, 3.753257, 4.400772, 5.562568]
_UT2 = [-1.105128, -1.258304e5, -274.2390, -1.265969, -3.069097, -1.113085, -1.356116, -1.801317]
_AM = [
    [[5.292616, -2.751910, -2.488990], [0.9714424, 0.01011827, -0.01023660], [-16.51006, 7.959721, 8.810563],
     [-16.43394, 5.892854, 9.348874], [30.67422, 4.235796, -0.5112136], [23.52526, -5.305168, -11.69174],
     [-10.95451, 3.006577, 5.638136], [-11.72251, -2.183624, 4.955794], [0.01662533, 0.007622870, -0.0004895887]],
    [[0.9905300, -0.4502235, 0.1624441], [0.8867534, 0.01630829, -0.04049085], [0.8547974, 0.3336301, 0.1371388],
     [0.2941113, -1.527905, 0.2331879], [33.84235, 3.715315, 0.8276930], [6.230115, 3.134639, -1.729099],
     [-1.186928, -0.3282460, 0.1052020], [-8.545702, -6.247947, 3.692561], [0.01724598, 0.007120465, 0.00004003646]],
    [[119.3572, -3.886845, -1.133965], [-94.21449, 3.995885, 1.607363], [4.206383, 0.2485954, 0.2497468],
     [121.0557, -3.015765, -1.423651], [-101.3897, -0.7113478, 0.2621865], [-1.312404, -0.9297691, -0.1562531],
     [1.627137, 0.4954111, -0.6387009], [0.1537698, -0.2487878, 0.8305947], [0.02496448, 0.002457823, 0.0008234276]],
    [[26.47441, 10.59277, -0.9176654], [1.990636, 0.08558918, 0.04248667], [-14.76095, -32.76255, 1.558110],
     [-2.966889, -36.49037, 1.195914], [-100.0519, -2.464635, 0.1964849], [37.18331, 47.00389, -2.772142],
     [-18.72722, -22.91189, 1.089052], [-16.28146, -18.23993, 2.537369], [-1.156300, -0.1280495, 0.05153245]],
    [[-0.6556775, 0.2490190, 0.03966485], [1.305102, -0.1188925, -0.004600870], [-2.371436, 0.3566814, -0.2834683],
     [-6.152826, 0.8339877, -0.7233230], [-8.346558, 2.892168, 0.2137099], [12.79530, 0.1021114, 0.5787439],
     [0.5858816, -1.940375, -0.4029269], [-27.95725, -0.5263392, 1.290229], [0., 0., 0.]],
    [[1.580931, -2.273826, -1.822245], [2.702644, 0.6763243, 0.007231586], [-18.57924, 3.907500, 5.850109],
     [-30.44793, 2.639332, 5.566644], [-4.258011, -5.429244, 0.4418946], [34.65259, -5.532604, -4.904153],
     [-16.58858, 2.923275, 2.266286], [-11.49263, 2.877475, -0.7999105], [0., 0., 0.]],
    [[-0.8293661, -3.982375, -0.06494283], [2.754618, 0.8338636, -0.06885160], [-16.57987, 14.39143, -0.6887240],
     [-28.00703, 15.35966, -0.7377693], [-6.460216, -4.783019, 0.4913297], [31.41830, -31.78031, 7.136013],
     [-18.02509, 18.62163, -4.632843], [-12.40412, 25.65386, -10.66570], [0., 0., 0.]],
    [[-6.031237, 1.992727, -1.076331], [2.933912, 0.5839674, 0.07509435], [-8.284919, 1.488593, -0.8251678],
     [-19.25986, 2.805753, -3.015446], [-9.480483, -0.9767837, -1.165544], [21.93195, -17.88518, 9.460908],
     [-13.27377, 12.01754, -6.277844], [0., 0., 0.], [0., 0., 0.]]]
_SQRT_S, _PT_MIN, _ALPHAS_MZ, _CONV, _N_QUARK_NEW = 13000.0, 20.0, 0.13, 0.389380, 3
_MASK32 = 0xFFFFFFFF


def _philox(points, iteration, stream, seed):
    """Philox-4x32-10 words of int64 point indices: four int64 tensors of 32-bit values."""
    c = [points & _MASK32, (points >> 32) & _MASK32, torch.full_like(points, iteration), torch.full_like(points, stream)]
    k0, k1 = seed & _MASK32, (seed >> 32) & _MASK32
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & _MASK32, (k1 + 0xBB67AE85) & _MASK32
        # the 64-bit products wrap in int64; the masks take their halves
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & _MASK32) ^ c[1] ^ k0, p1 & _MASK32, ((p0 >> 32) & _MASK32) ^ c[3] ^ k1, p0 & _MASK32]
    return c


def _u24(w):
    return (w >> 8).double() * 2.0 ** -24


def _map(words, edges, half=0.0):
    """VEGAS map of the words: x (3 tensors), the Jacobian, the bins; edges [3, nb + 1] double."""
    nb = edges.shape[1] - 1
    x, jac, bins = [], 1.0, []
    for d in range(3):
        m = (words[d] >> 8) * nb
        b, frac = m >> 24, ((m & 0xFFFFFF).double() + half) * 2.0 ** -24
        lo, hi = edges[d][b], edges[d][b + 1]
        x.append(lo + frac * (hi - lo))
        jac = jac * (nb * (hi - lo))
        bins.append(b)
    return x, jac, bins


def _cteq5l(lnx, q2):
    """x f of {d, u, g, ubar, dbar, s, c, b} at ln x and Q^2 (clamped as the parametrisation says)."""
    q2 = q2.clamp(1.0, 1e8)
    lnx = lnx.clamp(math.log(1e-6), -1e-10)
    q, lnq = q2.sqrt(), 0.5 * q2.log()
    x, omx, y = lnx.exp(), -torch.expm1(lnx), -lnx
    u, lny, x1l = lnx + math.log(1e5), y.log(), omx.log()
    f = []
    for i in range(8):
        sb1 = (lnq - math.log(_ALPHA[i])).log() - 1.2
        af = [a[0] + sb1 * (a[1] + sb1 * a[2]) for a in _AM[i]]
        part1 = af[1] * ((1.0 + 0.01 * af[4]) * lny).exp() * (1.0 + af[8] * u)
        part2 = af[0] * omx + af[3] * x
        part3 = x * omx * (af[5] + omx * (af[6] + af[7] * x))
        part4 = _UT1[i] * x1l + af[2] * (x1l if _UT2[i] < -100.0 else (omx + math.exp(_UT2[i])).log())
        ans = x * (part1 + part2 + part3 + part4).exp()
        if _QMIN[i] > 0.0:
            ans = torch.where(q > _QMIN[i], ans * (1.0 - _QMIN[i] / q), torch.zeros_like(ans))
        f.append(ans)
    f = [ans if i == 4 else x * ans for i, ans in enumerate(f)]
    both, ratio = f[3], f[4]
    f[3], f[4] = both / (1.0 + ratio), both * ratio / (1.0 + ratio)
    return [v.clamp_min(0.0) for v in f]


def _alphas(q2, alphas_mz):
    """First-order running coupling with thresholds at 1.5, 4.8 and 171 GeV."""
    l5 = 91.188 * torch.exp(-6.0 * math.pi / (23.0 * alphas_mz))
    l6 = l5 * (l5 / 171.0) ** (2.0 / 21.0)
    l4 = l5 * (4.8 / l5) ** (2.0 / 25.0)
    l3 = l4 * (1.5 / l4) ** (2.0 / 27.0)
    q2 = torch.maximum(q2, torch.full_like(q2, (1.07 * float(l3)) ** 2))
    b0 = torch.where(q2 > 171.0 ** 2, 21.0, torch.where(q2 > 4.8 ** 2, 23.0, torch.where(q2 > 1.5 ** 2, 25.0, 27.0)))
    lam = torch.where(q2 > 171.0 ** 2, l6, torch.where(q2 > 4.8 ** 2, l5, torch.where(q2 > 1.5 ** 2, l4, l3)))
    return 12.0 * math.pi / (b0 * (q2.log() - 2.0 * lam.log()))


def _channels(tp, up, a, b):
    """Sum over the five processes and their pairs of bracket x f_a f_b, at t/s and u/s."""
    rt, ru = 1.0 / tp, 1.0 / up
    tu, ut = tp * ru, up * rt
    square = lambda v: v * v  # noqa: E731
    gg2gg = 1.125 * (square(tp + 1) + square(rt + 1) + square(up + 1) + square(ru + 1) + square(tu + 1)
                     + square(ut + 1) + 3.0)
    gg2qq = _N_QUARK_NEW * ((ut + tu) / 6.0 - 0.375 * (up * up + tp * tp))
    qg2qg = (up * up + 1.0) * rt * rt - (4.0 / 9.0) * (up + ru)
    qq2gg = 0.5 * ((32.0 / 27.0) * (ut + tu) - (8.0 / 3.0) * (up * up + tp * tp))
    t_, u_ = (4.0 / 9.0) * (1.0 + up * up) * rt * rt, (4.0 / 9.0) * (1.0 + tp * tp) * ru * ru
    tu_, st_ = -(8.0 / 27.0) * rt * ru, -(8.0 / 27.0) * up * up * rt
    qa = a[0] + a[1] + a[3] + a[4] + 2.0 * (a[5] + a[6] + a[7])
    qb = b[0] + b[1] + b[3] + b[4] + 2.0 * (b[5] + b[6] + b[7])
    sea = 2.0 * (a[5] * b[5] + a[6] * b[6] + a[7] * b[7])
    same = a[0] * b[0] + a[1] * b[1] + a[3] * b[3] + a[4] * b[4] + sea
    opposite = a[0] * b[4] + a[4] * b[0] + a[1] * b[3] + a[3] * b[1] + sea
    return (a[2] * b[2] * (gg2gg + gg2qq) + qg2qg * (qa * b[2] + a[2] * qb) + qa * qb * t_
            + same * 0.5 * (u_ + tu_ - t_) + opposite * (st_ + qq2gg))


def _theta(device="cuda"):
    """alpha_s(mZ), the renormalisation-scale factor and the pT cut as 0-dim tensors."""
    return [torch.tensor(v, dtype=torch.float64, device=device) for v in (_ALPHAS_MZ, 1.0, _PT_MIN)]


def _weight(x, theta=None, scales=False):
    """f J_base (mb) at x in [0, 1]^3; with `scales` the six scale-variation ratios instead."""
    alphas_mz, k_ren, pt_min = theta if theta is not None else _theta(x[0].device)
    s = _SQRT_S ** 2
    ln_tau_min = (4.0 * pt_min * pt_min / s).log()
    ln_tau = (1.0 - x[0]) * ln_tau_min
    tau = ln_tau.exp()
    a0 = x[0] * ln_tau_min
    r, z_max = a0.exp(), (-torch.expm1(a0)).clamp_min(1e-300).sqrt()   # 0 at x0 = 0, with a finite slope
    omz_max = r / (1.0 + z_max)
    omz, opz = omz_max + 2.0 * z_max * (1.0 - x[2]), omz_max + 2.0 * z_max * x[2]
    tp, up = -0.5 * omz, -0.5 * opz
    pt2 = 0.25 * tau * s * omz * opz
    lnx1, lnx2 = ln_tau * (1.0 - x[1]), ln_tau * x[1]
    alpha = _alphas(k_ren * pt2, alphas_mz)
    b = _channels(tp, up, _cteq5l(lnx1, pt2), _cteq5l(lnx2, pt2))
    if scales:
        ren = [(_alphas(k * pt2, alphas_mz) / alpha) ** 2 for k in (4.0, 0.25)]
        fac = [_channels(tp, up, _cteq5l(lnx1, k * pt2), _cteq5l(lnx2, k * pt2)) / b for k in (4.0, 0.25)]
        return torch.stack(ren + fac + [ren[0] * fac[0], ren[1] * fac[1]], 1)
    k0 = 2.0 * math.pi * _CONV * (-ln_tau_min) / s
    return k0 * alpha * alpha * b * (-0.5 * ln_tau) * z_max / tau


_COUPLINGS = (((0,), (1, 2)), ((1, 2), (0,)), ((1,), (0, 2)), ((0, 2), (1,)))   # condition, transform
_PER = 5768


def _flow(x, jac, params):
    """The flow after the VEGAS map: v (3 tensors) and the total Jacobian."""
    x = [v.clamp(2.0 ** -24, 1.0 - 2.0 ** -24) for v in x]
    ld = jac.log() - sum(v.log() + torch.log1p(-v) for v in x)
    z = [v.log() - torch.log1p(-v) for v in x]
    for c, (cond, move) in enumerate(_COUPLINGS):
        q = params[c * _PER:(c + 1) * _PER]
        w1, b1 = q[:1024].view(16, 64)[:len(cond)], q[1024:1088]
        w2, b2, w3, b3 = q[1088:5184].view(64, 64), q[5184:5248], q[5248:5760].view(64, 8), q[5760:5768]
        h = torch.relu(torch.stack([z[d] for d in cond], 1) @ w1 + b1)
        h = torch.relu(h @ w2 + b2)
        o = h @ w3 + b3
        for j, d in enumerate(move):
            scale = 4.0 * torch.tanh(o[:, j] / 4.0)
            z[d] = z[d] * scale.exp() + o[:, len(move) + j]
            ld = ld + scale
    ld = ld + sum(torch.nn.functional.logsigmoid(v) + torch.nn.functional.logsigmoid(-v) for v in z)
    return [torch.sigmoid(v) for v in z], ld.exp()


def _points(lo, hi):
    return torch.arange(lo, hi, dtype=torch.int64, device="cuda")


def _chunks(n, size=1 << 21):
    return [(lo, min(n, lo + size)) for lo in range(0, n, size)]


def _edges(grid):
    return torch.as_tensor(np.asarray(grid), dtype=torch.float64, device="cuda")


def _refine(edges, hist, alpha=1.5):
    """Classic refinement of one dimension (numpy, doubles)."""
    nb = len(hist)
    sm = np.empty(nb)
    sm[0], sm[-1] = (hist[0] + hist[1]) / 2, (hist[-2] + hist[-1]) / 2
    sm[1:-1] = (hist[:-2] + hist[1:-1] + hist[2:]) / 3
    d = sm / sm.sum()
    inner = (d > 0) & (d < 1)
    r = np.where(d >= 1, 1.0, 0.0)
    r[inner] = ((d[inner] - 1) / np.log(d[inner])) ** alpha
    cum = np.concatenate([[0.0], np.cumsum(r)])
    new = np.interp(np.arange(1, nb) * (cum[-1] / nb), cum, edges)
    return np.concatenate([edges[:1], new, edges[-1:]])


def _result(s1, s2, wmax, n):
    mean = s1 / n
    err = math.sqrt(max((s2 / n - mean * mean) / (n - 1), 0.0))
    return {"sigma": mean, "sigma_err": err, "sum_w": s1, "sum_w2": s2, "w_max": wmax, "n_points": None,
            "n_bad": None, "eta": mean / wmax}


def _exact_integrate(case, seed):
    nb, n, key = case["bins"], case["n_points"], 1 + int(seed)
    grid = np.tile(np.arange(nb + 1) / nb, (3, 1))
    per = []
    for it in range(case["n_iter"]):
        e = _edges(grid)
        s1 = s2 = wmax = 0.0
        hist = torch.zeros((3, nb), dtype=torch.float64, device="cuda")
        qhist = torch.zeros(4096, dtype=torch.int64, device="cuda")
        for lo, hi in _chunks(n):
            x, jac, bins = _map(_philox(_points(lo, hi), it, 0, key), e)
            w = _weight(x) * jac
            s1, s2, wmax = s1 + float(w.sum()), s2 + float((w * w).sum()), max(wmax, float(w.max()))
            for d in range(3):
                hist[d] += torch.bincount(bins[d], weights=w * w, minlength=nb)
            # weight histogram: the top 14 bits of the single-precision weight, from 2^-64
            q = (w[w > 0].float().view(torch.int32) >> 18) - ((127 - 64) << 5)
            qhist += torch.bincount(q.clamp(0, 4095), minlength=4096)
        per.append(_result(s1, s2, wmax, n))
        grid = np.stack([_refine(grid[d], hist[d].cpu().numpy()) for d in range(3)])
    kept = per[case["n_iter"] // 3:]
    w2 = sum(1.0 / r["sigma_err"] ** 2 for r in kept)
    comb = _result(sum(r["sum_w"] for r in kept), sum(r["sum_w2"] for r in kept), max(r["w_max"] for r in kept),
                   n * len(kept))
    comb["sigma"] = sum(r["sigma"] / r["sigma_err"] ** 2 for r in kept) / w2
    comb["sigma_err"] = 1.0 / math.sqrt(w2)
    comb["eta"] = comb["sigma"] / comb["w_max"]
    q = qhist.cpu().numpy()
    above = np.cumsum(q[::-1])[::-1]                       # points in this bin or above
    b = int(np.nonzero(above > (1.0 - 0.999) * q.sum())[0][-1])
    threshold = float(np.array((b + 1 + ((127 - 64) << 5)) << 18, np.uint32).view(np.float32))
    return {"per_iteration": np.array([[r["sigma"], r["sigma_err"], r["w_max"], r["eta"]] for r in per]),
            "combined": comb, "threshold": threshold, "grid": grid}


def _exact_produce(case, seed):
    st = prepare(dict(case, n_points=2) if case["op"] == "produce" else case, seed)   # the plan: grid, flow, threshold
    it, wmax, n, key = st["it"], st["wmax"], case["n_points"], 1 + int(seed)
    e = _edges(it.grid)
    params = torch.as_tensor(it.flow_params, device="cuda").double() if case["form"] == "flow" else None
    s1 = s2 = se = seen = 0.0
    acc, ratios = 0, []
    for lo, hi in _chunks(n, 1 << 20):
        words = _philox(_points(lo, hi), PRODUCTION_ITERATION, 0, key)
        x, jac, _ = _map(words, e, 0.5 if params is not None else 0.0)
        if params is not None:
            x, jac = _flow(x, jac, params)
        w = _weight(x) * jac
        keep = _u24(words[3]) * wmax < w
        s1, s2, seen = s1 + float(w.sum()), s2 + float((w * w).sum()), max(seen, float(w.max()))
        se += float((w[keep] / wmax).clamp_min(1.0).sum())
        acc += int(keep.sum())
        if case["form"] == "scale":
            ratios.append(_weight([v[keep] for v in x], scales=True))
    r = _result(s1, s2, seen, n)
    stats = {"sigma": r["sigma"], "sigma_err": r["sigma_err"], "sigma_unweighted": wmax * se / n, "w_max": wmax,
             "w_max_seen": seen, "eta": acc / n, **{k: None for k in _INT_STATS}}
    out = {"records": None, "stats": stats}
    if ratios:
        out["ratios"] = torch.cat(ratios + [ratios[0].new_zeros((_room(case) - acc, 6))])
    return out


def _exact_train(case, seed):
    # two trainings that differ by a rounding part after some tens of Adam steps: longer runs have
    # no 64-bit value, and the parameters have none at all (Adam's first steps follow the sign of
    # gradients that the kernels form from BF16 activations)
    if case["steps"] > 20:
        return None
    st = prepare(case, seed)
    it, key, n, p = st["it"], 1 + int(seed), case["batch"], case["moment"]
    it.flow_init(7)
    theta = torch.as_tensor(it.flow_params, device="cuda").double()
    e, used = _edges(st["grid"]), torch.zeros(4 * _PER, dtype=torch.bool, device="cuda")
    for c, (cond, move) in enumerate(_COUPLINGS):
        q = used[c * _PER:(c + 1) * _PER]
        q[:64 * len(cond)] = True
        q[1024:5248] = True
        q[5248:5760].view(64, 8)[:, :2 * len(move)] = True
        q[5760:5760 + 2 * len(move)] = True
    m, v, losses = torch.zeros_like(theta), torch.zeros_like(theta), []
    for step in range(case["steps"]):
        x, jac, _ = _map(_philox(_points(0, n), step, 2, key), e, 0.5)
        theta.requires_grad_(True)
        y, j = _flow(x, jac, theta)
        w = _weight(y) * j
        losses.append(float((w * w).mean() / w.mean() ** 2))
        # the pathwise gradient of <w^p> at fixed <w> scale, as the training objective is defined
        loss = (w / w.mean().detach()).pow(p).mean()
        g, = torch.autograd.grad(loss, theta)
        with torch.no_grad():
            g = torch.where(used, g, torch.zeros_like(g))
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            theta = theta.detach() - TRAIN_LR * (m / (1 - 0.9 ** (step + 1))) / (
                (v / (1 - 0.999 ** (step + 1))).sqrt() + 1e-8)
            theta = torch.where(used, theta, torch.zeros_like(theta))
    return {"loss": np.array(losses), "params": None}


def _gradients(grid, n, iteration, key, p=2.0):
    """sums w, w^p and their gradients with respect to (edges, theta) over points [0, n)."""
    e, theta = _edges(grid).requires_grad_(True), [t.requires_grad_(True) for t in _theta()]
    tot = [0.0, 0.0]
    grads = [None, None]
    for lo, hi in _chunks(n, 1 << 19):
        x, jac, _ = _map(_philox(_points(lo, hi), iteration, 0, key), e)
        w = _weight(x, theta) * jac
        for k, s in enumerate((w.sum(), w.pow(p).sum())):
            g = torch.autograd.grad(s, [e] + theta, retain_graph=k == 0)
            tot[k] += float(s.detach())
            grads[k] = list(g) if grads[k] is None else [a + b for a, b in zip(grads[k], g)]
    return tot, [[g.cpu().numpy() for g in v] for v in grads]


def _exact_adjoint(case, seed):
    n = case["n_points"]
    (s1, s2), (g1, g2) = _gradients(prepare(case, seed)["grid"], n, PRODUCTION_ITERATION, 1 + int(seed))
    mean = s1 / n
    dvar = [b / n - 2.0 * mean * a / n for a, b in zip(g1, g2)]
    return {"sigma": mean, "var": s2 / n - mean * mean, "n_bad": None, "dsigma": [float(g) / n for g in g1[1:]],
            "dvar": [float(g) for g in dvar[1:]], "dsigma_dedges": g1[0] / n, "dvar_dedges": dvar[0]}


def _exact_adapt(case, seed):
    n, p, grid, key = case["n_points"], case["moment"], prepare(case, seed)["grid"], 1 + int(seed)
    nb, lr, prev, hist = case["bins"], ADAPT_LR, None, []
    for step in range(case["steps"]):
        (s1, sp), (g1, gp) = _gradients(grid, n, 200 + step, key, p)
        mean, mp = s1 / n, sp / n
        rel = mp / mean ** p - 1.0
        # the variance for p = 2, otherwise the relative p-th moment (up to a factor)
        gv = gp[0] / n - (2.0 * mean if p == 2.0 else p * mp / mean) * g1[0] / n
        new = []
        for d in range(3):
            width = np.diff(grid[d])
            tail = np.concatenate([np.cumsum(gv[d][1:nb][::-1])[::-1], [0.0]])
            g = width * tail
            width = width * np.exp(-lr * g / np.abs(g).max())
            inner = np.cumsum(width / width.sum())[:-1]
            new.append(np.concatenate([[0.0], inner, [1.0]]))
        grid = np.stack(new)
        if prev is not None and rel > prev:
            lr *= 0.5
        prev = rel
        hist.append((rel, mean, lr))
    rel, sigma, lrs = (np.array(v) for v in zip(*hist))
    return {"rel_var": rel, "sigma": sigma, "lr": lrs, "grid": grid}


def _exact_hand_off(case, seed):
    st = prepare(case, seed)
    rec = cp.events_view(st["records"])
    n = len(rec)
    out = {k: None for k in st["events"]}
    zero, pin = np.zeros(n), rec["pz_in"].astype(np.float64)
    p3, p4 = rec["p3"].astype(np.float64), rec["p4"].astype(np.float64)
    out["px"] = np.stack([zero, zero, p3[:, 0], p4[:, 0]], 1).reshape(-1)
    out["py"] = np.stack([zero, zero, p3[:, 1], p4[:, 1]], 1).reshape(-1)
    out["pz"] = np.stack([pin[:, 0], pin[:, 1], p3[:, 2], p4[:, 2]], 1).reshape(-1)
    out["e"] = np.stack([np.abs(pin[:, 0]), np.abs(pin[:, 1]), p3[:, 3], p4[:, 3]], 1).reshape(-1)
    out["m"] = np.zeros(4 * n)
    out["scale"] = rec["pt_hat"].astype(np.float64)
    out["x1"], out["x2"] = np.abs(pin[:, 0]) * 2 / _SQRT_S, np.abs(pin[:, 1]) * 2 / _SQRT_S
    weight = rec["weight"].astype(np.float64)[:, None]
    if st["ratios"] is not None:
        weight = weight * np.concatenate([np.ones((n, 1)), st["ratios"].cpu().numpy().astype(np.float64)], 1)
    out["weight"] = weight.reshape(-1)
    return out


def _splitmix(z):
    """SplitMix64 of int64 counters; int64 products wrap, logical shifts by mask."""
    z = z + (0x9E3779B97F4A7C15 - (1 << 64))
    z = (z ^ ((z >> 30) & ((1 << 34) - 1))) * (0xBF58476D1CE4E5B9 - (1 << 64))
    z = (z ^ ((z >> 27) & ((1 << 37) - 1))) * (0x94D049BB133111EB - (1 << 64))
    return z ^ ((z >> 31) & ((1 << 33) - 1))


def _exact_partonic(case, seed):
    shat, cmax, conv = 100.0 ** 2, 0.9, 0.3893793721
    n = case["threads"] * case["draws"]
    alphas = 0.13 if case["rng"] == "philox" else 0.118
    s1 = s2 = wmax = 0.0
    for lo, hi in _chunks(n, 1 << 24):
        i = _points(lo, hi)
        if case["rng"] == "philox":
            w = _philox(i, 0, 0, 42 + int(seed))
            u = ((w[1] << 21) | (w[0] >> 11)).double() * 2.0 ** -53
        else:
            k = i % case["draws"]
            z = _splitmix((0xABCDEF01 + int(seed)) + (i // case["draws"]) * 0x100000001B3 + k)
            u = ((z >> 11) & ((1 << 53) - 1)).double() * 2.0 ** -53
        c = (2.0 * u - 1.0) * cmax
        t = -0.5 * shat * (1.0 - c)
        v = -shat - t
        me = 4.5 * (3.0 - t * v / shat ** 2 - shat * v / t ** 2 - shat * t / v ** 2)
        w = math.pi / shat ** 2 * alphas ** 2 * 0.5 * me * (2.0 * cmax) * (shat / 2.0) * conv
        s1, s2, wmax = s1 + float(w.sum()), s2 + float((w * w).sum()), max(wmax, float(w.max()))
    return _result(s1, s2, wmax, n)


def exact(case, seed):
    op = case["op"]
    if op == "integrate":
        return _exact_integrate(case, seed)
    if op in ("produce", "host"):
        return _exact_produce(case, seed)
    if op == "train":
        return _exact_train(case, seed)
    if op == "adjoint":
        return _exact_adjoint(case, seed)
    if op == "adapt":
        return _exact_adapt(case, seed)
    return _exact_hand_off(case, seed) if op == "hand_off" else _exact_partonic(case, seed)
