"""Cases of the library's public entry points, as a program that computes spectral functions and
conductivities calls them: scGD0 self-consistency, the ladder solves, the training of the warm start's
network.

Two models, both of `epspectral_gb300.synthetic`: the 1D Holstein chain of the tests and examples, and the
3-band cubic t2g model on N^3 k points (15 modes in [10, 80] meV, log-normal g2) of the benchmark. A case
names its family (one of FAMILIES) and that family's sizes; `prepare` makes the model from the seed and
sets up the plans a program keeps between runs, `run` makes one pass.

Outputs have the precision of the path that makes them: Σ, μ and σ in FP64 on the FP64 paths; on the
tensor-core paths, whose products and vertices are FP32, Σ as complex64 and μ and σ as float32 (the
library's arrays hold them in FP64). On those paths Σ stays on the device, where a torch program goes on
with it.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "epspectral.jl_gb300"))

from epspectral_gb300 import FrequencyGrid, api, graded_frequency_grid, synthetic, warmstart  # noqa: E402

K_B = 8.617333262e-5  # eV per K
ETA_INIT = 0.01
OMEGA_AC = 1e-4

# Each family's sizes: (smallest, largest) of what is drawn over the logarithm, or a tuple of choices.
#   N        k points per axis (t2g) or in all (chain)       dw       finest grid step in eV
#   modes    phonon modes      temps  temperatures in one run      omegas   probe frequencies
#   rtol     GMRES tolerance   rows   training rows               batch    right-hand sides together
FAMILIES = {
    # the chain through the default (direct FP64) path: the smallest model users start with
    "chain": dict(N=(16, 96), dw=(0.01, 0.04), temps=(1, 2), path=("direct_fp64",)),
    "chain_ladder": dict(N=(8, 48), dw=(0.02, 0.04), omegas=(1, 3), path=("direct_fp64",)),
    # the t2g model in FP64, dispersionless modes: reference-quality runs of medium models
    "scgd0_fp64": dict(N=(5, 12), dw=(0.002, 0.01), modes=(4, 15), temps=(1, 2), path=("gemm_fp64",)),
    "ladder_fp64": dict(N=(4, 8), dw=(0.005, 0.01), modes=(4, 15), omegas=(1, 2), path=("gemm_fp64",)),
    # dispersive modes: term by term, in FP64 and on the tensor-core plan
    "disp_fp64": dict(N=(3, 5), dw=(0.01, 0.04), modes=(3, 8), temps=(1, 1), path=("direct_fp64",)),
    "disp": dict(N=(4, 8), dw=(0.004, 0.02), modes=(4, 15), temps=(1, 2), path=("gemm_bf16",)),
    # the tensor-core path: one temperature, and a temperature scan in one run
    "scgd0": dict(N=(5, 16), dw=(0.002, 0.01), modes=(4, 15), temps=(1, 1), path=("gemm_bf16",)),
    "scan": dict(N=(5, 12), dw=(0.003, 0.01), modes=(4, 15), temps=(3, 8), path=("gemm_bf16",)),
    # σ(Ω) from a host Σ, the Ωs one after the other, and all (T, Ω) pairs together
    "ladder": dict(N=(5, 14), dw=(0.003, 0.01), modes=(4, 15), omegas=(1, 4), path=("gemm_tf32", "gemm_bf16")),
    "ladder_batch": dict(N=(4, 10), dw=(0.004, 0.01), modes=(4, 15), omegas=(4, 16), temps=(1, 3), batch=(8, 32),
                         path=("gemm_tf32", "gemm_bf16")),
    # the whole step: scGD0 to tol, then σ(Ω) from the Σ left on the device
    "step": dict(N=(6, 16), dw=(0.002, 0.01), modes=(4, 15), path=("gemm_tf32", "gemm_bf16")),
    # training of the warm start's network (forward, backward, Adam)
    "train": dict(nw=(101, 1251), rows=(500, 6000), width=(64, 128, 256)),
}


def listed():
    return [
        # the tests' chain: 33 outer states, 401 nodes
        dict(name="chain", family="chain", N=64, dw=0.02, temps=1, path="direct_fp64", filling=0.85),
        # the chain's σ(Ω) through the default path, as the examples compute it
        dict(name="chain_ladder", family="chain_ladder", N=16, dw=0.02, omegas=2, path="direct_fp64"),
        # a converged FP64 reference run of a medium model
        dict(name="scgd0_fp64", family="scgd0_fp64", N=8, dw=0.005, modes=15, temps=1, path="gemm_fp64"),
        # an FP64 σ(Ω) to check a mixed-precision one against
        dict(name="ladder_fp64", family="ladder_fp64", N=6, dw=0.008, modes=15, omegas=1, path="gemm_fp64"),
        # dispersive modes, an odd k grid: the FP64 parity run of a small model, and the production run
        dict(name="disp_fp64", family="disp_fp64", N=5, dw=0.02, modes=5, temps=1, path="direct_fp64"),
        dict(name="disp", family="disp", N=8, dw=0.005, modes=15, temps=1, path="gemm_bf16"),
        # the GPU tests' medium model (105 outer states), and the benchmark's temperature scan on a ragged one
        dict(name="scgd0", family="scgd0", N=8, dw=0.005, modes=15, temps=1, path="gemm_bf16"),
        dict(name="scan", family="scan", N=11, dw=0.004, modes=13, temps=8, path="gemm_bf16"),
        # a few σ(Ω) of a medium model in BF16x3, and a (T, Ω) map as simultaneous right-hand sides
        dict(name="ladder", family="ladder", N=9, dw=0.004, modes=15, omegas=3, path="gemm_bf16"),
        dict(name="ladder_batch", family="ladder_batch", N=8, dw=0.005, modes=15, omegas=8, temps=2, batch=16,
             path="gemm_tf32"),
        # the benchmark's step: 495 outer states, 1251 nodes
        dict(name="step", family="step", N=16, dw=0.002, modes=15, path="gemm_tf32"),
        # two epochs over a few runs' rows of the benchmark's network
        dict(name="train", family="train", nw=1251, rows=4096, width=256),
    ]


def draw(rng):
    family = rng.choice(sorted(FAMILIES))
    case = dict(family=family)
    for key, lim in FAMILIES[family].items():
        if isinstance(lim[0], str) or len(lim) != 2:
            case[key] = rng.choice(lim)
        elif isinstance(lim[0], int):
            case[key] = min(lim[1], int(math.exp(rng.uniform(math.log(lim[0]), math.log(lim[1] + 1)))))
        else:
            case[key] = round(math.exp(rng.uniform(math.log(lim[0]), math.log(lim[1]))), 4)
    if family not in ("train", "chain_ladder"):
        case["filling"] = round(rng.uniform(0.7, 1.3), 3)
    return case


# ---- inputs ----


def _chain(case):
    return case["family"].startswith("chain")


def _temperatures(case):
    n = case.get("temps", 1)
    if _chain(case):
        return [0.1 * (1 + k) for k in range(n)]
    if case["family"] == "ladder_batch":
        return [(300 + 100 * k) * K_B for k in range(n)]
    return [300 * K_B] if n == 1 else [(100 + 700 * k / (n - 1)) * K_B for k in range(n)]


def _probe_frequencies(case):
    n = case.get("omegas", 1)
    return [0.1] if n == 1 else [0.5 * k / n for k in range(n)]


def _model(case, seed):
    rng = np.random.default_rng(seed)
    dw = case["dw"]
    if _chain(case):
        n = int(round(4.0 / dw))
        return synthetic.holstein_1d_setup(case["N"], 1.0, rng.uniform(0.16, 0.24), rng.uniform(0.15, 0.25),
                                           FrequencyGrid.from_nodes(np.arange(-n, n + 1) * dw))
    ws = graded_frequency_grid([(-0.5, 0.5, dw), (-3.0, 3.0, 5 * dw), (-8.0, 8.0, 20 * dw)])
    s = synthetic.cubic_t2g_setup(N=case["N"], nmodes=case["modes"], ws=ws, seed=seed, g2_chunk=768,
                                  g2_dtype=np.float64 if case["path"].endswith("fp64") else np.float32)
    return synthetic.with_dispersion(s, case["N"], 0.2) if case["family"].startswith("disp") else s


def _occupation(case, Ts):
    return dict(Tlist=Ts, nlist=[0.0] * len(Ts), nelec=case.get("filling", 1.0), spin_degeneracy=2.0, type="metal")


def _mu_start(case, s, Ts):
    return [0.0 if _chain(case) else synthetic.bare_mu(s, T, case.get("filling", 1.0)) for T in Ts]


def _self_energy(s, nT, seed):
    """A causal Σ [nω, ni, nT] of broad poles over the band per state, of the size that scGD0 leaves for the model's
    coupling (15 modes: |Im Σ| of about 0.2 eV in the bands, rising with the temperature)."""
    rng = np.random.default_rng([seed, 7])
    w, ni, nm = _nodes(s["omegas"]), len(s["eps_i"]), s["g2"].shape[0]
    half, size = (2.4, 0.04) if nm == 1 else (1.6, 0.03 * nm / 15)
    S = np.zeros((len(w), ni, nT), dtype=np.complex128, order="F")
    for x in np.linspace(-half, half, 8):
        pole = 1.0 / (w - x - rng.uniform(-0.1, 0.1) + 1j * rng.uniform(0.25, 0.4))
        S += pole[:, None, None] * (size * rng.uniform(0.7, 1.3, size=(ni, 1)) * (1 + 0.5 * np.arange(nT)))[None]
    return S


def _training_set(case, seed):
    rng = np.random.default_rng(seed)
    d = 2 * case["nw"] + 4
    X = rng.standard_normal((case["rows"], d), dtype=np.float32)
    mix = rng.standard_normal((d, 8), dtype=np.float32) / np.float32(math.sqrt(d))
    Y = np.tanh(X @ mix) @ rng.standard_normal((8, d - 4), dtype=np.float32)
    return X, Y.astype(np.float32), [d] + [case["width"]] * 3 + [d - 4]


def _first_parameters(dims, seed):
    return warmstart.init_params(dims, seed % 1000)


def _row_orders(case):
    return np.stack([np.random.default_rng(e).permutation(case["rows"]) for e in range(2)])


def prepare(case, seed):
    family = case["family"]
    if family == "train":
        X, Y, dims = _training_set(case, seed)
        net = warmstart.Network(dims)
        return dict(case=case, X=X, Y=Y, net=net, p0=_first_parameters(dims, seed), perm=_row_orders(case))
    s = _model(case, seed)
    Ts = _temperatures(case)
    st = dict(case=case, Ts=Ts, occ=_occupation(case, Ts), mu0=_mu_start(case, s, Ts), Om=_probe_frequencies(case))
    if family in ("chain_ladder", "ladder_fp64", "ladder", "ladder_batch"):
        st["sigma"] = _self_energy(s, len(Ts), seed)
    else:
        path = "gemm_bf16" if family == "step" else case["path"]
        st["scgd0"] = api.Scgd0Plan(s, path=path, omega_acoustic=OMEGA_AC)
    if family == "step" or "sigma" in st:
        st["ladder"] = api.LadderPlan(s, path=case["path"], omega_acoustic=OMEGA_AC)
    return st


class _DeviceArray:
    """A DeviceSigma as an array that torch takes over without a copy."""

    def __init__(self, sigma):
        nw, ni, nT = sigma.shape
        self.__cuda_array_interface__ = dict(shape=(nT, ni, nw), typestr="<c16", data=(sigma.address, False), version=3)


def run(state):
    case = state["case"]
    family = case["family"]
    if family == "train":
        state["net"].set_params(state["p0"])
        hist = state["net"].train(state["X"], state["Y"], epochs=2, batch=256, lr=1e-4, perm=state["perm"])
        return dict(params=state["net"].get_params(), loss=np.float32(hist))
    out = {}
    sigma, mu = state.get("sigma"), state["mu0"]
    if "scgd0" in state:
        fp64 = case["path"].endswith("fp64")
        r = state["scgd0"].run(state["occ"], eta_init=ETA_INIT if not _chain(case) else 0.05, tol=1e-6, maxiter=50,
                               mu_start=state["mu0"], sigma_to_host=fp64)
        sigma, mu = r["sigma"], r["mu"]
        out["mu"] = mu if fp64 else np.float32(mu)
        out["converged"] = r["converged"]
        if fp64:
            out["sigma"] = sigma
        elif family != "step":
            out["sigma"] = torch.as_tensor(_DeviceArray(sigma), device="cuda").to(torch.complex64)
            torch.cuda.current_stream().synchronize()  # the plan's next run writes Σ on the library's own stream
    if "ladder" in state:
        r = state["ladder"].run(sigma, mu, state["Ts"], state["Om"], rtol=1e-2, maxiter=30, batch_rhs=case.get("batch"))
        kind = np.float64 if case["path"].endswith("fp64") else np.float32
        out["sigma_bubble"] = kind(r["sigma_bubble"])
        out["sigma_ladder"] = kind(r["sigma_ladder"])
        out["solved"] = r["converged"]
    return out


# ---- what a pass cannot do without ----


def _sizes(case):
    if _chain(case):
        n, N = 2 * int(round(4.0 / case["dw"])) + 1, case["N"]
        return n, n, N // 2 + 1, N, 1
    dw, N = case["dw"], case["N"]
    h = N // 2 + 1
    ni = 3 * (h * (h + 1) * (h + 2) // 6)
    return int(1.0 / dw) + int(5.0 / (5 * dw)) + int(10.0 / (20 * dw)) + 1, int(16.0 / dw) + 1, ni, 3 * N ** 3, case["modes"]


def work(case):
    """The sums of a pass in their cheapest form: a dispersionless Fan-Migdal sum as nω ni nm columns, a dispersive
    one as its terms (30 operations each), ten iterations to tol; one operator application per solve; the network's
    products forward and back."""
    if case["family"] == "train":
        d = 2 * case["nw"] + 4
        p = d * case["width"] + 2 * case["width"] ** 2 + case["width"] * (d - 4)
        return {"bytes": 4.0 * (2 * case["rows"] * (2 * d - 4) + 2 * p), "flops": 2.0 * 6 * p * case["rows"]}
    nw, nwa, ni, nf, nm = _sizes(case)
    nT, nO = case.get("temps", 1), case.get("omegas", 1)
    flops, size = 0.0, 0.0
    if "ladder" not in case["family"]:
        terms = nw * ni * nm * (nf * 30.0 if case["family"].startswith("disp") else ni * 2.0)
        flops += 10 * nT * (terms + 2.0 * nw * nw * ni + 10.0 * nwa * ni)
        size += 16.0 * nw * ni * nT + 4.0 * nm * ni * (nf if case["family"].startswith("disp") else ni) + 8.0 * nw * nw
    if "ladder" in case["family"] or case["family"] == "step":
        pair = 2.0 * 16 * nw * (3 * ni) ** 2 * nm + 2.0 * nw * nw * 24 * ni
        flops += nT * nO * pair
        size += 16.0 * nw * ni * nT + 4.0 * nm * 9 * ni * ni + 8.0 * nw * nw
    return {"bytes": size, "flops": flops}


# ---- the same in 64 bits, in plain torch and numpy ----


def _nodes(g):
    return g.origin + np.asarray(g.offsets, dtype=np.float64) * g.unit


def _gpu(x):
    return torch.as_tensor(np.ascontiguousarray(x), device="cuda")


def _fermi(x, T):
    return 1.0 / (torch.exp(torch.clamp(x / T, max=700.0)) + 1.0)


def _trapezoid(w):
    W = np.zeros(len(w))
    W[:-1] += 0.5 * np.diff(w)
    W[1:] += 0.5 * np.diff(w)
    return W


def _hilbert(w):
    """ReΣ = H ImΣ: the principal value of ImΣ's hat functions on w, padded by one spacing at either end."""
    x = np.concatenate([[2 * w[0] - w[1]], w, [2 * w[-1] - w[-2]]])

    def xlogx(v):
        return np.where(v == 0, 0.0, v * np.log(np.abs(np.where(v == 0, 1.0, v))))

    a, b, c = x[None, :-2], x[None, 1:-1], x[None, 2:]
    y = w[:, None]
    return _gpu((xlogx(a - y) / (b - a) - xlogx(b - y) * (c - a) / (b - a) / (c - b) + xlogx(c - y) / (c - b)) / math.pi)


def _cells(w, x):
    """Lower node and weight of linear interpolation on w at x, flat outside."""
    j = torch.clamp(torch.searchsorted(w, x, right=True) - 1, 0, len(w) - 2)
    t = torch.clamp((x - w[j]) / (w[j + 1] - w[j]), 0.0, 1.0)
    return j, t


def _coupling(s):
    g2 = s["g2"]
    return _gpu(np.asarray(g2).transpose(2, 1, 0)).double()  # [f, i, ν]


def _exact_scgd0(case, s, Ts, mu0):
    w_h, wa_h = _nodes(s["omegas"]), _nodes(s["omegas_spectral"])
    w, wa = _gpu(w_h), _gpu(wa_h)
    Wa, H = _gpu(_trapezoid(wa_h)), _hilbert(w_h)
    eps, wi = _gpu(s["eps_i"]), _gpu(s["w_i"])
    fi = _gpu(s["f_to_i"]).long()
    nw, ni, nm = len(w_h), len(s["eps_i"]), s["g2"].shape[0]
    wph = _gpu(s["omega_ph"])
    dispersive = case["family"].startswith("disp")
    g2 = _coupling(s) * _gpu(s["w_f"])[:, None, None]
    if dispersive:
        q = _gpu(s["iq_kk"]).long()[_gpu(s["iks_i"]).long()][:, _gpu(s["iks_f"]).long()]  # [i, f]
    else:  # sum over each star: its inner states share energy and Σ
        G = torch.zeros((ni, ni, nm), dtype=torch.float64, device="cuda").index_add_(0, fi, g2)  # [c, i, ν]
        del g2
    ja, ta = _cells(w, wa)

    def fan_migdal(S, mu, T):
        im = torch.zeros((nw, ni), dtype=torch.float64, device="cuda")
        if not dispersive:
            for nu in range(nm):
                wq = wph[nu, 0]
                nb = 1.0 / torch.expm1(wq / T)
                K = 0
                for x, n in ((w + wq, nb + _fermi(w + wq - mu, T)), (w - wq, nb + 1 - _fermi(w - wq - mu, T))):
                    j, t = _cells(w, x)
                    Sx = (1 - t)[:, None] * S[j] + t[:, None] * S[j + 1]
                    K = K + (1.0 / (x[:, None] - eps[None, :] - Sx)).imag * n[:, None]
                im += K @ G[:, :, nu]
            return im
        St = S.t().contiguous()  # [state, ω]
        for i in range(ni):
            wq = wph[:, q[i]]  # [ν, f]
            nb = 1.0 / torch.expm1(wq / T)
            for nu in range(nm):
                acc = 0
                for sign in (1.0, -1.0):
                    x = w[None, :] + sign * wq[nu][:, None]  # [f, ω]
                    j, t = _cells(w, x)
                    Sf = St[fi]
                    Sx = (1 - t) * torch.gather(Sf, 1, j) + t * torch.gather(Sf, 1, j + 1)
                    f = _fermi(x - mu, T)
                    n = nb[nu][:, None] + (f if sign > 0 else 1 - f)
                    acc = acc + (1.0 / (x - eps[fi][:, None] - Sx)).imag * n
                im[:, i] += g2[:, i, nu] @ acc
        return im

    def root(D, T):
        target = case.get("filling", 1.0)
        lo, hi = wa_h[0] - 0.1, wa_h[-1] + 0.1
        for _ in range(80):
            mid = 0.5 * (lo + hi)
            x = np.clip((wa_h - mid) / T, -700, 700)
            if 2.0 * (np.sum(D / (np.exp(x) + 1.0)) + s["nstates_base"]) < target:
                lo = mid
            else:
                hi = mid
        return 0.5 * (lo + hi)

    out, mus, done = [], [], []
    for T, mu in zip(Ts, mu0):
        S = torch.full((nw, ni), -1j * (0.05 if _chain(case) else ETA_INIT), dtype=torch.complex128, device="cuda")
        ok = False
        for _ in range(50):
            im = fan_migdal(torch.complex(S.real, torch.clamp(S.imag, max=0.0)), mu, T)
            new = torch.complex(H @ im, im)
            for m in s["multiplets"]:
                new[:, m] = new[:, m].mean(dim=1, keepdim=True)
            Sa = (1 - ta)[:, None] * new[ja] + ta[:, None] * new[ja + 1]
            A = -(1.0 / (wa[:, None] - eps[None, :] - Sa)).imag / math.pi
            mu = root(((A @ wi) * Wa).cpu().numpy(), T)
            err = float((new - S).abs().max())
            S = new
            if err < 1e-6:
                ok = True
                break
        out.append(S)
        mus.append(mu)
        done.append(ok)
    return torch.stack(out), np.array(mus), np.array(done)  # Σ [T, ω, i]


def _exact_ladder(case, s, Ts, Om, sigma, mus):
    """σ_bubble and σ_ladder [3, 3, nΩ, nT]: GMRES on (1 - L) J = J0 as the solver runs it, from the Ω before unless
    the pairs are solved together."""
    grid = s["omegas"]
    w_h, off, h = _nodes(grid), np.asarray(grid.offsets, dtype=np.int64), grid.unit
    w, H, W = _gpu(w_h), _hilbert(w_h), _gpu(_trapezoid(w_h))
    eps, wi, v = _gpu(s["eps_i"]), _gpu(s["w_i"]), _gpu(s["v"])
    nw, ni, nm = len(w_h), len(s["eps_i"]), s["g2"].shape[0]
    fi = _gpu(s["f_to_i"]).long()
    wph = np.asarray(s["omega_ph"])[:, 0]
    # G̃_ν[(i', b), (i, a)] = Σ_{f in star(i')} R_f[a, b] w_f g2[ν, i, f]
    g2, R = _coupling(s) * _gpu(s["w_f"])[:, None, None], _gpu(s["R"])
    Gt = torch.zeros((nm, ni, 3, ni, 3), dtype=torch.float64, device="cuda")
    for b in range(3):
        for a in range(3):
            Gt[:, :, b, :, a].permute(1, 2, 0).copy_(
                torch.zeros((ni, ni, nm), dtype=torch.float64, device="cuda").index_add_(0, fi, R[a, b][:, None, None] * g2))
    del g2
    Gt = Gt.reshape(nm, 3 * ni, 3 * ni)

    def shifts(nu, sign):
        """The interpolation matrix [nω, nω] of J at ω ± ω_ν on the grid of shifts, as node indices and weights."""
        x = wph[nu] / h
        lo = math.floor(x)
        idx, wts = [], []
        for m, tent in ((lo, 1 - (x - lo)), (lo + 1, x - lo)):
            p = off + sign * m
            k = np.clip(np.searchsorted(off, p, side="right"), 1, nw - 1) - 1
            t = (p - off[k]) / (off[k + 1] - off[k])
            inside = (p >= off[0]) & (p <= off[-1])
            idx += [k, k + 1]
            wts += [tent * np.where(inside, 1 - t, 0.0), tent * np.where(inside, t, 0.0)]
        return [_gpu(k) for k in idx], [_gpu(x) for x in wts]

    tables = [[shifts(nu, 1), shifts(nu, -1)] for nu in range(nm)]

    def greens(S, x, mu, T):
        j, t = _cells(w, x)
        GR = 1.0 / (x[:, None] - eps[None, :] - ((1 - t)[:, None] * S[j] + t[:, None] * S[j + 1]))
        GA = GR.conj()
        GK = (GR - GA) * (1 - 2 * _fermi(x - mu, T))[:, None]
        # [c1, c2] blocks: 11, 12 / 21, 22, each [ω, i]
        return torch.stack([torch.stack([GR + GA + GK, GA - GR + GK]), torch.stack([GR - GA + GK, GK - GR - GA])]) / 2

    def operator(J, Gm, Gp, T):
        """L(J) of J [c1, c2, c0, ω, i, b]."""
        K = torch.zeros_like(J)
        Y = torch.zeros((2,) + J.shape[2:], dtype=J.dtype, device="cuda")
        flat = torch.view_as_real(J).permute(0, 1, 2, 6, 3, 4, 5).reshape(-1, 3 * ni)  # rows (c1, c2, c0, re/im, ω)
        for nu in range(nm):
            n = 1.0 / math.expm1(wph[nu] / T)
            Z = (flat @ Gt[nu]).reshape(2, 2, 2, 2, nw, ni, 3).permute(0, 1, 2, 4, 5, 6, 3).contiguous()
            Z = torch.view_as_complex(Z)
            up, dn = (sum(t[:, None, None] * Z[:, :, :, k] for k, t in zip(*tab)) for tab in tables[nu])
            for d in range(2):
                Y[d] += (up[d, d] - dn[d, d]) / 2
                K[d, d] -= (0.5 + n) * (up[d, d] + dn[d, d])
            K[1, 0] += n * up[1, 0] + (1 + n) * dn[1, 0]
            K[0, 1] += (1 + n) * up[0, 1] + n * dn[0, 1]
            del Z, up, dn
        HY = torch.einsum("xw,dcwr->dcxr", H.to(Y.dtype), Y.reshape(2, 2, nw, 3 * ni)).reshape(Y.shape)
        K[0, 0] -= 1j * HY[0]
        K[1, 1] += 1j * HY[1]
        return -torch.einsum("abwi,bcqwik,cdwi->adqwik", Gm, K, Gp)

    def conductivity(J, Omega, T):
        y = torch.einsum("w,wib->ib", W.to(J.dtype), J[1, 1, 0] + J[0, 0, 1])
        F = 1j / (4 * T) if Omega == 0 else -1.0 / (2j * Omega * (1 + 2 / math.expm1(Omega / T)))
        S = torch.einsum("ai,i,ib->ab", v.to(J.dtype), wi.to(J.dtype), y)
        return (F / (2j * math.pi) * S).real.cpu().numpy()

    def gmres(op, b, x0, rtol, maxiter):
        r = b - op(x0) if x0 is not None else b
        atol, beta = rtol * float(torch.linalg.vector_norm(b)), float(torch.linalg.vector_norm(r))
        if beta <= atol:
            return (x0 if x0 is not None else torch.zeros_like(b)), True
        V, Hs, y = [r / beta], np.zeros((maxiter + 1, maxiter), dtype=complex), None
        for k in range(maxiter):
            q = op(V[k])
            for i, u in enumerate(V):
                Hs[i, k] = complex(torch.vdot(u.reshape(-1), q.reshape(-1)))
                q = q - Hs[i, k] * u
            Hs[k + 1, k] = float(torch.linalg.vector_norm(q))
            rhs = np.zeros(k + 2, dtype=complex)
            rhs[0] = beta
            y = np.linalg.lstsq(Hs[:k + 2, :k + 1], rhs, rcond=None)[0]
            solved = np.linalg.norm(rhs - Hs[:k + 2, :k + 1] @ y) <= atol
            if solved:
                break
            V.append(q / Hs[k + 1, k].real)
        x = sum(complex(c) * u for c, u in zip(y, V))
        return (x if x0 is None else x0 + x), bool(solved)

    sb, sl = np.zeros((3, 3, len(Om), len(Ts))), np.zeros((3, 3, len(Om), len(Ts)))
    done = np.zeros((len(Om), len(Ts)), dtype=bool)
    for iT, (T, mu) in enumerate(zip(Ts, mus)):
        J = None
        for iO, Omega in enumerate(Om):
            Gm, Gp = greens(sigma[iT], w - Omega / 2, mu, T), greens(sigma[iT], w + Omega / 2, mu, T)
            J0 = torch.einsum("aqwi,ki,qdwi->adqwik", Gm, v.to(Gm.dtype), Gp)
            J, done[iO, iT] = gmres(lambda x: x - operator(x, Gm, Gp, T), J0, None if case.get("batch") else J, 1e-2, 30)
            sb[:, :, iO, iT], sl[:, :, iO, iT] = conductivity(J0, Omega, T), conductivity(J, Omega, T)
    return sb, sl, done


def _exact_train(case, seed):
    """Two epochs of Adam on the mean squared error in FP64, the products with the weights rounded to BF16."""
    X, Y, dims = _training_set(case, seed)
    X, Y = _gpu(X).double(), _gpu(Y).double()
    p = _gpu(_first_parameters(dims, seed)).double()
    m, u, hist, step = torch.zeros_like(p), torch.zeros_like(p), [], 0
    for order in _row_orders(case):
        total = 0.0
        for r0 in range(0, case["rows"], 256):
            idx = _gpu(order[r0:r0 + 256])
            x, y = X[idx], Y[idx]
            acts, at = [], 0
            for l, (a, b) in enumerate(zip(dims[:-1], dims[1:])):
                Wq = p[at:at + a * b].float().bfloat16().double().reshape(b, a)
                z = x @ Wq.t() + p[at + a * b:at + a * b + b]
                acts.append((x, z, Wq))
                at += a * b + b
                x = z * torch.sigmoid(z) if l + 2 < len(dims) else z
            e = x - y
            total += float((e * e).sum())
            dz, grads = 2 * e / e.numel(), []
            for l in range(len(acts) - 1, -1, -1):
                x, _, Wq = acts[l]
                grads.insert(0, torch.cat([(dz.t() @ x).reshape(-1), dz.sum(0)]))
                if l:
                    z = acts[l - 1][1]
                    sg = torch.sigmoid(z)
                    dz = (dz @ Wq) * (sg * (1 + z * (1 - sg)))
            g = torch.cat(grads)
            step += 1
            m, u = 0.9 * m + 0.1 * g, 0.999 * u + 0.001 * g * g
            p = p - 1e-4 * (m / (1 - 0.9 ** step)) / (torch.sqrt(u / (1 - 0.999 ** step)) + 1e-8)
        hist.append(total / Y.numel())
    return dict(params=p, loss=np.array(hist))


def exact(case, seed):
    if case["family"] == "train":
        return _exact_train(case, seed)
    s = _model(case, seed)
    Ts = _temperatures(case)
    mu0 = _mu_start(case, s, Ts)
    out = {}
    ladder = "ladder" in case["family"]
    if ladder:
        sigma, mus = _gpu(_self_energy(s, len(Ts), seed).transpose(2, 0, 1)), mu0
    else:
        sigma, mus, done = _exact_scgd0(case, s, Ts, mu0)
        out.update(mu=mus, converged=done)
        if case["path"].endswith("fp64"):
            out["sigma"] = sigma.permute(1, 2, 0).contiguous()
        elif case["family"] != "step":
            out["sigma"] = sigma.transpose(1, 2).contiguous()
    if ladder or case["family"] == "step":
        sb, sl, done = _exact_ladder(case, s, Ts, _probe_frequencies(case), sigma, mus)
        out.update(sigma_bubble=sb, sigma_ladder=sl, solved=done)
    return out
