"""The work that users of this solver have it do, as cases that can be timed and compared.

Each case is a dict of plain values; prepare() makes the inputs and the solver handle that a
program would keep, run() is one call (or one sequence of stage calls) through the public
Python binding, exact() the same result as a plain FP64 direct sum where that is affordable.

Distributions are those of the package's datasets module (and of the reference's Dataset):
a cube with charges of zero mean, a Plummer sphere of equal charges, a spherical surface with
charges in [0, 1].  They are drawn on the GPU, so that inputs of millions of bodies are quick
to make.
"""
import importlib
import math

import numpy as np
import torch

fmm = importlib.import_module("exafmm-dev_b200")

# opening angle per order that holds mixed requests to a relative error of 1e-4 (the serving
# workload of bench.py), and the default of the configuration for the orders beside them
SERVE_THETA = {4: 0.22, 6: 0.22, 8: 0.30, 10: 0.35, 12: 0.40}


def listed():
    return [
        # the smallest request of the serving workload, one call on host arrays: latency
        dict(name="request_1k_host", call="host", basis="spherical", P=6, theta=0.22, ncrit=64,
             prec="f32", ropt=0, dist="plummer", n=1000),
        # a request of the middle of that range, odd size, highest of its orders
        dict(name="request_31k_host", call="host", basis="spherical", P=10, theta=0.35, ncrit=64,
             prec="f32", ropt=0, dist="cube", n=31607),
        # a simulation step of a mid-size system whose bodies stay on the device
        dict(name="cube_200k_p8", call="device", basis="spherical", P=8, theta=0.30, ncrit=64,
             prec="f32", ropt=0, dist="cube", n=200003),
        # the plain FP64 configuration (cube of 16,384 bodies), driven stage by stage as
        # examples/serial.cxx of the reference does
        dict(name="cube_16k_f64_stages", call="stages", basis="spherical", P=6, theta=0.4,
             ncrit=64, prec="f64", ropt=0, dist="cube", n=16384),
        # the benchmark's headline: 2^20 bodies, P = 10, FP32 with compensated sums
        dict(name="plummer_1m_p10", call="device", basis="spherical", P=10, theta=0.35, ncrit=64,
             prec="f32", ropt=1, dist="plummer", n=1 << 20),
        # the same bodies in plain FP64
        dict(name="plummer_1m_p10_f64", call="device", basis="spherical", P=10, theta=0.35,
             ncrit=64, prec="f64", ropt=1, dist="plummer", n=1 << 20),
        # the Cartesian basis on a surface: deep, unbalanced trees and long near lists
        dict(name="sphere_4m_cart_p5", call="device", basis="cartesian", P=5, theta=0.5, ncrit=32,
             prec="f32", ropt=0, dist="sphere", n=1 << 22),
        # 256 independent solves of uneven size in one call
        dict(name="batch_256_p8", call="batch", basis="spherical", P=8, theta=0.4, ncrit=64,
             prec="f32", ropt=0, dist="mixed", n=200000, nmin=1000, solves=256, sizes=44),
        # a molecular-dynamics box with periodic images, host arrays (the wrappers' call)
        dict(name="periodic_30k_host", call="host", basis="spherical", P=8, theta=0.4, ncrit=32,
             prec="f32", ropt=0, dist="cube", n=30003, images=2),
        # targets against other sources (two trees), FP64, host arrays (the PetIGA wrapper's)
        dict(name="ij_20k_50k_f64_host", call="ij", basis="spherical", P=8, theta=0.4, ncrit=64,
             prec="f64", ropt=0, dist="cube", n=50021, targets=20011),
        # the uniform Morton tree on a homogeneous box
        dict(name="uniform_250k_p6", call="device", basis="spherical", P=6, theta=0.4, ncrit=64,
             prec="f32", ropt=0, dist="cube", n=250007, tree="uniform"),
        # the accuracy check of a large solve: an FP64 direct sum of sampled targets
        dict(name="direct_1k_x_1m", call="direct", prec="f64", dist="plummer", n=1 << 20,
             targets=1024),
    ]


def _log_int(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return n | 1 if rng.random() < 0.75 else n


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "cart", "batch", "periodic", "ij", "uniform",
                       "direct"])
    prec = rng.choice(["f32", "f32", "f64"])
    ncrit = rng.choice([32, 48, 64, 64, 96, 128])
    P = rng.choice([4, 6, 8, 10, 10, 12])
    dist = rng.choice(["cube", "plummer", "sphere"])
    top = 1000000 if prec == "f32" else 400000
    base = dict(basis="spherical", P=P, theta=SERVE_THETA[P], ncrit=ncrit, prec=prec, dist=dist,
                ropt=0 if dist == "cube" else rng.choice([0, 1]))
    if kind == "solve":
        return dict(base, call=rng.choice(["device", "device", "host", "stages"]),
                    n=_log_int(rng, 1000, top))
    if kind == "cart":
        return dict(base, call=rng.choice(["device", "host"]), basis="cartesian",
                    P=rng.choice([3, 4, 5, 5, 6, 7]), theta=rng.choice([0.4, 0.5]),
                    n=_log_int(rng, 1000, 4000000 if prec == "f32" else 400000))
    if kind == "batch":
        return dict(base, call="batch", dist="mixed", ropt=0, prec="f32", nmin=1000,
                    n=_log_int(rng, 2000, 100000), solves=rng.randint(2, 100),
                    sizes=rng.randint(1, 1000))
    if kind == "periodic":
        return dict(base, call=rng.choice(["device", "host"]), dist="cube", ropt=0,
                    theta=0.4, n=_log_int(rng, 1000, 200000), images=rng.choice([1, 2, 3]))
    if kind == "ij":
        return dict(base, call="ij", ropt=0, n=_log_int(rng, 1000, 300000),
                    targets=_log_int(rng, 1000, 300000))
    if kind == "uniform":
        return dict(base, call="device", dist="cube", ropt=0, tree="uniform",
                    n=_log_int(rng, 1000, 500000))
    return dict(call="direct", prec="f64", dist=dist, n=_log_int(rng, 10000, 1000000),
                targets=_log_int(rng, 64, 4096))


# ---------------------------------------------------------------- inputs
def _bodies(dist, n, gen, prec):
    """(n, 4) FP64 tensor of x, y, z, q whose values the working precision holds exactly."""
    d = dict(generator=gen, dtype=torch.float64, device="cuda")
    if dist == "cube":
        x = torch.rand((n, 3), **d) * 2 - 1
        q = torch.rand(n, **d) * 2 - 1
        q -= q.mean()
    elif dist == "plummer":
        u = torch.rand((n, 3), **d)
        u[:, 0] *= 1.01 ** -1.5  # the radii below ten times the scale, by the inverse CDF
        r = (u[:, 0].clamp_min(1e-12) ** (-2.0 / 3.0) - 1).rsqrt()
        z = (1 - 2 * u[:, 1]) * r
        s = (r * r - z * z).clamp_min(0).sqrt()
        x = torch.stack([s * torch.cos(2 * math.pi * u[:, 2]),
                         s * torch.sin(2 * math.pi * u[:, 2]), z], 1)
        x -= x.mean(0)
        q = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    else:
        x = torch.randn((n, 3), **d)
        x /= x.norm(dim=1, keepdim=True)
        q = torch.rand(n, **d)
    b = torch.cat([x, q[:, None]], 1)
    return b.float().double() if prec == "f32" else b


def _counts(case):
    rng = np.random.default_rng(case["sizes"])
    lo, hi = math.log(case["nmin"]), math.log(case["n"])
    return np.rint(np.exp(rng.uniform(lo, hi, case["solves"]))).astype(np.int32)


def _solver(case):
    kw = dict(basis=case["basis"], P=case["P"], theta=case["theta"], ncrit=case["ncrit"],
              use_ropt=case["ropt"], precision=case["prec"])
    if case.get("images"):
        kw.update(images=case["images"], cycle=2.0)
    if case.get("tree"):
        kw.update(tree=case["tree"])
    return fmm.Solver(**kw)


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    if case["call"] == "batch":
        kinds = ("cube", "plummer", "sphere")
        return torch.cat([_bodies(kinds[i % 3], int(c), gen, case["prec"])
                          for i, c in enumerate(_counts(case))])
    b = _bodies(case["dist"], case["n"], gen, case["prec"])
    if case["call"] == "ij":
        return _bodies(case["dist"], case["targets"], gen, case["prec"]), b
    return b


def _host(b):
    h = b.cpu().numpy()
    return np.ascontiguousarray(h[:, :3]), np.ascontiguousarray(h[:, 3])


def prepare(case, seed):
    b = _inputs(case, seed)
    st = dict(case=case, call=case["call"])
    if case["call"] == "direct":
        x, q = _host(b)
        step = max(1, case["n"] // case["targets"])
        st.update(x=x, q=q, xt=np.ascontiguousarray(x[:step * case["targets"]:step]))
        return st
    st["solver"] = _solver(case)
    if case["call"] in ("device", "batch"):
        st["bodies"] = b if case["prec"] == "f64" else b.float()
        st["out"] = torch.empty_like(st["bodies"])
        st["solver"].set_stream(torch.cuda.current_stream().cuda_stream)
        if case["call"] == "batch":
            st["counts"] = _counts(case)
    elif case["call"] == "ij":
        st["xt"], st["qt"] = _host(b[0])
        st["x"], st["q"] = _host(b[1])
    else:
        st["x"], st["q"] = _host(b)
    return st


def run(st):
    call = st["call"]
    if call == "direct":
        return fmm.direct(st["xt"], st["x"], st["q"])
    s = st["solver"]
    if call == "device":
        s.solve_device(st["bodies"].shape[0], st["bodies"].data_ptr(), st["out"].data_ptr())
        return _fields(st["out"])
    if call == "batch":
        s.solve_batch_device(st["counts"], st["bodies"].data_ptr(), st["out"].data_ptr())
        return _fields(st["out"])
    if call == "host":
        return _fields(s.solve(st["x"], st["q"]))
    if call == "ij":
        return _fields(s.solve_ij(st["xt"], st["qt"], st["x"], st["q"]))
    s.set_bodies(st["x"], st["q"])
    s.build_tree()
    s.upward_pass()
    s.traverse()
    s.downward_pass()
    return _fields(s.trg())


def _fields(t):
    """Potential and gradient apart: their scales differ."""
    return {"potential": t[:, 0], "gradient": t[:, 1:]}


def exact(case, seed):
    b = _inputs(case, seed)
    if case["call"] == "batch" or case.get("images"):
        return None
    if case["call"] == "ij":
        t, s = b
    elif case["call"] == "direct":
        step = max(1, case["n"] // case["targets"])
        t, s = b[:step * case["targets"]:step], b
    else:
        t, s = b, b
    if float(t.shape[0]) * s.shape[0] > 7e10:
        return None
    out = torch.empty((t.shape[0], 4), dtype=torch.float64, device="cuda")
    rows = max(1, 50000000 // s.shape[0])
    for i in range(0, t.shape[0], rows):
        e = t[i:i + rows]
        d = [s[None, :, k] - e[:, None, k] for k in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        inv = torch.where(r2 > 0, r2.rsqrt(), 0.0)
        q1 = s[None, :, 3] * inv
        out[i:i + rows, 0] = q1.sum(1)
        q1 *= inv * inv
        for k in range(3):
            out[i:i + rows, 1 + k] = (q1 * d[k]).sum(1)
    if case["call"] == "direct":
        return out
    return _fields(out)


def work(case):
    """Bodies read and results written once; the pair sums' flops, from interaction counts per
    body that go as theta^-3 (theta^-2 on a surface) and were read off solves of these kinds."""
    size = 4 if case["prec"] == "f32" else 8
    n = case["n"]
    if case["call"] == "direct":
        return {"bytes": 32.0 * n + 56.0 * case["targets"], "flops": 20.0 * n * case["targets"]}
    if case["call"] == "batch":
        n = int(_counts(case).sum())
    nt = case.get("targets", n)
    dim = 2 if case["dist"] == "sphere" else 3
    near = min(n, 0.7 * case["ncrit"] * case["theta"] ** -dim)
    far = min(n / case["ncrit"], 170.0 * (case["theta"] / 0.35) ** -dim) * 4.0 / case["ncrit"]
    P = case["P"]
    if case["basis"] == "spherical":  # two multiply-adds per (j, k, n, m) term, j + n < P
        pair = 4.0 * math.comb(P + 3, 4)
    else:
        terms = lambda p: p * (p + 1) * (p + 2) // 6
        pair = 2.0 * sum((o + 1) * (o + 2) // 2 * terms(P - o) for o in range(P))
    moved = size * 4.0 * ((n if case["call"] != "ij" else n + nt) + nt)
    return {"bytes": moved, "flops": nt * (20.0 * near + far * pair)}
