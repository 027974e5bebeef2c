"""The evaluations this framework is timed on: FMM3d evals, batches, direct sums
and the one-call form, through the public entry points of ``kifmm``.

A case is a dict of plain values.  Its ``kind`` says which entry point runs:

* ``eval``    ``FMM3d.eval``: host arrays in, host array out, as the reference's
  own driver calls it;
* ``device``  ``FMM3d.eval_device``: densities and potentials in device memory on
  the caller's stream, ``nrhs`` density vectors, as an iterative solver calls it;
* ``batch``   ``Batch.eval``: several set-up instances in one call;
* ``direct``  ``FMM3d.direct``: the direct sum that checks an evaluation;
* ``mex``     ``fmm3d_mex``: setup, evaluation and check in one call, for a
  geometry that is used once.

Point clouds and densities come from the package's seeded generators.  The FP64
engine is the default precision; the mixed engine is the option.
"""
import math
import os
import sys

import numpy as np
import torch

for _p in list(sys.path):
    _d = os.path.join(_p or os.getcwd(), "kernel-independent-fast-multipole-method_b200")
    if os.path.isdir(_d):
        if _d not in sys.path:
            sys.path.insert(0, _d)
        break

import kifmm  # noqa: E402
import workloads  # noqa: E402

COEFS = {111: [1.0], 121: [1.0], 311: [1.0], 312: [1.0], 321: [1.0], 322: [1.0], 511: [1.0, 0.3], 521: [1.0, 0.3]}
DOUBLE_LAYER = (121, 321, 322, 521)
GEOMETRIES = {"sphere": workloads.sphere, "ellipsoid": workloads.ellipsoid, "cube": workloads.cube,
              "cube_plummer": workloads.cube_plummer, "plummer_ball": workloads.plummer_ball}


def listed():
    return [
        # a small cloud, the size of the test fixtures and of a first try: latency
        {"name": "laplace_sphere_np4_2k_fp64_host", "kind": "eval", "kt": 111, "np": 4, "ptsmax": 100,
         "precision": "fp64", "geometry": "sphere", "n": 2000},
        # the low-accuracy surface configuration at its size
        {"name": "laplace_sphere_np4_32k_fp64_host", "kind": "eval", "kt": 111, "np": 4, "ptsmax": 100,
         "precision": "fp64", "geometry": "sphere", "n": 32768},
        # the Stokes double-layer configuration: a boundary-integral matvec inside a solver
        {"name": "stokes_dl_ellipsoid_np6_262k_fp64", "kind": "device", "kt": 321, "np": 6, "ptsmax": 100,
         "precision": "fp64", "geometry": "ellipsoid", "n": 262144, "nt": 0, "nrhs": 1},
        # the high-accuracy elasticity configuration at its size
        {"name": "navier_sphere_np8_1m_fp64", "kind": "device", "kt": 511, "np": 8, "ptsmax": 150,
         "precision": "fp64", "geometry": "sphere", "n": 1048576, "nt": 0, "nrhs": 1},
        # the headline cloud in the reference's own arithmetic, largest size
        {"name": "laplace_cube_plummer_np6_4m_fp64", "kind": "device", "kt": 111, "np": 6, "ptsmax": 64,
         "precision": "fp64", "geometry": "cube_plummer", "n": 4194304, "nt": 0, "nrhs": 1},
        # the headline cloud in mixed precision, at the largest size whose direct sum can be checked
        {"name": "laplace_cube_plummer_np6_1m_mixed", "kind": "device", "kt": 111, "np": 6, "ptsmax": 64,
         "precision": "mixed", "geometry": "cube_plummer", "n": 1048576, "nt": 0, "nrhs": 1},
        # the same cloud at an ordinary size, through the host call
        {"name": "laplace_cube_plummer_np6_262k_mixed_host", "kind": "eval", "kt": 111, "np": 6, "ptsmax": 64,
         "precision": "mixed", "geometry": "cube_plummer", "n": 262144},
        # a block solver: several Stokes density vectors per call, a ragged count
        {"name": "stokes_cube_np6_100k_mixed_x4", "kind": "device", "kt": 311, "np": 6, "ptsmax": 100,
         "precision": "mixed", "geometry": "cube", "n": 100003, "nt": 0, "nrhs": 4},
        # a double layer on a surface, its potential wanted at other points in the volume
        {"name": "laplace_dl_ellipsoid_np6_150k_to_40k_mixed", "kind": "device", "kt": 121, "np": 6, "ptsmax": 100,
         "precision": "mixed", "geometry": "ellipsoid", "n": 150001, "nt": 40009, "nrhs": 1},
        # independent instances of several sizes, kernels and shapes, eight density vectors each
        {"name": "batch_10_instances_x8_mixed", "kind": "batch", "instances": 10, "stokes": 3, "lo": 10000, "hi": 100000,
         "precision": "mixed", "nrhs": 8},
        # the check of an evaluation: the direct sum at 1,000 of its targets
        {"name": "direct_laplace_262k_to_1000", "kind": "direct", "kt": 111, "np": 6, "ptsmax": 100, "precision": "fp64",
         "geometry": "cube", "n": 262144, "nt": 1000},
        # a geometry that is used once: setup, evaluation and check in one call
        {"name": "mex_laplace_cube_np4_20k_fp64", "kind": "mex", "kt": 111, "np": 4, "precision": "fp64",
         "geometry": "cube", "n": 20011},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("eval", "eval", "device", "device", "device", "device", "device", "batch", "direct", "mex"))
    kt = rng.choice((111, 111, 111, 121, 311, 312, 321, 322, 511, 521))
    precision = rng.choice(("fp64", "mixed"))
    geometry = rng.choice(tuple(GEOMETRIES))
    np_ = rng.choice((4, 6, 6, 8))
    ptsmax = rng.choice((50, 64, 100, 150))
    if kind == "eval":
        return {"kind": kind, "kt": kt, "np": np_, "ptsmax": ptsmax, "precision": precision, "geometry": geometry,
                "n": _log_int(rng, 1500, 200000)}
    if kind == "device":
        big = 1000000 if kt in (111, 121) and np_ < 8 else 250000
        n, nrhs = _log_int(rng, 3000, big), rng.choice((1, 1, 1, 2, 5))
        nt = rng.choice((0, 0, 0, max(1000, int(n * rng.uniform(0.1, 1.5)))))
        return {"kind": kind, "kt": kt, "np": np_, "ptsmax": ptsmax, "precision": precision, "geometry": geometry,
                "n": n if nrhs == 1 else max(3000, n // 4), "nt": nt if nrhs == 1 else nt // 4, "nrhs": nrhs}
    if kind == "batch":
        return {"kind": kind, "instances": rng.randint(3, 9), "stokes": rng.randint(0, 3), "lo": 5000,
                "hi": rng.randint(20000, 80000), "precision": precision, "nrhs": rng.choice((1, 3, 8))}
    if kind == "direct":
        return {"kind": kind, "kt": kt, "np": 4, "ptsmax": 100, "precision": "fp64", "geometry": geometry,
                "n": _log_int(rng, 5000, 500000), "nt": _log_int(rng, 20, 4096)}
    return {"kind": kind, "kt": kt, "np": rng.choice((4, 6)), "precision": precision, "geometry": geometry,
            "n": _log_int(rng, 2000, 40000)}


class State:
    pass


def _cloud(geometry, n, seed):
    p, nor = GEOMETRIES[geometry](n, seed)
    return p, nor if geometry in ("sphere", "ellipsoid") else p


def _dofs(kt):
    return kifmm.Kernel3d.DOFS[kt]


def _inputs(case, seed):
    """Sources, normals, targets, densities of a case with one instance."""
    src, nor = _cloud(case["geometry"], case["n"], seed)
    trg = src
    if case.get("nt"):
        trg = workloads.cube(case["nt"], seed + 1000003)[0] * 0.999
    den = workloads.densities(case["n"] * case.get("nrhs", 1), _dofs(case["kt"])[0], "uniform", seed + 2000003)
    return src, nor, trg, den


def _instance(kt, np_, ptsmax, precision, src, nor, trg):
    f = kifmm.FMM3d("fmm3d_")
    f.srcpos, f.srcnor, f.trgpos = src, nor, trg
    f.knl = kifmm.Kernel3d(kt, COEFS[kt])
    f.setup({"-fmm3d_np": str(np_), "-fmm3d_let3d_ptsmax": str(ptsmax), "-fmm3d_let3d_maxlevel": "10",
             "-fmm3d_precision": precision})
    return f


def _members(case, seed):
    """(kt, sources, normals, densities) of a batch's instances: sizes evenly spread over their logarithm."""
    k, out = case["instances"], []
    for i in range(k):
        n = int(round(case["lo"] * (case["hi"] / case["lo"]) ** (i / max(1, k - 1))))
        geometry = ("sphere", "cube", "plummer_ball")[i % 3]
        kt = 311 if i % 3 == 1 and i // 3 < case["stokes"] else 111
        src, nor = _cloud(geometry, n, seed + 17 * i)
        out.append((kt, src, nor, workloads.densities(n * case["nrhs"], _dofs(kt)[0], "uniform", seed + 2000003 + i)))
    return out


def prepare(case, seed):
    s = State()
    s.kind = case["kind"]
    if s.kind == "batch":
        s.fmms, s.den, s.out = [], [], []
        for kt, src, nor, den in _members(case, seed):
            s.fmms.append(_instance(kt, 6, 100, case["precision"], src, nor, src))
            s.den.append(torch.from_numpy(den).cuda())
            s.out.append(torch.zeros(len(src) * case["nrhs"] * _dofs(kt)[1], device="cuda", dtype=torch.float64))
        s.batch, s.nrhs = kifmm.Batch(s.fmms), case["nrhs"]
        return s
    src, nor, trg, den = _inputs(case, seed)
    sd, td = _dofs(case["kt"])
    if s.kind == "mex":
        s.args = (np.ascontiguousarray(src.T), np.ascontiguousarray(nor.T), np.ascontiguousarray(trg.T), (0.0, 0.0, 0.0), 0,
                  (case["kt"], COEFS[case["kt"]]), case["np"], den)
        s.precision = case["precision"]
        return s
    if s.kind == "direct":
        s.fmm = _instance(case["kt"], case["np"], case["ptsmax"], case["precision"], src, nor, src)
        s.den, s.trg = den, trg
        return s
    s.fmm = _instance(case["kt"], case["np"], case["ptsmax"], case["precision"], src, nor, trg)
    if s.kind == "eval":
        s.den, s.out = den, np.zeros(len(trg) * td)
    else:
        s.nrhs = case["nrhs"]
        s.den = torch.from_numpy(den).cuda()
        s.out = torch.zeros(s.nrhs * len(trg) * td, device="cuda", dtype=torch.float64)
    return s


def run(s):
    if s.kind == "eval":
        s.fmm.eval(s.den, s.out)
        return s.out
    if s.kind == "device":
        s.fmm.eval_device(s.den.data_ptr(), s.out.data_ptr(), s.nrhs, torch.cuda.current_stream().cuda_stream, sync=False)
        return s.out
    if s.kind == "batch":
        s.batch.eval([d.data_ptr() for d in s.den], [o.data_ptr() for o in s.out], s.nrhs,
                     torch.cuda.current_stream().cuda_stream, sync=False)
        return s.out
    if s.kind == "direct":
        return s.fmm.direct(s.den, s.trg)
    return kifmm.fmm3d_mex(*s.args, precision=s.precision)


# ---------------------------------------------------------------------------
# Operations of one pass: kernel evaluations of the direct neighbours and the
# leaf surfaces, and the V-list products in the frequency domain, for a cloud
# refined to `ptsmax` points a leaf.
_FLOPS = {111: 11, 121: 19, 311: 29, 312: 17, 321: 30, 322: 27, 511: 29, 521: 55}


def _fmm_work(kt, np_, ptsmax, precision, geometry, n, nt, nrhs):
    sd, td = _dofs(kt)
    esd, etd = {111: (1, 1), 311: (4, 3), 511: (3, 3)}[111 if kt in (111, 121, 312, 322) else 311 if kt in (311, 321) else 511]
    surface = geometry in ("sphere", "ellipsoid")
    leaf = 0.5 * ptsmax
    near, pairs = (9.0, 30.0) if surface else (27.0, 150.0)
    nsurf = np_ ** 3 - (np_ - 2) ** 3
    nodes = 1.2 * n / leaf
    nfc = 4 * np_ ** 3 + 4
    flops = nt * near * leaf * _FLOPS[kt] + 2 * max(n, nt) * nsurf * _FLOPS[kt] + nodes * pairs * nfc * 8 * esd * etd
    flops += nodes * 8 * (nsurf * max(esd, etd)) ** 2
    size = 8 if precision == "fp64" else 4
    spectra = 2 * nodes * nfc * (esd + etd) * 2 * size  # written once, read once
    points = 8 * (nrhs * (n * sd + nt * td)) + size * ((n + nt) * 3 + (3 * n if kt in DOUBLE_LAYER else 0))
    return points + nrhs * spectra, nrhs * flops


def work(case):
    if case["kind"] == "batch":
        b = f = 0.0
        k = case["instances"]
        for i in range(k):
            n = int(round(case["lo"] * (case["hi"] / case["lo"]) ** (i / max(1, k - 1))))
            kt = 311 if i % 3 == 1 and i // 3 < case["stokes"] else 111
            x, y = _fmm_work(kt, 6, 100, case["precision"], ("sphere", "cube", "plummer_ball")[i % 3], n, n, case["nrhs"])
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    sd, td = _dofs(case["kt"])
    if case["kind"] == "direct":
        return {"bytes": 8 * (case["n"] * (3 + sd + (3 if case["kt"] in DOUBLE_LAYER else 0)) + case["nt"] * (3 + td)),
                "flops": float(case["n"]) * case["nt"] * _FLOPS[case["kt"]]}
    b, f = _fmm_work(case["kt"], case["np"], case.get("ptsmax", 150), case["precision"], case["geometry"], case["n"],
                     case.get("nt") or case["n"], case.get("nrhs", 1))
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# The sums themselves, pair by pair in 64 bits.
_COST = {111: 1.0, 121: 1.8, 311: 3.5, 312: 2.0, 321: 3.5, 322: 2.8, 511: 3.5, 521: 4.5}  # of one pair, against Laplace's


def _sums(kt, src, nor, den, trg, nrhs):
    sd, td = _dofs(kt)
    dev = "cuda"
    s = torch.from_numpy(src).to(dev).t().contiguous()
    t = s.clone() if trg is src else torch.from_numpy(np.ascontiguousarray(trg)).to(dev).t().contiguous()
    m = torch.from_numpy(nor).to(dev).t().contiguous()
    f = torch.from_numpy(den).to(dev).reshape(nrhs, src.shape[0], sd)
    mu, nu = COEFS[kt][0], COEFS[kt][-1]
    pi = math.pi
    ns, nt = s.shape[1], t.shape[1]
    out = torch.zeros(nrhs, nt, td, device=dev, dtype=torch.float64)
    block_t, block_s = min(nt, 2048), 4096
    for b in range(0, ns, block_s):
        S, N, F = s[:, b:b + block_s], m[:, b:b + block_s], f[:, b:b + block_s]
        for a in range(0, nt, block_t):
            T = t[:, a:a + block_t]
            o = out[:, a:a + block_t]
            d = [T[i][:, None] - S[i][None, :] for i in range(3)]
            r2 = d[0] * d[0]
            r2.addcmul_(d[1], d[1]).addcmul_(d[2], d[2])
            if trg is src and (a + block_t <= b or b + block_s <= a):
                ri = r2.rsqrt_()
            else:  # a source at the target itself adds nothing
                ri = r2.masked_fill_(r2 < 1e-16, math.inf).rsqrt_()
            if kt == 111:
                o += (ri @ F[:, :, 0].t()).t()[:, :, None] * (1 / (4 * pi))
                continue
            ri3 = ri * ri
            ri3 *= ri
            rn = nf = None
            if kt in DOUBLE_LAYER:
                rn = d[0] * N[0]
                rn.addcmul_(d[1], N[1].expand_as(rn)).addcmul_(d[2], N[2].expand_as(rn))
            if kt == 121:
                o += ((ri3 * rn) @ F[:, :, 0].t()).t()[:, :, None] * (-1 / (4 * pi))
                continue
            for k in range(nrhs):
                g = F[k]
                xf = d[0] * g[:, 0]
                xf.addcmul_(d[1], g[:, 1].expand_as(xf)).addcmul_(d[2], g[:, 2].expand_as(xf))
                if kt == 312:
                    o[k, :, 0] += (ri3 * xf).sum(1) * (1 / (4 * pi))
                    continue
                if kt in (311, 511):
                    c0, c1 = (1 / (8 * pi * mu),) * 2 if kt == 311 else (
                        (3 - 4 * nu) / (16 * pi * (1 - nu)) / mu, 1 / (16 * pi * (1 - nu)) / mu)
                    w = ri3 * xf
                    o[k] += (ri @ g) * c0
                    for i in range(3):
                        o[k, :, i] += (w * d[i]).sum(1) * c1
                    continue
                if kt == 322:
                    nf = (N * g.t()).sum(0)
                    w = ri3 * ri * ri * rn * xf
                    o[k, :, 0] += (ri3 @ nf - 3 * w.sum(1)) * (mu / (2 * pi))
                    continue
                if kt == 321:
                    w = ri3 * ri * ri * rn * xf
                    for i in range(3):
                        o[k, :, i] += (w * d[i]).sum(1) * (-6 / (8 * pi))
                    continue
                a1, a2 = (1 - 2 * nu) / (8 * pi * (1 - nu)), 3 / (8 * pi * (1 - nu))
                nf = (N * g.t()).sum(0)
                w = ri3 * nf * a1
                w -= ri3 * ri * ri * rn * xf * a2
                o[k] += ((ri3 * xf) @ N.t() - (ri3 * rn) @ g) * a1
                for i in range(3):
                    o[k, :, i] += (w * d[i]).sum(1)
    return out.reshape(-1)


def exact(case, seed):
    if case["kind"] == "batch":
        return [_sums(kt, src, nor, den, src, case["nrhs"]) for kt, src, nor, den in _members(case, seed)]
    nt, nrhs = case.get("nt") or case["n"], case.get("nrhs", 1)
    many = nrhs if case["kt"] not in (111, 121) else 1
    if float(case["n"]) * nt * _COST[case["kt"]] * many > 1.2e12:
        return None  # too many pairs for a direct sum in a few seconds
    src, nor, trg, den = _inputs(case, seed)
    return _sums(case["kt"], src, nor, den, trg, nrhs).cpu().numpy()
