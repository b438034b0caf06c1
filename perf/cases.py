"""Matvec cases of the framework, through its public Python entry points.

Every case is one matvec val = G den on a fixed geometry, the call that an
iterative boundary-integral solver makes over and over: the session (tree,
interaction lists, operators on the device) is what its program keeps, the
densities are new.  A case is

  form      "plain" (complex128 in and out, every pass in FP64) or "mixed"
            (complex64 in and out, FP32 state and tensor-core translations)
  io        "device" (tensors of the GPU, the caller's stream), "host" (host
            arrays, copies included) or "batch" (several mixed instances in
            one merged call, device tensors)
  geometry  "sphere", "ellipsoid" (semi-axes 1/2, 1/4, 1/8 of K) or "cluster"
            (half on a sphere, half in three tight blobs, a few coincident
            points: an adaptive tree with all four near-field lists)
  K, n      root-box width in wavelengths and number of points
  accu      1, 2, 3: 4, 6, 8 equivalent points per box edge
  kernel    0: exp(ir)/r, 1: exp(ir)
  ptsmax    points per leaf at most

Sizes are those of the repository's benchmark (sphere K=64, N=321,699, P=6),
of its test fixtures (K=4, 8, 16; N=1500 .. 5000) and of the mixes that its
batch and server tests use (25 points per square wavelength).
"""
import math
import os
import tempfile

import numpy as np
import torch

from ddfmm_b200 import _lib, precompute, wave3d

SHRINK = 1.0 - 1e-12  # keeps the surface off the faces of the root box


def _case(name, form, io, geometry, K, n, accu=1, kernel=0, ptsmax=100, count=1):
    return {"name": name, "form": form, "io": io, "geometry": geometry, "K": K, "n": n, "accu": accu,
            "kernel": kernel, "ptsmax": ptsmax, "count": count}


def listed():
    return [
        # the smallest instance: a few hundred boxes, where launches and latency count
        _case("plain_sphere_k4_p4", "plain", "device", "sphere", 4, 1500),
        # the driver's own small run, host arrays in and out as Wave3d.eval is called
        _case("plain_host_sphere_k8_p4", "plain", "host", "sphere", 8, 5000),
        # adaptive geometry: small leaves, deep low-frequency tree, U, V, W and X lists
        _case("plain_cluster_k8_p4", "plain", "device", "cluster", 8, 12007, ptsmax=8),
        # highest accuracy (P = 8) on a small surface
        _case("plain_sphere_k4_p8", "plain", "device", "sphere", 4, 1500, accu=3),
        # the other kernel, two high-frequency widths
        _case("plain_expr_sphere_k16_p4", "plain", "device", "sphere", 16, 20106, kernel=1),
        # an ordinary FP64 solve on a ragged, elongated surface
        _case("plain_ellipsoid_k32_p6", "plain", "device", "ellipsoid", 32, 56251, accu=2),
        # the benchmark's instance, FP64
        _case("plain_sphere_k64_p6", "plain", "device", "sphere", 64, 321699, accu=2),
        # mixed form: smallest, ordinary, the benchmark's instance
        _case("mixed_sphere_k8_p4", "mixed", "device", "sphere", 8, 5000),
        _case("mixed_ellipsoid_k16_p6", "mixed", "device", "ellipsoid", 16, 20106, accu=2),
        _case("mixed_sphere_k64_p6", "mixed", "device", "sphere", 64, 321699, accu=2),
        # many uneven instances in one call: spheres and ellipsoids, K cycling 4, 8, 16, 32 up to K
        _case("mixed_batch_k32_p6", "mixed", "batch", "sphere", 32, 80425, accu=2, count=8),
    ]


def draw(rng):
    form = rng.choice(["plain", "plain", "mixed"])
    geometry = rng.choice(["sphere", "sphere", "ellipsoid", "ellipsoid", "cluster"])
    accu = rng.choice([1, 1, 2, 2, 2, 3])
    kernel = 1 if accu == 1 and rng.random() < 0.25 else 0
    # K is a power of two; the widest boxes of the dearer operators are left out
    K = rng.choice([4, 8] if accu == 3 or geometry == "cluster" else [4, 8, 16, 32] if kernel else [4, 8, 16, 32, 64])
    # 6 to 30 points per square wavelength of the sphere of diameter K, 1000 points at least
    lo, hi = max(1000.0, 6 * math.pi * K * K), max(3000.0, 25 * math.pi * K * K)
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    io = rng.choice(["device", "device", "host"])
    if form == "mixed" and accu == 2 and K <= 32 and geometry != "cluster" and rng.random() < 0.4:
        return _drawn(_case("", form, "batch", "sphere", K, n, accu=accu, count=rng.randint(2, 8)))
    ptsmax = rng.choice([8, 16, 40]) if geometry == "cluster" else rng.choice([50, 100, 100])
    return _drawn(_case("", form, io, geometry, K, n, accu=accu, kernel=kernel, ptsmax=ptsmax))


def _drawn(case):
    return {k: v for k, v in case.items() if k != "name"}


def _instances(case):
    """(geometry, K, n, seed shift) of each instance: one, or a batch's mix."""
    if case["io"] != "batch":
        return [(case["geometry"], case["K"], case["n"], 0)]
    Ks = [k for k in (4, 8, 16, 32) if k <= case["K"]]
    out = []
    for j in range(case["count"]):
        K = Ks[-1 - j % len(Ks)]
        out.append(("sphere" if j % 2 == 0 else "ellipsoid", K, max(500, case["n"] * K * K // (case["K"] ** 2)), j))
    return out


def _points(geometry, K, n, seed):
    rng = np.random.default_rng([seed, n, K])
    if geometry == "sphere":
        v = rng.standard_normal((n, 3))
        v /= np.linalg.norm(v, axis=1, keepdims=True)
        return v * (0.5 * K * SHRINK)
    if geometry == "ellipsoid":  # uniform by area: rejection on the area element
        ax = np.array([0.5, 0.25, 0.125]) * (K * SHRINK)
        got, have = [], 0
        while have < n:
            u = rng.standard_normal((2 * n, 3))
            u /= np.linalg.norm(u, axis=1, keepdims=True)
            keep = rng.random(2 * n) * ax.prod() / ax.min() < ax.prod() * np.linalg.norm(u / ax, axis=1)
            got.append(u[keep] * ax)
            have += int(keep.sum())
        return np.concatenate(got)[:n]
    h = n // 2
    v = rng.standard_normal((h, 3))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    mid = np.array([[0.2, 0.1, -0.15], [-0.25, 0.2, 0.1], [0.05, -0.3, 0.3]]) * K
    blob = mid[np.arange(n - h - 8) % 3] + rng.standard_normal((n - h - 8, 3)) * (0.02 * K)
    pts = np.clip(np.concatenate([v * 0.4 * K, blob]), -0.5 * K * SHRINK, 0.5 * K * SHRINK)
    return np.concatenate([pts, pts[rng.choice(n - 8, size=8, replace=False)]])


def _density(n, seed, dtype):
    """N(0, 1) real and imaginary parts, as the benchmark's densities."""
    rng = np.random.default_rng([seed, n, 77])
    return (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(dtype)


def _cells(K):
    return min(8, K)


def _operators(case):
    """The operator files of the case's kernel and accuracy, made once per
    machine by the library's generator and kept in a scratch folder: files
    from another machine differ in the last bits of their factors."""
    folder = os.path.join(tempfile.gettempdir(), "ddfmm_operators_%d" % os.getuid())
    widest = 8 if case["accu"] < 3 and case["kernel"] == 0 else 4 if case["accu"] < 3 else 1
    return precompute.ensure_operators(folder, case["kernel"], case["accu"], widest)


def _session(case, pos, K):
    ld, hd = _operators(case)
    mlib = wave3d.Mlib3d()
    mlib.kernel = case["kernel"]
    mlib.setup({"-mlib3d_ldname": ld, "-mlib3d_hdname": hd, "-mlib3d_NPQ": "4"})
    w = wave3d.Wave3d(precision=_lib.PLAIN_FP64 if case["form"] == "plain" else _lib.MIXED)
    w.posptr, w.kernel, w.mlibptr, w.geomprtn = pos, case["kernel"], mlib, _cells(K)
    w.setup({"-wave3d_ACCU": str(case["accu"]), "-wave3d_NPQ": "4", "-wave3d_K": repr(float(K)),
             "-wave3d_ctr": "0 0 0", "-wave3d_ptsmax": str(case["ptsmax"]),
             "-wave3d_maxlevel": str(int(round(math.log2(K))) + 6)})
    return w


def prepare(case, seed):
    c64 = case["form"] == "mixed"
    dtype = np.complex64 if c64 else np.complex128
    waves, dens = [], []
    for geometry, K, n, j in _instances(case):
        waves.append(_session(case, _points(geometry, K, n, seed + 1000 * j), K))
        dens.append(_density(n, seed + 1000 * j, dtype))
    s = {"io": case["io"], "c64": c64, "waves": waves, "stream": torch.cuda.Stream()}
    if case["io"] == "host":
        s["den"], s["val"] = dens[0], np.zeros_like(dens[0])
        return s
    s["den"] = [torch.from_numpy(d).cuda() for d in dens]
    s["val"] = [torch.zeros_like(d) for d in s["den"]]
    if case["io"] == "batch":
        s["batch"] = wave3d.Batch(waves)
    torch.cuda.synchronize()
    return s


def run(s):
    if s["io"] == "host":
        s["waves"][0].eval(s["den"], s["val"])
        return s["val"]
    stream = s["stream"].cuda_stream
    if s["io"] == "batch":
        s["batch"].eval_device([d.data_ptr() for d in s["den"]], [v.data_ptr() for v in s["val"]], stream)
        return s["val"]
    s["waves"][0].eval_device(s["den"][0].data_ptr(), s["val"][0].data_ptr(), stream, s["c64"])
    return s["val"][0]


def work(case):
    """Points, densities and values once; the operations of the method's own
    counts on this geometry (host-only tree): 8 r^2 for each translation of a
    (box, wedge) of rank r = 45, 85, 140 at P = 4, 6, 8 -- the far pairs, and
    one skeleton product and about four child translations each way -- and 8
    per frequency of each pair of the V list.  The near field is small."""
    rank = {1: 45.0, 2: 85.0, 3: 140.0}[case["accu"]]
    grid = {1: 8 ** 3, 2: 12 ** 3, 3: 16 ** 3}[case["accu"]]
    size = 8 if case["form"] == "mixed" else 16
    total_bytes = flops = 0.0
    for geometry, K, n, j in _instances(case):
        t = _lib.tree_stats(_points(geometry, K, n, 1000 * j), float(K), case["ptsmax"],
                            int(round(math.log2(K))) + 6, _cells(K))
        total_bytes += n * (24.0 + 2 * size)
        for level in t["levels"]:
            flops += 8 * rank * rank * (level["far_pairs"] + 5.0 * (level["out_dirs"] + level["inc_dirs"]))
            flops += 8 * grid * level["v_pairs"]
        flops += 20.0 * n * 60
    return {"bytes": total_bytes, "flops": flops}


def _direct(pos, den, kernel):
    """sum_j G(p_i, p_j) den_j in 64 bits; coincident points count as r = 1."""
    p = torch.from_numpy(pos).cuda()
    d = torch.view_as_real(torch.from_numpy(den.astype(np.complex128)).cuda())
    n = p.shape[0]
    x, y, z = (p[:, k].contiguous() for k in range(3))
    out = torch.empty((n, 2), dtype=torch.float64, device="cuda")
    step = max(1, min(n, (1 << 27) // n))
    for a in range(0, n, step):
        r = (x[a:a + step, None] - x).square_()
        r += (y[a:a + step, None] - y).square_()
        r += (z[a:a + step, None] - z).square_()
        r[r < 1e-16] = 1.0
        r.sqrt_()
        ph = r * (2 * math.pi)
        re, im = torch.cos(ph), torch.sin(ph)
        if kernel == 0:
            re /= r
            im /= r
        u, v = re @ d, im @ d
        out[a:a + step, 0] = u[:, 0] - v[:, 1]
        out[a:a + step, 1] = u[:, 1] + v[:, 0]
    return torch.view_as_complex(out)


def exact(case, seed):
    """The direct sum.  None for exp(ir), where the method's own error is some
    tens of percent (its low-frequency scheme represents Helmholtz fields and
    exp(ir) is not one), and where the sum would take too long."""
    if case["kernel"] == 1:
        return None
    got = []
    for geometry, K, n, j in _instances(case):
        if n > 150000:
            return None
        den = _density(n, seed + 1000 * j, np.complex64 if case["form"] == "mixed" else np.complex128)
        got.append(_direct(_points(geometry, K, n, seed + 1000 * j), den, case["kernel"]))
    return got if case["io"] == "batch" else got[0].cpu().numpy() if case["io"] == "host" else got[0]
