"""Measured cases: the work a user of this framework has it do, through its public entry points.

A case is a dict of plain values; ``op`` names the family:

* ``einsum``   binary_einsum of two neighbouring MPS sites (theta = A·B)
* ``lattice``  binary_einsum of a 2-D lattice's boundary tensor with the next site
* ``svd``      tensor_svd_thin of a two-site tensor, truncated, and the approximation it gives
* ``canonize`` canonize(psi, site) of one MPS
* ``compress`` compress(psi; maxdim) of one MPS and the checks a user makes on the result
* ``tebd``     one brickwork layer of two-site gates on a batch of MPS, then amplitudes
* ``overlap``  overlap(psi, phi) and one amplitude
* ``dmrg``     one two-site DMRG sweep
* ``group``    canonize, compress, norm of a ragged batch of MPS
* ``serve``    a burst of queries to the query server

Singular vectors are defined up to a phase, so what depends on them is returned in the form
that does not (the approximated tensor, singular values, amplitudes); QR's Q and R follow
LAPACK's sign convention and come as they are.
"""

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tenet.jl_gb300"))

import tenetgb  # noqa: E402
from tenetgb import serve as tenet_serve  # noqa: E402
from tenetgb.group import MPSGroup  # noqa: E402

Z = np.array([[1, 0], [0, -1]], dtype=np.complex128)
X = np.array([[0, 1], [1, 0]], dtype=np.complex128)


def listed():
    return [
        # the smallest call: theta of two sites of a small MPS, where latency counts
        {"name": "einsum_chi12", "op": "einsum", "dtype": "complex128", "precision": "native", "l": 12, "k": 12, "r": 12},
        # the heavy step of contracting an 8x8 lattice of bond 8: the boundary tensor (8 open
        # legs) absorbs the next site, on the tensor cores
        {"name": "lattice_bond8_mixed", "op": "lattice", "precision": "mixed", "bond": 8, "legs": 8, "at": 3},
        # the same step of an odd-sized lattice in plain single precision, the accurate choice
        {"name": "lattice_bond7_fp32", "op": "lattice", "precision": "native", "bond": 7, "legs": 8, "at": 3},
        # truncated SVD of a two-site tensor, sizes not a power of two, double precision
        {"name": "svd_chi100", "op": "svd", "precision": "native", "l": 100, "r": 100, "keep": 100},
        # the plain small configuration: canonize an MPS of 32 sites, bond 64
        {"name": "canonize_L32_chi64", "op": "canonize", "L": 32, "chi": 64, "centre": 32},
        # the same MPS compressed to half its bond and checked
        {"name": "compress_L32_chi64", "op": "compress", "L": 32, "chi": 64, "maxdim": 32},
        # TEBD at bond 256: one MPS in double precision
        {"name": "tebd_fp64_L20_chi256", "op": "tebd", "precision": "native", "B": 1, "L": 20, "chi": 256, "start": 1,
         "reverse": False},
        # TEBD at bond 256: 16 circuits in lockstep, mixed precision (the headline workload's form)
        {"name": "tebd_mixed_b16_L28_chi256", "op": "tebd", "precision": "mixed", "B": 16, "L": 28, "chi": 256,
         "start": 1, "reverse": False},
        # overlap of two saturated MPS of the TEBD workload
        {"name": "overlap_L64_chi256", "op": "overlap", "L": 64, "chi_a": 256, "chi_b": 256},
        # ground-state search: one two-site sweep of a transverse-field Ising chain
        {"name": "dmrg2_L24_chi32", "op": "dmrg", "L": 24, "chi": 32, "h": 1.3},
        # many MPS of uneven length and bond dimension
        {"name": "group_16_chi8to72", "op": "group", "B": 16, "L_min": 12, "L_max": 28, "chi_min": 8, "chi_max": 72,
         "shape_seed": 5},
        # query serving: a burst of amplitudes, expectation values and overlaps
        {"name": "serve_burst64", "op": "serve", "precision": "native", "pairs": 2, "L_min": 24, "L_max": 48,
         "chi_max": 128, "queries": 64, "shape_seed": 6},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["einsum", "einsum", "lattice", "svd", "canonize", "compress", "tebd", "tebd", "overlap", "dmrg",
                     "group", "serve"])
    if op == "einsum":
        dtype, precision = rng.choice([("complex128", "native"), ("complex128", "mixed"), ("complex128", "split_bf16"),
                                       ("complex64", "native"), ("complex64", "mixed"), ("complex64", "tf32")])
        return {"op": op, "dtype": dtype, "precision": precision, "l": _log_int(rng, 6, 400), "k": _log_int(rng, 6, 400),
                "r": _log_int(rng, 6, 400)}
    if op == "lattice":
        legs = rng.randint(4, 8)
        return {"op": op, "precision": rng.choice(["native", "mixed", "tf32"]), "bond": rng.randint(4, 8), "legs": legs,
                "at": rng.randint(0, legs - 2)}
    if op == "svd":
        l, r = _log_int(rng, 8, 160), _log_int(rng, 8, 160)
        return {"op": op, "precision": rng.choice(["native", "native", "mixed"]), "l": l, "r": r,
                "keep": max(1, int(rng.uniform(0.3, 1.0) * min(l, r)))}
    if op == "canonize":
        L = rng.randint(8, 40)
        return {"op": op, "L": L, "chi": _log_int(rng, 8, 160), "centre": rng.choice([1, L // 2, L])}
    if op == "compress":
        chi = _log_int(rng, 8, 80)
        return {"op": op, "L": rng.randint(8, 32), "chi": chi, "maxdim": max(2, int(chi * rng.uniform(0.3, 0.8)))}
    if op == "tebd":
        precision = rng.choice(["native", "mixed"])
        return {"op": op, "precision": precision, "B": rng.choice([1, 2, 5]) if precision == "native" else rng.choice([1, 4, 16]),
                "L": rng.randint(8, 20), "chi": _log_int(rng, 12, 160), "start": rng.randint(1, 2),
                "reverse": rng.random() < 0.5}
    if op == "overlap":
        return {"op": op, "L": rng.randint(12, 64), "chi_a": _log_int(rng, 8, 256), "chi_b": _log_int(rng, 8, 256)}
    if op == "dmrg":
        return {"op": op, "L": rng.randint(10, 24), "chi": _log_int(rng, 8, 32), "h": round(rng.uniform(1.2, 1.6), 3)}
    if op == "group":
        return {"op": op, "B": rng.randint(4, 24), "L_min": 8, "L_max": rng.randint(12, 24), "chi_min": 8,
                "chi_max": rng.randint(24, 72), "shape_seed": rng.randint(0, 10**6)}
    return {"op": op, "precision": rng.choice(["native", "mixed"]), "pairs": rng.randint(1, 3), "L_min": 8,
            "L_max": rng.randint(16, 48), "chi_max": _log_int(rng, 16, 128), "queries": _log_int(rng, 4, 128),
            "shape_seed": rng.randint(0, 10**6)}


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _gauss(gen, n, dtype=torch.complex128):
    """n complex Gaussians of unit variance on the GPU."""
    return torch.randn(n, generator=gen, device="cuda", dtype=dtype)


class _Wrapped:
    """A library tensor shown to torch (column-major, flat) without a copy."""

    def __init__(self, t):
        self.t = t
        self.__cuda_array_interface__ = {"shape": (t.size,), "typestr": {16: "<c16", 8: "<c8"}[t.dtype.itemsize]
                                         if t.dtype.kind == "c" else "<f8",
                                         "data": (t.ptr, False), "version": 2}


def _out(t):
    return torch.as_tensor(_Wrapped(t), device="cuda")


def _in(flat, shape, inds):
    """A library tensor over a flat torch tensor in column-major order (which it keeps alive)."""
    t = tenetgb.DeviceTensor(tenetgb.default_context(), shape, np.complex128 if flat.dtype == torch.complex128 else np.complex64,
                             inds, ptr=flat.data_ptr())
    t.storage = flat
    return t


def _view(flat, shape):
    """The column-major tensor behind a flat buffer, as a torch view."""
    return flat.reshape(tuple(reversed(shape))).permute(*reversed(range(len(shape))))


def _bonds(L, chi, d=2):
    return [1] + [min(chi, d ** min(i, L - i, 40)) for i in range(1, L)] + [1]


def _split_sites(flat, b, d=2):
    """Site tensors (chi_l, d, chi_r) as numpy arrays in column-major order from one flat buffer."""
    host, out, o = flat.cpu().numpy(), [], 0
    for i in range(len(b) - 1):
        n = b[i] * d * b[i + 1]
        out.append(host[o:o + n].reshape((b[i], d, b[i + 1]), order="F"))
        o += n
    return out


def _gauss_mps(gen, L, chi, d=2):
    """Gaussian sites scaled so that the norm stays O(1), not in a canonical form."""
    b = _bonds(L, chi)
    parts = [_gauss(gen, b[i] * d * b[i + 1]) / math.sqrt(d * b[i]) for i in range(L)]
    return _split_sites(torch.cat(parts), b)


def _circuit_mps(gen, B, L, chi, d=2):
    """B random MPS of right-isometric sites: their Schmidt values fall from 1 to about 0.2, as
    those of a random circuit's state at its bond limit do.  The isometries are Gaussians
    orthogonalised by Newton-Schulz steps in single precision (the library brings the state
    to its canonical form)."""
    b = _bonds(L, chi)
    parts = []
    for i in range(L):
        g = _gauss(gen, B * b[i] * d * b[i + 1], torch.complex64).reshape(B, d * b[i + 1], b[i])
        g = g / (math.sqrt(b[i]) + math.sqrt(d * b[i + 1]))
        for _ in range(12 if i < L - 8 else 24):
            g = 1.5 * g - 0.5 * (g @ (g.mH @ g))
        parts.append(g.to(torch.complex128).reshape(B, -1))
    flat = torch.cat(parts, dim=1)
    return [_split_sites(flat[k], b) for k in range(B)]


def _gates(seed, count):
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(count):
        q, r = np.linalg.qr(rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4)))
        q = q * (np.diagonal(r) / np.abs(np.diagonal(r)))[None, :]
        out.append(np.ascontiguousarray(q.reshape(2, 2, 2, 2)))
    return out


def _bit_strings(seed, L, count):
    rng = np.random.default_rng(seed + 77)
    return ["".join(rng.choice(["0", "1"], L)) for _ in range(count)]


def _lattice_labels(case):
    """Boundary tensor legs a0..; it shares leg ``at`` and its last leg with the site (x, y, u, v)."""
    legs = ["a%d" % i for i in range(case["legs"])]
    legs[case["at"]] = "x"
    legs[-1] = "y"
    return legs


def _group_shapes(case):
    rng = np.random.default_rng(case["shape_seed"])
    Ls = [int(v) for v in rng.integers(case["L_min"], case["L_max"] + 1, case["B"])]
    chis = [int(round(math.exp(v))) for v in rng.uniform(math.log(case["chi_min"]), math.log(case["chi_max"]), case["B"])]
    return Ls, chis


def _pool_shapes(case):
    rng = np.random.default_rng(case["shape_seed"])
    out = []
    for _ in range(case["pairs"]):
        L = int(rng.integers(case["L_min"], case["L_max"] + 1))
        for _ in range(2):
            out.append((L, max(8, int(case["chi_max"] * rng.uniform(0.5, 1.0)))))
    return out


def _queries(case, shapes, seed):
    """(kind, mps, argument) by the served mix: 60 % amplitudes, 30 % <O_i>, 10 % overlaps."""
    rng = np.random.default_rng(seed + 7)
    out = []
    for q in range(case["queries"]):
        m = int(rng.integers(len(shapes)))
        kind = ("amp", "amp", "exp", "amp", "amp", "exp", "amp", "exp", "amp", "ovl")[q % 10]
        if kind == "amp":
            out.append((kind, m, rng.integers(0, 2, shapes[m][0])))
        elif kind == "exp":
            o = rng.standard_normal((2, 2)) + 1j * rng.standard_normal((2, 2))
            out.append((kind, m, (int(rng.integers(1, shapes[m][0] + 1)), (o + o.conj().T) / 2)))
        else:
            out.append((kind, 2 * (m // 2), 2 * (m // 2) + 1))
    return out


def _inputs(case, seed):
    """The plain arrays of a case (what exact() starts from too)."""
    op = case["op"]
    gen = _generator(seed)
    if op == "einsum":
        dt = getattr(torch, case["dtype"])
        return {"A": _gauss(gen, case["l"] * 2 * case["k"], dt) / math.sqrt(2 * case["k"]),
                "B": _gauss(gen, case["k"] * 2 * case["r"], dt) / math.sqrt(2 * case["r"])}
    if op == "lattice":
        D = case["bond"]
        return {"A": _gauss(gen, D ** case["legs"], torch.complex64) / D, "B": _gauss(gen, D**4, torch.complex64) / D}
    if op == "svd":
        # theta of two sites whose shared bond carries a decaying spectrum
        l, r = case["l"], case["r"]
        k = 2 * min(l, r)
        a, b = _gauss(gen, 2 * l * k).reshape(k, 2 * l), _gauss(gen, 2 * r * k).reshape(2 * r, k)
        w = torch.exp(-5.0 * torch.arange(k, device="cuda", dtype=torch.float64) / k) / math.sqrt(l * r)
        return {"A": ((b * w[None, :]) @ a).reshape(-1)}  # column-major (l, 2, 2, r)
    if op in ("canonize", "compress"):
        return {"sites": _gauss_mps(gen, case["L"], case["chi"])}
    if op == "tebd":
        n = (case["L"] - case["start"] + 1) // 2
        return {"sites": _circuit_mps(gen, case["B"], case["L"], case["chi"]),
                "gates": _gates(seed, n), "bits": _bit_strings(seed, case["L"], 4)}
    if op == "overlap":
        return {"a": _gauss_mps(gen, case["L"], case["chi_a"]), "b": _gauss_mps(gen, case["L"], case["chi_b"]),
                "bits": _bit_strings(seed, case["L"], 1)[0]}
    if op == "dmrg":
        return {"sites": _gauss_mps(gen, case["L"], case["chi"])}
    if op == "group":
        return {"instances": [_gauss_mps(gen, L, chi) for L, chi in zip(*_group_shapes(case))]}
    shapes = _pool_shapes(case)
    return {"pool": [_gauss_mps(gen, L, chi) for L, chi in shapes], "queries": _queries(case, shapes, seed)}


def prepare(case, seed):
    op, x = case["op"], _inputs(case, seed)
    s = {"case": case}
    if op == "einsum":
        s["A"] = _in(x["A"], (case["l"], 2, case["k"]), ["l", "p", "k"])
        s["B"] = _in(x["B"], (case["k"], 2, case["r"]), ["k", "q", "r"])
    elif op == "lattice":
        D = case["bond"]
        s["A"] = _in(x["A"], (D,) * case["legs"], _lattice_labels(case))
        s["B"] = _in(x["B"], (D,) * 4, ["x", "y", "u", "v"])
    elif op == "svd":
        s["A"] = _in(x["A"], (case["l"], 2, 2, case["r"]), ["l", "p", "q", "r"])
    elif op in ("canonize", "compress", "dmrg"):
        s["psi"] = tenetgb.MPS(x["sites"], max_bond=case["chi"])
        if op == "dmrg":
            s["H"] = tenetgb.ising_1d_mpo(case["L"], case["h"], 1.0)
    elif op == "tebd":
        s["psi"] = tenetgb.MPS.batched(x["sites"], max_bond=case["chi"], precision=case["precision"])
        # a running circuit has its orthogonality centre where the layer begins
        s["psi"].canonize_(case["L"] if case["reverse"] else 1)
        s["layer"] = (case["start"], x["gates"], case["reverse"])
        s["bits"] = x["bits"]
    elif op == "overlap":
        s["a"], s["b"], s["bits"] = tenetgb.MPS(x["a"]), tenetgb.MPS(x["b"]), x["bits"]
    elif op == "group":
        s["instances"] = x["instances"]
        s["maxdim"] = [max(4, chi // 2) for chi in _group_shapes(case)[1]]
    else:
        s["server"] = tenet_serve.Server(work_bytes=1 << 28, precision=case["precision"])
        s["ids"] = [s["server"].add_mps(m) for m in x["pool"]]
        s["queries"] = x["queries"]
    return s


# ---------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    op = case["op"]
    if op == "einsum":
        return _out(tenetgb.binary_einsum(s["A"], s["B"], dims=["k"], precision=case["precision"]))
    if op == "lattice":
        return _out(tenetgb.binary_einsum(s["A"], s["B"], dims=["x", "y"], precision=case["precision"]))
    if op == "svd":
        u, sv, v = tenetgb.tensor_svd_thin(s["A"], ["l", "p"], ["q", "r"], "s", precision=case["precision"],
                                           maxdim=case["keep"])
        return {"s": _out(sv), "approximation": _out(tenetgb.binary_einsum(tenetgb.hadamard(u, sv), v, dims=["s"]))}
    if op == "canonize":
        return tenetgb.canonize(s["psi"], case["centre"]).sites()
    if op == "compress":
        phi = tenetgb.compress(s["psi"], maxdim=case["maxdim"])
        lam = phi.lambda_()
        phi.canonize_(case["L"])
        return {"bonds": np.array(phi.bondsizes()), "schmidt": lam, "overlap": phi.overlap(s["psi"]) * np.ones(1),
                "z": phi.local_expectations(Z)}
    if op == "tebd":
        phi = s["psi"].copy()
        phi.evolve_brickwork_([s["layer"]], maxdim=case["chi"], threshold=1e-12)
        amps = np.stack([np.atleast_1d(phi.amplitude(b)) for b in s["bits"]], axis=1)
        return {"bonds": np.array(phi.bondsizes()), "amplitudes": [a for a in amps]}
    if op == "overlap":
        return {"overlap": s["a"].overlap(s["b"]) * np.ones(1), "amplitude": s["a"].amplitude(s["bits"]) * np.ones(1)}
    if op == "dmrg":
        phi, energy, history = tenetgb.dmrg(s["psi"], s["H"], 1, method=tenetgb.Dmrg2, maxdim=case["chi"], history=True)
        return {"energy": float(energy), "history": history, "x": phi.local_expectations(X)}
    if op == "group":
        g = MPSGroup.from_arrays(s["instances"])
        norms = g.canonize_compress_norm(s["maxdim"])
        return {"norms": norms, "schmidt": [g.lambda_(b) for b in range(g.B)]}
    sv, tickets = s["server"], []
    for kind, m, arg in s["queries"]:
        if kind == "amp":
            tickets.append(sv.submit_amplitude(s["ids"][m], arg))
        elif kind == "exp":
            tickets.append(sv.submit_expectation(s["ids"][m], *arg))
        else:
            tickets.append(sv.submit_overlap(s["ids"][m], s["ids"][arg]))
    got = {"amp": [], "exp": [], "ovl": []}
    for (kind, _, _), t in zip(s["queries"], tickets):
        got[kind].append(sv.wait(t)[0])
    # a mixed server's amplitudes and overlaps carry single precision
    dt = np.complex128 if case["precision"] == "native" else np.complex64
    return {k: np.array(v, dtype=np.complex128 if k == "exp" else dt) for k, v in got.items() if v}


# ---------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------
def _gemm(m, n, k):
    return 8.0 * m * n * k


def _qr(m, n):
    m, n = max(m, n), min(m, n)
    return 8.0 * (2.0 * m * n * n - 2.0 * n**3 / 3.0)


def _svd(m, n):
    m, n = max(m, n), min(m, n)
    return 4.0 * (4.0 * m * m * n + 8.0 * m * n * n + 9.0 * n**3)


def _sites_bytes(b, d=2):
    return sum(16.0 * b[i] * d * b[i + 1] for i in range(len(b) - 1))


def _sweep(b, maxdim=None, d=2):
    """QR sweep over an MPS of bonds b, and with maxdim the truncated SVD sweep back."""
    f = sum(_qr(d * b[i + 1], b[i]) + _gemm(d * b[i - 1], b[i], b[i]) for i in range(1, len(b) - 1))
    if maxdim:
        prev = 1
        for i in range(1, len(b) - 1):
            r = min(maxdim, prev * d, b[i])
            f += _svd(prev * d, b[i]) + _gemm(r, b[i], b[i]) + _gemm(r, d * b[i + 1], b[i])
            prev = r
    return f


def _overlap(a, b, d=2):
    return sum(_gemm(b[i], d * a[i + 1], a[i]) + _gemm(b[i + 1], a[i + 1], d * b[i]) for i in range(len(a) - 1))


def work(case):
    op = case["op"]
    if op == "einsum":
        l, k, r, e = case["l"], case["k"], case["r"], 16 if case["dtype"] == "complex128" else 8
        return {"bytes": e * (2.0 * l * k + 2.0 * k * r + 4.0 * l * r), "flops": _gemm(2 * l, 2 * r, k)}
    if op == "lattice":
        D, n = float(case["bond"]), case["legs"]
        return {"bytes": 8 * (2 * D**n + D**4), "flops": _gemm(D ** (n - 2), D * D, D * D)}
    if op == "svd":
        m, n, r = 2.0 * case["l"], 2.0 * case["r"], case["keep"]
        return {"bytes": 32 * m * n + 8 * r, "flops": _svd(m, n) + _gemm(m, n, r)}
    if op == "canonize":
        b = _bonds(case["L"], case["chi"])
        f, c = 0.0, case["centre"]
        for i in range(1, case["L"]):
            f += (_qr(2 * b[i - 1], b[i]) + _gemm(b[i], 2 * b[i + 1], b[i])) if i < c else (
                _qr(2 * b[i + 1], b[i]) + _gemm(2 * b[i - 1], b[i], b[i]))
        return {"bytes": 2 * _sites_bytes(b), "flops": f}
    if op == "compress":
        b = _bonds(case["L"], case["chi"])
        c = _bonds(case["L"], case["maxdim"])
        return {"bytes": _sites_bytes(b) + _sites_bytes(c), "flops": _sweep(b, case["maxdim"]) + _overlap(b, c) + 2 * _overlap(c, c)}
    if op == "tebd":
        b, f = _bonds(case["L"], case["chi"]), 0.0
        for a in range(case["start"], case["L"], 2):
            m, n = 2 * b[a - 1], 2 * b[a + 1]
            f += _gemm(m, n, b[a]) + 32.0 * m * n + _svd(m, n) + _gemm(min(case["chi"], m, n), n, m)
            f += _qr(m, b[a]) + _gemm(b[a], 2 * b[a + 1], b[a])
        return {"bytes": 2.0 * case["B"] * _sites_bytes(b), "flops": f * case["B"]}
    if op == "overlap":
        a, b = _bonds(case["L"], case["chi_a"]), _bonds(case["L"], case["chi_b"])
        return {"bytes": _sites_bytes(a) + _sites_bytes(b), "flops": min(_overlap(a, b), _overlap(b, a))}
    if op == "dmrg":
        b, f = _bonds(case["L"], case["chi"]), 0.0
        for i in range(1, case["L"]):  # 2 updates per bond and sweep, 6 products with H each
            m, n = 2.0 * b[i - 1], 2.0 * b[i + 1]
            f += 2 * (6 * (_gemm(m, 3 * n, b[i - 1]) + _gemm(m, n, 3 * b[i + 1])) + _svd(m, n))
        return {"bytes": 2 * _sites_bytes(b), "flops": f}
    if op == "group":
        f = by = 0.0
        for L, chi in zip(*_group_shapes(case)):
            b = _bonds(L, chi)
            f += 2 * _sweep(b) + _sweep(b, max(4, chi // 2)) - _sweep(b)
            by += 2 * _sites_bytes(b)
        return {"bytes": by, "flops": f}
    f = by = 0.0
    shapes = _pool_shapes(case)
    for kind, m, arg in _queries(case, shapes, 0):
        b = _bonds(*shapes[m])
        if kind == "amp":
            f += _sites_bytes(b) / 2
        elif kind == "exp":
            f += 8.0 * 4 * shapes[m][1] ** 2
            by += 64.0 * shapes[m][1] ** 2
        else:
            f += _overlap(b, _bonds(*shapes[arg]))
    return {"bytes": by + sum(_sites_bytes(_bonds(*x)) for x in shapes), "flops": f}


# ---------------------------------------------------------------------------------------
# the same in plain 64-bit numpy / torch
# ---------------------------------------------------------------------------------------
def _right_canonical(sites):
    out = [np.array(s) for s in sites]
    for i in range(len(out) - 1, 0, -1):
        l, d, r = out[i].shape
        q, rr = np.linalg.qr(out[i].reshape(l, d * r).conj().T)
        out[i] = q.conj().T.reshape(-1, d, r)
        out[i - 1] = np.tensordot(out[i - 1], rr.conj().T, (2, 0))
    return out


def _np_overlap(a, b):
    """<b|a>"""
    f = np.ones((1, 1), complex)
    for x, y in zip(a, b):
        t = np.tensordot(f, x, (1, 0))
        f = np.tensordot(y.conj(), t, ((0, 1), (0, 1)))
    return f[0, 0]


def _np_expect(sites, op):
    L = len(sites)
    right = [None] * (L + 1)
    right[L] = np.ones((1, 1), complex)
    for i in range(L - 1, -1, -1):
        right[i] = np.einsum("asb,bd,csd->ac", sites[i], right[i + 1], sites[i].conj(), optimize=True)
    f, out = np.ones((1, 1), complex), []
    for i in range(L):
        t = np.einsum("ca,asb->csb", f, sites[i])
        out.append(np.einsum("csb,ts,bd,ctd->", t, op, right[i + 1], sites[i].conj(), optimize=True))
        f = np.einsum("csb,csd->db", t, sites[i].conj(), optimize=True)
    return np.array(out) / f[0, 0]


def _np_amplitude(sites, bits):
    v = np.ones((1,), complex)
    for s, c in zip(sites, bits):
        v = v @ s[:, int(c), :]
    return v[0]


def _svd_sweep(sites, maxdim):
    """Truncated left-to-right SVD sweep of a right-canonical MPS; the last Schmidt values."""
    out, s = [np.array(x) for x in sites], None
    for i in range(len(out) - 1):
        l, d, r = out[i].shape
        u, s, v = np.linalg.svd(out[i].reshape(l * d, r), full_matrices=False)
        k = min(maxdim, s.size)
        u, s, v = u[:, :k], s[:k], v[:k]
        out[i] = u.reshape(l, d, k)
        out[i + 1] = np.tensordot(s[:, None] * v, out[i + 1], (1, 0))
    return out, s


def _np_layer(sites, gates, start, reverse, chi):
    L = len(sites)
    if reverse:  # mirrored chain: the sites, the gates and their legs the other way round
        flip = [np.transpose(s, (2, 1, 0)) for s in reversed(sites)]
        g = [np.transpose(G, (1, 0, 3, 2)) for G in reversed(gates)]
        last = start + 2 * (len(gates) - 1)
        return [np.transpose(s, (2, 1, 0)) for s in reversed(_np_layer(flip, g, L - last, False, chi))]
    out = _right_canonical(sites)
    centre = 0
    for q, G in enumerate(gates):
        a = start - 1 + 2 * q
        while centre < a:
            l, d, r = out[centre].shape
            u, rr = np.linalg.qr(out[centre].reshape(l * d, r))
            out[centre] = u.reshape(l, d, -1)
            out[centre + 1] = np.tensordot(rr, out[centre + 1], (1, 0))
            centre += 1
        th = np.einsum("abcd,lcdr->labr", G, np.tensordot(out[a], out[a + 1], (2, 0)), optimize=True)
        l, d, _, r = th.shape
        u, s, v = np.linalg.svd(th.reshape(l * d, d * r), full_matrices=False)
        k = max(1, int(np.sum(s[:chi] > 1e-12)))
        out[a], out[a + 1] = u[:, :k].reshape(l, d, k), (s[:k, None] * v[:k]).reshape(k, d, r)
        centre = a + 1
    return out


def exact(case, seed):
    op = case["op"]
    if op in ("dmrg",):  # the unfinished eigensolves follow every detail of the iteration
        return None
    x = _inputs(case, seed)
    if op == "einsum":
        a = _view(x["A"].to(torch.complex128), (case["l"] * 2, case["k"]))
        b = _view(x["B"].to(torch.complex128), (case["k"], 2 * case["r"]))
        return (a @ b).T.reshape(-1)
    if op == "lattice":
        D, labels = case["bond"], _lattice_labels(case)
        a = _view(x["A"].to(torch.complex128), (D,) * case["legs"])
        b = _view(x["B"].to(torch.complex128), (D,) * 4)
        c = torch.tensordot(a, b, dims=([labels.index("x"), labels.index("y")], [0, 1]))
        return c.permute(*reversed(range(c.dim()))).reshape(-1)
    if op == "svd":
        a = _view(x["A"], (2 * case["l"], 2 * case["r"])).cpu().numpy()
        u, s, v = np.linalg.svd(a, full_matrices=False)
        k = case["keep"]
        return {"s": s[:k], "approximation": ((u[:, :k] * s[:k]) @ v[:k]).reshape(-1, order="F")}
    if op == "canonize":
        out, c = [np.array(s) for s in x["sites"]], case["centre"] - 1
        for i in range(c):
            l, d, r = out[i].shape
            if r == 1:
                continue
            q, rr = np.linalg.qr(out[i].reshape((l * d, r), order="F"))
            out[i] = q.reshape((l, d, -1), order="F")
            out[i + 1] = np.tensordot(rr, out[i + 1], (1, 0))
        for i in range(len(out) - 1, c, -1):
            l, d, r = out[i].shape
            q, rr = np.linalg.qr(out[i].reshape((l, d * r), order="F").conj().T)
            out[i] = q.conj().T.reshape((-1, d, r), order="F")
            out[i - 1] = np.tensordot(out[i - 1], rr.conj().T, (2, 0))
        return out
    if op == "compress":
        phi, s = _svd_sweep(_right_canonical(x["sites"]), case["maxdim"])
        return {"bonds": None, "schmidt": s, "overlap": _np_overlap(phi, x["sites"]) * np.ones(1), "z": _np_expect(phi, Z)}
    if op == "tebd":
        limit = 1e11  # flops: about ten seconds of numpy
        done = max(0, min(case["B"], int(limit / (work(case)["flops"] / case["B"]))))
        if done == 0:
            return None
        amps = []
        for b in range(done):
            phi = _np_layer(x["sites"][b], x["gates"], case["start"], case["reverse"], case["chi"])
            amps.append(np.array([_np_amplitude(phi, bits) for bits in x["bits"]]))
        return {"bonds": None, "amplitudes": amps + [None] * (case["B"] - done)}
    if op == "overlap":
        return {"overlap": _np_overlap(x["a"], x["b"]) * np.ones(1), "amplitude": _np_amplitude(x["a"], x["bits"]) * np.ones(1)}
    if op == "group":
        norms, lams = [], []
        for sites, chi in zip(x["instances"], _group_shapes(case)[1]):
            phi, s = _svd_sweep(_right_canonical(sites), max(4, chi // 2))
            norms.append(np.linalg.norm(phi[-1]))
            lams.append(s)
        return {"norms": np.array(norms), "schmidt": lams}
    got = {"amp": [], "exp": [], "ovl": []}
    for kind, m, arg in x["queries"]:
        psi = x["pool"][m]
        if kind == "amp":
            got[kind].append(_np_amplitude(psi, "".join(str(int(v)) for v in arg)))
        elif kind == "exp":
            got[kind].append(_np_expect(psi, arg[1])[arg[0] - 1])
        else:
            got[kind].append(_np_overlap(psi, x["pool"][arg]))
    return {k: np.array(v) for k, v in got.items() if v}
