"""Performance cases: the work a user of permgpu has it do, timed through the
public entry points.

  listed()            the cases that are timed
  draw(rng)           one more case of the same ranges
  prepare(case, s)    inputs on seed s, as a program holds them before the call
  run(state)          one pass through the public entry points
  work(case)          bytes and operations that one pass cannot do without
  exact(case, s)      the floating results in 64 bits, by another algorithm

Integer results come back as little-endian two's-complement bytes, so that
values of any width compare exactly.
"""

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "rivin-perm_gb300"))

import permgpu  # noqa: E402
from permgpu import batch, f64, mod3  # noqa: E402

RESULT_BYTES = 256     # widest integer result: 25 rows of 25 entries of 41 bits

# Box grids whose biadjacency matrices (half the vertices) have orders 18..40;
# an axis is periodic when its length is even and above 2.
GRIDS = ("3x4x3", "6x6", "4x4x3", "6x4x2", "6x8", "6x10", "5x6x2", "8x8", "4x4x4", "5x7x2",
         "6x4x3", "8x10", "4x4x5")


def listed():
    return [
        # one small matrix, the whole call: latency and launches
        {"name": "generic8", "kind": "generic", "n": 8, "mag": 8},
        # the 24x24 configuration: one short launch
        {"name": "generic24", "kind": "generic", "n": 24, "mag": 8},
        # the headline: exact permanent of a 32x32 matrix, entries in [-8, 8]
        {"name": "generic32", "kind": "generic", "n": 32, "mag": 8},
        # entries far beyond 32-bit row sums: residues and CRT, odd order
        {"name": "wide25", "kind": "generic", "n": 25, "mag": (1 << 38) + 11},
        # one Schur residue of prime order, through the extension drop-in
        {"name": "schur37", "kind": "schur", "n": 37},
        # perfect matchings of a 4x4x5 grid with a few bonds missing: a sparse 0/1
        # matrix, the largest call
        {"name": "grid40", "kind": "grid", "dims": "4x4x5"},
        # a dense 0/1 matrix
        {"name": "bernoulli36", "kind": "bernoulli", "n": 36, "density": 0.5},
        # many uneven matrices in one call, entries in [-3, 3]
        {"name": "batch1024", "kind": "batch", "count": 1024, "n_lo": 12, "n_hi": 26, "mag": 3},
        # FP64 permanents of a batch, forward and backward
        {"name": "grad26", "kind": "real", "n": 26, "batch": 16, "grad": True},
        # complex permanents of a batch, odd order, forward only
        {"name": "complex21", "kind": "complex", "n": 21, "batch": 32},
        # exact rook polynomial of a 0/1 board, odd order
        {"name": "rook25", "kind": "rook", "n": 25, "density": 0.5},
        # permanents modulo 3 one after the other, rows wider than one word, odd order
        {"name": "mod3_35", "kind": "mod3", "n": 35, "count": 8},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["generic", "generic", "wide", "schur", "grid", "bernoulli", "batch",
                       "real", "real", "complex", "rook", "mod3"])
    if kind == "generic":
        # orders span the walk's length on a logarithmic scale already
        return {"kind": "generic", "n": rng.randint(6, 33), "mag": _log_int(rng, 3, 1000)}
    if kind == "wide":
        return {"kind": "generic", "n": rng.randint(6, 25), "mag": _log_int(rng, 1 << 31, 1 << 40)}
    if kind == "schur":
        return {"kind": "schur", "n": rng.choice([23, 25, 27, 29, 31, 37])}
    if kind == "grid":
        return {"kind": "grid", "dims": rng.choice(GRIDS)}
    if kind == "bernoulli":
        return {"kind": "bernoulli", "n": rng.randint(16, 37),
                "density": round(rng.uniform(0.25, 0.75), 3)}
    if kind == "batch":
        lo = rng.randint(2, 14)
        return {"kind": "batch", "count": _log_int(rng, 16, 1024), "n_lo": lo,
                "n_hi": rng.randint(lo + 2, 26), "mag": _log_int(rng, 1, 20)}
    if kind == "real":
        n = rng.randint(4, 26)
        top = min(1024, 16 << (26 - n))
        return {"kind": "real", "n": n, "batch": _log_int(rng, 1, top),
                "grad": rng.random() < 0.5}
    if kind == "complex":
        n = rng.randint(4, 23)
        return {"kind": "complex", "n": n, "batch": _log_int(rng, 1, min(512, 32 << (23 - n)))}
    if kind == "rook":
        return {"kind": "rook", "n": rng.randint(6, 26), "density": round(rng.uniform(0.25, 0.75), 3)}
    return {"kind": "mod3", "n": rng.randint(8, 35), "count": 8}


def grid_biadjacency(dims):
    """Edges of the box grid between its even and odd vertices."""
    size = [int(d) for d in dims.split("x")]
    cells = list(np.ndindex(*size))
    even = {c: i for i, c in enumerate(c for c in cells if sum(c) % 2 == 0)}
    odd = {c: i for i, c in enumerate(c for c in cells if sum(c) % 2 == 1)}
    m = np.zeros((len(even), len(odd)), dtype=np.int64)
    for c, i in even.items():
        for axis, length in enumerate(size):
            for step in (-1, 1):
                v = list(c)
                v[axis] += step
                if length % 2 == 0 and length > 2:
                    v[axis] %= length
                if tuple(v) in odd:
                    m[i, odd[tuple(v)]] = 1
    return m


def _schur_prime(n, rng):
    """The largest prime = 1 (mod n) below a random number of 30 bits."""
    p = int(rng.integers(1 << 29, 1 << 30)) // n * n + 1
    while p % 2 == 0 or any(p % d == 0 for d in range(3, math.isqrt(p) + 1, 2)):
        p -= n
    return p


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "generic":
        a = rng.integers(-case["mag"], case["mag"] + 1, (case["n"], case["n"]), dtype=np.int64)
        return kind, a.tolist()
    if kind == "schur":
        n = case["n"]
        p = _schur_prime(n, rng)
        g = int(rng.integers(2, p - 1))
        while any(pow(pow(g, (p - 1) // n, p), d, p) == 1 for d in range(1, n)):
            g += 1
        return kind, (permgpu.GpuExt(), n, pow(g, (p - 1) // n, p), p)
    if kind == "grid":
        m = grid_biadjacency(case["dims"])
        bonds = np.argwhere(m)
        for i, j in bonds[rng.choice(len(bonds), 3, replace=False)]:
            m[i, j] = 0
        return kind, m[rng.permutation(len(m))][:, rng.permutation(len(m))].tolist()
    if kind in ("bernoulli", "rook"):
        return kind, (rng.random((case["n"], case["n"])) < case["density"]).astype(np.int64).tolist()
    if kind == "batch":
        orders = rng.integers(case["n_lo"], case["n_hi"] + 1, case["count"])
        return kind, [rng.integers(-case["mag"], case["mag"] + 1, (int(n), int(n)), dtype=np.int64)
                      for n in orders]
    if kind in ("real", "complex"):
        a, g = _float_inputs(case, seed)
        return kind, (a.cuda(), g.cuda(), bool(case.get("grad")))
    return kind, rng.integers(-50, 51, (case["count"], case["n"], case["n"]), dtype=np.int64)


def _float_inputs(case, seed):
    """(matrices, incoming gradients): entries of variance 1/n."""
    rng = np.random.default_rng(seed)
    n, b = case["n"], case["batch"]
    a = rng.normal(0.0, 1.0 / math.sqrt(n), (b, n, n))
    if case["kind"] == "complex":
        a = (a + 1j * rng.normal(0.0, 1.0 / math.sqrt(n), (b, n, n))) / math.sqrt(2.0)
    return torch.from_numpy(a), torch.from_numpy(rng.normal(0.0, 1.0, b))


def _whole(value):
    return np.frombuffer(int(value).to_bytes(RESULT_BYTES, "little", signed=True), dtype=np.uint8)


def run(state):
    kind, x = state
    if kind == "generic":
        return _whole(permgpu.matrix_permanent(x))
    if kind == "schur":
        ext, n, omega, p = x
        return ext.schur_permanent_mod_p(n, omega, p)
    if kind in ("grid", "bernoulli"):
        return _whole(permgpu.binary_permanent(x))
    if kind == "batch":
        return np.concatenate([_whole(v) for v in batch.batch_permanents(x, tune=None)])
    if kind == "real":
        a, g, grad = x
        if not grad:
            return [f64.glynn_permanent(a)]
        a = a.detach().requires_grad_()
        per = f64.glynn_permanent(a)
        per.backward(g)
        return [per.detach(), a.grad]
    if kind == "complex":
        return list(f64.permanent_c64(x[0]))
    if kind == "rook":
        return np.concatenate([_whole(v) for v in permgpu.rook_polynomial(x)])
    return np.array([mod3.permanent_mod3_fast(m) for m in x])


def work(case):
    """Operations of the walk over sign vectors (one update and one product
    per row), the polynomial walk's n/2 coefficient updates per row, one
    gradient row sum and product per row; bytes of the inputs and results."""
    kind = case["kind"]
    if kind == "grid":
        n = math.prod(int(d) for d in case["dims"].split("x")) // 2
    else:
        n = case.get("n", 0)
    if kind == "batch":
        orders = range(case["n_lo"], case["n_hi"] + 1)
        each = case["count"] / len(orders)
        return {"bytes": each * sum(8 * n * n + RESULT_BYTES for n in orders),
                "flops": each * sum(2.0 * n * 2.0 ** (n - 1) for n in orders)}
    states = 2.0 ** (n - 1)
    flops = 2.0 * n * states
    size = 8.0 * n * n + RESULT_BYTES
    if kind == "generic" and case["mag"] >= 1 << 31:
        # bits of the signed range the result can take, in 31-bit primes
        flops *= math.ceil((n * math.log2(n * case["mag"]) + 1) / 31)
    elif kind == "schur":
        size = 24.0
        # prime orders from 37 up take one sign word of each rotation class
        flops = states if n >= 37 else (n - 1) * states
    elif kind == "real":
        size = case["batch"] * 8.0 * (n * n + 1) * (2 if case["grad"] else 1)
        flops *= case["batch"] * (2 if case["grad"] else 1)
    elif kind == "complex":
        size = case["batch"] * 8.0 * (2 * n * n + 3)
        flops *= 4 * case["batch"]
    elif kind == "rook":
        flops = n * n * states * max(1, math.ceil(2 * n * math.log2(n) / 60))
        size += RESULT_BYTES * n
    elif kind == "mod3":
        flops = 2.0 * n * states * case["count"]
        size = (8.0 * n * n + 8) * case["count"]
    return {"bytes": size, "flops": flops}


# ---- 64-bit values of the floating results --------------------------------
# per(A) by the sum over column subsets S of the permanents of the first |S|
# rows on S: 2^n values, no signs, so none of the Glynn sum's cancellation.

def _subset_permanents(rows):
    """f[S] = permanent of the first |S| of `rows` on the columns S."""
    n = rows.shape[1]
    total = torch.zeros(1 << n, dtype=rows.dtype, device=rows.device)
    total[0] = 1
    layer = total.clone()
    for i in range(n):
        new = torch.zeros_like(layer)
        for j in range(n):
            new.view(-1, 2, 1 << j)[:, 1] += rows[i, j] * layer.view(-1, 2, 1 << j)[:, 0]
        total += new
        layer = new
    return total


def _gradient(a, f):
    """d per / d a_ij = sum over |S| = i without j of f[S] times the permanent
    of the rows below i on the columns outside S and j."""
    n = a.shape[0]
    h = _subset_permanents(a.flip(0)).flip(0)
    idx = torch.arange(1 << (n - 1), device=a.device)
    pop = torch.zeros_like(idx, dtype=torch.int32)
    for b in range(n - 1):
        pop += ((idx >> b) & 1).to(torch.int32)
    order = torch.argsort(pop)
    ends = [0] + torch.bincount(pop, minlength=n).cumsum(0).tolist()
    grad = torch.empty_like(a)
    for j in range(n):
        p = (f.view(-1, 2, 1 << j)[:, 0] * h.view(-1, 2, 1 << j)[:, 1]).reshape(-1)[order]
        for i in range(n):
            grad[i, j] = p[ends[i]:ends[i + 1]].sum()
    return grad


def exact(case, seed):
    if case["kind"] not in ("real", "complex"):
        return None
    n, b = case["n"], case["batch"]
    if b * n * n * 2.0 ** n > 4e12 or b * n * n > 2e5:
        return None
    a, g = _float_inputs(case, seed)
    a, g = a.cuda(), g.cuda()
    if case["kind"] == "complex":
        per = torch.stack([_subset_permanents(m)[-1] for m in a])
        return [per, None]            # no 64-bit value of the sum of |terms|
    if not case["grad"]:
        return [torch.stack([_subset_permanents(m)[-1] for m in a])]
    per, grad = [], []
    for m, scale in zip(a, g):
        f = _subset_permanents(m)
        per.append(f[-1])
        grad.append(scale * _gradient(m, f))
    return [torch.stack(per), torch.stack(grad)]
