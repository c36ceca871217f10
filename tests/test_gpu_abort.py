"""Host-side abort of long launches: pg_abort() called from another host
thread while a multi-second traversal runs makes the call return PG_EABORT
within a fraction of a second (the kernels read the host-mapped abort word
once per 2^16 states, or per chunk, after each thread's first period);
pg_clear_abort() re-arms the library and
the next call computes the right value.  The failure is made on the host:
no kernel is broken, nothing waits on anything that is not set."""

import threading
import time

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _aborted_after(lib, fn, delay=0.2):
    timer = threading.Timer(delay, lib.load().pg_abort)
    t0 = time.perf_counter()
    timer.start()
    try:
        with pytest.raises(lib.PermGpuError) as err:
            fn()
    finally:
        timer.join()
        lib.load().pg_clear_abort()
    return err.value.status, time.perf_counter() - t0


def test_abort_exact_engine(lib):
    # 40 x 40 0/1 matrix: 2^39 Gray states, about 2.6 s uninterrupted
    a = (np.random.default_rng(301).random((40, 40)) < 0.5).astype(np.int64)
    lib.load().pg_clear_abort()
    status, took = _aborted_after(lib, lambda: lib.exact_permanent(a, lib.exact_limbs(a)))
    assert status == lib.PG_EABORT
    assert took < 1.5
    b = np.random.default_rng(7).integers(-8, 9, (20, 20), dtype=np.int64)
    assert lib.exact_permanent(b, lib.exact_limbs(b)) == oracle.exact_permanent(b.tolist())


def test_abort_residue_engine(lib):
    # one 31-bit prime over a 40 x 40 matrix: about 7 s uninterrupted
    a = np.random.default_rng(302).integers(-8, 9, (40, 40), dtype=np.int64)
    lib.load().pg_clear_abort()
    status, took = _aborted_after(lib, lambda: lib.residues(a, [2_147_483_647]))
    assert status == lib.PG_EABORT
    assert took < 1.5
    b = np.random.default_rng(8).integers(-8, 9, (16, 16), dtype=np.int64)
    p = 2_147_483_647
    assert lib.residues(b, [p]) == [oracle.exact_permanent(b.tolist()) % p]


def test_abort_batched_engine(lib):
    # 256 matrices of order 32, entries in [-3, 3]: about 2 s of one
    # persistent launch; its warps read the word once per 8 tasks
    mats = [np.random.default_rng(600 + i).integers(-3, 4, (32, 32), dtype=np.int64)
            for i in range(256)]
    lib.load().pg_clear_abort()
    status, took = _aborted_after(lib, lambda: lib.batch_exact(mats))
    assert status == lib.PG_EABORT
    assert took < 1.5
    small = [np.random.default_rng(700 + i).integers(-3, 4, (n, n), dtype=np.int64)
             for i, n in enumerate((12, 17, 21))]
    assert lib.batch_exact(small) == [oracle.exact_permanent(m.tolist()) for m in small]


def test_abort_flag_left_set_stops_the_next_launch_at_once(lib):
    # a raised word that nobody cleared makes every later long launch stop at
    # its first poll (after each thread's first 2^16 states: a 36 x 36 walk
    # gives every thread several hundred thousand); clearing it restores
    # normal service.  Launches too short for a poll complete as usual.
    a = np.random.default_rng(9).integers(-8, 9, (36, 36), dtype=np.int64)
    h = lib.load()
    h.pg_abort()
    try:
        t0 = time.perf_counter()
        with pytest.raises(lib.PermGpuError) as err:
            lib.exact_permanent(a, lib.exact_limbs(a))
        assert err.value.status == lib.PG_EABORT
        assert time.perf_counter() - t0 < 1.0
        b = np.random.default_rng(10).integers(-8, 9, (16, 16), dtype=np.int64)
        assert lib.exact_permanent(b, lib.exact_limbs(b)) == oracle.exact_permanent(b.tolist())
    finally:
        h.pg_clear_abort()
    c = np.random.default_rng(9).integers(-8, 9, (20, 20), dtype=np.int64)
    assert lib.exact_permanent(c, lib.exact_limbs(c)) == oracle.exact_permanent(c.tolist())


def _raised_before(lib, fn):
    # status of a call that starts with the word already raised
    lib.load().pg_abort()
    try:
        with pytest.raises(lib.PermGpuError) as err:
            fn()
    finally:
        lib.load().pg_clear_abort()
    return err.value.status


def _fp64(kind, n, batch):
    import torch
    from permgpu import f64
    a = torch.from_numpy(np.random.default_rng(n).normal(0, n ** -0.5, (batch, n, n))).cuda()
    if kind == "complex":
        return f64.permanent_c64(a.to(torch.complex128) * (1 - 0.5j))
    return f64.permanent_f64(a, want_grad=kind == "gradient")


@pytest.mark.parametrize("kind,n,batch", [
    ("forward", 32, 1), ("complex", 30, 1), ("gradient", 28, 1),    # several ranges a warp
    ("forward", 34, 1), ("complex", 34, 1),                         # the kernel of orders 33..63
])
def test_abort_word_raised_before_fp64_walks(lib, kind, n, batch):
    # the lanes of a warp vote on the word and leave together: a status, not a
    # partial sum, and the next call is right again
    want = [x.cpu() for x in _fp64(kind, 12, 2) if x is not None]
    assert _raised_before(lib, lambda: _fp64(kind, n, batch)) == lib.PG_EABORT
    got = [x.cpu() for x in _fp64(kind, 12, 2) if x is not None]
    assert all((x == y).all() for x, y in zip(want, got))


@pytest.mark.parametrize("kind,n,batch", [("forward", 30, 512), ("complex", 28, 512),
                                          ("gradient", 28, 512)])
def test_abort_fp64_walks(lib, kind, n, batch):
    # two to four seconds uninterrupted
    lib.load().pg_clear_abort()
    status, took = _aborted_after(lib, lambda: _fp64(kind, n, batch))
    assert status == lib.PG_EABORT
    assert took < 1.5


@pytest.mark.parametrize("kind,n,batch", [
    ("forward", 4, 200_000), ("forward", 12, 20_000), ("forward", 13, 200_000),
    ("complex", 5, 200_000), ("complex", 12, 50_000),
    ("gradient", 4, 200_000), ("gradient", 10, 50_000), ("gradient", 15, 10_000),
])
def test_abort_word_raised_before_batches_of_small_matrices(lib, kind, n, batch):
    # a warp walks one range only: blocks beyond the first wave ask before
    # they start
    want = [x.cpu() for x in _fp64(kind, n, 4) if x is not None]
    assert _raised_before(lib, lambda: _fp64(kind, n, batch)) == lib.PG_EABORT
    got = [x.cpu() for x in _fp64(kind, n, 4) if x is not None]
    assert all((x == y).all() for x, y in zip(want, got))


@pytest.mark.parametrize("kind", ["general40", "binary44", "mod3_48"])
def test_abort_integer_walks_of_seconds(lib, kind):
    # three to five seconds uninterrupted
    rng = np.random.default_rng(44)
    a = {"general40": lambda: rng.integers(-8, 9, (40, 40)),
         "binary44": lambda: (rng.random((44, 44)) < 0.5).astype(np.int64),
         "mod3_48": lambda: rng.integers(0, 3, (48, 48))}[kind]()
    call = lib.permanent_mod3 if kind == "mod3_48" else lambda m: lib.exact_permanent(m, lib.exact_limbs(m))
    if kind == "binary44":
        plan = lib.ExactPlan(a)
        assert lib.load().pg_exact_plan_bit_planes(plan._h) >= 2
        plan.close()
    lib.load().pg_clear_abort()
    status, took = _aborted_after(lib, lambda: call(a))
    assert status == lib.PG_EABORT
    assert took < 1.0
    b = a[:18, :18].copy()
    want = oracle.exact_permanent(b.tolist())
    assert call(b) == (want % 3 if kind == "mod3_48" else want)


def test_abort_word_raised_before_wide_and_polynomial_walks(lib):
    # the 64-bit exact kernel asks in blocks beyond the first wave, the exact
    # polynomial kernel from a block's second task on
    rng = np.random.default_rng(45)
    a = rng.integers(-(1 << 42), 1 << 42, (28, 28))
    assert _raised_before(lib, lambda: lib.exact_wide_permanent(a, lib.exact_limbs(a))) == lib.PG_EABORT
    L = (rng.random((28, 28)) < 0.5).astype(np.int64)
    ones = np.ones((28, 28), dtype=np.int64)
    assert _raised_before(lib, lambda: lib.affine_residues(ones, L, [1_000_003])) == lib.PG_EABORT
    b = a[:14, :14].copy()
    assert lib.exact_wide_permanent(b, 40) == oracle.exact_permanent(b.tolist())
    m = L[:14, :14].copy()
    assert lib.affine_residues(ones[:14, :14], m, [1_000_003])[0] == \
        oracle.affine_mod_p(ones[:14, :14], m, 1_000_003)
