"""GPU parity of the mod-3 engine (pg_permanent_mod3, pg_permanent_mod3_cols)
against the reference's mod-3 results, the oracle, and exact identities."""

import math

import numpy as np
import pytest

import oracle
from conftest import golden

pytestmark = pytest.mark.gpu


def test_reference_golden_cases(lib):
    from permgpu import mod3
    for c in golden("mod3.json")["cases"]:
        assert mod3.permanent_mod3_fast(c["matrix"]) == c["mod3"], len(c["matrix"])


@pytest.mark.parametrize("n", list(range(2, 25)))
def test_random_vs_oracle(lib, n):
    rng = np.random.default_rng(300 + n)
    a = rng.integers(-(1 << 62), 1 << 62, (n, n))
    assert lib.permanent_mod3(a) == oracle.permanent_mod_p(a, 3, 8)


def test_column_entry_matches_matrix_entry(lib):
    from permgpu import mod3
    rng = np.random.default_rng(9)
    for n in (3, 16, 31, 32, 33, 35):
        a = rng.integers(0, 3, (n, n))
        mags, sgns = mod3.encode_matrix_f3(a)
        assert lib.permanent_mod3_cols(mags, sgns, n) == lib.permanent_mod3(a)


def test_identities_up_to_order_40(lib):
    for n in (3, 20, 33, 40):
        assert lib.permanent_mod3(np.ones((n, n), np.int64)) == math.factorial(n) % 3
        assert lib.permanent_mod3(np.eye(n, dtype=np.int64)) == 1
        assert lib.permanent_mod3(2 * np.eye(n, dtype=np.int64)) == pow(2, n, 3)
        p = np.eye(n, dtype=np.int64)[np.random.default_rng(n).permutation(n)]
        assert lib.permanent_mod3(-p) == pow(2, n, 3)


@pytest.mark.parametrize("n", [3, 5, 6, 7, 10, 11, 12, 15, 16, 17, 20, 21, 24])
def test_many_survivors_at_table_edges(lib, n):
    # orders around the table's edges (word bits, lanes, the 32 high states of
    # a batch, the last row group) with repeated rows, so that most states
    # keep every row nonzero and reach the sign words
    rng = np.random.default_rng(900 + n)
    base = rng.integers(1, 3, (2, n))
    a = base[rng.integers(0, 2, n)]
    assert lib.permanent_mod3(a) == oracle.permanent_mod_p(a, 3, 8)
    a[n // 2, : n // 2] = 0
    assert lib.permanent_mod3(a) == oracle.permanent_mod_p(a, 3, 8)


def test_expansion_beyond_one_word(lib):
    # per of a block-diagonal matrix is the product of the blocks', at orders
    # whose rows take more than one 32-bit word
    rng = np.random.default_rng(33)
    for n, k in ((33, 13), (36, 18), (38, 19)):
        a = np.zeros((n, n), np.int64)
        a[:k, :k] = rng.integers(0, 3, (k, k))
        a[k:, k:] = rng.integers(0, 3, (n - k, n - k))
        want = lib.permanent_mod3(a[:k, :k]) * lib.permanent_mod3(a[k:, k:]) % 3
        p, q = rng.permutation(n), rng.permutation(n)
        assert lib.permanent_mod3(a[p][:, q]) == want


@pytest.mark.parametrize("n", [25, 26, 28, 29, 31, 32, 33, 34])
def test_many_survivors_with_tables(lib, n):
    # orders that take tables, rows of one word and of two, the last batch and
    # row group; rows that differ in few places, so that many states keep every
    # row nonzero; against the exact engine
    rng = np.random.default_rng(2500 + n)
    row = rng.integers(1, 3, n)
    a = np.where(rng.random((n, n)) < 0.12, rng.integers(0, 3, (n, n)), row)
    a *= rng.integers(1, 3, (n, 1))
    want = lib.exact_permanent(a, lib.exact_limbs(a)) % 3
    assert lib.permanent_mod3(a) == want
    assert lib.permanent_mod3(a.T.copy()) == want
