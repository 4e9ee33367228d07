"""Halton draws whose index passed 2^31 (a sample number times the stride wraps after some 69000 samples): the digits are
those of the index as 32 unsigned bits, each operation rounded to FP32 in the order of the reference's loop.

A film of one pixel has stride 1, so the sample number is the index.  The digit tables come from the oracle's draws
of one-digit indices, and the loop below is first held against the oracle where the index is positive."""
import numpy as np
import pytest

from crystal2_gb300 import Context, scenes
from crystal2_gb300 import _native as N
from oracle import bindings as B

pytestmark = pytest.mark.gpu

PRIMES = [p for p in range(2, 542) if all(p % q for q in range(2, p))]
F = np.float32


def _oracle(index, dim):
    z = np.zeros(len(index), np.int32)
    return B.oracle_halton(1, 1, z, z, index.astype(np.int32), dim + 1)[:, dim]


def _table(dim):
    base = PRIMES[dim]
    if dim == 1:
        return np.arange(3)
    draws = _oracle(np.arange(base), dim).astype(np.float64)
    tail = draws[0]  # index 0 has no digits: T[0] / base / (1 - 1 / base)
    return np.rint(np.concatenate([[tail * (base - 1)], draws[1:] * base - tail])).astype(np.int64)


def _draw(index, dim, table):
    base, inv = F(PRIMES[dim]), F(1) / F(PRIMES[dim])
    v = index.astype(np.uint32).astype(np.int64)
    result, inv_n = np.zeros(len(v), F), np.ones(len(v), F)
    while np.any(v):
        live = v > 0
        result = np.where(live, result * base + table[v % PRIMES[dim]].astype(F), result)
        inv_n = np.where(live, inv_n * inv, inv_n)
        v //= PRIMES[dim]
    if dim > 1:
        result = result + inv * F(table[0]) / (F(1) - inv)
    return np.minimum(result * inv_n, F(np.nextafter(F(1), F(0))))


@pytest.mark.parametrize("dim", [1, 2, 3, 9, 40, 96, 97, 98, 99])
def test_wrapped_indices(tmp_path, dim):
    rng = np.random.default_rng(dim)
    below = np.concatenate([np.arange(1, 400), rng.integers(1, 2 ** 31, 3000), [2 ** 31 - 1]]).astype(np.int64)
    above = np.concatenate([np.arange(2 ** 31, 2 ** 31 + 400), rng.integers(2 ** 31, 2 ** 32, 3000), [2 ** 32 - 1, 2 ** 32 - 2]]).astype(np.int64)
    table = _table(dim)
    assert sorted(table) == list(range(PRIMES[dim]))
    assert np.array_equal(_draw(below, dim, table).view(np.uint32), _oracle(below, dim).view(np.uint32))
    cp, sp = scenes.cornell(str(tmp_path), width=1, height=1, spp=1)
    with Context(0) as ctx:
        ctx.load(cp, sp, tree=N.TREE_SAH)
        for index in (below, above):
            s = index.astype(np.uint32).view(np.int32)
            z = np.zeros(len(s), np.int32)
            want = _draw(index, dim, table)
            assert np.array_equal(ctx.sampler_values(z, z, s, dim, two_d=False).view(np.uint32), want.view(np.uint32))
            pair = ctx.sampler_values(z, z, s, dim, two_d=True)
            assert np.array_equal(np.ascontiguousarray(pair[:, 0]).view(np.uint32), want.view(np.uint32))
