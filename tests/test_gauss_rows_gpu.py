"""The Gaussian smoother's kernel (unshifted weights of -power(a - b, 2) scores,
finite values) against the general tile kernel (EINFOLD_TILES_GENERAL=1) and
the oracle, at the edges of its blocks, groups and key chunks, and on rows it
hands back to the exact kernel."""
import numpy as np
import pytest

from einfold_b200 import ir, kernels as K
from oracle import oracle
from tests import pipelines as P
from tests.tables import rows_of

pytestmark = pytest.mark.gpu

GE, LT = ir.Comparison.GREATER_OR_EQUAL, ir.Comparison.LESS


def _run(case, monkeypatch, general=False):
    if general:
        monkeypatch.setenv("EINFOLD_TILES_GENERAL", "1")
    got = K.pipeline(case.pipeline, [K.Relation(*case.q), K.Relation(*case.k), K.Relation(*case.v)])
    monkeypatch.delenv("EINFOLD_TILES_GENERAL", raising=False)
    if got is None:
        return None
    t = rows_of(got.batches)
    return (got.tiles_visited, got.tiles), t, t.column(t.num_columns - 1).to_numpy(zero_copy_only=False)


def _case(l, lk, nb, d, c, scale, conditions=(), normalizer=ir.Normalizer.KEPT_GROUPS, far=0):
    def q(n):
        x = oracle.Rng.seeded(41, 2).units(n)
        if far:
            x[::far] = 60.0
        return x

    return P.attention(l, d=d, lk=lk, nb=nb, c=c, scores=P.gaussian_scores(), conditions=list(conditions),
                       weight=ir.Weight.exp(scale, ir.Shift.NONE), normalizer=normalizer, q_value=q,
                       k_value=lambda n: oracle.Rng.seeded(42, 2).units(n),
                       v_value=lambda n: oracle.Rng.seeded(43, 2).units(n) * 2 - 1)


CASES = {
    # rows and keys a batch, batches, features, value columns, scale, conditions
    "one_pair": (1, 1, 1, 1, 1, ir.Scale.over(0.05), ()),
    "groups_of_threads": (257, 129, 3, 2, 8, ir.Scale.over(0.05), ()),
    "masked": (300, 255, 2, 3, 2, ir.Scale.times(7.5), ((GE, -30), (LT, 60))),
    "no_key_at_first": (140, 140, 1, 1, 1, ir.Scale.one(), ((GE, 20),)),
    "a_row_a_thread": (27000, 33, 3, 1, 1, ir.Scale.over(0.05), ()),
    "two_rows_a_thread": (33001, 131, 5, 1, 3, ir.Scale.over(0.05), ()),
}


@pytest.mark.parametrize("normalizer", [ir.Normalizer.KEPT_GROUPS, ir.Normalizer.NONE])
@pytest.mark.parametrize("name", list(CASES))
def test_the_smoothers_kernel_matches_the_general_one(name, normalizer, monkeypatch):
    l, lk, nb, d, c, scale, conditions = CASES[name]
    case = _case(l, lk, nb, d, c, scale, conditions, normalizer)
    tiles, table, got = _run(case, monkeypatch)
    tiles_g, table_g, want = _run(case, monkeypatch, general=True)
    assert tiles == tiles_g and table.num_rows == table_g.num_rows
    for i in range(table.num_columns - 1):
        assert table.column(i).equals(table_g.column(i))
    # Scores lie within 20·d of 0; the general kernel rounds the scaled score
    # (half a unit of up to 20·d in the exponent), both round each weight,
    # product and sum (at most lk + 4 units each).
    unit = 2.0 ** -53
    tol = (20 * d + 2 * (lk + 4)) * unit * case.v_scale * (lk if normalizer == ir.Normalizer.NONE else 1)
    assert np.max(np.abs(got - want)) <= tol
    if l <= 300:
        assert P.run_oracle(case) is not None


@pytest.mark.parametrize("normalizer", [ir.Normalizer.KEPT_GROUPS, ir.Normalizer.NONE])
def test_rows_without_weight_go_to_the_exact_kernel(normalizer, monkeypatch):
    # Every 40th row lies 59 away from every key: its weights exp(-59²/0.05)
    # are all zero, below what the fast kernel's clamp can tell.
    case = _case(200, 130, 2, 1, 1, ir.Scale.over(0.05), (), normalizer, far=40)
    got, want, exact = _run(case, monkeypatch), _run(case, monkeypatch, general=True), P.run_oracle(case)
    assert (got is None) == (want is None) == (exact is None)
    if got is not None:
        assert got[0] == want[0]
        assert np.array_equal(np.isnan(got[2]), np.isnan(want[2]))
        seen = ~np.isnan(want[2])
        assert np.max(np.abs(got[2][seen] - want[2][seen])) <= 1e-13 * case.v_scale * (
            130 if normalizer == ir.Normalizer.NONE else 1)
