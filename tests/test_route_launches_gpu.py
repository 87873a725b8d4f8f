"""The routing launches at the sizes where they change, against the CPU oracle: the blocks of the single launch, two launches up
to 1,024 chunks of 256 tokens, three beyond."""

import numpy as np
import pytest

from oracle import routing as oracle_routing
from tests.test_routing_gpu import _native, run_route

pytestmark = pytest.mark.gpu


def check(ids, rank, num_experts, m_mult, capacity=None):
    ep = ids.shape[0]
    disp = [(s + 1) << 40 for s in range(ep)]
    comb = [((s + 1) << 40) | (1 << 39) for s in range(ep)]
    out = run_route(ids, rank, num_experts, disp, comb, 1024, 1024, 1024, m_mult, capacity=capacity)
    assert out["status"][0] == 0, out["status"]
    t = oracle_routing.route(ids, rank, num_experts, disp, comb, 1024, 1024, 1024, m_mult)
    rows = int(t.expert_offsets[-1])
    np.testing.assert_array_equal(out["counts"], t.counts)
    np.testing.assert_array_equal(out["per_rank"], t.per_rank)
    np.testing.assert_array_equal(out["offsets"], t.expert_offsets)
    for key in ("fwd", "bwd", "sct"):
        np.testing.assert_array_equal(out[key][:rows], getattr(t, key))
        assert (out[key][rows:] == -5).all(), key  # nothing past the last segment
    return rows


@pytest.mark.parametrize("ep,T,K,E,m_mult", [
    (1, 1025, 2, 5, 0),       # first size past the single launch, a remainder of one token
    (1, 1280, 8, 300, 128),   # more experts than threads
    (1, 262144, 2, 7, 128),   # 1,024 chunks
    (1, 262145, 2, 7, 128),   # 1,025: three launches
    (8, 32768, 3, 24, 0),     # 1,024 chunks over eight ranks
    (8, 32769, 3, 24, 0),     # 1,032
    (2, 700, 1, 2, 128),      # one expert per rank
    (1, 2000, 4, 513, 0),     # past the two-launch limit on experts
])
def test_tables_are_the_oracles(ep, T, K, E, m_mult):
    rng = np.random.default_rng(ep * 100003 + T)
    ids = np.argsort(-rng.standard_normal((ep, T, E)), axis=-1)[..., :K].astype(np.int64)
    ids[rng.random(ids.shape) < 0.05] = -1
    for rank in sorted({0, ep - 1}):
        check(ids, rank, E, m_mult)


@pytest.mark.parametrize("ep,T,K,E,m_mult", [
    (1, 5, 2, 4, 128),      # 508 padding rows: one block
    (1, 5, 2, 5, 128),      # 635: two
    (1, 1024, 9, 512, 128),  # the largest of everything: 32 blocks, an id past the eighth
    (4, 33, 3, 64, 128),
])
def test_single_launch_over_several_blocks(ep, T, K, E, m_mult):
    rng = np.random.default_rng(T + E)
    ids = np.argsort(-rng.standard_normal((ep, T, E)), axis=-1)[..., :K].astype(np.int64)
    ids[rng.random(ids.shape) < 0.05] = -1
    for rank in sorted({0, ep - 1}):
        rows = check(ids, rank, E, m_mult)
    disp, comb = [(s + 1) << 40 for s in range(ep)], [(s + 1) << 41 for s in range(ep)]
    out = run_route(ids, ep - 1, E, disp, comb, 1024, 1024, 1024, m_mult, capacity=rows - 1)
    assert out["status"][0] == 2 and out["status"][1] == rows
    assert not out["offsets"].any() and not out["counts"].any() and (out["fwd"] == -5).all()


def test_every_token_on_one_expert_and_no_token_at_all():
    ids = np.full((1, 1500, 1), 3, dtype=np.int64)
    rows = check(ids, 0, 8, 128)
    assert rows == 1536
    assert check(np.full((1, 1500, 1), -1, dtype=np.int64), 0, 8, 128) == 0


@pytest.mark.parametrize("T", [1500, 262200])
def test_capacity_is_exact_and_an_overflow_leaves_no_rows(T):
    rng = np.random.default_rng(T)
    ids = rng.integers(0, 16, size=(1, T, 1)).astype(np.int64)
    rows = check(ids, 0, 16, 128)
    assert check(ids, 0, 16, 128, capacity=rows) == rows
    out = run_route(ids, 0, 16, [1 << 40], [1 << 41], 1024, 1024, 1024, 128, capacity=rows - 1)
    assert out["status"][0] == 2 and out["status"][1] == rows
    assert not out["offsets"].any() and not out["counts"].any()
    assert (out["fwd"] == -5).all() and (out["sct"] == -5).all()


def test_repeated_ids_count_as_routes_of_the_rank_alike_on_both_forms():
    """A token that lists an expert twice holds one row of it; the routes per rank count what was listed, on either side of the limit."""
    for T in (1500, 262200):
        ids = np.tile(np.array([2, 2], dtype=np.int64), (1, T, 1))
        out = run_route(ids, 0, 4, [1 << 40], [1 << 41], 1024, 1024, 1024, 0)
        assert out["counts"].tolist() == [0, 0, T, 0]
        assert out["per_rank"].tolist() == [2 * T]


def test_launches_reported_on_either_side_of_the_limits():
    launches = _native().route_launches
    assert [launches(1, t, 64) for t in (1024, 1025, 262144, 262145)] == [1, 2, 2, 3]
    assert [launches(8, t, 12) for t in (128, 129, 32768, 32769)] == [1, 2, 2, 3]
    assert [launches(1, 2000, e) for e in (512, 513)] == [2, 3]
