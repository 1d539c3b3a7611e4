"""How the Linear backward cuts its work, as linear_sm100_backward_plan (include/linear_sm100.h) says it does: host arithmetic."""
import ctypes

import pytest

SMS = 148


def plan(pkg, M, N, K, want_dx=1, want_dw=1, sms=SMS):
    out = (ctypes.c_int * 9)()
    assert pkg.lib().linear_sm100_backward_plan(M, N, K, want_dx, want_dw, sms, out) == 0
    names = ("together", "views", "ctas", "team", "down", "dx_pieces", "dx_fixed_order", "dw_of_a_cta", "dw_sum")
    return dict(zip(names, out))


# shapes that dx, dW and db share one launch at, and its teams: (M, N, K, CTAs of a team, below each other)
TEAMS = [
    (8001, 760, 3072, 6, 1), (6867, 243, 2208, 2, 1),  # a padded copy of dy; its last tile has one row in use
    (5420, 3326, 160, 2, 0), (4500, 3072, 768, 3, 0),
    (173, 1365, 5216, 1, 0),                           # tiles of dW only 6 blocks deep
    (7146, 8, 288, 1, 0), (8776, 344, 32, 1, 0),       # one tile row, one block of columns
    (1025, 129, 4288, 1, 0),
]


@pytest.mark.parametrize("M,N,K,team,down", TEAMS)
def test_one_launch(pkg, M, N, K, team, down):
    p = plan(pkg, M, N, K)
    assert (p["together"], p["views"], p["team"], p["down"]) == (1, 1, team, down)


@pytest.mark.parametrize("M,N,K,views", [(8192, 50257, 768, 4), (1024, 50257, 768, 4), (37, 50257, 768, 1), (8192, 50304, 768, 1)])
def test_views(pkg, M, N, K, views):
    assert plan(pkg, M, N, K)["views"] == views


# dx as whole tiles, or the sum of two pieces, by products of its own: the same bits in every call, and with and without dW
FIXED = [(3838, 16861, 160), (3250, 20003, 384), (24797, 3050, 160), (9695, 20359, 864)]


@pytest.mark.parametrize("M,N,K", FIXED + [(16384, 50257, 768), (32768, 50257, 768), (14839, 12887, 896), (2300, 50257, 768),
                                           (900, 5120, 1280)])
def test_dx_in_a_fixed_order(pkg, M, N, K):
    both, alone = plan(pkg, M, N, K), plan(pkg, M, N, K, want_dw=0)
    assert both["dx_fixed_order"] == alone["dx_fixed_order"] == 1
    assert both["dx_pieces"] == alone["dx_pieces"]


# a CTA takes longer ranges of dW's contraction than one accumulator sums up
LONG = [(40998, 3796, 32), (11087, 2470, 672)]


@pytest.mark.parametrize("M,N,K", LONG + [(18917, 6368, 544)])
def test_sums_of_dw_stay_short(pkg, M, N, K):
    """At most 160 contraction blocks of 32 rows, where pieces of one size for all SMs would be no longer."""
    assert plan(pkg, M, N, K)["dw_of_a_cta"] > 160
    assert max(plan(pkg, M, N, K, want_dx=want_dx)["dw_sum"] for want_dx in (0, 1)) <= 160


# few tiles, so that every CTA has one piece of dW of the same size, in contraction blocks
EVEN = [(640, 33, 32, 1), (506, 384, 384, 2), (700, 512, 512, 4), (2187, 44, 768, 4), (1205, 160, 736, 4), (512, 768, 768, 4)]


@pytest.mark.parametrize("M,N,K,blocks", EVEN)
def test_pieces_of_one_size(pkg, M, N, K, blocks):
    for want_dx in (0, 1):
        assert plan(pkg, M, N, K, want_dx=want_dx)["dw_of_a_cta"] == blocks


def test_plan_arguments(pkg):
    L, out = pkg.lib(), (ctypes.c_int * 9)()
    assert L.linear_sm100_backward_plan(8, 8, 32, 1, 1, SMS, None) == -1
    for bad in ((0, 8, 32, 1, 1, SMS), (8, 8, 32, 0, 0, SMS), (8, 8, 32, 1, 1, 0), (65536, 65536, 32, 1, 1, SMS)):
        assert L.linear_sm100_backward_plan(*bad, out) == -2
    assert L.linear_sm100_backward_plan(8, 8, 40, 1, 1, SMS, out) == -3
