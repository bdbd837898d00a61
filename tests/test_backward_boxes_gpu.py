"""Backward at the edges of its window-sum tiles (64 x 32 outputs, 16 columns and 8 rows a thread):
images smaller than a tile and one pixel past it, windows narrower than a thread's run of columns,
and areas without energy beside bright ones, whose outputs have no derivative. Bar: 1e-4 of the
gradient's largest entry against the long-double CPU adjoint, as in test_backward_gpu.py."""
import numpy as np
import pytest

from test_backward_gpu import ADJ_TOL, backward, oracle_adjoint, rel_max

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W", [(33, 65), (32, 64), (31, 127), (97, 129), (64, 193)])
@pytest.mark.parametrize("th,tw", [(7, 15), (8, 16), (9, 17), (31, 12), (5, 33)])
def test_box_edges_match_cpu_adjoint(ocip, ctx, H, W, th, tw):
    ctx.make_current()
    ctx.set_path(ocip.PATH_TENSOR)
    rng = np.random.default_rng(H * W + th)
    S = (0.1 + rng.random((H, W))).astype(np.float32)
    T = (0.1 + rng.random((th, tw))).astype(np.float32)
    G1, G2 = (rng.standard_normal(S.shape).astype(np.float32) for _ in range(2))
    dS, dT = backward(ocip, S, T, G1, G2)
    ctx.set_path(ocip.PATH_PLAIN)
    rS, rT = oracle_adjoint(S, T, G1, G2)
    assert rel_max(dS, rS) <= ADJ_TOL and rel_max(dT, rT) <= ADJ_TOL


@pytest.mark.parametrize("th,tw", [(9, 17), (32, 32)])
def test_zero_windows_contribute_nothing(ocip, ctx, th, tw):
    """The window energies of the dark area must be exactly 0 (no residue of the bright one): the
    gradients are those without the upstream gradient there. (The CPU adjoint has 0 / 0 there.)"""
    ctx.make_current()
    ctx.set_path(ocip.PATH_TENSOR)
    rng = np.random.default_rng(th)
    S = (1e3 * (0.1 + rng.random((150, 280)))).astype(np.float32)
    S[40:120, 90:230] = 0
    T = (0.1 + rng.random((th, tw))).astype(np.float32)
    G2 = rng.standard_normal(S.shape).astype(np.float32)
    padded = np.pad(S, ((th // 2, th - 1 - th // 2), (tw // 2, tw - 1 - tw // 2)))
    live = np.lib.stride_tricks.sliding_window_view(padded, (th, tw)).max((2, 3)) > 0
    assert 0 < (~live).sum() < live.size / 2
    dS, dT = backward(ocip, S, T, None, G2)
    eS, eT = backward(ocip, S, T, None, np.where(live, G2, 0).astype(np.float32))
    ctx.set_path(ocip.PATH_PLAIN)
    assert np.array_equal(dS, eS)
    assert rel_max(dT, eT) <= ADJ_TOL
