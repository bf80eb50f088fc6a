"""The selected-negative operators (scores of chosen pairs forward and backward, tournament selection) against the oracle's
restatement of the reference's kernels for them (distmult_selected_neg_cuda.cu / .cpp).  fp32 sums in another order than the
oracle's float64: 1e-5 of the largest magnitude; selected columns must agree except on float ties."""
import numpy as np
import pytest
import torch

import ge2_oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-5

# (chunks, rows per chunk, negatives, D, selected per row)
PAIR_SHAPES = [(3, 50, 120, 32, 12), (2, 130, 1000, 100, 100), (1, 5, 7, 128, 1), (4, 9, 3, 1, 2), (2, 300, 64, 50, 7)]


def _pairs(rng, C, R, N, D, K):
    q = rng.standard_normal((C, R, D)).astype(np.float32)
    n = rng.standard_normal((C, N, D)).astype(np.float32)
    sel = rng.integers(0, N, (C, R * K)).astype(np.int64)
    if K >= 2:
        sel[0, 1] = sel[0, 0]  # one negative chosen twice by a row: its gradient adds up
    n[C - 1, sel[C - 1, 0]] = q[C - 1, 0]  # a pair at distance 0: the L2 score is the floor and passes no gradient
    return q, n, sel


def _close(got, want):
    got = got.cpu().numpy()
    assert got.shape == want.shape
    assert np.abs(got - want).max() <= TOL * max(1.0, np.abs(want).max())


@pytest.mark.parametrize("C,R,N,D,K", PAIR_SHAPES)
@pytest.mark.parametrize("kind,code", [("DOT", O.SELECTED_DOT), ("L2", O.SELECTED_L2)])
def test_selected_scores_forward_and_backward(capi, cuda_device, C, R, N, D, K, kind, code):
    rng = np.random.default_rng(C * 1000 + D)
    q, n, sel = _pairs(rng, C, R, N, D, K)
    grad = rng.standard_normal((C * R, K)).astype(np.float32)
    t = lambda a: torch.from_numpy(a).to(cuda_device)  # noqa: E731
    status = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    _close(capi.selected_neg_scores(kind, t(q), t(n), t(sel), status), O.selected_neg_scores(q, n, sel, code))
    dq, dn = capi.selected_neg_scores_backward(kind, t(grad), t(q), t(n), t(sel), status)
    exp_dq, exp_dn = O.selected_neg_scores_backward(grad, q, n, sel, code)
    _close(dq, exp_dq)
    _close(dn, exp_dn)
    assert int(status.item()) == 0


@pytest.mark.parametrize("C,R,N,D,K", [
    (100, 9, 7, 128, 5), (80, 33, 130, 101, 17), (74, 70, 1664, 128, 200),  # one slice; a ragged row; four slices of the negatives
    (149, 3, 5, 1, 33), (60, 100, 3300, 18, 300), (3, 700, 64, 50, 100),    # more chunks than SMs; the narrowest slice; many CTAs a chunk
])
@pytest.mark.parametrize("kind,code", [("DOT", O.SELECTED_DOT), ("L2", O.SELECTED_L2)])
def test_rows_resident_in_shared_memory(capi, cuda_device, C, R, N, D, K, kind, code):
    assert capi.load_library().ge2_selected_neg_backward_workspace_bytes(code, C, R, N, K, D) > 0  # this form can take them
    rng = np.random.default_rng(N + D)
    q, n, sel = _pairs(rng, C, R, N, D, K)
    grad = rng.standard_normal((C * R, K)).astype(np.float32)
    sel[C - 1, R * K - 1], grad[C * R - 1, K - 1] = 0, 0.0
    exp_s, (exp_dq, exp_dn) = O.selected_neg_scores(q, n, sel, code), O.selected_neg_scores_backward(grad, q, n, sel, code)
    sel[C - 1, R * K - 1] = N  # the last pair does not exist
    exp_s[C * R - 1, K - 1] = 0.0
    t = lambda a: torch.from_numpy(a).to(cuda_device)  # noqa: E731
    status = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    _close(capi.selected_neg_scores(kind, t(q), t(n), t(sel), status), exp_s)
    assert int(status.item()) == 8
    dq, dn = capi.selected_neg_scores_backward(kind, t(grad), t(q), t(n), t(sel), status)
    _close(dq, exp_dq)
    _close(dn, exp_dn)


@pytest.mark.parametrize("C,R,N,D,K,resident", [
    (148, 400, 130, 101, 60, True), (74, 600, 1664, 128, 250, True), (149, 400, 5, 1, 90, True),   # a ragged row; many slices of the negatives; two waves
    (74, 400, 3300, 18, 300, True), (3, 3000, 64, 50, 100, True), (62, 900, 299, 128, 90, True),     # the narrowest slice; many CTAs a chunk
    (7, 1428, 2310, 128, 4, False), (203, 60, 300, 99, 7, False), (1, 40, 50, 16, 3, False),       # few pairs a negative, a second wave, next to nothing
])
@pytest.mark.parametrize("kind,code", [("DOT", O.SELECTED_DOT), ("L2", O.SELECTED_L2)])
def test_the_form_that_the_estimate_takes(capi, cuda_device, C, R, N, D, K, resident, kind, code):
    """Gradients of either form against the oracle; which one ran shows in the scratch, which only the form with resident rows writes."""
    lib = capi.load_library()
    rng = np.random.default_rng(N + D)
    q, n, sel = _pairs(rng, C, R, N, D, K)
    grad = rng.standard_normal((C * R, K)).astype(np.float32)
    t = lambda a: torch.from_numpy(a).to(cuda_device)  # noqa: E731
    dq, dn, scores = torch.empty((C, R, D), device=cuda_device), torch.empty((C, N, D), device=cuda_device), None
    tq, tn, ts, tg = t(q), t(n), t(sel), t(grad)
    status = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    scores = capi.selected_neg_scores(kind, tq, tn, ts, status)
    need = lib.ge2_selected_neg_backward_workspace_bytes(code, C, R, N, K, D)
    assert need > 0 or not resident
    ws = torch.full((max(need, 12 * C * R * K),), 0xCD, dtype=torch.uint8, device=cuda_device)
    capi.check(lib.ge2_selected_neg_scores_backward_ws(code, tg.data_ptr(), tq.data_ptr(), tn.data_ptr(), ts.data_ptr(), C, R, N, K, D, dq.data_ptr(),
                                                       dn.data_ptr(), status.data_ptr(), ws.data_ptr(), ws.numel(), capi.cur_stream()), "backward")
    torch.cuda.synchronize()
    assert int(status) == 0
    if kind == "DOT":
        assert bool((ws != 0xCD).any()) == resident
    some = sorted({0, C // 2, C - 1})  # the oracle for a few chunks: they do not interact
    pick = lambda a: np.ascontiguousarray(a[some])  # noqa: E731
    rows = lambda a: np.concatenate([a[c * R:(c + 1) * R] for c in some])  # noqa: E731
    exp_s = O.selected_neg_scores(pick(q), pick(n), pick(sel), code)
    exp_dq, exp_dn = O.selected_neg_scores_backward(rows(grad), pick(q), pick(n), pick(sel), code)
    _close(torch.cat([scores[c * R:(c + 1) * R] for c in some]), exp_s)
    _close(dq[some], exp_dq)
    _close(dn[some], exp_dn)


def test_selected_column_out_of_range_is_reported_and_skipped(capi, cuda_device):
    rng = np.random.default_rng(3)
    C, R, N, D, K = 2, 20, 30, 40, 4
    q, n, sel = _pairs(rng, C, R, N, D, K)
    bad = sel.copy()
    bad[0, 5], bad[1, 7] = N, -1
    grad = rng.standard_normal((C * R, K)).astype(np.float32)
    t = lambda a: torch.from_numpy(a).to(cuda_device)  # noqa: E731
    status = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    scores = capi.selected_neg_scores("DOT", t(q), t(n), t(bad), status).cpu().numpy()
    assert int(status.item()) == 8  # GE2_STATUS_BAD_INDEX
    exp = O.selected_neg_scores(q, n, sel, O.SELECTED_DOT)
    exp[5 // K, 5 % K] = 0.0
    exp[R + 7 // K, 7 % K] = 0.0
    assert np.abs(scores - exp).max() <= TOL * np.abs(exp).max()
    status.zero_()
    dq, dn = capi.selected_neg_scores_backward("DOT", t(grad), t(q), t(n), t(bad), status)
    assert int(status.item()) == 8
    masked = grad.copy()  # a zero upstream gradient on the valid stand-in columns gives the same sums
    masked[5 // K, 5 % K] = 0.0
    masked[R + 7 // K, 7 % K] = 0.0
    exp_dq, exp_dn = O.selected_neg_scores_backward(masked, q, n, sel, O.SELECTED_DOT)
    _close(dq, exp_dq)
    _close(dn, exp_dn)


def _check_tournament(scores, idx, q, n, K, score_q=None, score_n=None):
    C, R, _ = q.shape
    N = n.shape[1]
    T = N // K
    exp_scores, exp_idx = O.tournament_selected_scores(q, n, K)
    scores, idx = scores.cpu().numpy(), idx.cpu().numpy()
    assert scores.shape == (C * R, K) and idx.shape == (C, R * K)
    sel_all = np.einsum("crd,cnd->crn", q.astype(np.float64), n.astype(np.float64))
    got = np.take_along_axis(sel_all, idx.reshape(C, R, K), axis=2)
    want = np.take_along_axis(sel_all, exp_idx.reshape(C, R, K), axis=2)
    scale = max(1.0, np.abs(sel_all).max())
    assert np.abs(got - want).max() <= TOL * scale  # another winner only on a float tie
    assert (idx != exp_idx).mean() <= 0.01
    assert np.array_equal(idx.reshape(C, R, K) // T, np.broadcast_to(np.arange(K), (C, R, K)))  # one winner from every group
    if score_q is None:
        assert np.abs(scores - exp_scores).max() <= TOL * scale
    else:
        exp = O.selected_neg_scores(score_q, score_n, idx, O.SELECTED_DOT)  # the winners scored by the scorer's rows
        assert np.abs(scores - exp).max() <= TOL * max(1.0, np.abs(exp).max())


@pytest.mark.parametrize("C,R,N,D,K", [
    (3, 50, 120, 32, 12),     # groups of 10: six whole groups a tile
    (2, 130, 128, 100, 64),   # groups of 2
    (1, 64, 256, 16, 4),      # groups of exactly one tile
    (2, 70, 96, 100, 96),     # groups of 1: every negative is kept
    (2, 130, 1000, 100, 4),   # groups of 250: a running winner over four tiles, the last one ragged
    (3, 17, 130, 128, 2),     # groups of 65: one column into the second tile
    (1, 200, 1000, 50, 1),    # one group: the best negative of the chunk
    (5, 3, 33, 7, 11),        # fewer rows than a tile, groups of 3, odd D
    (2, 100, 1000, 100, 100), # the benchmarked step's chunk shape, a tenth kept
])
def test_tournament_selection_matches_oracle(capi, cuda_device, C, R, N, D, K):
    rng = np.random.default_rng(N + K)
    q = rng.standard_normal((C, R, D)).astype(np.float32)
    n = rng.standard_normal((C, N, D)).astype(np.float32)
    scores, idx = capi.tournament_select(torch.from_numpy(q).to(cuda_device), torch.from_numpy(n).to(cuda_device), K)
    _check_tournament(scores, idx, q, n, K)


def test_tournament_with_a_separate_scorer(capi, cuda_device):
    rng = np.random.default_rng(9)
    C, R, N, D, K = 2, 90, 200, 64, 20
    q, n, sq, sn = (rng.standard_normal(s).astype(np.float32) for s in ((C, R, D), (C, N, D), (C, R, D), (C, N, D)))
    t = lambda a: torch.from_numpy(a).to(cuda_device)  # noqa: E731
    scores, idx = capi.tournament_select(t(q), t(n), K, score_chunked=t(sq), score_negatives=t(sn))
    _check_tournament(scores, idx, q, n, K, sq, sn)


def test_tournament_rejects_uneven_groups_and_accepts_empty_input(capi, cuda_device):
    q = torch.zeros((2, 5, 8), device=cuda_device)
    n = torch.zeros((2, 10, 8), device=cuda_device)
    with pytest.raises(capi.Ge2Error):
        capi.tournament_select(q, n, 3)
    scores, idx = capi.tournament_select(q[:, :0].contiguous(), n, 5)
    assert scores.shape == (0, 5) and idx.shape == (2, 0)
    # all scores equal: the first negative of every group wins
    scores, idx = capi.tournament_select(q, n, 5)
    torch.cuda.synchronize()
    assert torch.equal(idx.cpu().view(2, 5, 5), (torch.arange(5) * 2).expand(2, 5, 5)) and float(scores.abs().max()) == 0.0


@pytest.mark.parametrize("C,R,N,D,K", [
    (1, 127, 64, 63, 64), (2, 129, 65, 65, 5), (1, 1, 1, 1, 1), (300, 3, 20, 8, 4),  # one past a tile each way; more items than SMs
    (3, 256, 640, 128, 5), (1, 128, 4096, 66, 64),                                    # groups over several tiles, shares cut inside a row tile
])
def test_tournament_at_tile_edges_and_on_ties(capi, cuda_device, C, R, N, D, K):
    rng = np.random.default_rng(C + R + N + D)
    q = rng.standard_normal((C, R, D)).astype(np.float32)
    n = rng.standard_normal((C, N, D)).astype(np.float32)
    n[:, N // 2:] = n[:, :N - N // 2]  # every negative twice: equal scores, within a group when there is one, and the first must win
    scores, idx = capi.tournament_select(torch.from_numpy(q).to(cuda_device), torch.from_numpy(n).to(cuda_device), K)
    _check_tournament(scores, idx, q, n, K)
    if K == 1 and N > 1:
        assert int(idx.max()) < N // 2


@pytest.mark.parametrize("T,K", [(5, 31), (8, 33), (9, 1), (15, 40), (16, 12), (17, 9), (48, 3), (49, 7), (63, 2), (64, 5), (65, 4), (127, 3), (500, 1)])
def test_tournament_groups_read_in_parts(capi, cuda_device, T, K):
    """Groups whose parts begin and end at every place of a tile, one or an odd number of them in a share; scores that are NaN never win, and a
    group without any other has the value of nothing at its first column, on the path of the short groups (a group of four here) as well."""
    C, R, D = 3, 140, 20
    for T, K in ((T, K), (4, T)):
        N = T * K
        rng = np.random.default_rng(T * 1000 + K)
        q = rng.standard_normal((C, R, D)).astype(np.float32)
        n = rng.standard_normal((C, N, D)).astype(np.float32)
        n[:, N // 2:] = n[:, :N - N // 2]
        scores, idx = capi.tournament_select(torch.from_numpy(q).to(cuda_device), torch.from_numpy(n).to(cuda_device), K)
        _check_tournament(scores, idx, q, n, K)
        n[:, ::3] = np.nan
        n[1, :T] = np.nan
        scores, idx = (x.cpu().numpy().reshape(C, R, K) for x in capi.tournament_select(torch.from_numpy(q).to(cuda_device), torch.from_numpy(n).to(cuda_device), K))
        assert np.isneginf(scores[1, :, 0]).all() and (idx[1, :, 0] == 0).all()
        exact = np.einsum("crd,cnd->crn", q.astype(np.float64), n.astype(np.float64)).reshape(C, R, K, T)
        live = ~np.isnan(exact).all(-1)
        at = np.take_along_axis(exact.reshape(C, R, N), idx, 2)
        best = np.fmax.reduce(exact, -1)
        assert (idx // T == np.arange(K)).all() and np.abs(at - best)[live].max() < 1e-5 * np.abs(best[live]).max()  # fp32 sums of 20 products
        assert np.abs(scores - at)[live].max() < 1e-5 * np.abs(best[live]).max()
