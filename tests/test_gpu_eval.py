"""ge2_eval_ranks against the oracle's restatement of the reference's evaluation (node_corrupt_forward scores, the global
filter of compute_filter_corruption, ranks as LinkPredictionReporter::computeRanks): integer ranks, bit-exact."""
import numpy as np
import pytest
import torch

import ge2_oracle as O
import workloads

pytestmark = pytest.mark.gpu


def _case(rng, nodes, R, D, n_all, B, scale=0.5):
    table = (rng.standard_normal((nodes, D)) * scale).astype(np.float32)
    rel = (rng.standard_normal((max(R, 1), D)) * scale + 1).astype(np.float32)
    inv = (rng.standard_normal((max(R, 1), D)) * scale + 1).astype(np.float32)
    src = workloads.zipf_ids(rng, n_all, nodes, 1.0)
    dst = workloads.zipf_ids(rng, n_all, nodes, 1.0)
    if R > 0:
        all_edges = np.stack([src, workloads.zipf_ids(rng, n_all, R, 1.2), dst], 1).astype(np.int64)
    else:
        all_edges = np.stack([src, dst], 1).astype(np.int64)
    return table, rel, inv, all_edges, all_edges[:B].copy()


@pytest.mark.parametrize("kind,nodes,R,D,B,inverse", [
    ("DISTMULT", 5000, 40, 50, 200, True),     # two sides, tiles cut ragged on both axes
    ("COMPLEX", 3001, 11, 100, 130, True),
    ("COMPLEX", 4096, 7, 100, 64, False),      # one side although the edges carry relations
    ("DISTMULT", 2500, 0, 100, 257, False),    # Dot: two-column edges
    ("DISTMULT", 900, 5, 128, 70, True),
    ("DISTMULT", 700, 3, 6, 10, True),
])
def test_filtered_ranks_match_oracle(capi, cuda_device, kind, nodes, R, D, B, inverse):
    rng = np.random.default_rng(nodes + D)
    table, rel, inv, all_edges, edges = _case(rng, nodes, R, D, 20 * B, B)
    fd = O.global_filter(all_edges, edges, False)
    fs = O.global_filter(all_edges, edges, True) if (R > 0 and inverse) else None
    exp_d, exp_s = O.eval_ranks(kind, table, rel if R > 0 else None, inv if (R > 0 and inverse) else None, edges, fd, fs)
    t = lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a)).to(cuda_device)
    status = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    got_d, got_s = capi.eval_ranks(kind, t(table), t(edges), t(rel) if R > 0 else None, t(inv) if (R > 0 and inverse) else None,
                                   dst_filter=t(fd), src_filter=t(fs), status=status)
    torch.cuda.synchronize()
    assert int(status) == 0
    assert np.array_equal(got_d.cpu().numpy(), exp_d)
    if exp_s is None:
        assert got_s is None
    else:
        assert np.array_equal(got_s.cpu().numpy(), exp_s)
    # filtered evaluation removes the positive's own node: no rank can exceed the number of nodes
    assert int(got_d.max()) <= nodes and int(got_d.min()) >= 1


def test_unfiltered_counts_the_positive_itself_and_duplicate_pairs_change_nothing(capi, cuda_device):
    rng = np.random.default_rng(5)
    table, rel, inv, all_edges, edges = _case(rng, 1500, 9, 50, 2000, 100)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda_device)
    exp_d, exp_s = O.eval_ranks("DISTMULT", table, rel, inv, edges)
    got_d, got_s = capi.eval_ranks("DISTMULT", t(table), t(edges), t(rel), t(inv))
    assert np.array_equal(got_d.cpu().numpy(), exp_d) and np.array_equal(got_s.cpu().numpy(), exp_s)
    assert int(got_d.min()) >= 2  # the candidate equal to the positive's destination scores exactly the positive score
    fd = O.global_filter(all_edges, edges, False)
    twice = np.concatenate([fd, fd[::-1], fd[:7]])
    once, _ = capi.eval_ranks("DISTMULT", t(table), t(edges), t(rel), t(inv), dst_filter=t(fd))
    dup, _ = capi.eval_ranks("DISTMULT", t(table), t(edges), t(rel), t(inv), dst_filter=t(twice))
    assert torch.equal(once, dup)


def test_candidate_list_and_bad_ids(capi, cuda_device):
    rng = np.random.default_rng(6)
    table, rel, inv, all_edges, edges = _case(rng, 2000, 4, 100, 1000, 50)
    neg_ids = rng.choice(2000, 333, replace=False).astype(np.int64)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda_device)
    filt = np.stack([rng.integers(0, 50, 40), rng.integers(0, 333, 40)], 1).astype(np.int64)
    exp_d, exp_s = O.eval_ranks("COMPLEX", table, rel, inv, edges, filt, None, neg_ids=neg_ids)
    got_d, got_s = capi.eval_ranks("COMPLEX", t(table), t(edges), t(rel), t(inv), dst_filter=t(filt), neg_ids=t(neg_ids))
    assert np.array_equal(got_d.cpu().numpy(), exp_d) and np.array_equal(got_s.cpu().numpy(), exp_s)
    bad = edges.copy()
    bad[3, 0] = 2000      # source out of range
    bad[7, 1] = -1        # relation out of range
    status = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    got_d, got_s = capi.eval_ranks("COMPLEX", t(table), t(bad), t(rel), t(inv), status=status)
    torch.cuda.synchronize()
    assert int(status) & 8
    assert int(got_d[3]) == 0 and int(got_d[7]) == 0 and int(got_s[3]) == 0
    ok = np.ones(50, bool)
    ok[[3, 7]] = False
    exp_d, _ = O.eval_ranks("COMPLEX", table, rel, inv, edges)
    assert np.array_equal(got_d.cpu().numpy()[ok], exp_d[ok])


@pytest.mark.parametrize("nodes,B,D,scale", [
    (255, 127, 64, 1.0), (256, 128, 65, 1e-3), (257, 129, 128, 30.0),   # edges of the score tiles; odd, half and full row widths
    (513, 1, 2, 1.0), (40, 300, 100, 1e-12), (5000, 40, 98, 1e6),       # few candidates, few queries, values far from one
    (148 * 256 + 1, 3, 100, 1.0), (77_000, 130, 66, 1.0), (115_000, 2, 65, 1.0),  # several wide candidate tiles a CTA, staged ahead
])
def test_ranks_are_exact_at_tile_edges_and_on_ties(capi, cuda_device, nodes, B, D, scale):
    """The counting pass compares scores computed on the tensor cores and evaluates only what those leave open: ranks must still be
    those of the fp32 chains, ties included."""
    rng = np.random.default_rng(nodes * 1000 + B)
    table = (rng.standard_normal((nodes, D)) * scale).astype(np.float32)
    table[nodes // 2] = table[0]                      # equal candidates
    table[nodes - 1] = np.nextafter(table[0], np.float32(np.inf))  # and one that differs in the last bits
    table[1] = 0.0                                    # every score equals its positive's
    table[2] *= 1000.0                                # a row far larger than its neighbours
    edges = rng.integers(0, nodes, (B, 2)).astype(np.int64)
    edges[0] = (1, 0)
    edges[-1] = (nodes - 1, 0)
    filt = np.stack([rng.integers(0, B, 3 * B), rng.integers(0, nodes, 3 * B)], 1).astype(np.int64)
    exp, _ = O.eval_ranks("DISTMULT", table, None, None, edges, filt, None)
    t = lambda a: torch.from_numpy(a).to(cuda_device)  # noqa: E731
    got, none = capi.eval_ranks("DISTMULT", t(table), t(edges), dst_filter=t(filt))
    assert none is None and np.array_equal(got.cpu().numpy(), exp)


@pytest.mark.parametrize("D,size", [(64, 1e-23), (64, 3e-23), (100, 1e-22), (50, 1e-28), (64, 2e-36), (128, 1e-36), (64, 1e-38), (64, 1e-41), (100, 1e19), (64, 3e37)])
def test_ranks_are_exact_for_query_rows_of_any_size(capi, cuda_device, D, size):
    """Query rows (source times relation) so small that their squares vanish, down to numbers that are not normal, and so large that they
    overflow: a comparison may be decided on the tensor cores only by a bound that holds there too."""
    rng = np.random.default_rng(D)
    nodes, R, B = 700, 4, 150
    cand = 5e-3 if size < 1 else 1.0
    table = (rng.standard_normal((nodes, D)) * cand).astype(np.float32)
    table[5] = table[6]
    rel = (rng.standard_normal((R, D)) * (size / cand)).astype(np.float32)
    edges = np.stack([rng.integers(0, nodes, B), rng.integers(0, R, B), rng.integers(0, nodes, B)], 1).astype(np.int64)
    filt = np.stack([rng.integers(0, B, B), rng.integers(0, nodes, B)], 1).astype(np.int64)
    with np.errstate(over="ignore", invalid="ignore", under="ignore"):
        exp_d, exp_s = O.eval_ranks("DISTMULT", table, rel, rel, edges, filt, filt)
    t = lambda a: torch.from_numpy(a).to(cuda_device)  # noqa: E731
    got_d, got_s = capi.eval_ranks("DISTMULT", t(table), t(edges), t(rel), t(rel), dst_filter=t(filt), src_filter=t(filt))
    assert np.array_equal(got_d.cpu().numpy(), exp_d) and np.array_equal(got_s.cpu().numpy(), exp_s)


@pytest.mark.parametrize("nodes,D", [(148 * 256 + 1, 100), (77_000, 66), (300, 128)])
def test_a_workspace_without_the_optional_part_will_do(capi, cuda_device, monkeypatch, nodes, D):
    """the last 148 x 128 KB, in which wide candidate tiles are split ahead; one byte less than that is refused"""
    lib = capi.load_library()

    class Less:
        def __init__(self, less):
            self.less = less

        def __getattr__(self, name):
            return getattr(lib, name)

        def ge2_eval_workspace_bytes(self, d):
            return lib.ge2_eval_workspace_bytes(d) - self.less

    rng = np.random.default_rng(nodes)
    table = rng.standard_normal((nodes, D)).astype(np.float32)
    edges = rng.integers(0, nodes, (130, 2)).astype(np.int64)
    exp, _ = O.eval_ranks("DISTMULT", table, None, None, edges, np.empty((0, 2), np.int64), None)
    t_table, t_edges = torch.from_numpy(table).to(cuda_device), torch.from_numpy(edges).to(cuda_device)
    for less in (1, 148 * 131072):
        monkeypatch.setattr(capi, "load_library", lambda less=less: Less(less))
        got, _ = capi.eval_ranks("DISTMULT", t_table, t_edges)
        assert np.array_equal(got.cpu().numpy(), exp)
    monkeypatch.setattr(capi, "load_library", lambda: Less(148 * 131072 + 1))
    with pytest.raises(capi.Ge2Error):
        capi.eval_ranks("DISTMULT", t_table, t_edges)
