"""GPU parity of the fused link-prediction step (through the C ABI) against the reference fixtures and the oracle."""
from pathlib import Path

import numpy as np
import pytest

import ge2_oracle as O
import workloads
from gpu_helpers import rel_err, run_lp_step

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).resolve().parent / "golden"

# 1e-4 relative for the fp32 path, 1e-2 for 16-bit tensor tiles
TOL = {"fp32": 1e-4, "f16": 1e-2}


def check_against(res, ref, tol, S):
    assert res["status"] == 0
    assert abs(res["loss"] - ref["loss"]) <= tol * abs(ref["loss"])
    assert rel_err(res["node_grad"], ref["node_grad"]) < tol
    if "rel_grad" in ref and ref["rel_grad"] is not None:
        assert rel_err(res["rel_grad"], ref["rel_grad"]) < tol
    if S == 2:
        assert rel_err(res["inv_rel_grad"], ref["inv_rel_grad"]) < tol
    if "neg_scores" in res:
        masked = ref["neg_scores"] == O.MASK_VALUE
        assert np.array_equal(res["neg_scores"] == O.MASK_VALUE, masked)
        scale = np.abs(ref["neg_scores"][~masked]).max()
        assert np.abs(res["neg_scores"][~masked] - ref["neg_scores"][~masked]).max() < tol * scale
        assert rel_err(res["pos_scores"], ref["pos_scores"]) < tol
        if S == 2:
            assert np.abs(res["inv_neg_scores"][~masked] - ref["inv_neg_scores"][~masked]).max() < tol * np.abs(ref["inv_neg_scores"][~masked]).max()
            assert rel_err(res["inv_pos_scores"], ref["inv_pos_scores"]) < tol


def golden_ref(name):
    g = np.load(GOLDEN / f"{name}.npz")
    ref = {k[4:]: g[k] for k in g.files if k.startswith("ref_")}
    ref["loss"] = float(ref["loss"])
    return ref


@pytest.mark.parametrize("precision", ["fp32", "f16"])
@pytest.mark.parametrize("name", sorted(workloads.GOLDEN_CASES))
def test_golden_fixtures(capi, cuda_device, name, precision):
    case = workloads.golden_case(name)
    ref = golden_ref(name)
    S = 2 if case.src_negs is not None else 1
    res = run_lp_step(capi, case, cuda_device, precision=precision, filter_mode="pairs")
    check_against(res, ref, TOL[precision], S)


@pytest.mark.parametrize("name", ["complex_d100_deg_padded", "dot_d100_deg"])
def test_filter_from_degree_rows_and_row_index(capi, cuda_device, name):
    """The on-device filter derivation and the table-with-row-index addressing give the same result as the reference's forms."""
    case = workloads.golden_case(name)
    ref = golden_ref(name)
    S = 2 if case.src_negs is not None else 1
    res = run_lp_step(capi, case, cuda_device, filter_mode="deg_rows", indirect=True)
    check_against(res, ref, TOL["fp32"], S)


@pytest.mark.parametrize("precision", ["fp32", "f16"])
@pytest.mark.parametrize("kind,B,C,N,D,R,U,n_deg,relations,inverse", [
    ("DISTMULT", 1000, 10, 1000, 50, 1345, 14951, 0, True, True),     # configuration 1 shape
    ("COMPLEX", 2000, 2, 1000, 100, 1000, 30000, 500, True, True),    # configuration 2 shape, fewer chunks
    ("DISTMULT", 1001, 7, 130, 128, 50, 900, 30, True, True),          # ragged: B % C != 0, N % 64 != 0
    ("DISTMULT", 3000, 3, 1000, 100, 0, 20000, 500, False, False),     # Dot decoder, configuration 3 shape
    ("COMPLEX", 64, 1, 5, 6, 3, 40, 2, True, True),                    # tiny everything
])
def test_against_oracle(capi, cuda_device, precision, kind, B, C, N, D, R, U, n_deg, relations, inverse):
    case = workloads.make_case(kind, B, C, N, D, max(R, 1), U, n_deg, seed=B + N + D, relations=relations, inverse=inverse, alpha=1.1)
    S = 2 if case.src_negs is not None else 1
    o = O.lp_train_forward_backward(case.kind, case.edges, case.emb, case.rel, case.inv_rel, case.dst_negs, case.src_negs, case.filt,
                                    case.filt if S == 2 else None)
    ref = dict(loss=o.loss, node_grad=o.node_grad, rel_grad=o.rel_grad, inv_rel_grad=o.inv_rel_grad, neg_scores=o.neg_scores,
               pos_scores=o.pos_scores, inv_neg_scores=o.inv_neg_scores, inv_pos_scores=o.inv_pos_scores)
    res = run_lp_step(capi, case, cuda_device, precision=precision, filter_mode="deg_rows" if n_deg else "none")
    check_against(res, ref, TOL[precision], S)
    # without the score dump the training outputs are unchanged
    res2 = run_lp_step(capi, case, cuda_device, precision=precision, filter_mode="pairs", dump_scores=False)
    assert abs(res2["loss"] - res["loss"]) <= 1e-6 * abs(res["loss"]) + 1e-6
    assert rel_err(res2["node_grad"], res["node_grad"]) < 1e-5


@pytest.mark.parametrize("emb_scale", [0.6, 0.75])
def test_peaked_softmax_on_the_tensor_path(capi, cuda_device, emb_scale):
    """Trained-looking inputs: |embedding| up to 3 and more, scores up to +-60...90, and rows whose softmax mass sits on a
    dozen or fewer of the 1 000 negatives.  The fp16 probabilities of the gradient pass carry a power-of-two scale so that the small
    ones stay out of the subnormal range; the stated 1e-2 bound must hold here as it does on the mild fixtures."""
    case = workloads.make_case("COMPLEX", 1000, 2, 1000, 100, 200, 20000, 500, seed=5, relations=True, inverse=True, alpha=1.1, emb_scale=emb_scale)
    o = O.lp_train_forward_backward(case.kind, case.edges, case.emb, case.rel, case.inv_rel, case.dst_negs, case.src_negs, case.filt, case.filt)
    ns = o.neg_scores.astype(np.float64).copy()
    ns[o.neg_scores == O.MASK_VALUE] = -np.inf
    p = np.exp(ns - ns.max(1, keepdims=True))
    p /= p.sum(1, keepdims=True)
    k90 = ((np.sort(p, 1)[:, ::-1].cumsum(1) < 0.9).sum(1) + 1)
    assert np.median(k90) <= 12 and np.abs(case.emb).max() > 2.8  # the case is what the docstring says
    ref = dict(loss=o.loss, node_grad=o.node_grad, rel_grad=o.rel_grad, inv_rel_grad=o.inv_rel_grad, neg_scores=o.neg_scores,
               pos_scores=o.pos_scores, inv_neg_scores=o.inv_neg_scores, inv_pos_scores=o.inv_pos_scores)
    res = run_lp_step(capi, case, cuda_device, precision="f16", filter_mode="deg_rows")
    check_against(res, ref, TOL["f16"], 2)
    res = run_lp_step(capi, case, cuda_device, precision="fp32", filter_mode="deg_rows")
    check_against(res, ref, TOL["fp32"], 2)


def test_relation_grads_accumulate(capi, cuda_device):
    """rel_grad is accumulated into, like autograd's .grad across train_batch(call_step=false) calls."""
    import torch

    from gpu_helpers import dev

    case = workloads.golden_case("distmult_d50_uniform")
    ref = golden_ref("distmult_d50_uniform")
    B, C, N, D, R, U = case.dims
    edges = dev(case.edges, cuda_device)
    node_grad = torch.empty((U, D), device=cuda_device)
    loss = torch.empty(1, device=cuda_device)
    rg = torch.ones((R, D), device=cuda_device)
    irg = torch.zeros((R, D), device=cuda_device)
    # the descriptor holds raw pointers only: keep every tensor alive until the step has run
    emb, dn, sn, rel, inv = (dev(a, cuda_device) for a in (case.emb, case.dst_negs, case.src_negs, case.rel, case.inv_rel))
    d = capi.make_lp_desc(decoder=case.kind, precision="fp32", B=B, Cn=C, N=N, D=D, R=R, U=U, node_emb=emb,
                          src_ids=edges, dst_ids=edges[:, 2], rel_ids=edges[:, 1], edge_stride=3, rel_stride=3,
                          dst_negs=dn, src_negs=sn, rel=rel, inv_rel=inv, node_grad=node_grad, rel_grad=rg, inv_rel_grad=irg, loss=loss)
    ws = torch.empty(capi.lp_workspace_bytes(d), dtype=torch.uint8, device=cuda_device)
    d.workspace, d.workspace_bytes = ws.data_ptr(), ws.numel()
    capi.lp_step(d)
    capi.lp_step(d)
    torch.cuda.synchronize()
    assert rel_err(rg.cpu().numpy(), 1.0 + 2.0 * ref["rel_grad"]) < 1e-4
    assert rel_err(irg.cpu().numpy(), 2.0 * ref["inv_rel_grad"]) < 1e-4
    assert rel_err(node_grad.cpu().numpy(), ref["node_grad"]) < 1e-4  # node_grad is overwritten, not accumulated


def test_bad_inputs_set_status_without_faulting(capi, cuda_device):
    case = workloads.golden_case("dot_d100_deg")
    B, C, N, D, R, U = case.dims
    bad = workloads.golden_case("dot_d100_deg")
    bad.edges = bad.edges.copy()
    bad.edges[3, 0] = U + 5      # out-of-range local id
    bad.dst_negs = bad.dst_negs.copy()
    bad.dst_negs[1, 2] = -4
    res = run_lp_step(capi, bad, cuda_device, filter_mode="none")
    assert res["status"] & 8
    dup = workloads.golden_case("dot_d100_deg")
    dup.filt = np.array([[0, 1], [5, 1]], np.int64)  # two rows of chunk 0 masked in the same column
    res = run_lp_step(capi, dup, cuda_device, filter_mode="pairs")
    assert res["status"] & 4


def test_argument_validation(capi, cuda_device):
    import torch

    t = torch.zeros(16, device=cuda_device)
    i = torch.zeros(16, dtype=torch.int64, device=cuda_device)
    with pytest.raises(capi.Ge2Error):  # D > 128
        d = capi.make_lp_desc(decoder="DISTMULT", precision="fp32", B=2, Cn=1, N=2, D=200, R=0, U=2, node_emb=t, src_ids=i, dst_ids=i,
                              dst_negs=i, node_grad=t, loss=t)
        capi.lp_workspace_bytes(d)
    with pytest.raises(capi.Ge2Error):  # odd D with the complex operator
        d = capi.make_lp_desc(decoder="COMPLEX", precision="fp32", B=2, Cn=1, N=2, D=5, R=1, U=2, node_emb=t, src_ids=i, dst_ids=i,
                              rel_ids=i, dst_negs=i, rel=t, node_grad=t, rel_grad=t, loss=t)
        capi.lp_workspace_bytes(d)
    d = capi.make_lp_desc(decoder="DISTMULT", precision="fp32", B=2, Cn=1, N=2, D=4, R=0, U=2, node_emb=t, src_ids=i, dst_ids=i,
                          dst_negs=i, node_grad=t, loss=t)
    with pytest.raises(capi.Ge2Error):  # no workspace
        capi.lp_step(d)


@pytest.mark.parametrize("precision,B,C,N,D,R,U,n_deg", [
    ("fp32", 10_000, 10, 1000, 100, 1000, 60_000, 500),   # the benchmark's batch
    ("f16", 10_000, 10, 1000, 100, 1000, 60_000, 500),
    ("f16", 12_800, 10, 2000, 128, 300, 90_000, 1000),    # d = 128, 2 000 negatives per chunk (ragged last tile), 200 row blocks
])
def test_full_size_step_is_the_sum_of_its_chunks(capi, cuda_device, precision, B, C, N, D, R, U, n_deg):
    """Size-independent property at the benchmark's full batch (ComplEx d=100, B=10 000, 10 chunks x 1 000 shared negatives,
    half of them degree-based, both corruption sides): chunks do not interact, so the loss and every gradient of the whole
    step equal the sums over ten single-chunk steps.  The whole step runs 160 row blocks (one full round of unsplit blocks
    plus split leftovers on the tensor path), a single chunk runs 16 blocks split over several CTAs each -- different
    launch shapes of the same kernels."""
    case = workloads.make_case("COMPLEX", B, C, N, D, R, U, n_deg, seed=77, relations=True, inverse=True, alpha=1.1)
    whole = run_lp_step(capi, case, cuda_device, precision=precision, filter_mode="pairs", dump_scores=False)
    assert whole["status"] == 0
    npc = B // C
    loss = 0.0
    node_grad = np.zeros((U, D), np.float64)
    rel_grad = np.zeros((R, D), np.float64)
    inv_rel_grad = np.zeros((R, D), np.float64)
    for c in range(C):
        rows = slice(c * npc, (c + 1) * npc)
        f = case.filt[(case.filt[:, 0] >= c * npc) & (case.filt[:, 0] < (c + 1) * npc)].copy()
        f[:, 0] -= c * npc
        part = workloads.BatchCase(case.kind, case.edges[rows], case.emb, case.state, case.rel, case.inv_rel, case.dst_negs[c:c + 1],
                                   case.src_negs[c:c + 1], None, f)
        res = run_lp_step(capi, part, cuda_device, precision=precision, filter_mode="pairs", dump_scores=False)
        assert res["status"] == 0
        loss += res["loss"]
        node_grad += res["node_grad"]
        rel_grad += res["rel_grad"]
        inv_rel_grad += res["inv_rel_grad"]
    tol = 2e-4 if precision == "fp32" else 2e-3  # both sides run the same arithmetic; only the order of fp32 additions differs
    assert abs(whole["loss"] - loss) <= tol * abs(loss)
    assert rel_err(whole["node_grad"], node_grad) < tol
    assert rel_err(whole["rel_grad"], rel_grad) < tol
    assert rel_err(whole["inv_rel_grad"], inv_rel_grad) < tol
    assert np.abs(node_grad).max() > 0


@pytest.mark.parametrize("kind,B,C,N,D", [
    ("DISTMULT", 129, 1, 63, 64), ("DISTMULT", 128, 1, 65, 65), ("COMPLEX", 257, 2, 1, 66),   # one row, one negative past a tile
    ("DISTMULT", 7, 3, 200, 1), ("COMPLEX", 1500, 2, 900, 128), ("DISTMULT", 60, 1, 2000, 17),  # blocks cut between CTAs; narrow rows
])
def test_split_operand_tiles_at_their_edges(capi, cuda_device, kind, B, C, N, D):
    """The fp32 path's exact bf16 splitting and its tile sums: gradients to a few fp32 roundings of float64 contractions."""
    case = workloads.make_case(kind, B, C, N, D, 5, 150, N // 2, 31 + D)
    o = O.lp_train_forward_backward(case.kind, case.edges, case.emb, case.rel, case.inv_rel, case.dst_negs, case.src_negs, case.filt, case.filt)
    exp = dict(loss=o.loss, node_grad=o.node_grad, rel_grad=o.rel_grad, inv_rel_grad=o.inv_rel_grad)
    got = run_lp_step(capi, case, cuda_device, "fp32", "pairs")
    assert got["status"] == 0
    assert abs(got["loss"] - exp["loss"]) <= 2e-6 * abs(exp["loss"])
    for key in ("node_grad", "rel_grad", "inv_rel_grad"):
        assert rel_err(got[key], exp[key]) <= 5e-6, key


@pytest.mark.parametrize("kind,B,C,N,D", [
    ("DISTMULT", 38400, 300, 40, 50),    # a tile a block, four blocks a CTA: every block brings its own rows, and one issuing warp has none of some
    ("COMPLEX", 38400, 300, 40, 100),    # the same with two 64-column blocks a row, the halves of the rows through one buffer
    ("DISTMULT", 51300, 300, 100, 128),  # two tiles a block, blocks of 128 and of 43 rows
    ("COMPLEX", 25000, 125, 150, 66),    # three tiles a block: as many as are under way
])
def test_short_blocks_of_the_split_operand_scores(capi, cuda_device, kind, B, C, N, D):
    """Many short blocks a CTA, so that rows, tiles and scores of several are under way at once; twice, for what one pass leaves to the next."""
    case = workloads.make_case(kind, B, C, N, D, 20, 5000, 0, seed=B + N + D, relations=True, inverse=True, alpha=1.1)
    o = O.lp_train_forward_backward(case.kind, case.edges, case.emb, case.rel, case.inv_rel, case.dst_negs, case.src_negs, case.filt, case.filt)
    for _ in range(2):
        res = run_lp_step(capi, case, cuda_device, "fp32", "pairs", dump_scores=False)
        check_against(res, dict(loss=o.loss, node_grad=o.node_grad, rel_grad=o.rel_grad, inv_rel_grad=o.inv_rel_grad), TOL["fp32"], 2)


@pytest.mark.parametrize("kind,B,C,N,D", [("DISTMULT", 130, 1, 66001, 128), ("COMPLEX", 210, 70, 1000, 66), ("DISTMULT", 300, 2, 70001, 50), ("COMPLEX", 1290, 10, 7003, 100)])
def test_streaming_softmax_tiles_at_their_edges(capi, cuda_device, kind, B, C, N, D):
    """The fp16 path with a dK that does not stay in the L2 (which of its forms a shape gets: lp_uses_flash; the streaming one at sizes of its
    own below): blocks shared by many CTAs, chunks of three rows, one row past a tile; then scores large enough that the reference of a row
    has to move."""
    for scale in (1.0, 6.0):
        case = workloads.make_case(kind, B, C, N, D, 5, 150, N // 2, 77 + D)
        case.emb *= np.float32(scale)
        o = O.lp_train_forward_backward(case.kind, case.edges, case.emb, case.rel, case.inv_rel, case.dst_negs, case.src_negs, case.filt, case.filt)
        got = run_lp_step(capi, case, cuda_device, "f16", "pairs", dump_scores=False)
        assert got["status"] == 0
        assert abs(got["loss"] - o.loss) <= 1e-2 * abs(o.loss)
        for key in ("node_grad", "rel_grad", "inv_rel_grad"):
            assert rel_err(got[key], getattr(o, key)) <= 1e-2, key


@pytest.mark.parametrize("kind,B,C,N,D", [
    ("DISTMULT", 98, 49, 2000, 128), ("DISTMULT", 136, 68, 2000, 128),      # one row block a chunk, many tiles: either side of the line
    ("COMPLEX", 9472, 74, 1000, 66), ("COMPLEX", 9576, 76, 1000, 66),       # as many chunk sides as SMs, so no block is cut, and a few more
    ("DISTMULT", 1500, 500, 300, 66), ("DISTMULT", 1440, 480, 300, 66),     # a last tile that is mostly padding
    ("DISTMULT", 200, 90, 2000, 50), ("DISTMULT", 200, 70, 2000, 50),       # rows of 64 columns
    ("DISTMULT", 10368, 27, 1300, 50), ("DISTMULT", 9984, 26, 1300, 50),    # ... and 12 tiles a CTA
    ("COMPLEX", 24064, 47, 2000, 66), ("COMPLEX", 23552, 46, 2000, 66),     # 40 of wider rows
])
def test_both_fp16_forms_where_the_rule_between_them_lies(capi, cuda_device, kind, B, C, N, D):
    case = workloads.make_case(kind, B, C, N, D, 5, 150, min(N, 50), 9 + D)
    o = O.lp_train_forward_backward(case.kind, case.edges, case.emb, case.rel, case.inv_rel, case.dst_negs, case.src_negs, case.filt, case.filt)
    got = run_lp_step(capi, case, cuda_device, "f16", "pairs", dump_scores=False)
    assert got["status"] == 0
    assert abs(got["loss"] - o.loss) <= 1e-2 * abs(o.loss)
    for key in ("node_grad", "rel_grad", "inv_rel_grad"):
        assert rel_err(got[key], getattr(o, key)) <= 1e-2, key


@pytest.mark.parametrize("kind,B,C,N,D", [
    ("DISTMULT", 3870, 30, 4001, 128), ("COMPLEX", 330, 110, 1000, 66), ("DISTMULT", 7740, 60, 3001, 50), ("COMPLEX", 640, 160, 1000, 50)])
def test_streaming_softmax_where_it_is_taken(capi, cuda_device, kind, B, C, N, D):
    """as test_streaming_softmax_tiles_at_their_edges, at sizes that the rule gives to that form: blocks cut between many CTAs, chunks of three
    rows, one row past a tile, scores large enough that the reference of a row has to move"""
    for scale in (1.0, 6.0):
        case = workloads.make_case(kind, B, C, N, D, 5, 150, min(N, 500), 77 + D)
        case.emb *= np.float32(scale)
        o = O.lp_train_forward_backward(case.kind, case.edges, case.emb, case.rel, case.inv_rel, case.dst_negs, case.src_negs, case.filt, case.filt)
        got = run_lp_step(capi, case, cuda_device, "f16", "pairs", dump_scores=False)
        assert got["status"] == 0
        assert abs(got["loss"] - o.loss) <= 1e-2 * abs(o.loss)
        for key in ("node_grad", "rel_grad", "inv_rel_grad"):
            assert rel_err(got[key], getattr(o, key)) <= 1e-2, key


@pytest.mark.parametrize("kind,B,C,N,D", [("DISTMULT", 330, 110, 1000, 128), ("DISTMULT", 1400, 700, 100, 128), ("COMPLEX", 660, 220, 1100, 64)])
@pytest.mark.parametrize("rising", [True, False])
def test_streaming_softmax_reference_moves(capi, cuda_device, kind, B, C, N, D, rising):
    """Scores that grow along a chunk's negatives by dozens of octaves: the reference of a row has to follow in either half of nearly every tile;
    falling ones leave it where the first scores put it.  The second shape has one tile a block."""
    case = workloads.make_case(kind, B, C, N, D, 5, 150, min(N, 50), 21)
    case.emb *= np.linspace(0.1, 4.0, len(case.emb), dtype=np.float32)[:, None]
    for negs in (case.dst_negs, case.src_negs):
        negs.sort(axis=1)
        if not rising:
            negs[:] = negs[:, ::-1].copy()
    case = workloads.BatchCase(case.kind, case.edges, case.emb, case.state, case.rel, case.inv_rel, case.dst_negs, case.src_negs, None, case.filt[:0])
    o = O.lp_train_forward_backward(case.kind, case.edges, case.emb, case.rel, case.inv_rel, case.dst_negs, case.src_negs, case.filt, case.filt)
    got = run_lp_step(capi, case, cuda_device, "f16", "pairs", dump_scores=False)
    assert got["status"] == 0
    # |q| |k| of up to 190 over 128 terms with operands of 11 bits: 190 / sqrt(128) * 2^-11 = 0.01 in a score, so in a probability
    assert abs(got["loss"] - o.loss) <= 1e-2 * abs(o.loss)
    for key in ("node_grad", "rel_grad", "inv_rel_grad"):
        assert np.isfinite(got[key]).all(), key
        assert np.linalg.norm(got[key] - getattr(o, key)) <= 2e-2 * np.linalg.norm(getattr(o, key)), key


@pytest.mark.parametrize("B,C,N,D", [(600, 200, 1000, 128), (1400, 1400, 100, 128), (990, 330, 1100, 64), (1400, 350, 1100, 50)])
@pytest.mark.parametrize("order", ["drawn", "rising", "masked"])
def test_streaming_softmax_row_by_row(capi, cuda_device, B, C, N, D, order):
    """dQ of every row against float64, relative to that row, however far its positive leads the largest negative: 0 to 70 nats (beyond 80 a
    probability leaves fp32).  Sources and destinations use other coordinates than the negatives, so the gradient of a source in the negatives'
    coordinates is dQ alone; operands are multiples of 2^-6 and at most 4, so fp16 holds them and fp32 their products.  "masked": the first 128
    negatives are masked for every row that has a chunk to itself (those the filter words can mask).
    Bound: P is rounded to 11 bits, and where it is small to a multiple of at most 2^-25 of a row's largest (N of them); four arguments of exp2 and the
    lse, of up to 2^8, are rounded to 24 bits; N / 16 sums in tensor memory are cut off after 23; nothing cancels, since the negatives' rows are positive."""
    rng = np.random.default_rng(B + D)
    npc, h = -(-B // C), D // 2
    U = 2 * B + C * N
    grid = lambda a: np.round(a * 64) / 64  # noqa: E731
    emb = np.zeros((U, D), np.float32)
    src, dst, negs = np.arange(B), B + np.arange(B), (2 * B + np.arange(C * N)).reshape(C, N)
    emb[src, :h] = grid(rng.uniform(-0.5, 0.5, (B, h)))
    emb[negs.ravel(), :h] = grid(rng.uniform(0.5, 2.0, (C * N, h)))
    chunk = np.arange(B) // npc
    scores = np.einsum("bd,bnd->bn", emb[src, :h].astype(np.float64), emb[negs[chunk], :h].astype(np.float64))
    if order == "rising":
        by = np.argsort(scores[np.arange(C) * npc], axis=1)  # for the first row of every chunk
        negs = np.take_along_axis(negs, by, axis=1)
        scores = np.take_along_axis(scores, by[chunk], axis=1)
    filt = np.empty((0, 2), np.int64)
    if order == "masked":
        rows = np.arange(0, B, npc)
        filt = np.stack([np.repeat(rows, min(N - 1, 128)), np.tile(np.arange(min(N - 1, 128)), len(rows))], 1)
        scores[filt[:, 0], filt[:, 1]] = -np.inf
    lead = rng.choice([0.0, 4.0, 9.0, 14.0, 20.0, 28.0, 45.0, 70.0], B)
    emb[src, h:h + 8], emb[dst, h:h + 8] = 4.0, grid((lead + scores.max(1)) / 32)[:, None]  # eight products of 4 and a multiple of 2^-6
    pos = 32 * emb[dst, h].astype(np.float64)
    lse = np.logaddexp(pos, np.logaddexp.reduce(scores, axis=1))
    want = np.einsum("bn,bnd->bd", np.exp(scores - lse[:, None]), emb[negs[chunk], :h].astype(np.float64))
    case = workloads.BatchCase("DISTMULT", np.stack([src, dst], 1).astype(np.int64), emb, np.zeros_like(emb), None, None, negs.astype(np.int64), None, None, filt)
    got = run_lp_step(capi, case, cuda_device, "f16", "pairs", dump_scores=False)
    assert got["status"] == 0
    err = np.abs(got["node_grad"][src, :h] - want).max(1) / want.max(1)
    bound = 2.0**-11 + N * 2.0**-25 + 4 * 2.0**-17 + N / 16 * 2.0**-23
    assert err.max() <= bound, [(x, float(err[lead == x].max())) for x in np.unique(lead)]


@pytest.mark.parametrize("kind,B,C,N,D", [("DISTMULT", 10368, 27, 1300, 50), ("COMPLEX", 330, 110, 1000, 66)])
def test_streaming_softmax_gives_way_where_its_parts_have_no_room(capi, cuda_device, kind, B, C, N, D):
    """shapes of the streaming form with a workspace of the two-pass form's size, and a byte less than that"""
    case = workloads.make_case(kind, B, C, N, D, 5, 150, min(N, 50), 9 + D)
    o = O.lp_train_forward_backward(case.kind, case.edges, case.emb, case.rel, case.inv_rel, case.dst_negs, case.src_negs, case.filt, case.filt)
    parts = 148 * 2 * 128 * (64 if D <= 64 else 128) * 4
    got = run_lp_step(capi, case, cuda_device, "f16", "pairs", dump_scores=False, less_workspace=parts)
    assert got["status"] == 0
    assert abs(got["loss"] - o.loss) <= 1e-2 * abs(o.loss)
    for key in ("node_grad", "rel_grad", "inv_rel_grad"):
        assert rel_err(got[key], getattr(o, key)) <= 1e-2, key
    with pytest.raises(capi.Ge2Error):
        run_lp_step(capi, case, cuda_device, "f16", "pairs", dump_scores=False, less_workspace=parts + 1)


@pytest.mark.parametrize("kind,B,C,N,D", [("COMPLEX", 600, 3, 300, 50), ("COMPLEX", 500, 2, 7001, 100), ("DISTMULT", 300, 2, 3000, 128), ("DISTMULT", 257, 2, 640, 3)])
def test_one_node_in_most_edges_and_negatives(capi, cuda_device, kind, B, C, N, D):
    """Rows of a node that most edges and degree negatives have are added up where they meet, and leave as sums."""
    case = workloads.make_case(kind, B, C, N, D, 5, 400, int(0.9 * N), seed=B + D, relations=True, inverse=True, alpha=3.0)
    o = O.lp_train_forward_backward(case.kind, case.edges, case.emb, case.rel, case.inv_rel, case.dst_negs, case.src_negs, case.filt, case.filt)
    res = run_lp_step(capi, case, cuda_device, "fp32", "deg_rows", dump_scores=False)
    assert res["status"] == 0
    assert abs(res["loss"] - o.loss) <= 1e-5 * abs(o.loss)
    for key in ("node_grad", "rel_grad", "inv_rel_grad"):
        assert rel_err(res[key], getattr(o, key)) <= 1e-4, key
