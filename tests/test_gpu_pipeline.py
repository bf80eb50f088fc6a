"""Whole training steps on the GPU (sampler -> unique-map -> fused decoder -> Adagrad scatter) against the oracle's
restatement of the reference trainer loop, fed with the negatives the device sampler drew."""
import numpy as np
import pytest
import torch

import ge2_oracle as O
import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("decoder,D,R,deg", [("DISTMULT", 50, 40, 0.0), ("COMPLEX", 100, 25, 0.5), ("DISTMULT", 100, 1, 0.5)])
def test_three_steps_match_oracle(ge2, cuda_device, decoder, D, R, deg):
    from importlib import import_module

    pipeline = import_module("ge-2_b200.pipeline")
    rng = np.random.default_rng(11)
    nodes, B, C, N = 5000, 600, 3, 200
    table = (0.3 * rng.standard_normal((nodes, D))).astype(np.float32)
    # non-zero starting state: with state = 0 the first Adagrad step is -lr * sign(g), which turns rounding noise in a
    # near-zero gradient into a 0.2-wide difference and says nothing about parity
    state = (0.01 + 0.05 * rng.random((nodes, D))).astype(np.float32)
    has_rel = R > 1
    rel = (1 + 0.2 * rng.standard_normal((R, D))).astype(np.float32) if has_rel else None
    inv_rel = (1 + 0.2 * rng.standard_normal((R, D))).astype(np.float32) if has_rel else None
    cfg = pipeline.PipelineConfig(decoder=decoder, B=B, C=C, N=N, degree_fraction=deg, D=D, R=R, domain=nodes, lr=0.1, precision="fp32")
    t = lambda a: None if a is None else torch.from_numpy(a.copy()).to(cuda_device)
    d_table, d_state, d_rel, d_inv = t(table), t(state), t(rel), t(inv_rel)
    d_rel_state = torch.zeros_like(d_rel) if has_rel else None
    d_inv_state = torch.zeros_like(d_inv) if has_rel else None
    pipe = pipeline.BatchPipeline(cfg, d_table, d_state, d_rel, d_rel_state, d_inv, d_inv_state)
    rel_state = np.zeros_like(rel) if has_rel else None
    inv_state = np.zeros_like(inv_rel) if has_rel else None
    for step in range(3):
        cols = [workloads.zipf_ids(rng, B, nodes, 1.0)] + ([workloads.zipf_ids(rng, B, R, 1.2)] if has_rel else []) + [workloads.zipf_ids(rng, B, nodes, 1.0)]
        edges = np.stack(cols, axis=1).astype(np.int64)
        pipe.step(torch.from_numpy(edges).to(cuda_device), step)
        torch.cuda.synchronize()
        # replay the device sampler's draws through the oracle
        packed = pipe.packed.cpu().numpy()
        CN = C * N
        S = cfg.sides
        src_negs = packed[2 * B:2 * B + CN].reshape(C, N) if S == 2 else None
        dst_negs = packed[2 * B + (S - 1) * CN:].reshape(C, N)
        filt = O.deg_negative_local_filter(pipe.deg_rows.cpu().numpy(), B) if cfg.n_deg > 0 else None
        loss, U = O.train_step(decoder, table, state, rel, rel_state, inv_rel, inv_state, edges, dst_negs, src_negs, filt, filt, 0.1, nodes)
        assert int(pipe.count[0]) == U and int(pipe.count[1]) == 0 and int(pipe.status) == 0
        assert abs(float(pipe.loss) - loss) <= 1e-4 * abs(loss)
        assert np.abs(d_table.cpu().numpy() - table).max() <= 1e-4 * np.abs(table).max()
        assert np.abs(d_state.cpu().numpy() - state).max() <= 1e-4 * max(np.abs(state).max(), 1e-12)
        if has_rel:
            assert np.abs(d_rel.cpu().numpy() - rel).max() <= 1e-4 * np.abs(rel).max()
            assert np.abs(d_inv.cpu().numpy() - inv_rel).max() <= 1e-4 * np.abs(inv_rel).max()


def test_graph_replay_equals_host_issued_steps(ge2, cuda_device):
    """The resident form reads its batch index from device memory; a captured CUDA graph replayed three times must leave
    the tables where three host-issued steps leave them (up to the order of the gradient atomics)."""
    from importlib import import_module

    pipeline = import_module("ge-2_b200.pipeline")
    rng = np.random.default_rng(21)
    nodes, B, C, N, D, R, nb = 6000, 512, 2, 256, 100, 17, 5
    table = (0.3 * rng.standard_normal((nodes, D))).astype(np.float32)
    state = (0.01 + 0.05 * rng.random((nodes, D))).astype(np.float32)
    rel = (1 + 0.2 * rng.standard_normal((R, D))).astype(np.float32)
    edges = np.stack([workloads.zipf_ids(rng, nb * B, nodes, 1.0), workloads.zipf_ids(rng, nb * B, R, 1.2),
                      workloads.zipf_ids(rng, nb * B, nodes, 1.0)], axis=1).astype(np.int64)
    d_edges = torch.from_numpy(edges).to(cuda_device)
    results = []
    for mode in ("host", "graph", "pipelined"):
        cfg = pipeline.PipelineConfig("COMPLEX", B, C, N, 0.5, D, R, nodes, lr=0.1, precision="fp32")
        t = lambda a: torch.from_numpy(a.copy()).to(cuda_device)
        d_table, d_state, d_rel, d_inv = t(table), t(state), t(rel), t(rel)
        pipe = pipeline.BatchPipeline(cfg, d_table, d_state, d_rel, torch.zeros_like(d_rel), d_inv, torch.zeros_like(d_inv))
        if mode == "host":
            for _ in range(3):
                pipe.enqueue_resident(d_edges, nb)
        else:
            # one host-issued step, then the capture; the pipelined form draws batch t+1 on a side stream during step t
            g = pipe.capture_resident(d_edges, nb) if mode == "graph" else pipe.capture_pipelined(d_edges, nb)
            g.replay()
            g.replay()
        pipe.check_status()
        assert pipe.step_dev.tolist() == [3, 4]
        results.append((d_table.cpu().numpy(), d_state.cpu().numpy(), d_rel.cpu().numpy(), float(g.loss if mode == "pipelined" else pipe.loss)))
    for other in results[1:]:
        for a, b in zip(results[0][:3], other[:3]):
            assert np.abs(a - b).max() <= 1e-5 * np.abs(a).max()
        assert abs(results[0][3] - other[3]) <= 1e-5 * abs(results[0][3])
    assert np.abs(results[0][0] - table).max() > 0  # and the steps did train


@pytest.mark.parametrize("decoder,R,B,C,N,ids_an_sm,idle", [
    ("COMPLEX", 200, 592, 74, 64, None, False),  # a tile for every SM: none is left over, the next batch is drawn behind the scores
    ("COMPLEX", 200, 600, 60, 64, None, True),   # 28 SMs are left over, for 8 880 ids
    ("COMPLEX", 200, 600, 60, 64, 317, False),   # four ids too many
    ("COMPLEX", 200, 600, 60, 64, 318, True),
    ("DOT", 1, 600, 60, 64, 57, False),         # 88 SMs, 5 040 ids
    ("DOT", 1, 600, 60, 64, 58, True),
])
def test_next_batch_drawn_on_idle_sms_or_behind_the_scores(ge2, cuda_device, monkeypatch, decoder, R, B, C, N, ids_an_sm, idle):
    """both places that a pipelined step has for the next batch's sampler and unique-map train the same tables as host-issued steps.
    Bound: a gradient is a sum of n <= 24 terms (uniform ids; asserted) of size 2 and less, in any order: two of them are n 2^-24 of 2 n apart at most, from either
    side of the sum, and lr / sqrt(state) <= 1; four steps.  Another batch's ids would move rows by 0.01 and more."""
    from importlib import import_module

    pipeline = import_module("ge-2_b200.pipeline")
    rng = np.random.default_rng(B + C)
    nodes, D, nb, steps = 6000, 64, 5, 4
    if ids_an_sm is not None:
        monkeypatch.setattr(pipeline.BatchPipeline, "IDS_PER_IDLE_SM", ids_an_sm)
    table = (0.3 * rng.standard_normal((nodes, D))).astype(np.float32)
    state = (0.01 + 0.05 * rng.random((nodes, D))).astype(np.float32)
    rel = (1 + 0.2 * rng.standard_normal((2, R, D))).astype(np.float32)
    rel_state = (0.01 + 0.05 * rng.random((2, R, D))).astype(np.float32)
    perm = lambda n: np.concatenate([rng.permutation(n) for _ in range(-(-nb * B // n))])[: nb * B]  # noqa: E731
    cols = [perm(nodes)] + ([perm(R)] if R > 1 else []) + [perm(nodes)]
    d_edges = torch.from_numpy(np.stack(cols, axis=1).astype(np.int64)).to(cuda_device)
    t = lambda a: torch.from_numpy(a.copy()).to(cuda_device)  # noqa: E731
    results, places, losses = [], [], []
    for pipelined in (False, True):
        cfg = pipeline.PipelineConfig(decoder, B, C, N, 0.5, D, R, nodes, lr=0.1, precision="fp32")
        tables = [t(table), t(state)]
        if R > 1:
            tables += [t(rel[0]), t(rel_state[0]), t(rel[1]), t(rel_state[1])]
        pipe = pipeline.BatchPipeline(cfg, *tables)
        if pipelined:
            front = pipe._front
            monkeypatch.setattr(pipe, "_front", lambda *a, **k: (places.append(k.get("sms", 0)) if torch.cuda.is_current_stream_capturing() else None, front(*a, **k)))
            run = pipe.capture_pipelined(d_edges, nb)
            for _ in range(steps - 1):
                run.replay()
        else:
            for _ in range(steps):
                pipe.enqueue_resident(d_edges, nb)
        pipe.check_status()
        assert int(torch.bincount(pipe.packed).max()) <= 24
        results.append([a.cpu().numpy() for a in tables])
        losses.append(run.loss.item() if pipelined else pipe.loss.item())
    assert len(places) == 2 and all((sms > 0) == idle for sms in places)
    for a, b in zip(*results):
        assert np.abs(a - b).max() <= 4 * 2 * 24 * 2.0**-24 * 2 * 24
    assert abs(losses[0] - losses[1]) <= 1e-5 * abs(losses[0])
    assert np.abs(results[0][0] - table).max() > 0.01


@pytest.mark.gpu
def test_host_feed_trains_the_same_batches_as_the_resident_form(cuda_device):
    """Batches fed from pinned host memory through the pipelined graphs (copies on side streams) give the tables and the
    per-step losses of the resident form stepping over the same batches in the same order."""
    from importlib import import_module

    pipeline = import_module("ge-2_b200.pipeline")
    rng = np.random.default_rng(33)
    nodes, B, C, N, D, R, nb = 5000, 384, 2, 128, 64, 11, 6
    table = (0.3 * rng.standard_normal((nodes, D))).astype(np.float32)
    state = (0.01 + 0.05 * rng.random((nodes, D))).astype(np.float32)
    rel = (1 + 0.2 * rng.standard_normal((R, D))).astype(np.float32)
    edges = np.stack([workloads.zipf_ids(rng, nb * B, nodes, 1.0), workloads.zipf_ids(rng, nb * B, R, 1.2),
                      workloads.zipf_ids(rng, nb * B, nodes, 1.0)], axis=1).astype(np.int64)
    host = torch.from_numpy(edges).reshape(nb, B, 3).pin_memory()
    d_edges = torch.from_numpy(edges).to(cuda_device)
    out = []
    for mode in ("resident", "host_feed"):
        cfg = pipeline.PipelineConfig("DISTMULT", B, C, N, 0.5, D, R, nodes, lr=0.1, precision="fp32")
        t = lambda a: torch.from_numpy(a.copy()).to(cuda_device)
        d_table, d_state, d_rel, d_inv = t(table), t(state), t(rel), t(rel)
        pipe = pipeline.BatchPipeline(cfg, d_table, d_state, d_rel, torch.zeros_like(d_rel), d_inv, torch.zeros_like(d_inv))
        losses = torch.zeros(nb, dtype=torch.float32).pin_memory()
        if mode == "resident":
            for i in range(nb - 1):
                pipe.enqueue_resident(d_edges, nb)
                losses[i:i + 1].copy_(pipe.loss)
        else:
            feed = pipeline.HostFeed(pipe, 3)
            feed.start(host[0], host[1])  # trains batch 0
            losses[0:1].copy_(pipe.loss)
            for i in range(1, nb - 1):
                feed.step(host[i + 1], losses[i:i + 1])  # trains batch i, draws batch i+1
            feed.drain()
        pipe.check_status()
        out.append((d_table.cpu().numpy(), d_state.cpu().numpy(), d_rel.cpu().numpy(), losses.numpy().copy()))
    for a, b in zip(out[0], out[1]):
        assert np.abs(a - b).max() <= 1e-5 * np.abs(a).max()
    assert (out[0][3][: nb - 1] > 0).all()


@pytest.mark.parametrize("decoder,D,R,B,C,N,nodes", [("COMPLEX", 50, 9, 33, 2, 30, 300), ("COMPLEX", 128, 3, 1, 1, 1, 5), ("DISTMULT", 101, 7, 700, 3, 65, 90000),
                                                      ("DISTMULT", 62, 300, 16, 1, 600, 900), ("DOT", 128, 1, 17, 1, 40, 100), ("DOT", 3, 1, 500, 7, 33, 2000)])
def test_rows_finished_in_the_backward_pass(ge2, cuda_device, decoder, D, R, B, C, N, nodes):
    """Rows with one occurrence updated where their gradient arises, the others through the gradient buffer: the tables are those of the
    form that sends every row through the buffer."""
    from importlib import import_module

    pipeline = import_module("ge-2_b200.pipeline")
    gen = torch.Generator(device=cuda_device)
    gen.manual_seed(D + B)
    start = [torch.rand((r, D), generator=gen, device=cuda_device) * 0.5 + 0.1 for r in (nodes, nodes, R, R, R, R)]
    edges = torch.stack([torch.randint(m, (B,), generator=gen, device=cuda_device) for m in ((nodes, R, nodes) if R > 1 else (nodes, nodes))], 1).contiguous()
    cfg = pipeline.PipelineConfig(decoder=decoder, B=B, C=C, N=N, degree_fraction=0.3, D=D, R=R, domain=nodes, lr=0.1, precision="fp32")
    results = []
    for fused in (True, False):
        tables = [t.clone() for t in start]
        pipe = pipeline.BatchPipeline(cfg, *(tables if R > 1 else tables[:2]))
        if fused:
            pipe.step(edges, 3)
        else:
            capi = ge2.capi
            capi.sample_negatives(edges, edges[:, -1], edges.shape[1], B, C, N, cfg.n_deg, nodes, cfg.sides == 2, cfg.seed, 3, pipe.packed, pipe.deg_rows)
            pipe._unique(pipe.ids[0])
            d = pipe._make_desc(edges)
            d.node_state = d.row_shared = None
            capi.lp_step(d)
            capi.adagrad_scatter(pipe.table, pipe.state, pipe.unique, pipe.node_grad, 0.1, U=pipe.cap, U_dev=pipe.count, clear_grad=True)
            pipe._update_relations()
        torch.cuda.synchronize()
        assert int(pipe.status) == 0 and int(pipe.node_grad.abs().max() > 0) == 0
        results.append(tables)
    for a, b, s in zip(*results, start):
        assert (a - b).abs().max() <= 2e-5 * max(1e-3, float((a - s).abs().max()))


@pytest.mark.parametrize("decoder,precision,D,R,form", [
    ("COMPLEX", "f16", 100, 9, "issued"), ("DISTMULT", "fp32", 64, 9, "resident"), ("DOT", "f16", 50, 1, "resident"), ("COMPLEX", "fp32", 50, 9, "lp_step"),
    ("DOT", "f16", 100, 1, "lp_step")])
def test_ids_past_the_table_are_reported_and_write_nothing(ge2, cuda_device, decoder, precision, D, R, form):
    """The id domain may be larger than the table (a partition buffer that is not full): an id between the two is flagged, and neither the
    rows behind the table nor the gradient buffer are touched, whether the id occurs once in the batch or more often."""
    from importlib import import_module

    pipeline = import_module("ge-2_b200.pipeline")
    rng = np.random.default_rng(D)
    nodes, past, B, C, N = 700, 900, 96, 3, 64
    both = [torch.from_numpy(rng.random((nodes + past, D), dtype=np.float32) + 0.1).to(cuda_device) for _ in range(2)]
    before = [t.clone() for t in both]
    rels = [torch.from_numpy(rng.random((R, D), dtype=np.float32)).to(cuda_device) for _ in range(4)] if R > 1 else []
    cfg = pipeline.PipelineConfig(decoder, B, C, N, 0.5, D, R, nodes + past, lr=0.1, precision=precision)
    pipe = pipeline.BatchPipeline(cfg, both[0][:nodes], both[1][:nodes], *rels)
    cols = [rng.integers(0, nodes, B)] + ([rng.integers(0, R, B)] if R > 1 else []) + [rng.integers(0, nodes, B)]
    edges = torch.from_numpy(np.stack(cols, 1).astype(np.int64)).to(cuda_device)
    edges[3, 0] = nodes + 5                    # once (unless it is drawn too) and twice, as source and destination
    edges[7, -1] = edges[9, 0] = nodes + past - 1
    if form == "issued":
        pipe.step(edges, 0)
    elif form == "resident":
        pipe.enqueue_resident(edges, 1)
    else:                                      # the entry points one by one, every id of the domain mapped: the kernels' own check
        capi = ge2.capi
        capi.sample_negatives(edges, edges[:, -1], edges.shape[1], B, C, N, cfg.n_deg, cfg.domain, cfg.sides == 2, 1, 0, pipe.packed, pipe.deg_rows)
        capi.unique_bitmap(pipe.packed, cfg.domain, out_unique=pipe.unique, out_inverse=pipe.inverse, out_count=pipe.count, out_shared=pipe.ids[0].shared,
                           twins=pipe.ids[0].twins)
        capi.lp_step(pipe._make_desc(edges))
        pipe._update()
    torch.cuda.synchronize()
    drawn = pipe.packed[2 * B:]
    assert int((drawn >= nodes).sum()) > 0     # uniform negatives fall there as well
    assert int(pipe.status) & 8
    for t, old in zip(both, before):
        assert torch.equal(t[nodes:], old[nodes:])
        assert bool(torch.isfinite(t[:nodes]).all()) and not torch.equal(t[:nodes], old[:nodes])
    assert float(pipe.node_grad.abs().max()) == 0.0


@pytest.mark.parametrize("change", [dict(seed=7), dict(degree_fraction=0.25), dict(domain=2500), dict(decoder="COMPLEX"), dict(lr=0.01), dict(dense_lr=0.02)])
def test_issued_steps_follow_changes_of_the_configuration(ge2, cuda_device, change):
    """step() keeps its launch arguments between calls: a field that the caller changes in between counts from the next step on, as in a
    pipeline that was made with it."""
    from dataclasses import replace
    from importlib import import_module

    pipeline = import_module("ge-2_b200.pipeline")
    nodes, B, C, N, D, R = 3000, 200, 2, 64, 32, 6
    gen = torch.Generator(device=cuda_device)
    gen.manual_seed(5)
    start = [torch.rand((r, D), generator=gen, device=cuda_device) * 0.5 + 0.1 for r in (nodes, nodes, R, R, R, R)]
    edges = [torch.stack([torch.randint(m, (B,), generator=gen, device=cuda_device) for m in (2500, R, 2500)], 1).contiguous() for _ in range(2)]
    results = []
    for made_with_it in (False, True):
        cfg = pipeline.PipelineConfig("DISTMULT", B, C, N, 0.5, D, R, nodes, lr=0.1)
        tables = [t.clone() for t in start]
        pipe = pipeline.BatchPipeline(cfg, *tables)
        pipe.step(edges[0], 0)
        if made_with_it:
            pipe = pipeline.BatchPipeline(replace(cfg, **change), *tables)
        else:
            for name, value in change.items():
                setattr(cfg, name, value)
        pipe.step(edges[1], 1)
        pipe.check_status()
        results.append([pipe.packed.clone()] + tables)
    assert torch.equal(results[0][0], results[1][0])
    for a, b in zip(results[0][1:], results[1][1:]):
        assert (a - b).abs().max() <= 2e-5 * b.abs().max()  # sums of gradients in another order


def test_timing_a_phase_trains_nothing(ge2, cuda_device):
    from importlib import import_module

    pipeline = import_module("ge-2_b200.pipeline")
    nodes, B, C, N, D, R = 3000, 200, 2, 64, 100, 6
    gen = torch.Generator(device=cuda_device)
    gen.manual_seed(8)
    tables = [torch.rand((r, D), generator=gen, device=cuda_device) + 0.1 for r in (nodes, nodes, R, R, R, R)]
    edges = torch.stack([torch.randint(m, (B,), generator=gen, device=cuda_device) for m in (nodes, R, nodes)], 1).contiguous()
    pipe = pipeline.BatchPipeline(pipeline.PipelineConfig("COMPLEX", B, C, N, 0.5, D, R, nodes, precision="f16"), *tables)
    pipe.enqueue_resident(edges, 1)
    kept = tables + [pipe.node_grad, pipe.rel_grads, pipe.loss]
    before = [t.clone() for t in kept]
    for phase in (4, 1, 2):
        assert pipe.time_scores_phase(edges, 3, phase) > 0
    for t, old in zip(kept, before):
        assert torch.equal(t, old)
    pipe.check_status()
