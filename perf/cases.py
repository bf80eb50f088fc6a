"""What the performance of this framework is measured on: the work a user has it do, through its public entry points.

Kinds of case
  step    one training step of pipeline.BatchPipeline on resident edges.  mode "issued": step(), launch by launch, as in an
          exploratory loop; "graph": the captured, software-pipelined steps of an epoch (capture_pipelined); "feed": the same
          with every batch arriving in pinned host memory and the loss read back (HostFeed)
  host    one training step through the C++ host layer in the reference's call order (getBatch, train_batch, updateEmbeddings)
  eval    filtered ranks of a batch of test edges against every node (capi.eval_ranks)
  tour    tournament selection of negatives (capi.tournament_select)
  pairs   scores of chosen negatives and their gradients (capi.selected_neg_scores, _backward)
  state   what happens between two supersteps of partitioned training on one GPU: the partition swap and the rebuild of the
          state's edge list (partition.RelayBuffer.swap, capi.build_state_edges), as PartitionedTrainer.run_epoch calls them

Sizes are those of the five configurations in BASELINE.json (per GPU, where a configuration spans several), of the operator sweeps
in bench.py, and ragged ones between them.  Graphs are synthetic: power-law node and relation ids, seeded; tables are in the
state they have in the middle of a training run (an Adagrad state that is no longer zero)."""
import importlib
import importlib.util
import math
from pathlib import Path

import numpy as np
import torch

ge2 = importlib.import_module("ge-2_b200")
capi = ge2.capi
pipeline = importlib.import_module("ge-2_b200.pipeline")
partition = importlib.import_module("ge-2_b200.partition")

LR = 0.1
RESIDENT_BATCHES = 8  # batches of the resident edge list a training case cycles through
_host_module = None


def _host_layer():
    """The C++ host layer's Python binding (loaded once; it sits beside the package's modules)."""
    global _host_module
    if _host_module is None:
        so = Path(ge2.__file__).resolve().parent / "ge2_host.so"
        spec = importlib.util.spec_from_file_location("ge2_host", so)
        _host_module = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(_host_module)
    return _host_module


# ---------------------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------------------
def _step(name, mode, precision, decoder, nodes, R, D, B, C, N, deg, alpha):
    return dict(name=name, kind="step", mode=mode, precision=precision, decoder=decoder, nodes=nodes, R=R, D=D, B=B, C=C, N=N, deg=deg, alpha=alpha)


def listed():
    return [
        # configuration 1, the smallest step: a loop over batches of a thousand edges, launch by launch, in the default precision
        _step("kg15k_issued_fp32", "issued", "fp32", "DISTMULT", 14_951, 1345, 50, 1000, 10, 1000, 0.0, 1.0),
        # configuration 2: the epoch's step on one GPU, tensor path, and the same epoch in the default precision
        _step("kg1m_graph_f16", "graph", "f16", "COMPLEX", 1_000_000, 1000, 100, 10_000, 10, 1000, 0.5, 1.1),
        _step("kg1m_graph_fp32", "graph", "fp32", "COMPLEX", 1_000_000, 1000, 100, 10_000, 10, 1000, 0.5, 1.1),
        # configuration 3's share of a GPU (four of sixteen partitions), no relations, batches from the host
        _step("social_feed_f16", "feed", "f16", "DOT", 1_211_896, 1, 100, 50_000, 50, 1000, 0.0, 0.5),
        # configuration 5's share of a GPU (four of thirty-two partitions): the largest batch, table and chunk
        _step("kg100m_graph_f16", "graph", "f16", "DISTMULT", 12_500_000, 10_000, 128, 100_000, 100, 2000, 0.0, 1.1),
        # sizes that divide nothing: a middle-sized graph explored launch by launch
        _step("ragged_issued_f16", "issued", "f16", "COMPLEX", 300_007, 237, 50, 7919, 7, 653, 0.5, 1.1),
        # configuration 2 driven by a C++ trainer that keeps the reference's call order
        dict(_step("kg1m_host_f16", "", "f16", "COMPLEX", 1_000_000, 1000, 100, 10_000, 10, 1000, 0.5, 1.1), kind="host"),
        # filtered evaluation: a batch of configuration 1's test edges, and the same on configuration 2's graph
        dict(name="kg15k_eval", kind="eval", decoder="DISTMULT", nodes=14_951, R=1345, D=50, B=1000, per_row=30),
        dict(name="kg1m_eval", kind="eval", decoder="COMPLEX", nodes=1_000_000, R=1000, D=100, B=1000, per_row=30),
        # negatives chosen by tournament for a batch of 50 000 query rows, and training on the chosen ones
        dict(name="tournament", kind="tour", chunks=10, rows=5000, N=1000, K=100, D=100),
        dict(name="pairs_dot", kind="pairs", score="DOT", chunks=10, rows=5000, N=1000, K=100, D=100),
        # configuration 3 between two supersteps, all sixteen partitions at home on one GPU
        dict(name="social_state", kind="state", parts=16, rows=302_974, D=100, edges=68_993_773, cols=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dim(rng, even):
    d = rng.choice([50, 64, 80, 100, 128, rng.randint(16, 128), rng.randint(16, 128)])
    return d + (d & 1) if even else d


def _draw_step(rng, kind):
    decoder = rng.choice(["DISTMULT", "COMPLEX", "DOT"])
    precision = rng.choice(["f16", "f16", "fp32"])
    mode = "" if kind == "host" else rng.choice(["issued", "graph", "graph", "feed"])
    while True:
        B, N = _log(rng, 1000, 100_000), _log(rng, 100, 2000)
        C = max(1, min(100, round(B / _log(rng, 100, 2000))))
        D = _dim(rng, decoder == "COMPLEX")
        sides = 1 if decoder == "DOT" else 2
        if 6 * sides * B * N * D <= (3.0e11 if precision == "f16" else 4.0e10):
            break
    deg = rng.choice([0.0, 0.5, round(rng.uniform(0.1, 0.9), 2)])
    R = 1 if decoder == "DOT" else _log(rng, 10, 10_000)
    case = _step(None, mode, precision, decoder, _log(rng, 10_000, 4_000_000), R, D, B, C, N, deg, round(rng.uniform(0.5, 1.1), 2))
    del case["name"]
    case["kind"] = kind
    return case


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["host", "eval", "eval", "tour", "pairs", "state"])
    if kind in ("step", "host"):
        return _draw_step(rng, kind)
    if kind == "eval":
        decoder = rng.choice(["DISTMULT", "COMPLEX", "DOT"])
        D = _dim(rng, decoder == "COMPLEX")
        nodes = _log(rng, 3000, 1_000_000)
        B = min(_log(rng, 50, 2000), int(4.0e11 / (4 * nodes * D)))
        return dict(kind="eval", decoder=decoder, nodes=nodes, R=1 if decoder == "DOT" else _log(rng, 10, 5000), D=D, B=B, per_row=rng.randint(1, 60))
    if kind == "state":
        parts = rng.choice([8, 16, 32])
        return dict(kind="state", parts=parts, rows=4 * (_log(rng, 10_000, 4_800_000 // parts) // 4), D=_dim(rng, False), edges=_log(rng, 1_000_000, 60_000_000),
                    cols=rng.choice([2, 3]))
    D, rows, chunks = _dim(rng, False), _log(rng, 50, 5000), rng.randint(1, 20)
    T = rng.choice([1, 2, 5, 10, 20, 50, 100, 250])  # negatives a group
    K = max(1, min(500 if kind == "pairs" else 1000, _log(rng, 100, 2000) // T))
    chunks = max(1, min(chunks, 50_000 // rows))
    if kind == "tour":
        return dict(kind="tour", chunks=chunks, rows=rows, N=K * T, K=K, D=D)
    return dict(kind="pairs", score=rng.choice(["DOT", "L2"]), chunks=chunks, rows=rows, N=K * T, K=K, D=D)


# ---------------------------------------------------------------------------------------------------------------------
# inputs, made on the GPU from the seed alone
# ---------------------------------------------------------------------------------------------------------------------
def _power_law(gen, n, domain, alpha):
    """n ids in [0, domain) whose rank-frequency law falls as rank^-alpha (inverse CDF of the continuous law), the ranks scattered
    over the ids by multiplication with a constant that shares no factor with the domain."""
    u = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)
    if abs(alpha - 1.0) < 1e-6:
        x = torch.exp(u * math.log(domain + 1.0))
    else:
        x = (1.0 + u * ((domain + 1.0) ** (1.0 - alpha) - 1.0)).pow(1.0 / (1.0 - alpha))
    rank = (x.floor().long() - 1).clamp_(0, domain - 1)
    step = max(1, int(0.6180339887 * domain))
    while math.gcd(step, domain) != 1:
        step += 1
    return (rank * step + domain // 3) % domain


def _normal(gen, shape, scale, mean=0.0):
    return torch.randn(shape, generator=gen, device="cuda").mul_(scale).add_(mean)


def _adagrad_state(gen, shape):
    return torch.rand(shape, generator=gen, device="cuda").mul_(0.05).add_(0.01)


def _edges(gen, n, nodes, R, alpha):
    cols = [_power_law(gen, n, nodes, alpha)]
    if R > 1:
        cols.append(_power_law(gen, n, R, 1.2))
    cols.append(_power_law(gen, n, nodes, alpha))
    return torch.stack(cols, 1).contiguous()


def _relation_tables(gen, R, D):
    """Relation and inverse-relation table back to back, and their states: the layout a trainer keeps them in."""
    rel, state = _normal(gen, (2, R, D), 0.2, 1.0), _adagrad_state(gen, (2, R, D))
    return rel, state


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return globals()["_prepare_" + case["kind"]](case, gen)


def _prepare_step(case, gen):
    nodes, R, D, B = case["nodes"], case["R"], case["D"], case["B"]
    table, state = _normal(gen, (nodes, D), 0.3), _adagrad_state(gen, (nodes, D))
    rel = rel_state = None
    if R > 1:
        rel, rel_state = _relation_tables(gen, R, D)
    cfg = pipeline.PipelineConfig(decoder=case["decoder"], B=B, C=case["C"], N=case["N"], degree_fraction=case["deg"], D=D, R=R, domain=nodes, lr=LR,
                                  precision=case["precision"])
    tables = (table, state) if R <= 1 else (table, state, rel[0], rel_state[0], rel[1], rel_state[1])
    pipe = pipeline.BatchPipeline(cfg, *tables)
    edges = _edges(gen, RESIDENT_BATCHES * B, nodes, R, case["alpha"])
    s = dict(case=case, pipe=pipe, edges=edges, table=table, state=state, rel=rel, rel_state=rel_state, t=0)
    if case["mode"] == "graph":
        s["runner"] = pipe.capture_pipelined(edges, RESIDENT_BATCHES)
    elif case["mode"] == "feed":
        s["host"] = [b.cpu().pin_memory() for b in edges.view(RESIDENT_BATCHES, B, -1)]
        s["losses"] = torch.zeros(RESIDENT_BATCHES).pin_memory()
        s["feed"] = pipeline.HostFeed(pipe, edges.shape[1])
        s["feed"].start(s["host"][0], s["host"][1])
        s["t"] = 2
    else:  # the first step sizes the workspace
        s["batches"] = list(edges.view(RESIDENT_BATCHES, B, -1))
        pipe.step(s["batches"][0], 0)
        s["t"] = 1
    return s


def _prepare_host(case, gen):
    H = _host_layer()
    nodes, R, D, B = case["nodes"], case["R"], case["D"], case["B"]
    model = H.Model(H.DecoderType.COMPLEX if case["decoder"] == "COMPLEX" else H.DecoderType.DISTMULT, R, D, R > 1, LR, LR, torch.device("cuda:0"),
                    case["precision"])
    rel, rel_state = _relation_tables(gen, R, D)
    model.relations, model.relations_state = rel[0], rel_state[0]
    if R > 1:
        model.inverse_relations, model.inverse_relations_state = rel[1], rel_state[1]
    table, state = H.InMemory(_normal(gen, (nodes, D), 0.3)), H.InMemory(_adagrad_state(gen, (nodes, D)))
    edges = _edges(gen, RESIDENT_BATCHES * B, nodes, R, case["alpha"])
    loader = H.DataLoader(edges, table, state, B, case["C"], case["N"], case["deg"], R > 1, 20260)
    s = dict(case=case, model=model, table=table, state=state, loader=loader)
    _run_host(s)  # the first step sizes the workspaces
    return s


def _prepare_eval(case, gen):
    nodes, R, D, B = case["nodes"], case["R"], case["D"], case["B"]
    s = dict(case=case, table=_normal(gen, (nodes, D), 0.3), edges=_edges(gen, B, nodes, R, 1.0))
    if R > 1:
        s["rel"], s["inv_rel"] = _normal(gen, (R, D), 0.2, 1.0), _normal(gen, (R, D), 0.2, 1.0)
    # the true neighbours of every edge: its own endpoint, and on average per_row more, drawn by degree (some of them twice)
    for key, col in (("dst_filter", -1), ("src_filter", 0)):
        rows = torch.randint(B, (B * case["per_row"],), generator=gen, device="cuda").sort().values
        pairs = torch.stack([rows, _power_law(gen, B * case["per_row"], nodes, 1.0)], 1)
        own = torch.stack([torch.arange(B, device="cuda"), s["edges"][:, col]], 1)
        s[key] = torch.cat([pairs, own]).contiguous()
    if R <= 1:
        del s["src_filter"]
    return s


def _prepare_tour(case, gen):
    C, R, N, D = case["chunks"], case["rows"], case["N"], case["D"]
    return dict(case=case, queries=_normal(gen, (C, R, D), 0.3), negatives=_normal(gen, (C, N, D), 0.3))


def _prepare_pairs(case, gen):
    C, R, N, K = case["chunks"], case["rows"], case["N"], case["K"]
    s = _prepare_tour(case, gen)
    # what a tournament leaves: one negative from each of K groups of consecutive ones
    T = N // K
    s["selected"] = (torch.randint(T, (C, R, K), generator=gen, device="cuda") + T * torch.arange(K, device="cuda")).view(C, R * K)
    s["grad"] = _normal(gen, (C * R, K), 0.01)  # softmax probabilities, about
    s["status"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    return s


def _prepare_state(case, gen):
    P, rows, D, cols = case["parts"], case["rows"], case["D"], case["cols"]
    home = [_normal(gen, (P * rows, D), 0.3), _adagrad_state(gen, (P * rows, D))]
    relay = partition.RelayBuffer(home, rows, P, 0, 1)
    # bucket-sorted edges with global ids; bucket sizes vary by a factor of three
    share = 1.0 + 0.5 * np.sin(1.7 * np.arange(P * P))
    sizes = (share / share.sum() * case["edges"]).astype(np.int64)
    bucket = torch.repeat_interleave(torch.arange(P * P, device="cuda"), torch.from_numpy(sizes).cuda())
    n = bucket.numel()
    column = [bucket // P * rows + torch.randint(rows, (n,), generator=gen, device="cuda")]
    if cols == 3:
        column.append(torch.randint(1000, (n,), generator=gen, device="cuda"))
    column.append(bucket % P * rows + torch.randint(rows, (n,), generator=gen, device="cuda"))
    edges = torch.stack(column, 1).contiguous()
    supersteps = partition.make_supersteps(P, 1)
    buckets = partition.state_buckets(supersteps, P, sizes)
    most = max(int(sizes[b[0]].sum()) for b in buckets)
    s = dict(case=case, relay=relay, edges=edges, begin=np.concatenate([[0], np.cumsum(sizes)])[:-1], sizes=sizes, supersteps=supersteps, buckets=buckets,
             state_edges=torch.zeros((most, cols), dtype=torch.int64, device="cuda"), slots=torch.full((P,), -1, dtype=torch.int64, device="cuda"),
             status=torch.zeros(1, dtype=torch.int32, device="cuda"), k=0)
    _run_state(s)  # from here on there is a state to swap out
    return s


# ---------------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------------
def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


def _run_step(s):
    pipe, t = s["pipe"], s["t"]
    s["t"] = t + 1
    mode = s["case"]["mode"]
    if mode == "graph":
        s["runner"].replay()
        loss = s["runner"].loss
    elif mode == "feed":
        loss = s["losses"][t % RESIDENT_BATCHES:][:1]
        s["feed"].step(s["host"][t % RESIDENT_BATCHES], loss)
    else:
        pipe.step(s["batches"][t % RESIDENT_BATCHES], t)
        loss = pipe.loss
    return dict(loss=loss, table=s["table"], state=s["state"], rel=s["rel"], rel_state=s["rel_state"], status=pipe.status)


def _run_host(s):
    batch = s["loader"].getBatch()
    s["model"].train_batch(batch, True)
    s["loader"].updateEmbeddings(batch)
    m = s["model"]
    return dict(loss=batch.loss, edges=batch.edges, table=s["table"].data, state=s["state"].data, rel=m.relations,
                rel_state=m.relations_state, inv_rel=m.inverse_relations, inv_rel_state=m.inverse_relations_state)


def _run_eval(s):
    return capi.eval_ranks(s["case"]["decoder"], s["table"], s["edges"], s.get("rel"), s.get("inv_rel"), s["dst_filter"], s.get("src_filter"))


def _run_tour(s):
    return capi.tournament_select(s["queries"], s["negatives"], s["case"]["K"])


def _run_pairs(s):
    kind = s["case"]["score"]
    scores = capi.selected_neg_scores(kind, s["queries"], s["negatives"], s["selected"], s["status"])
    return (scores,) + capi.selected_neg_scores_backward(kind, s["grad"], s["queries"], s["negatives"], s["selected"], s["status"])


def _run_state(s):
    relay, k = s["relay"], s["k"] % len(s["supersteps"])
    s["k"] += 1
    relay.swap(s["supersteps"][k])
    mine = s["buckets"][k][0]
    s["slots"].copy_(torch.tensor(relay.slot_table(), dtype=torch.int64))
    total = capi.build_state_edges(s["edges"], [int(s["begin"][b]) for b in mine], [int(s["sizes"][b]) for b in mine], s["slots"], relay.rows,
                                   1 + 7919 * s["k"], s["state_edges"], s["status"])
    return relay.buf(0), relay.buf(1), s["state_edges"][:total], s["status"]


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how closely two correct implementations agree
# ---------------------------------------------------------------------------------------------------------------------
def _expected_distinct(case):
    """Distinct node ids of a batch: 2 B endpoints (and C * N * deg degree-drawn ones, which repeat them) by the power law,
    the rest uniform over the nodes."""
    n, alpha = case["nodes"], case["alpha"]
    uniform = case["C"] * (case["N"] - int(case["N"] * case["deg"]))
    edges = np.unique(np.concatenate([[1.0], np.logspace(0, math.log10(n + 1), 4000)]))
    cdf = np.log(edges) / math.log(n + 1) if abs(alpha - 1) < 1e-6 else (edges ** (1 - alpha) - 1) / ((n + 1.0) ** (1 - alpha) - 1)
    width = np.diff(edges)
    missed = np.exp(-2.0 * case["B"] * np.diff(cdf) / width - uniform / n)
    return float((width * (1.0 - missed)).sum())


def work(case):
    kind, D = case["kind"], case["D"]
    if kind in ("step", "host"):
        S = 2 if case["R"] > 1 else 1
        ids = 8 * case["B"] * (3 if case["R"] > 1 else 2)
        tables = 16 * D * (_expected_distinct(case) + (S * case["R"] if case["R"] > 1 else 0))
        return dict(bytes=ids + tables, flops=6 * S * case["B"] * case["N"] * D)
    if kind == "eval":
        S = 2 if case["R"] > 1 else 1
        return dict(bytes=4 * D * (case["nodes"] + 2 * case["R"]) + S * case["B"] * (32 + 16 * (case["per_row"] + 1)), flops=2 * S * case["B"] * case["nodes"] * D)
    if kind == "state":
        # a swap replaces all four partitions of the state (with eight partitions, three on average): each comes in from home, and the
        # one it replaces goes home
        moved = 4 if case["parts"] > 8 else 3
        return dict(bytes=2 * 2 * 2 * moved * case["rows"] * D * 4 + 16 * case["cols"] * case["edges"] / len(partition.make_supersteps(case["parts"], 1)), flops=0)
    rows = case["chunks"] * case["rows"]
    vectors = 4 * D * (rows + case["chunks"] * case["N"])
    if kind == "tour":
        return dict(bytes=vectors + 12 * rows * case["K"], flops=2 * rows * case["N"] * D)
    return dict(bytes=2 * vectors + 16 * rows * case["K"], flops=6 * rows * case["K"] * D)


def tolerance(case):
    kind = case["kind"]
    if kind in ("eval", "state"):
        return "exact"  # ranks, node ids and whole slabs
    if kind == "tour":
        return dict(rel=1e-5, max=1e-4, differ=1e-4)  # another winner of a group only where two scores are equal to the last bits
    if kind == "pairs":
        return dict(rel=1e-5, max=1e-3)  # the L2 gradient of a pair that nearly coincides
    if case["precision"] == "f16":  # fp16 operands of the contractions (11 bits), fp32 sums
        return dict(rel=1e-3, max=5e-2)
    return dict(rel=1e-5, max=1e-3)
