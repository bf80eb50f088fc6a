"""Per-batch training pipeline on one GPU: the sequence SynchronousTrainer::train runs for every batch
(cpp/src/engine/trainer.cpp:170-211 of the reference project), issued as a fixed list of launches on the current
CUDA stream with no host synchronisation in between:

    sample negatives + pack ids  ->  unique-map  ->  fused decoder forward/loss/backward  ->  sparse Adagrad scatter
    ->  dense Adagrad on the relation tables

Torch tensors are used as device memory only; every arithmetic step is a kernel of libge2_b200.so.
"""
from __future__ import annotations

import ctypes
from dataclasses import dataclass
from typing import Optional

import torch

from . import capi


@dataclass
class PipelineConfig:
    decoder: str            # "DISTMULT" | "COMPLEX" ("DOT" = DISTMULT on 2-column edges)
    B: int                  # batch size
    C: int                  # num_chunks
    N: int                  # negatives_per_positive (per chunk)
    degree_fraction: float  # share of degree-based negatives
    D: int
    R: int                  # number of relations (0/1 => relation-free, 2-column edges)
    domain: int             # nodes resident on the device (rows of the table)
    lr: float = 0.1
    dense_lr: Optional[float] = None
    precision: str = "fp32"
    seed: int = 20260
    inverse: bool = True

    @property
    def has_relations(self):
        return self.R > 1

    @property
    def sides(self):
        return 2 if (self.has_relations and self.inverse) else 1

    @property
    def n_deg(self):
        return int(self.N * self.degree_fraction)  # negative.cpp:945 of the reference project

    @property
    def n_ids(self):
        return 2 * self.B + self.sides * self.C * self.N


class _IdSet:
    """The per-batch id buffers: packed ids, unique map, inverse (and its column slices), device-side count, degree rows,
    relation column.  The pipeline owns two sets so that batch t+1 can be sampled and deduplicated while batch t trains."""

    def __init__(self, cfg: "PipelineConfig", cap: int, dev):
        n_ids, CN, B = cfg.n_ids, cfg.C * cfg.N, cfg.B
        i64 = dict(dtype=torch.int64, device=dev)
        self.packed = torch.empty(n_ids, **i64)
        self.deg_rows = torch.empty((cfg.C, max(cfg.n_deg, 1)), **i64)
        self.unique = torch.empty(cap, **i64)
        self.inverse = torch.empty(n_ids, **i64)
        self.shared = torch.empty(cap, dtype=torch.uint8, device=dev)  # per unique id: 1 = more than one occurrence in the batch
        self.twins = (2 * B, CN) if cfg.sides == 2 else (0, 0)  # the sides' negatives, node for node where they are drawn uniformly
        self.count = torch.zeros(2, dtype=torch.int32, device=dev)
        self.rel_ids = torch.empty(max(B, 1), **i64)  # the batch's relation column, copied by the sampler
        self.loss = torch.zeros(1, dtype=torch.float32, device=dev)  # loss of the batch trained from this set
        self.uws = capi.unique_workspace(cfg.domain, dev)  # one per set: two unique-maps may be in flight at the same time
        self.src_local = self.inverse[0:B]
        self.dst_local = self.inverse[B:2 * B]
        off = 2 * B
        self.src_negs_local = None
        if cfg.sides == 2:
            self.src_negs_local = self.inverse[off:off + CN]
            off += CN
        self.dst_negs_local = self.inverse[off:off + CN]


class PeerGradients:
    """Relation-gradient buffers that every rank of a node can read over NVLink (one process per GPU): the sum over ranks
    and the dense optimizer step then take one launch per rank (ge2_dense_adagrad_peers) instead of a collective call
    between two halves of the step, and the whole multi-GPU step fits in one CUDA graph.  Replaces Model::all_reduce of
    the reference (model.cpp:174-204).  Layout of each rank's buffer: two halves of `numel` floats (the step whose counter
    is t accumulates into half t & 1), then one 8-byte flag per rank, the verdict word and the wait-time counter.

    The buffers are torch symmetric memory: every rank's allocation is mapped into this process's address space with
    access granted to this rank's GPU, which is what a kernel needs to load from it.  (A legacy CUDA IPC import of a
    peer's tensor is mapped in the context of the peer's device and faulted when a kernel of this rank's device read it.)
    No multicast object is bound to the buffers: the kernel uses plain peer loads and stores."""

    def __init__(self, dist, numel: int, device):
        import os

        os.environ.setdefault("TORCH_SYMM_MEM_DISABLE_MULTICAST", "1")
        import torch.distributed._symmetric_memory as symm_mem

        assert numel % 2 == 0, "the flag row behind the two halves must be 8-byte aligned"
        self.rank, self.world, self.numel = dist.get_rank(), dist.get_world_size(), numel
        self.buf = symm_mem.empty(2 * numel + 2 * self.world + 32, dtype=torch.float32, device=device)
        self.buf.zero_()
        torch.cuda.synchronize(device)
        self.handle = symm_mem.rendezvous(self.buf, dist.group.WORLD)  # collective; keeps the peers' mappings alive
        self.ptrs = [int(p) for p in self.handle.buffer_ptrs]
        if len(self.ptrs) != self.world or self.ptrs[self.rank] != self.buf.data_ptr():
            raise RuntimeError("symmetric memory rendezvous returned an unexpected set of buffers")
        dist.barrier()  # every rank has zeroed and mapped every buffer before anybody launches on them
        torch.cuda.synchronize(device)

    def half(self, parity: int):
        return self.buf[parity * self.numel:(parity + 1) * self.numel]

    def waited_ns(self) -> int:
        """nanoseconds this rank's announcing kernels have spent waiting for the slowest rank so far (synchronises)"""
        return int(self.buf[2 * self.numel:2 * self.numel + 2 * self.world + 4].view(torch.int64)[self.world + 1].item())


class BatchPipeline:
    """Owns the per-batch scratch (ids, unique map, gradients, workspaces); tables are owned by the caller."""

    # Ids of a batch for every SM that the scores kernels leave over, up to which the next batch's sampler and unique-map run there.  They take
    # about 11 us and 0.7 us for every thousand ids an SM, beside scores of 13 us and more.  The pipelined step at 320 shapes (1 000 ... 60 000
    # edges, 60 ... 2 000 negatives, both precisions), on those SMs : behind the scores, mean ratio by ids an SM: up to 6 000 0.92;
    # 6 000 ... 16 384 0.98; to 20 000 0.99; to 26 000 1.01; to 40 000 1.06; to 70 000 1.10; above 1.35.  In us: fp16, 3 061 edges, Dot 64,
    # 5 700 ids an SM 35.4 : 42.9; fp32, 47 126, Dot 64, 13 400 121.1 : 132.2; fp16, 10 751, Dot 100, 14 700 127.0 : 118.6 (finish is long there);
    # fp32, 7 144, ComplEx 50, 17 200 150.3 : 155.8; fp16, 12 413, ComplEx 50, 30 200 138.0 : 138.5; 14 711, ComplEx 64, 39 200 122.3 : 109.9.
    # The way that is taken is 0.7 % slower than the better one on average (never there: 6.4 %, always: 4.7), at worst 9.5 % on those SMs (5 642
    # edges, DistMult 50, 2.9 M nodes: 63.4 : 57.9) and 22 % behind the scores (4 060, DistMult 64, 19 300 ids an SM: 62.5 : 76.2).  A linear
    # rule on the measured times of these kernels, the scores and finish in place of the ids: 0.5 % on average, 11 % at worst.
    IDS_PER_IDLE_SM = 16384

    def __init__(self, cfg: PipelineConfig, table, state, rel=None, rel_state=None, inv_rel=None, inv_rel_state=None):
        capi.load_library()
        self.cfg = cfg
        dev = table.device
        self.device = dev
        self.table, self.state = table, state
        self.rel, self.rel_state, self.inv_rel, self.inv_rel_state = rel, rel_state, inv_rel, inv_rel_state
        assert table.is_cuda and table.dtype == torch.float32 and table.shape[1] == cfg.D and table.is_contiguous()
        n_ids, CN = cfg.n_ids, cfg.C * cfg.N
        self.cap = min(n_ids, cfg.domain)
        self.ids = [_IdSet(cfg, self.cap, dev), _IdSet(cfg, self.cap, dev)]
        first = self.ids[0]  # the non-pipelined forms use the first set only; its buffers keep their plain names
        self.packed, self.deg_rows, self.unique, self.inverse, self.count, self.rel_ids = (
            first.packed, first.deg_rows, first.unique, first.inverse, first.count, first.rel_ids)
        self.status = torch.zeros(1, dtype=torch.int32, device=dev)
        self.node_grad = torch.zeros((self.cap, cfg.D), dtype=torch.float32, device=dev)
        self.loss = first.loss
        self.uws = first.uws
        if cfg.has_relations:
            # one contiguous buffer for both relation-gradient tables: a single all-reduce serves them in the multi-GPU trainer
            self.rel_grads = torch.zeros((cfg.sides,) + tuple(rel.shape), dtype=rel.dtype, device=dev)
            self.rel_grad = self.rel_grads[0]
            self.inv_rel_grad = self.rel_grads[1] if cfg.sides == 2 else None
            # when the caller keeps the two relation tables (and their states) back to back in one allocation, the dense
            # optimizer step is one launch over both
            self._rel_tables_adjacent = False
            if cfg.sides == 2 and rel.is_contiguous() and inv_rel.is_contiguous() and rel_state.is_contiguous() and inv_rel_state.is_contiguous():
                n = rel.numel()
                adj = lambda a, b: (b.data_ptr() == a.data_ptr() + n * a.element_size()
                                    and a.untyped_storage().data_ptr() == b.untyped_storage().data_ptr())
                if adj(rel, inv_rel) and adj(rel_state, inv_rel_state):
                    both = lambda a: torch.as_strided(a, (2,) + tuple(a.shape), (n,) + tuple(a.stride()))
                    self._rel_both, self._rel_state_both = both(rel), both(rel_state)
                    self._rel_tables_adjacent = True
        else:
            self.rel_grad = self.inv_rel_grad = None
            self._rel_tables_adjacent = False
        # device-side batch counters of the graph-replay forms: {t, t + 1}
        self.step_dev = torch.tensor([0, 1], dtype=torch.int64, device=dev)
        self._graph = None
        self._desc = None
        self._ws = None
        self.grad_scale = 1.0  # 1 / #GPUs when relation gradients are all-reduced (model.cpp:188-192 of the reference project)
        self.peer: Optional[PeerGradients] = None
        self._t_host = 0       # host mirror of step_dev[0]; only the peer-gradient form needs it (which half a step writes)
        # number of batches of the resident edge list, on the device: a partition-buffer state replaces the list by one of
        # another length without the captured launches changing (set_num_batches); None = the host-side count is used
        self.nb_dev = None
        self._ids_parity = 0   # which id set holds the batch drawn ahead (shared by every pipelined runner of this pipeline)

    def set_num_batches(self, num_batches: int):
        """Stream-ordered update of the device-side batch count used by the resident / pipelined forms."""
        if self.nb_dev is None:
            self.nb_dev = torch.zeros(1, dtype=torch.int64, device=self.device)
        self.nb_dev.fill_(max(1, int(num_batches)))

    def _unique(self, ids: "_IdSet"):
        capi.unique_bitmap(ids.packed, self._mapped_domain(), workspace=ids.uws, out_unique=ids.unique, out_inverse=ids.inverse, out_count=ids.count,
                           out_shared=ids.shared, twins=ids.twins)

    def _mapped_domain(self):
        """ids that get a local id: those with a row in the table (others are flagged, and neither read nor written)"""
        return min(self.cfg.domain, self.table.shape[0])

    def use_peer_gradients(self, peer: PeerGradients):
        """Multi-GPU: relation gradients go into `peer`'s buffer (alternating halves) and the dense optimizer step sums them
        over the ranks itself.  Supported by enqueue_resident and capture_pipelined; needs the relation tables (and their
        states) back to back when there are two."""
        cfg = self.cfg
        assert cfg.has_relations and (cfg.sides == 1 or self._rel_tables_adjacent)
        assert peer.numel == cfg.sides * self.rel.numel()
        self.peer = peer
        self.grad_scale = 1.0 / peer.world
        self._t_host = int(self.step_dev[0].item())
        self._peer_views = [peer.half(h).view((cfg.sides,) + tuple(self.rel.shape)) for h in (0, 1)]

    def _make_desc(self, edges, rel_ids=None, rel_stride=None, ids: Optional[_IdSet] = None, parity: Optional[int] = None):
        cfg = self.cfg
        ids = ids or self.ids[0]
        rel_grad, inv_rel_grad = self.rel_grad, self.inv_rel_grad
        if self.peer is not None:
            view = self._peer_views[(self._t_host if parity is None else parity) & 1]
            rel_grad, inv_rel_grad = view[0], (view[1] if cfg.sides == 2 else None)
        cols = edges.shape[1]
        if rel_ids is None and cfg.has_relations:
            rel_ids, rel_stride = edges[:, 1], cols
        d = capi.make_lp_desc(
            decoder=cfg.decoder, precision=cfg.precision, B=cfg.B, Cn=cfg.C, N=cfg.N, D=cfg.D, R=cfg.R if cfg.has_relations else 0,
            U=self.cap, node_emb=self.table, row_index=ids.unique, emb_stride=cfg.D, src_ids=ids.src_local, dst_ids=ids.dst_local,
            rel_ids=rel_ids if cfg.has_relations else None, edge_stride=1, rel_stride=rel_stride or 1, dst_negs=ids.dst_negs_local,
            src_negs=ids.src_negs_local, deg_sample_rows=ids.deg_rows if cfg.n_deg > 0 else None, n_deg=cfg.n_deg,
            rel=self.rel, inv_rel=self.inv_rel if cfg.sides == 2 else None, node_grad=self.node_grad, rel_grad=rel_grad,
            inv_rel_grad=inv_rel_grad, loss=ids.loss, status=self.status, node_grad_is_zero=True,
            node_state=self.state, row_shared=ids.shared, node_lr=cfg.lr)
        if self._ws is None:
            self._ws = torch.empty(capi.lp_workspace_bytes(d), dtype=torch.uint8, device=self.device)
        d.workspace, d.workspace_bytes = self._ws.data_ptr(), self._ws.numel()
        return d

    def step(self, edges, batch_index: int, scores_events=None, rel_hook=None):
        """edges: [B, 2|3] int64 device tensor with resident-table row ids (global ids, or buffer-local ids with a
        partition buffer).  Enqueues one training step; returns nothing (loss stays in self.loss).
        scores_events: optional (start, end) torch.cuda.Event pair recorded around the scores kernel alone.
        rel_hook: optional callable run after the backward pass and before the dense optimizer step (the multi-GPU
        trainer all-reduces the relation gradients there, Model::all_reduce of the reference)."""
        cfg = self.cfg
        cols = edges.shape[1]
        assert edges.shape[0] == cfg.B and edges.dtype == torch.int64 and edges.is_contiguous()
        if scores_events is None and rel_hook is None and self.peer is None:
            t = self._train_desc(edges)
            t.edges, t.batch_index = edges.data_ptr(), batch_index
            if cfg.has_relations:
                self._train_lp.rel_ids = t.edges + 8  # column 1
            capi.train_step(t)
            return
        capi.sample_negatives(edges, edges[:, cols - 1], cols, cfg.B, cfg.C, cfg.N, cfg.n_deg, cfg.domain, cfg.sides == 2, cfg.seed,
                              batch_index, self.packed, self.deg_rows if cfg.n_deg > 0 else None)
        self._unique(self.ids[0])
        self._backward_and_update(self._make_desc(edges), scores_events, rel_hook)

    def _train_desc(self, edges):
        """The arguments of a whole host-issued step: laid out once, and again whenever a table was replaced or any field of the
        configuration changed; of the rest only the batch's address and number change from step to step."""
        cfg = self.cfg
        key = (*vars(cfg).values(), self.table.data_ptr(), self.table.shape[0], self.state.data_ptr(), self.node_grad.data_ptr(), self.status.data_ptr(),
               self.grad_scale, edges.shape[1])
        if cfg.has_relations:
            tabs = (self.rel, self.rel_state, self.rel_grad) + ((self.inv_rel, self.inv_rel_state, self.inv_rel_grad) if cfg.sides == 2 else ())
            key += (self.rel.numel(), *(a.data_ptr() for a in tabs))
        if key == getattr(self, "_train_key", None):
            return self._train
        ids = self.ids[0]
        self._train_lp = self._make_desc(edges)
        t = capi.TrainDesc()
        t.lp = ctypes.pointer(self._train_lp)
        t.cols, t.n_deg, t.domain, t.seed = edges.shape[1], cfg.n_deg, cfg.domain, cfg.seed
        t.packed, t.deg_rows, t.n_ids = ids.packed.data_ptr(), ids.deg_rows.data_ptr() if cfg.n_deg > 0 else None, ids.packed.numel()
        t.unique_ws, t.unique_ws_bytes = ids.uws.data_ptr(), ids.uws.numel()
        t.unique, t.inverse, t.count, t.shared = (a.data_ptr() for a in (ids.unique, ids.inverse, ids.count, ids.shared))
        t.twin_begin, t.twin_len = ids.twins
        t.table, t.state, t.table_rows, t.lr, t.grad_scale = self.table.data_ptr(), self.state.data_ptr(), self.table.shape[0], cfg.lr, self.grad_scale
        if cfg.has_relations:
            t.dense_lr = cfg.lr if cfg.dense_lr is None else cfg.dense_lr
            both = cfg.sides == 2 and self._rel_tables_adjacent
            t.num_dense = 2 if cfg.sides == 2 and not both else 1
            t.dense_numel = self.rel.numel() * (2 if both else 1)
            for k, (p, st, g) in enumerate(((self.rel, self.rel_state, self.rel_grad), (self.inv_rel, self.inv_rel_state, self.inv_rel_grad))[:t.num_dense]):
                t.dense_param[k], t.dense_state[k], t.dense_grad[k] = p.data_ptr(), st.data_ptr(), g.data_ptr()
        self._train, self._train_key = t, key
        return t

    def _backward_and_update(self, desc, scores_events=None, rel_hook=None):
        self._backward(desc, scores_events)
        if rel_hook is not None:
            rel_hook(self)
        self._update()

    def _backward(self, desc, scores_events=None):
        if scores_events is None:
            capi.lp_step(desc)
        else:  # same kernels, issued phase by phase so the scores kernel can be bracketed by events
            desc.phases = 1
            capi.lp_step(desc)
            desc.phases = 2
            scores_events[0].record()
            capi.lp_step(desc)
            scores_events[1].record()
            desc.phases = 4
            capi.lp_step(desc)

    def time_scores_phase(self, edges_all, reps: int = 20, phases: int = 2) -> float:
        """Milliseconds per scores phase (the clearing of dK plus the scores launches) as it runs inside a replayed graph:
        `reps` phases captured back to back on the operands the last step left in the workspace, bracketed by events.
        Host-issued launches of the same phase carry a few microseconds of launch gaps that a graph replay does not have.
        (phases: 1 = prepare, 2 = scores, 4 = finish, as in ge2_lp_desc.  The finish kernel trains rows and adds to the gradient
        buffers: it is timed on copies of them.)"""
        desc = self._make_desc(edges_all, self.ids[0].rel_ids, 1)
        desc.phases = phases
        scratch = []
        if phases & 4:
            def copy(name, t):
                scratch.append(t.clone())
                setattr(desc, name, scratch[-1].data_ptr())

            copy("node_emb", self.table), copy("node_state", self.state), copy("node_grad", self.node_grad), copy("loss", self.loss)
            if self.cfg.has_relations:
                copy("rel_grad", self.rel_grad)
                if self.cfg.sides == 2:
                    copy("inv_rel_grad", self.inv_rel_grad)
        capi.lp_step(desc)
        torch.cuda.synchronize(self.device)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for _ in range(reps):
                capi.lp_step(desc)
        g.replay()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        g.replay()
        b.record()
        torch.cuda.synchronize(self.device)
        desc.phases = 0
        return a.elapsed_time(b) / reps

    def _update(self, ids: Optional[_IdSet] = None):
        cfg = self.cfg
        if not cfg.has_relations or self.peer is not None:
            self._update_nodes(ids)
            self._update_relations()
            return
        ids = ids or self.ids[0]
        if cfg.sides == 2 and self._rel_tables_adjacent:
            # relation and inverse-relation tables (and their states) sit back to back, as the gradients do: one table
            dense = [(self._rel_both, self._rel_state_both, self.rel_grads)]
        else:
            dense = [(self.rel, self.rel_state, self.rel_grad)] + ([(self.inv_rel, self.inv_rel_state, self.inv_rel_grad)] if cfg.sides == 2 else [])
        capi.adagrad_step(self.table, self.state, ids.unique, self.node_grad, cfg.lr, dense, cfg.lr if cfg.dense_lr is None else cfg.dense_lr, U=self.cap,
                          U_dev=ids.count, status=self.status, row_shared=ids.shared, grad_scale=self.grad_scale)

    def _update_nodes(self, ids: Optional[_IdSet] = None):
        cfg = self.cfg
        ids = ids or self.ids[0]
        # rows with one occurrence were updated by the backward pass, where their whole gradient is at hand; this does the others.
        # clear_grad: the rows just consumed are zeroed in the same pass, so the next step needs no memset of the gradient buffer
        capi.adagrad_scatter(self.table, self.state, ids.unique, self.node_grad, cfg.lr, U=self.cap, U_dev=ids.count, clear_grad=True,
                             status=self.status, row_shared=ids.shared)

    def _update_relations(self):
        cfg = self.cfg
        if cfg.has_relations:
            dl = cfg.lr if cfg.dense_lr is None else cfg.dense_lr
            if self.peer is not None:
                # sum over the ranks' gradient buffers + Adagrad on both tables + clearing of the other half, one launch
                both = cfg.sides == 2
                capi.dense_adagrad_peers(self._rel_both if both else self.rel, self._rel_state_both if both else self.rel_state, self.peer.ptrs,
                                         self.peer.rank, self.peer.numel, self.step_dev, dl, self.status, grad_scale=self.grad_scale)
                return
            if cfg.sides == 2 and self._rel_tables_adjacent:
                # relation and inverse-relation tables (and their states) sit back to back, as the gradients do: one launch
                capi.dense_adagrad(self._rel_both, self._rel_state_both, self.rel_grads, dl, grad_scale=self.grad_scale, clear_grad=True)
                return
            capi.dense_adagrad(self.rel, self.rel_state, self.rel_grad, dl, grad_scale=self.grad_scale, clear_grad=True)
            if cfg.sides == 2:
                capi.dense_adagrad(self.inv_rel, self.inv_rel_state, self.inv_rel_grad, dl, grad_scale=self.grad_scale, clear_grad=True)

    # ---- graph-replay form: the whole step is a fixed launch list that reads its batch index from device memory ----------
    def enqueue_resident(self, edges_all, num_batches: int, scores_events=None, rel_hook=None):
        """One training step on batch (*step_dev % num_batches) of the resident edge list edges_all[num_batches * B, cols];
        advances the device-side counter at the end.  No argument changes from step to step, so the launch list can be
        captured once into a CUDA graph (capture_resident) and replayed."""
        cfg = self.cfg
        self._front(self.ids[0], edges_all, num_batches, self.step_dev, advance=True)
        self._backward_and_update(self._make_desc(edges_all, self.rel_ids, 1), scores_events, rel_hook)
        if self.peer is not None:
            capi.advance_step(self.step_dev, 2)
        self._t_host += 1
        self._ids_parity = self._t_host & 1  # (a pipelined runner used after this needs refill(): nothing is drawn ahead)

    def capture_resident(self, edges_all, num_batches: int, rel_hook=None):
        """Captures one resident step into a CUDA graph (after one eager step, which also resolves driver entry points and
        function attributes outside the capture).  replay() then costs a single graph launch per step."""
        assert self.peer is None, "the peer-gradient form needs the alternating graphs of capture_pipelined"
        self.enqueue_resident(edges_all, num_batches, rel_hook=rel_hook)
        torch.cuda.synchronize(self.device)
        self._graph_edges = edges_all  # keep the captured pointers alive
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            self.enqueue_resident(edges_all, num_batches, rel_hook=rel_hook)
        self._graph = g
        return g

    def capture_resident_split(self, edges_all, num_batches: int, rel_hook):
        """Multi-GPU form: the step is captured as two graphs with the relation-gradient all-reduce (rel_hook, a host-issued
        NCCL call) between them -- sample/unique/forward/backward, then the optimizer updates and the counter bump."""
        self.enqueue_resident(edges_all, num_batches, rel_hook=rel_hook)
        torch.cuda.synchronize(self.device)
        self._graph_edges = edges_all
        cfg = self.cfg
        ga, gb = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(ga):
            self._front(self.ids[0], edges_all, num_batches, self.step_dev, advance=True)
            self._backward(self._make_desc(edges_all, self.rel_ids, 1))
        with torch.cuda.graph(gb):
            self._update()

        class _Split:
            def replay(_self):
                ga.replay()
                rel_hook(self)
                gb.replay()

        self._split = (ga, gb)
        return _Split()

    # ---- pipelined form: batch t+1 is sampled and deduplicated on a side stream while batch t trains -----------------
    def _front(self, ids: _IdSet, edges_all, num_batches: int, counter, advance: bool = False, sms: int = 0):
        """sampler + unique-map into one id set; `counter` is the device counter holding the batch number to use.  advance: both
        device counters go up by one at the end, unless the step's own exchange between ranks still reads them.  sms: SMs to keep to (0: all)."""
        cfg = self.cfg
        assert edges_all.dtype == torch.int64 and edges_all.is_contiguous() and edges_all.shape[1] in (2, 3)
        f = capi.FrontDesc()
        f.edges, f.cols, f.num_batches, f.sms = edges_all.data_ptr(), edges_all.shape[1], num_batches, sms
        f.num_batches_dev = None if self.nb_dev is None else self.nb_dev.data_ptr()
        f.step_dev, f.seed = counter.data_ptr(), cfg.seed
        f.B, f.C, f.N, f.n_deg, f.domain, f.mapped, f.want_src_negs = cfg.B, cfg.C, cfg.N, cfg.n_deg, cfg.domain, self._mapped_domain(), cfg.sides == 2
        f.packed, f.deg_rows, f.rel_ids = ids.packed.data_ptr(), ids.deg_rows.data_ptr(), ids.rel_ids.data_ptr() if cfg.has_relations else None
        f.unique_ws, f.unique_ws_bytes = ids.uws.data_ptr(), ids.uws.numel()
        f.unique, f.inverse, f.count, f.shared = (a.data_ptr() for a in (ids.unique, ids.inverse, ids.count, ids.shared))
        if advance and self.peer is None:
            f.counters, f.num_counters = self.step_dev.data_ptr(), 2
        capi.sample_unique(f)

    def idle_step(self):
        """A step of a lane that has no batch (lanes of a superstep have unequal batch counts): the relation-gradient
        exchange alone -- this rank's half of the gradient buffer is zero, so it contributes zeros, as the reference's
        zero-filled gradients do (model.cpp:182-187) -- and the counter bump, so that the replicas of the relation tables
        stay in step with the ranks that train."""
        self._update_relations()
        capi.advance_step(self.step_dev, 2)
        self._t_host += 1
        self._ids_parity = self._t_host & 1

    def capture_pipelined(self, edges_all, num_batches: int, rel_hook=None, front_after_scores: bool = True, tables=None, warm: bool = True):
        """tables: (table, state) to capture the graphs for, when not the pipeline's own -- a partition buffer that alternates
        between two active buffers keeps one runner per buffer; runners of one pipeline are interchangeable from step to
        step (they share the id sets, the counters and the rule "the step whose counter is t uses id set t & 1").
        warm = False skips the host-issued warm-up step (a later capture of a pipeline that has run already).

        Software-pipelined steps: while the decoder step of batch t runs, the ids of batch t+1 are drawn and deduplicated on a side stream into
        the other id set (on SMs that the scores kernels leave, or beside the finish kernel); the optimizer
        updates of batch t follow the join, so batch t+1 gathers the updated rows.  Two graphs alternate (one per id set);
        with rel_hook (the multi-GPU all-reduce, host-issued) each step is two graph launches around the hook.
        Returns an object with replay().  The same batches, negatives and arithmetic as the plain resident form."""
        own_tables = (self.table, self.state)
        if tables is not None:
            self.table, self.state = tables
        if warm:
            self.enqueue_resident(edges_all, num_batches, rel_hook=rel_hook)  # warm-up: driver entry points, function attributes
        torch.cuda.synchronize(self.device)
        self._graph_edges = edges_all
        cfg = self.cfg
        ctr_now, ctr_next = self.step_dev[0:1], self.step_dev[1:2]
        self._ids_parity = self._t_host & 1
        self._front(self.ids[self._ids_parity], edges_all, num_batches, ctr_now)  # ids of the first pipelined batch
        torch.cuda.synchronize(self.device)
        # Side streams are made once, outside any capture, and nothing is destroyed while a capture is open (a stream,
        # graph or tensor of an earlier capture dying inside a later one invalidates it): no garbage collection meanwhile.
        import gc

        if getattr(self, "_side_streams", None) is None:
            self._side_streams = (torch.cuda.Stream(device=self.device), torch.cuda.Stream(device=self.device))
        self._make_desc(edges_all, self.ids[0].rel_ids, 1)  # sizes the workspace before the capture
        gc.collect()
        gc_was_on = gc.isenabled()
        gc.disable()
        try:
            graphs = []
            if self.peer is not None:
                assert rel_hook is None and self._t_host == int(self.step_dev[0].item())
            for p in (0, 1):
                cur, nxt = self.ids[p], self.ids[1 - p]
                ga = torch.cuda.CUDAGraph()
                with torch.cuda.graph(ga):
                    main = torch.cuda.current_stream()
                    side, side2 = self._side_streams
                    # graph p trains the steps whose counter has parity p: id set p, half p of the peer gradient buffer
                    desc = self._make_desc(edges_all, cur.rel_ids, 1, ids=cur, parity=p)
                    if front_after_scores:
                        # The scores kernels own whole SMs (one CTA with all of its shared memory), and small kernels would delay their CTAs.
                        # Where they leave SMs over, and the batch is small enough for those, the sampler and the unique-map run there; else
                        # behind the scores, beside finish -- which fills the SMs first, so that what was left of this chain for the
                        # end of the step was 11 us: 88.0 us a step at configuration 2, 84.6 on the SMs left over.  (Beside prepare, which
                        # fills the SMs as well, it holds up the scores: 87.7.)
                        idle = capi.lp_idle_sms(desc)
                        idle = idle if cfg.n_ids <= self.IDS_PER_IDLE_SM * idle else 0
                        desc.phases = 1 if idle else 3
                        capi.lp_step(desc)
                        side.wait_stream(main)
                        with torch.cuda.stream(side):
                            self._front(nxt, edges_all, num_batches, ctr_next, advance=rel_hook is None, sms=idle)
                        if idle:
                            desc.phases = 2
                            capi.lp_step(desc)
                        desc.phases = 4
                        capi.lp_step(desc)
                        desc.phases = 0
                    else:
                        side.wait_stream(main)
                        with torch.cuda.stream(side):
                            self._front(nxt, edges_all, num_batches, ctr_next, advance=rel_hook is None)
                        self._backward(desc)
                        main.wait_stream(side)
                    if rel_hook is None:
                        if self.peer is None:
                            self._update(cur)
                        else:
                            # the two optimizer updates touch different tables: the dense one, with its wait for the other ranks' gradients,
                            # runs beside the sparse scatter
                            side2.wait_stream(main)
                            with torch.cuda.stream(side2):
                                self._update_relations()
                            self._update_nodes(cur)
                            main.wait_stream(side2)
                        main.wait_stream(side)
                        if self.peer is not None:
                            capi.advance_step(self.step_dev, 2)
                    if rel_hook is not None and front_after_scores:
                        main.wait_stream(side)
                gb = None
                if rel_hook is not None:
                    gb = torch.cuda.CUDAGraph()
                    with torch.cuda.graph(gb):
                        self._update(cur)
                        capi.advance_step(self.step_dev, 2)
                graphs.append((ga, gb))
        finally:
            if gc_was_on:
                gc.enable()
            self.table, self.state = own_tables
        pipe = self

        class _Pipelined:
            def replay(_self):
                ga, gb = graphs[pipe._ids_parity]
                ga.replay()
                if gb is not None:
                    rel_hook(pipe)
                    gb.replay()
                pipe._ids_parity ^= 1
                pipe._t_host += 1

            @property
            def loss(_self):
                """device scalar holding the loss of the batch trained by the last replay"""
                return pipe.ids[pipe._ids_parity ^ 1].loss

            def refill(_self):
                """Draws the ids of the coming batch again (host-issued): call after the resident edge list was replaced,
                e.g. at a partition swap, since the batch sampled ahead came from the old list."""
                pipe._front(pipe.ids[pipe._ids_parity], edges_all, num_batches, ctr_now)

        self._pipelined = graphs
        return _Pipelined()

    def replay(self):
        self._graph.replay()

    def launches_per_step(self, resident: bool = True) -> int:
        """Kernels of libge2_b200.so launched per step (memsets not counted)."""
        cfg = self.cfg
        n = 3                                  # sampler, which marks what it draws; unique-map: scan, inverse (and the counters)
        n += 1                                 # prepare (gather + relation operator + positive scores + filter words)
        n += 2                                 # scores: logsumexp pass + gradient pass, or both passes of the streaming form
        n += 1                                 # finish (operator backward + scatter)
        n += 1                                 # Adagrad: the rows, and without peers the relation tables
        if cfg.has_relations and self.peer is not None:
            n += 1 if (cfg.sides == 1 or self._rel_tables_adjacent) else 2
        return n + (1 if resident and self.peer is not None else 0)  # counters that the exchange between ranks still reads

    def check_status(self):
        """Synchronises and raises if any kernel flagged bad data (call between epochs, not per batch)."""
        torch.cuda.synchronize(self.device)
        word = int(self.status.item()) | int(self.ids[0].count[1].item()) | int(self.ids[1].count[1].item())
        if word:
            raise capi.Ge2Error("device status: " + capi.decode_status(word))


class HostFeed:
    """Trains batches that arrive in pinned host memory through the pipelined graphs, with the copies off the critical path.

    start(batch0, batch1) trains batch0 (host-issued, also the warm-up the capture needs) and draws the ids of batch1;
    every later step(next_batch, loss_out) trains the batch drawn ahead while, on a side stream, next_batch is drawn.
    The host-to-device copy of next_batch runs on its own stream during the previous step; the 4-byte loss read-back runs on
    a third stream.  Each loss slot and each staging slot is reused every second step; events order the reuse.
    Batches are trained exactly once, in the order given, with the same sampler counters as the resident forms."""

    def __init__(self, pipe: BatchPipeline, cols: int, rel_hook=None):
        self.pipe, self.rel_hook = pipe, rel_hook
        dev = pipe.device
        self.stage = torch.empty((2, pipe.cfg.B, cols), dtype=torch.int64, device=dev)
        self.h2d, self.d2h = torch.cuda.Stream(device=dev), torch.cuda.Stream(device=dev)
        self.copied = [torch.cuda.Event() for _ in range(2)]
        self.done = [torch.cuda.Event() for _ in range(2)]
        self.read = [torch.cuda.Event() for _ in range(2)]
        self.runner, self.j = None, 0

    def start(self, batch0, batch1, tables=None):
        """tables: (table, state) to train, when not the pipeline's own (a partition buffer's current pair)"""
        pipe = self.pipe
        c = int(pipe.step_dev[0].item())
        self.stage[c % 2].copy_(batch0)
        self.stage[(c + 1) % 2].copy_(batch1)
        self.slot0 = c + 2
        self.runner = pipe.capture_pipelined(self.stage.view(2 * pipe.cfg.B, -1), 2, rel_hook=self.rel_hook, tables=tables)
        torch.cuda.synchronize(pipe.device)
        self.j = 0

    def step(self, next_batch, loss_out=None):
        """next_batch: pinned host tensor [B, cols] (the batch after the one trained by this call);
        loss_out: pinned host tensor of one float receiving this step's loss (valid after a synchronize)."""
        j, main = self.j, torch.cuda.current_stream()
        k = j % 2
        if j >= 2:
            self.h2d.wait_event(self.done[k])  # the sampler of step j-2 was the last reader of this staging slot
        with torch.cuda.stream(self.h2d):
            self.stage[(self.slot0 + j) % 2].copy_(next_batch, non_blocking=True)
            self.copied[k].record()
        main.wait_event(self.copied[k])
        if j >= 2 and loss_out is not None:
            main.wait_event(self.read[k])      # this step overwrites the loss slot read back two steps ago
        self.runner.replay()
        self.done[k].record()
        if loss_out is not None:
            self.d2h.wait_event(self.done[k])
            with torch.cuda.stream(self.d2h):
                loss_out.copy_(self.runner.loss, non_blocking=True)
                self.read[k].record()
        self.j = j + 1

    def drain(self):
        """makes the current stream wait for the loss read-backs still in flight (call before timing stops or before reading them)"""
        torch.cuda.current_stream().wait_stream(self.d2h)

    def refill(self):
        self.runner.refill()
