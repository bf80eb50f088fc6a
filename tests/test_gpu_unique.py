"""GPU parity of the bitmap unique-map (through the C ABI) against the oracle: bit-exact integers."""
import numpy as np
import pytest
import torch

import ge2_oracle as O
import workloads

pytestmark = pytest.mark.gpu


def run(capi, ids_np, domain, device):
    ids = torch.from_numpy(ids_np.astype(np.int64)).to(device)
    u, inv, cnt = capi.unique_bitmap(ids, domain)
    torch.cuda.synchronize()
    count, status = (int(x) for x in cnt.cpu())
    return u.cpu().numpy()[:count], inv.cpu().numpy(), count, status


@pytest.mark.parametrize("n,domain", [(1, 1), (1, 64), (10, 64), (1000, 65), (4096, 63), (22000, 14951), (40000, 1_000_000),
                                      (150000, 1_211_896), (65536, 65536), (70000, 65537)])
def test_matches_oracle(capi, cuda_device, n, domain):
    rng = np.random.default_rng(n * 31 + domain)
    ids = rng.integers(0, domain, n)
    u, inv, count, status = run(capi, ids, domain, cuda_device)
    ou, oinv, _ = O.unique_map_bitmap(ids, domain)
    assert status == 0 and count == ou.size
    assert np.array_equal(u, ou) and np.array_equal(inv, oinv)


def test_skewed_and_degenerate_inputs(capi, cuda_device):
    domain = 1_000_000
    rng = np.random.default_rng(3)
    for ids in (workloads.zipf_ids(rng, 40000, domain, 1.1), np.full(5000, 777_777), np.arange(domain - 3000, domain),
                np.array([0, domain - 1, 0, domain - 1, 63, 64, 65])):
        u, inv, count, status = run(capi, ids, domain, cuda_device)
        ou, oinv = O.unique_map_sort(ids)
        assert status == 0 and np.array_equal(u, ou) and np.array_equal(inv, oinv)


def test_empty_input(capi, cuda_device):
    ids = torch.empty(0, dtype=torch.int64, device=cuda_device)
    u, inv, cnt = capi.unique_bitmap(ids, 100)
    torch.cuda.synchronize()
    assert cnt.cpu().tolist() == [0, 0] and inv.numel() == 0


def test_out_of_range_sets_status_without_faulting(capi, cuda_device):
    ids = np.array([5, 99, 100, -1, 7, 5])
    u, inv, count, status = run(capi, ids, 100, cuda_device)
    assert status & 1
    assert inv[2] == -1 and inv[3] == -1  # the reference's inverse kernel writes -1 there too before falling back to sort
    assert u.tolist() == [5, 7, 99] and inv[[0, 1, 4, 5]].tolist() == [0, 2, 1, 0]


def test_large_domain_properties(capi, cuda_device):
    """Largest configuration: 600 000 ids over a 12.5 M-node domain; checked through properties and the sort restatement."""
    domain, n = 12_500_000, 600_000
    ids = workloads.zipf_ids(np.random.default_rng(8), n, domain, 1.1)
    u, inv, count, status = run(capi, ids, domain, cuda_device)
    assert status == 0 and np.all(np.diff(u) > 0) and np.array_equal(u[inv], ids)
    ou, oinv = O.unique_map_sort(ids)
    assert count == ou.size and np.array_equal(u, ou) and np.array_equal(inv, oinv)


def test_workspace_reuse_back_to_back(capi, cuda_device):
    """The caller-owned workspace is reused across calls; the second call must not see the first call's bits."""
    domain = 100_000
    ws = capi.unique_workspace(domain, cuda_device)
    rng = np.random.default_rng(4)
    for _ in range(3):
        ids_np = rng.integers(0, domain, 20000)
        ids = torch.from_numpy(ids_np).to(cuda_device)
        u, inv, cnt = capi.unique_bitmap(ids, domain, workspace=ws)
        torch.cuda.synchronize()
        ou, oinv = O.unique_map_sort(ids_np)
        c = int(cnt[0])
        assert c == ou.size and np.array_equal(u.cpu().numpy()[:c], ou) and np.array_equal(inv.cpu().numpy(), oinv)


@pytest.mark.parametrize("n,domain", [(3, 2), (22000, 255), (22000, 257), (65536, 65536), (65537, 65537), (3000, 4_456_449)])
def test_repeated_ids_and_twins(capi, cuda_device, n, domain):
    """out_shared at the edges of words and tiles; the two equal halves of a twin count once."""
    rng = np.random.default_rng(n + domain)
    ids = rng.integers(0, domain, n)
    begin, length = n // 3, n // 4
    ids[begin + length:begin + 2 * length:2] = ids[begin:begin + length:2][:len(ids[begin + length:begin + 2 * length:2])]
    ou, oinv, _ = O.unique_map_bitmap(ids, domain)
    first = np.ones(n, bool)
    first[begin + length:begin + 2 * length] = ids[begin + length:begin + 2 * length] != ids[begin:begin + length]
    for twins, counted in (((0, 0), np.ones(n, bool)), ((begin, length), first)):
        shared = torch.full((min(n, domain),), 7, dtype=torch.uint8, device=cuda_device)
        u, inv, cnt = capi.unique_bitmap(torch.from_numpy(ids).to(cuda_device), domain, out_shared=shared, twins=twins)
        torch.cuda.synchronize()
        assert cnt.tolist() == [ou.size, 0]
        assert np.array_equal(u.cpu().numpy()[:ou.size], ou) and np.array_equal(inv.cpu().numpy(), oinv)
        assert np.array_equal(shared.cpu().numpy()[:ou.size], np.bincount(oinv[counted], minlength=ou.size) > 1)


@pytest.mark.parametrize("domain", [1, 64, 8192, 8193, 1_000_003])
def test_the_form_without_out_shared_needs_one_bitset(capi, cuda_device, domain):
    """scratch of control words, one bitset and the per-word offsets is enough where repeated ids are not asked for, and nothing behind it is
    written; with out_shared it is refused"""
    words, up = (domain + 63) // 64, lambda x: (x + 255) // 256 * 256
    small = up(((words + 127) // 128 + 4) * 4) + up(words * 8) + up(words * 4)
    rng = np.random.default_rng(domain)
    ids_np = rng.integers(0, domain, 5000)
    ids = torch.from_numpy(ids_np).to(cuda_device)
    ws = torch.full((small + 4096,), 0xCD, dtype=torch.uint8, device=cuda_device)
    u, inv, cnt = capi.unique_bitmap(ids, domain, workspace=ws[:small])
    torch.cuda.synchronize()
    ou, oinv = O.unique_map_sort(ids_np)
    assert cnt.tolist() == [ou.size, 0] and np.array_equal(u.cpu().numpy()[:ou.size], ou) and np.array_equal(inv.cpu().numpy(), oinv)
    assert bool((ws[small:] == 0xCD).all())
    with pytest.raises(capi.Ge2Error, match="workspace"):
        capi.unique_bitmap(ids, domain, workspace=ws[:small], out_shared=torch.empty(5000, dtype=torch.uint8, device=cuda_device))


@pytest.mark.parametrize("cols,want_src,n_deg,shared,mapped,sms,resident", [
    (3, True, 5, True, 300, 0, True), (3, True, 5, True, 300, 2, True), (3, False, 0, True, 300, 1, True), (2, False, 11, False, 300, 0, False),
    (3, True, 11, True, 300, 3, False), (2, True, 4, True, 250, 0, True), (3, True, 0, False, 300, 148, True)])
@pytest.mark.parametrize("B,C,N", [(1, 1, 11), (257, 3, 100), (1000, 2, 700)])
def test_drawing_and_mapping_in_one_go(capi, cuda_device, cols, want_src, n_deg, shared, mapped, sms, resident, B, C, N):
    """ge2_sample_unique leaves what the sampler and the unique-map leave one after the other, whatever the form, on all SMs or on a few."""
    domain, batches, dev = 300, 3, cuda_device
    rng = np.random.default_rng(B + N + n_deg)
    edges = torch.from_numpy(rng.integers(0, domain, ((batches if resident else 1) * B, cols))).to(dev)
    step, counters = torch.tensor([4], device=dev), torch.tensor([7, 8, 9], device=dev)
    nb = torch.tensor([batches], device=dev)
    n_ids = 2 * B + (2 if want_src else 1) * C * N
    i64 = dict(dtype=torch.int64, device=dev)

    def outputs():
        return dict(packed=torch.full((n_ids,), -7, **i64), deg_rows=torch.full((C * max(n_deg, 1),), -7, **i64), rel_ids=torch.full((B,), -7, **i64),
                    unique=torch.full((min(n_ids, mapped),), -7, **i64), inverse=torch.full((n_ids,), -7, **i64),
                    count=torch.full((2,), -7, dtype=torch.int32, device=dev), shared=torch.full((min(n_ids, mapped),), 9, dtype=torch.uint8, device=dev))

    want = outputs()
    deg = want["deg_rows"] if n_deg else None
    if resident:
        capi.sample_batch_dev(edges, nb, step, B, C, N, n_deg, domain, want_src, 99, want["packed"], deg, want["rel_ids"] if cols == 3 else None)
    else:
        capi.sample_negatives(edges, edges[:, cols - 1], cols, B, C, N, n_deg, domain, want_src, 99, 4, want["packed"], deg)
    capi.unique_bitmap(want["packed"], mapped, out_unique=want["unique"], out_inverse=want["inverse"], out_count=want["count"],
                       out_shared=want["shared"] if shared else None, twins=(2 * B, C * N) if want_src and shared else (0, 0))
    got = outputs()
    ws = capi.unique_workspace(mapped, dev).fill_(0xAB)
    f = capi.FrontDesc(edges=edges.data_ptr(), cols=cols, sms=sms, num_batches=batches, num_batches_dev=nb.data_ptr() if sms != 1 else None,
                       step_dev=step.data_ptr() if resident else None, seed=99, batch_index=4, B=B, C=C, N=N, n_deg=n_deg, domain=domain, mapped=mapped,
                       want_src_negs=want_src, num_counters=2, unique_ws=ws.data_ptr(), unique_ws_bytes=ws.numel(), counters=counters.data_ptr())
    for name in ("packed", "deg_rows", "unique", "inverse", "count"):
        setattr(f, name, got[name].data_ptr())
    f.rel_ids = got["rel_ids"].data_ptr() if resident else None
    f.shared = got["shared"].data_ptr() if shared else None
    capi.sample_unique(f)
    torch.cuda.synchronize()
    for name in want:
        assert torch.equal(want[name], got[name]), name
    assert counters.tolist() == [8, 9, 9] and (mapped < domain or int(want["count"][1]) == 0)


def test_drawing_and_mapping_refuses_what_does_not_fit(capi, cuda_device):
    import ctypes

    t = torch.zeros(64, dtype=torch.int64, device=cuda_device)
    ws = capi.unique_workspace(50, cuda_device)
    p = t.data_ptr()

    def call(**kw):
        a = dict(edges=p, cols=2, B=2, C=1, N=3, domain=50, mapped=50, packed=p, unique=p, inverse=p, count=p, unique_ws=ws.data_ptr(), unique_ws_bytes=ws.numel())
        return capi.load_library().ge2_sample_unique(ctypes.byref(capi.FrontDesc(**{**a, **kw})), None)

    for kw in (dict(B=0), dict(cols=4), dict(n_deg=4), dict(n_deg=1), dict(mapped=0), dict(sms=-1), dict(sms=149), dict(edges=None), dict(count=None),
               dict(step_dev=p), dict(num_counters=1), dict(num_counters=33, counters=p)):
        assert call(**kw) == 1, kw
    assert call(unique_ws=None) == 3 and call(unique_ws_bytes=ws.numel() // 4) == 3 and call(unique_ws=ws.data_ptr() + 8) == 3
