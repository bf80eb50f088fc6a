"""The C-ABI library loads without a GPU and exports every function include/ge2_b200.h declares."""
import ctypes
import re
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def declared_functions():
    text = (ROOT / "include" / "ge2_b200.h").read_text()
    return sorted(set(re.findall(r"GE2_API[^;(]*?\b(ge2_\w+)\s*\(", text)))


def test_header_declares_functions():
    names = declared_functions()
    assert "ge2_unique_bitmap" in names and "ge2_lp_step" in names and "ge2_adagrad_scatter" in names
    assert len(names) >= 17


def test_library_exports_every_declared_symbol(ge2):
    lib = ge2.load_library()
    for name in declared_functions():
        assert hasattr(lib, name), f"{name} declared in include/ge2_b200.h but not exported"
    assert sorted(ge2.capi.EXPORTS) == [n for n in declared_functions() if n in ge2.capi.EXPORTS]
    assert set(declared_functions()) <= set(ge2.capi.EXPORTS)


def test_host_only_entry_points(ge2):
    lib = ge2.load_library()
    assert lib.ge2_version().startswith(b"ge2_b200")
    assert lib.ge2_status_string(0) == b"ok"
    assert lib.ge2_unique_workspace_bytes(0) == 0
    assert lib.ge2_unique_workspace_bytes(1_000_000) >= 125_000 + 62_500
    # argument validation happens before any CUDA call
    assert lib.ge2_unique_bitmap(None, -1, 10, None, 0, None, None, None, None) == 1
    d = ge2.capi.LpDesc()
    out = ctypes.c_size_t(0)
    assert lib.ge2_lp_workspace_bytes(ctypes.byref(d), ctypes.byref(out)) == 1


def test_selected_negative_entry_points_validate_before_any_cuda_call(ge2):
    """Shapes the reference rejects with TORCH_CHECK (distmult_selected_neg_cuda.cpp:63-76, .cu:215-217) come back as
    GE2_ERR_INVALID_ARGUMENT; D above the kernels' 128 as GE2_ERR_UNSUPPORTED; empty inputs are accepted without a launch."""
    lib = ge2.load_library()
    p = 4096  # never dereferenced: every call below returns before it touches the device
    tour = lambda chunks, rows, negs, sel, D: lib.ge2_tournament_select(p, p, None, None, chunks, rows, negs, sel, D, p, p, None)  # noqa: E731
    assert tour(2, 5, 10, 3, 8) == 1       # negatives not divisible into groups
    assert tour(2, 5, 10, 0, 8) == 1
    assert tour(2, 5, 10, 5, 129) == 4     # D > 128
    assert tour(70000, 5, 10, 5, 8) == 4   # more chunks than a grid dimension holds
    assert tour(0, 5, 10, 5, 8) == 0 and tour(2, 0, 10, 5, 8) == 0
    fwd = lambda kind, chunks, rows, negs, sel, D: lib.ge2_selected_neg_scores(kind, p, p, p, chunks, rows, negs, sel, D, p, None, None)  # noqa: E731
    assert fwd(0, 1, 1, 1, 1, 8) == 1      # SelectedNegScoreKind::NONE
    assert fwd(3, 1, 1, 1, 1, 8) == 1
    assert fwd(1, 1, 1, 0, 1, 8) == 1      # no negatives to index
    assert fwd(2, 1, 1, 1, 1, 200) == 4
    assert fwd(1, 3, 0, 5, 2, 8) == 0 and fwd(2, 3, 4, 5, 0, 8) == 0
    assert lib.ge2_selected_neg_scores_backward(7, p, p, p, p, 1, 1, 1, 1, 8, p, p, None, None) == 1


def test_desc_struct_matches_header_size(ge2):
    """ctypes mirror and C struct agree in size (a C probe compiled against the header prints sizeof)."""
    import subprocess
    import tempfile

    src = '#include "ge2_b200.h"\n#include <stdio.h>\nint main(){printf("%zu %zu %zu", sizeof(ge2_lp_desc), offsetof(ge2_lp_desc, workspace), offsetof(ge2_lp_desc, rel));return 0;}'
    with tempfile.TemporaryDirectory() as td:
        c = Path(td) / "p.c"
        c.write_text(src)
        exe = Path(td) / "p"
        r = subprocess.run(["gcc", "-I", str(ROOT / "include"), str(c), "-o", str(exe)], capture_output=True, text=True)
        if r.returncode != 0:
            pytest.skip("no C compiler: " + r.stderr[:80])
        size, off_ws, off_rel = map(int, subprocess.run([str(exe)], capture_output=True, text=True).stdout.split())
    D = ge2.capi.LpDesc
    assert ctypes.sizeof(D) == size and D.workspace.offset == off_ws and D.rel.offset == off_rel


def test_swap_and_eval_structs_match_header(ge2):
    """the ctypes mirrors of ge2_swap_desc and ge2_eval_desc agree with the C structs in size and in the offsets of a few members"""
    import subprocess
    import tempfile

    src = ('#include "ge2_b200.h"\n#include <stdio.h>\n#include <stddef.h>\nint main(){printf("%zu %zu %zu %zu %zu %zu", sizeof(ge2_swap_desc), '
           'offsetof(ge2_swap_desc, slab_bytes), offsetof(ge2_swap_desc, status), sizeof(ge2_eval_desc), offsetof(ge2_eval_desc, neg_ids), '
           'offsetof(ge2_eval_desc, workspace));return 0;}')
    with tempfile.TemporaryDirectory() as td:
        c = Path(td) / "p.c"
        c.write_text(src)
        exe = Path(td) / "p"
        r = subprocess.run(["gcc", "-std=c99", "-I", str(ROOT / "include"), str(c), "-o", str(exe)], capture_output=True, text=True)
        if r.returncode != 0:
            pytest.skip("no C compiler: " + r.stderr[:80])
        s_size, s_slab, s_status, e_size, e_neg, e_ws = map(int, subprocess.run([str(exe)], capture_output=True, text=True).stdout.split())
    S, E = ge2.capi.SwapDesc, ge2.capi.EvalDesc
    assert ctypes.sizeof(S) == s_size and S.slab_bytes.offset == s_slab and S.status.offset == s_status
    assert ctypes.sizeof(E) == e_size and E.neg_ids.offset == e_neg and E.workspace.offset == e_ws


def _old_caller(code):
    """runs `code` in a process of its own with `lib` loaded, `D` the ctypes descriptor, and `d`: a valid descriptor as a caller built against
    version 0.1 lays it out, ending with workspace_bytes, on the last bytes of a page behind which nothing can be read"""
    import subprocess
    import sys

    head = f"""
import ctypes, importlib, mmap, sys
sys.path.insert(0, {str(ROOT)!r})
capi = importlib.import_module("ge-2_b200.capi")
lib, D = capi.load_library(), capi.LpDesc
size = D.node_state.offset
libc = ctypes.CDLL(None, use_errno=True)
pages = mmap.mmap(-1, 2 * mmap.PAGESIZE)
base = ctypes.addressof(ctypes.c_char.from_buffer(pages))
assert libc.mprotect(ctypes.c_void_p(base + mmap.PAGESIZE), mmap.PAGESIZE, 0) == 0
full = D(B=8, C=2, N=4, D=16, U=40, emb_stride=16, edge_stride=1)
for name in ("node_emb", "src_ids", "dst_ids", "dst_negs", "node_grad", "loss"):
    setattr(full, name, 4096)
at = base + mmap.PAGESIZE - size
ctypes.memmove(at, ctypes.addressof(full), size)
d = ctypes.cast(at, ctypes.POINTER(D))
need = ctypes.c_size_t()
"""
    return subprocess.run([sys.executable, "-c", head + code], capture_output=True, text=True)


def test_descriptor_of_version_0_1_is_read_no_further_than_it_reaches():
    r = _old_caller("""
assert lib.ge2_lp_workspace_bytes(d, ctypes.byref(need)) == 0 and need.value > 0
assert lib.ge2_lp_step(d, None) == 3  # no workspace: found out before any CUDA call, after the descriptor was copied
""")
    assert r.returncode == 0, (r.returncode, r.stderr)


def test_row_update_members_count_only_with_their_flag(ge2):
    """what lies behind an old descriptor must not switch the in-place optimizer on, nor have the call refused"""
    lib, capi = ge2.load_library(), ge2.capi
    d = capi.LpDesc(B=8, C=2, N=4, D=16, U=40, emb_stride=16, edge_stride=1)
    for name in ("node_emb", "src_ids", "dst_ids", "dst_negs", "node_grad", "loss"):
        setattr(d, name, 4096)
    d.node_state = 4096  # without row_shared
    need = ctypes.c_size_t()
    assert lib.ge2_lp_workspace_bytes(ctypes.byref(d), ctypes.byref(need)) == 0
    d.flags = capi.LP_HAS_ROW_UPDATE
    assert lib.ge2_lp_workspace_bytes(ctypes.byref(d), ctypes.byref(need)) == 1
    assert b" 0.1 " not in lib.ge2_version()


def test_row_update_needs_the_number_of_table_rows(ge2):
    lib, capi = ge2.load_library(), ge2.capi
    d = capi.LpDesc(B=8, C=2, N=4, D=16, U=40, emb_stride=16, edge_stride=1, flags=capi.LP_HAS_ROW_UPDATE)
    for name in ("node_emb", "src_ids", "dst_ids", "dst_negs", "node_grad", "loss", "node_state", "row_shared"):
        setattr(d, name, 4096)
    need = ctypes.c_size_t()
    for rows, rc in ((0, 1), (-1, 1), (40, 0)):
        d.table_rows = rows
        assert lib.ge2_lp_workspace_bytes(ctypes.byref(d), ctypes.byref(need)) == rc


def _train_desc(capi):
    """a whole step that is right in everything but its unique-map workspace, which is looked at last: GE2_ERR_WORKSPACE, and no launch"""
    p, q = 4096, 8192  # never dereferenced
    lp = capi.LpDesc(B=8, C=2, N=4, D=16, R=5, U=40, emb_stride=16, edge_stride=1, rel_stride=3, has_relations=1, use_inverse=1,
                     flags=capi.LP_HAS_ROW_UPDATE, node_lr=0.1, table_rows=100, node_emb=p, node_state=q, row_index=p, row_shared=p, deg_sample_rows=p,
                     n_deg=2, workspace=p, workspace_bytes=1 << 30)
    for name in ("src_ids", "dst_ids", "rel_ids", "dst_negs", "src_negs", "node_grad", "loss", "rel", "inv_rel", "rel_grad", "inv_rel_grad"):
        setattr(lp, name, p)
    t = capi.TrainDesc(lp=ctypes.pointer(lp), edges=p, cols=3, n_deg=2, domain=100, packed=p, deg_rows=p, n_ids=2 * 8 + 2 * 2 * 4, unique=p, inverse=p, count=p,
                       shared=p, twin_begin=16, twin_len=8, table=p, state=q, table_rows=100, lr=0.1, dense_lr=0.1, grad_scale=1.0, num_dense=2,
                       dense_numel=80)
    for k in range(2):
        t.dense_param[k] = t.dense_state[k] = t.dense_grad[k] = p
    return t, lp


def test_whole_step_refuses_what_does_not_fit_together(ge2):
    lib, capi = ge2.load_library(), ge2.capi
    call = lambda t: lib.ge2_train_step(ctypes.byref(t), None)  # noqa: E731
    t, lp = _train_desc(capi)
    assert call(t) == 3
    t.dense_param[1] = None
    assert call(t) == 1
    for name, value in [("num_dense", 3), ("num_dense", -1), ("n_ids", 31), ("n_ids", 24), ("shared", 8192), ("shared", None), ("lr", 0.2), ("table", 8192),
                        ("state", 4096), ("unique", 8192), ("table_rows", 99), ("table_rows", 0), ("domain", 0), ("cols", 0), ("n_deg", 5), ("n_deg", 1),
                        ("edges", None), ("packed", None), ("inverse", None), ("count", None), ("deg_rows", None), ("twin_len", 9), ("twin_begin", -1)]:
        t, lp = _train_desc(capi)
        setattr(t, name, value)
        assert call(t) == 1, (name, value)
    for name, value in [("B", 0), ("emb_stride", 32), ("flags", 0), ("node_lr", 0.3), ("table_rows", 101), ("use_inverse", 0)]:
        t, lp = _train_desc(capi)
        setattr(lp, name, value)
        assert call(t) == 1, (name, value)
    t, lp = _train_desc(capi)
    lp.workspace_bytes = 0
    assert call(t) == 3


def test_whole_step_takes_a_workspace_without_the_streaming_forms_parts(ge2):
    """the smaller of the two sizes that an fp16 step can do with; what is refused next is the missing edge list"""
    lib, capi = ge2.load_library(), ge2.capi
    t, lp = _train_desc(capi)
    lp.precision, lp.B, lp.C, lp.N, lp.D, lp.emb_stride, lp.n_deg, lp.deg_sample_rows = 1, 10368, 27, 1300, 50, 50, 0, None
    need = ctypes.c_size_t()
    assert lib.ge2_lp_workspace_bytes(ctypes.byref(lp), ctypes.byref(need)) == 0
    t.edges = None
    parts = 148 * 2 * 128 * 64 * 4
    for size, rc in ((need.value, 1), (need.value - parts, 1), (need.value - parts - 1, 3)):
        lp.workspace_bytes = size
        assert lib.ge2_train_step(ctypes.byref(t), None) == rc


def test_train_struct_matches_header(ge2):
    import subprocess
    import tempfile

    src = ('#include "ge2_b200.h"\n#include <stdio.h>\n#include <stddef.h>\nint main(){printf("%zu %zu %zu %zu", sizeof(ge2_train_desc), '
           'offsetof(ge2_train_desc, shared), offsetof(ge2_train_desc, num_dense), offsetof(ge2_train_desc, dense_numel));return 0;}')
    with tempfile.TemporaryDirectory() as td:
        c = Path(td) / "p.c"
        c.write_text(src)
        exe = Path(td) / "p"
        r = subprocess.run(["gcc", "-std=c99", "-I", str(ROOT / "include"), str(c), "-o", str(exe)], capture_output=True, text=True)
        if r.returncode != 0:
            pytest.skip("no C compiler: " + r.stderr[:80])
        size, shared, dense, numel = map(int, subprocess.run([str(exe)], capture_output=True, text=True).stdout.split())
    T = ge2.capi.TrainDesc
    assert ctypes.sizeof(T) == size and T.shared.offset == shared and T.num_dense.offset == dense and T.dense_numel.offset == numel


def test_comments_of_the_header_stand_where_they_belong():
    """a comment that runs on behind a #define must not swallow the declarations after it or be swallowed by them"""
    text = (ROOT / "include" / "ge2_b200.h").read_text()
    for line in text.splitlines():
        if line.startswith("#define") and "/*" in line and "GE2_PRECISION" not in line:
            assert line.rstrip().endswith("*/"), line
    kinds = text[text.index("#define GE2_SELECTED_DOT"):].splitlines()[:2]
    assert kinds[0].split()[:3] == ["#define", "GE2_SELECTED_DOT", "1"] and kinds[1].split() == ["#define", "GE2_SELECTED_L2", "2"]
