"""The mixture-of-experts FFN at the benchmark shape (512 routed experts, top-10 + shared, hidden 2048, expert FFN 512)
for the 24 rows of a configuration-5 verify pass, through the kernel-level C-ABI entry hp_moe_layer: bit for bit against
the CPU restatement (router GEMV, routing, per-(row, slot) expert GEMVs, SiLU, quantiser, slot-order combine) and,
for the routing, against the double-precision transcription of fn.hip:167-205."""
import ctypes

import numpy as np
import pytest
import torch

import hipster_b200 as hb
from hipster_b200 import kernels as K_, synth
from oracle import orc

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)


@pytest.mark.parametrize("n_expert,k,E,F,T", [(512, 10, 2048, 512, 24), (64, 4, 512, 256, 5), (512, 10, 2048, 512, 1)])
def test_moe_layer_bit_exact_vs_oracle(n_expert, k, E, F, T):
    rng = np.random.default_rng(n_expert + T)
    xn = rng.normal(0, 1, size=(T, E)).astype(np.float32)
    router = (rng.normal(0, 1, size=(n_expert + 1, E)) / np.sqrt(E)).astype(np.float32)     # router logits ~ N(0, 1)
    egu = synth.q4k_matrix(n_expert * 2 * F, E, seed=1).reshape(-1); edn = synth.q4k_matrix(n_expert * E, F, seed=2).reshape(-1)
    sgu = synth.q4k_matrix(2 * F, E, seed=3).reshape(-1); sdn = synth.q4k_matrix(E, F, seed=4).reshape(-1)
    d = lambda a: torch.from_numpy(a).cuda()
    ids, w, y = K_.moe_layer(d(xn), d(router), d(egu), d(edn), d(sgu), d(sdn), F, n_expert, k)
    K_.device_status()
    ids_o, w_o, y_o, lg = orc.moe_layer(xn, router, egu, edn, sgu, sdn, E, F, n_expert, k)
    assert np.array_equal(ids.cpu().numpy(), ids_o)
    assert np.array_equal(bits(w.cpu().numpy()), bits(w_o))
    assert np.array_equal(bits(y.cpu().numpy()), bits(y_o))
    # independent witness for the routing: same experts in the same order, weights within 1e-5 relative
    ids64, w64 = orc.ref64_moe_route(lg, n_expert, k)
    assert np.array_equal(ids64, ids_o)
    assert np.allclose(w_o, w64, rtol=1e-5, atol=0)


@pytest.mark.parametrize("n_expert,k,T", [(8, 2, 24), (4, 1, 19), (16, 3, 7)])
def test_experts_of_every_number_of_rows(n_expert, k, T):
    """Segments of 1 to 8 columns: up to 4 take the form that holds each column twice, more the full tile, and an expert
    of more than 8 rows both."""
    E, F = 512, 256
    rng = np.random.default_rng(T)
    xn = rng.normal(0, 1, size=(T, E)).astype(np.float32)
    router = (rng.normal(0, 1, size=(n_expert + 1, E)) / np.sqrt(E)).astype(np.float32)
    egu = synth.q4k_matrix(n_expert * 2 * F, E, seed=1).reshape(-1); edn = synth.q4k_matrix(n_expert * E, F, seed=2).reshape(-1)
    sgu = synth.q4k_matrix(2 * F, E, seed=3).reshape(-1); sdn = synth.q4k_matrix(E, F, seed=4).reshape(-1)
    d = lambda a: torch.from_numpy(a).cuda()
    ids, w, y = K_.moe_layer(d(xn), d(router), d(egu), d(edn), d(sgu), d(sdn), F, n_expert, k)
    K_.device_status()
    ids_o, _, y_o, _ = orc.moe_layer(xn, router, egu, edn, sgu, sdn, E, F, n_expert, k)
    assert np.array_equal(ids.cpu().numpy(), ids_o) and np.array_equal(bits(y.cpu().numpy()), bits(y_o))


def test_router_ties_go_to_the_lower_expert_id():
    """Two experts with identical router rows get identical probabilities: the lower id must be ranked first."""
    n_expert, k, E, F, T = 64, 4, 512, 256, 3
    rng = np.random.default_rng(5)
    xn = rng.normal(0, 1, size=(T, E)).astype(np.float32)
    router = (rng.normal(0, 1, size=(n_expert + 1, E)) / np.sqrt(E)).astype(np.float32)
    router[40] = router[7] = 0.5 * xn[0] / np.linalg.norm(xn[0])          # both win row 0 with exactly equal logits
    egu = synth.q4k_matrix(n_expert * 2 * F, E, seed=1).reshape(-1); edn = synth.q4k_matrix(n_expert * E, F, seed=2).reshape(-1)
    sgu = synth.q4k_matrix(2 * F, E, seed=3).reshape(-1); sdn = synth.q4k_matrix(E, F, seed=4).reshape(-1)
    d = lambda a: torch.from_numpy(a).cuda()
    ids, w, y = K_.moe_layer(d(xn), d(router), d(egu), d(edn), d(sgu), d(sdn), F, n_expert, k)
    ids_o, w_o, y_o, _ = orc.moe_layer(xn, router, egu, edn, sgu, sdn, E, F, n_expert, k)
    assert list(ids_o[0][:2]) == [7, 40]
    assert np.array_equal(ids.cpu().numpy(), ids_o) and np.array_equal(bits(y.cpu().numpy()), bits(y_o))


@pytest.mark.parametrize("n_expert,k,T", [(100, 10, 1), (512, 15, 3), (300, 3, 9)])
def test_rows_of_equal_probabilities_take_the_lowest_experts(n_expert, k, T):
    """More equal candidates than are ranked at once (a row of zeros: all probabilities the same), beside rows of the usual kind, for every number
    of warps per row."""
    E, F = 256, 256
    rng = np.random.default_rng(T)
    xn = rng.normal(0, 1, size=(T, E)).astype(np.float32); xn[T // 2] = 0.0
    router = (rng.normal(0, 1, size=(n_expert + 1, E)) / np.sqrt(E)).astype(np.float32)
    egu = synth.q4k_matrix(n_expert * 2 * F, E, seed=1).reshape(-1); edn = synth.q4k_matrix(n_expert * E, F, seed=2).reshape(-1)
    sgu = synth.q4k_matrix(2 * F, E, seed=3).reshape(-1); sdn = synth.q4k_matrix(E, F, seed=4).reshape(-1)
    d = lambda a: torch.from_numpy(a).cuda()
    ids, w, y = K_.moe_layer(d(xn), d(router), d(egu), d(edn), d(sgu), d(sdn), F, n_expert, k)
    K_.device_status()
    ids_o, w_o, y_o, _ = orc.moe_layer(xn, router, egu, edn, sgu, sdn, E, F, n_expert, k)
    assert list(ids_o[T // 2][:k]) == list(range(k))
    assert np.array_equal(ids.cpu().numpy(), ids_o) and np.array_equal(bits(w.cpu().numpy()), bits(w_o)) and np.array_equal(bits(y.cpu().numpy()), bits(y_o))


def test_unit_form_of_the_expert_gemv_matches_too():
    """The one-warp-per-unit form of the expert GEMVs (taken when the quads' activation buffers do not fit in shared
    memory, or with HIPSTER_B200_MOE_UNITS set) must give the same bits: the switch is read once per process, so the
    parity test of the small shape runs again in a child process with it set."""
    import os, subprocess, sys
    if os.environ.get("HIPSTER_B200_MOE_UNITS"):
        pytest.skip("already inside the child process")
    env = dict(os.environ, HIPSTER_B200_MOE_UNITS="1")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-m", "pytest", os.path.join(root, "tests", "test_moe_kernels_gpu.py"), "-q", "-m", "gpu", "-k", "bit_exact and 64-4"],
                       env=env, cwd=root, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    assert "1 passed" in r.stdout


class _Route(ctypes.Structure):   # MoeRouteParams of csrc/kernels.h
    _fields_ = [("W", ctypes.c_void_p), ("x", ctypes.c_void_p), ("logits", ctypes.c_void_p)] + [(n, ctypes.c_int) for n in ("E", "K", "k", "T")] + \
               [(n, ctypes.c_void_p) for n in ("ids", "w", "ticket", "row_tok", "row_pos", "row_slot")] + [("synth_key", ctypes.c_ulonglong)] + \
               [(n, ctypes.c_int) for n in ("e_lo", "e_hi", "own_shared")] + [(n, ctypes.c_void_p) for n in ("segs", "ctl", "touched", "err")]


# rows of a prompt chunk: one beyond a pass, a ragged last group of eight, the most pairs a thread takes (512 rows of 16 slots), one bucket more than
# threads, all rows on few experts, and a part of the experts without the shared one
@pytest.mark.parametrize("T,n_expert,k,lo,hi,shared", [(33, 64, 4, 0, 64, 1), (300, 512, 10, 0, 512, 1), (507, 1024, 15, 0, 1024, 1), (512, 16, 15, 0, 16, 1), (512, 512, 15, 128, 256, 0)])
def test_chunk_rows_are_grouped_by_expert(T, n_expert, k, lo, hi, shared):
    rng = np.random.default_rng(T + k)
    ids = np.full((T, k + 1), -1, dtype=np.int32)
    for t in range(T):
        ids[t, :k] = rng.choice(n_expert, size=k, replace=False)
    i32 = dict(dtype=torch.int32, device="cuda")
    d_ids, segs, ctl, touched = torch.from_numpy(ids).cuda(), torch.full((T * (k + 1), 16), 0x55, **i32), torch.full((4,), 7, **i32), torch.zeros(1, dtype=torch.int64, device="cuda")
    p = _Route(E=n_expert, k=k, T=T, ids=d_ids.data_ptr(), e_lo=lo, e_hi=hi, own_shared=shared, segs=segs.data_ptr(), ctl=ctl.data_ptr(), touched=touched.data_ptr())
    f = getattr(hb.lib(), "_ZN2hp14moe_group_rowsERKNS_14MoeRouteParamsEP11CUstream_st")
    hb.check(f(ctypes.byref(p), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    flat = ids.reshape(-1)
    want = {e: np.flatnonzero(flat == e) for e in list(range(lo, hi)) + ([-1] if shared else [])}
    want = {e: w for e, w in want.items() if len(w)}
    n = ctl[0].item()
    assert ctl[:3].tolist() == [sum((len(w) + 7) // 8 for w in want.values()), 0, 0]
    got, order = {}, []
    for expert, ncols, *cols in segs[:n, :10].tolist():
        assert 1 <= ncols <= 8 and (not order or order[-1] == expert or len(got[order[-1]]) == len(want[order[-1]]))
        got.setdefault(expert, []).extend(cols[:ncols]); order.append(expert)
    assert sorted(set(order), key=order.index) == list(want)                # in bucket order, the shared expert last
    assert all(np.array_equal(np.sort(got[e]), want[e]) for e in want)
    assert touched.item() == len(want)                                      # each matrix of the chunk counts once
