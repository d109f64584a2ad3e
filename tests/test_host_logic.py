"""Host-side logic that needs no GPU: the K-part rule of the GEMV (library vs the oracle's mirror), model presets, the
seeded draft substitution, the expected tokens per round, and the expert-parallel ownership map."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

import hipster_b200 as hb
from hipster_b200 import ep, kernels as K_, spec
from oracle import orc


def test_k_part_rule_matches_the_oracle_mirror_on_many_shapes():
    L = hb.lib(); O = orc.lib()
    for N in (16, 100, 512, 2368, 5120, 14336, 16480, 17408, 34816, 248320):
        for K in (256, 512, 1024, 2048, 5120, 6144, 10240, 17408):
            assert L.hp_gemv_parts(N, K) == O.orc_gemv_parts(N, K), (N, K)
    # the shapes of the dense configuration: down projection in 4 parts of 17 blocks, the big ones unsplit
    assert L.hp_gemv_parts(5120, 17408) == 4 and L.hp_gemv_parts(34816, 5120) == 1 and L.hp_gemv_parts(248320, 5120) == 1


def test_presets_carry_the_benchmark_shapes():
    c = hb.ModelCfg.preset("qwen35-27b")
    assert (c.n_layer, c.n_embd, c.n_ff, c.n_vocab, c.n_head, c.n_head_kv, c.gdn_qk_heads, c.gdn_v_heads) == (64, 5120, 17408, 248320, 24, 4, 16, 48)
    m = hb.ModelCfg.preset("flash-next")
    assert (m.n_layer, m.n_embd, m.n_expert, m.n_expert_used, m.expert_ff) == (48, 2048, 512, 10, 512)
    with pytest.raises(hb.HipsterError):
        hb.ModelCfg.preset("no-such-model")


def test_seeded_substitution_hits_the_requested_rate_exactly_at_the_extremes():
    plain = list(range(100, 200)); rng = np.random.default_rng(0)
    assert spec.seeded_substitutions(plain, 5, 4, 1.0, rng, 1000) == plain[5:9]
    wrong = spec.seeded_substitutions(plain, 5, 4, 0.0, rng, 1000)
    assert all(w != g for w, g in zip(wrong, plain[5:9]))
    hits = sum(a == b for _ in range(2000) for a, b in zip(spec.seeded_substitutions(plain, 5, 5, 0.7, rng, 1000), plain[5:10]))
    assert abs(hits / 10000 - 0.7) < 0.02


def test_expert_ranges_partition_the_experts():
    for world in (1, 2, 4, 8):
        owners = [ep.owner_of(e, world, 512) for e in range(512)]
        for r in range(world):
            lo, hi = ep.expert_range(r, world, 512)
            assert owners[lo:hi] == [r] * (hi - lo)
        assert sorted(set(owners)) == list(range(world))


def test_buffer_size_helpers():
    L = hb.lib()
    L.hp_argmax_scratch_bytes.restype = ctypes.c_size_t
    assert L.hp_xq8_q_bytes(1, 256) == 256 * 8 and L.hp_xq8_q_bytes(9, 256) == 2 * 256 * 8
    assert L.hp_argmax_scratch_bytes(6, 248320) > 0 and L.hp_argmax_scratch_bytes(0, 5) == 0


def test_package_imports_on_a_torch_build_without_cuda():
    code = ("import torch\n"
            "for n in ('_cuda_getCurrentRawStream', '_cuda_getDevice'):\n"
            "    delattr(torch._C, n)\n"                       # what a build without CUDA does not have
            "import hipster_b200\n"
            "print(hipster_b200.lib().hp_version())\n")
    r = subprocess.run([sys.executable, "-c", code], cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and int(r.stdout) >= 100, r.stderr[-2000:]


@pytest.mark.parametrize("native", [True, False])
def test_short_calls_work_with_and_without_the_native_entry_points(native):
    """The library alone serves the five calls too, and both forms refuse the same arguments (subprocess: the form is chosen once)."""
    code = ("import ctypes, sys\n"
            f"if not {native}: sys.modules['hipster_b200._calls'] = None\n"             # as if it had not been built
            "import hipster_b200 as hb\n"
            "from hipster_b200 import _lib\n"
            "H = _lib.hot(); L = hb.lib()\n"
            f"assert (H.__class__ is not ctypes.CDLL) == {native}\n"
            "def refused(f, *a):\n"
            "    try: f(*a)\n"
            "    except (TypeError, ctypes.ArgumentError): return True\n"
            "    return False\n"
            "for name, types in _lib._HOT.items():\n"
            "    f = getattr(H, name); null = [None if t == 'p' else 1 for t in types]\n"
            "    assert f(*null) == 1 and L.hp_last_error(), name\n"                     # refused by the library, before any CUDA call
            "    assert f(*[v if v is None else 2 ** 32 + 1 for v in null[:-1]], None) == 1, name\n"   # integers wrap as in C
            "    assert refused(f, *null[:-1]), name\n"
            "    for i, t in enumerate(types):\n"
            "        if t == 'i':\n"
            "            assert refused(f, *null[:i], None, *null[i + 1:]) and refused(f, *null[:i], 1.0, *null[i + 1:]), (name, i)\n"
            "        if t == 'p': assert refused(f, *null[:i], 1.0, *null[i + 1:]), (name, i)\n"
            "        if t == 'f': assert refused(f, *null[:i], None, *null[i + 1:]), (name, i)\n"
            f"if {native}:\n"
            "    try: H.bind('hp_version', 1)\n"
            "    except KeyError: print('ok')\n"
            "else: print('ok')\n")
    r = subprocess.run([sys.executable, "-c", code], cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr[-2000:]


@pytest.mark.parametrize("missing", ["headers", "compiler"])
def test_build_goes_on_without_the_native_entry_points(missing, monkeypatch, tmp_path, capfd):
    from hipster_b200 import build
    target = tmp_path / "_calls.so"
    target.write_bytes(b"of another interpreter")                                         # must not stay behind either
    monkeypatch.setattr(build, "CALLS", str(target))
    if missing == "headers":
        monkeypatch.setattr(build.sysconfig, "get_paths", lambda: {"include": str(tmp_path)})
    else:
        monkeypatch.setattr(build.shutil, "which", lambda name: str(tmp_path / "no-such-compiler"))
    assert build.build_calls(force=True) is None and not target.exists()
    assert "ctypes" in capfd.readouterr().err


def test_absent_tensors_are_refused_by_the_library(monkeypatch):
    monkeypatch.setattr(K_, "_raw_stream", lambda dev: 0); monkeypatch.setattr(K_, "_device", lambda: 0)   # refused before any CUDA call
    t = lambda *s: torch.zeros(s)  # noqa: E731
    with pytest.raises(hb.HipsterError, match="null pointer"):
        K_.gemv_q4k_q8(None, K_.XQ8(1, 256, "cpu"), 16, 256, t(1, 16))
    args = dict(q_norm=t(256), k_norm=t(256), rope=t(128, 32, 2), kc=t(1, 128, 256), vc=t(1, 128, 256))
    for name in args:
        with pytest.raises(hb.HipsterError, match="null pointer"):
            K_.attn_decode(t(1, 2 * 512 + 512), 0, 2, 1, 64, max_ctx=128, **{**args, name: None})


def test_sizes_that_were_asked_before_refuse_what_the_library_refuses(monkeypatch):
    """A number of another type is equal to the one that a size was computed for: it must not find that size."""
    monkeypatch.setattr(K_, "_raw_stream", lambda dev: 0); monkeypatch.setattr(K_, "_device", lambda: 0)
    monkeypatch.setattr(K_, "hot", lambda: type("Lib", (), {n: staticmethod(lambda *a: 0) for n in ("hp_argmax", "hp_attn_decode")}))
    t = torch.zeros(1, 2 * 512 + 512); x = torch.zeros((2, 512))
    attn = lambda ctx: K_.attn_decode(t, 0, 2, 1, 64, t, t, t, t, t, ctx)  # noqa: E731
    K_.XQ8(2, 512, "cpu"); K_.argmax(x, 512); attn(128)
    for other in (float, np.int64):
        for call in (lambda: K_.XQ8(other(2), 512, "cpu"), lambda: K_.XQ8(2, other(512), "cpu"), lambda: K_.argmax(x, other(512)), lambda: attn(other(128))):
            with pytest.raises(ctypes.ArgumentError):
                call()


def test_library_functions_take_any_ctypes_object():
    null = ctypes.c_size_t(0)   # an address as a size_t or an int64, as callers with their own bindings pass it
    L = hb.lib()
    assert L.hp_argmax(null, 1, ctypes.c_int64(1), 1, null, null, null, null) == 1 and b"null pointer" in L.hp_last_error()
    assert L.hp_gemv_q4k_q8(null, null, null, null, 16, 256, 1, 16, ctypes.c_uint64(0)) == 1 and b"null pointer" in L.hp_last_error()


def test_gdn_pass_over_several_sequences_needs_descriptors_and_takes_no_snapshots():
    """Several sequences would write the same snapshot rows, and without descriptors all would be the same sequence: refused before any CUDA call."""
    from test_gdn_gpu import _Gdn
    f = getattr(hb.lib(), "_ZN2hp11gdn_forwardERKNS_9GdnParamsEiP11CUstream_st")
    for nseq in (2, 3, 8):
        for fields in (dict(seq=4096, snap=4096), dict(seq=None, snap=None, imm_T=1)) + ((dict(seq=4100, snap=None),) if nseq > 2 else ()):   # three and more: read as 16-byte groups
            p = _Gdn(n_qk=1, n_v=2, **fields)
            assert f(ctypes.byref(p), nseq, ctypes.c_void_p(0)) == 1 and b"descriptors" in hb.lib().hp_last_error()


def test_argmax_hands_over_a_scratch_of_the_stated_size(monkeypatch):
    """A buffer of hp_argmax_scratch_bytes of its own wherever the library asks for one, no buffer where it asks for none."""
    L = hb.lib()
    assert L.hp_argmax_scratch_bytes(32, 65536) == 0 and L.hp_argmax_scratch_bytes(1, 65537) >= 8
    p = ctypes.c_void_p(4096)   # refused before any CUDA call
    assert L.hp_argmax(p, 1, 65537, 65537, p, None, None, None) == 1 and b"bad arguments" in L.hp_last_error()
    made, calls = [], []
    empty = torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, **k: made.append(empty(*a, **k)) or made[-1])
    monkeypatch.setattr(K_, "hot", lambda: type("Lib", (), {"hp_argmax": staticmethod(lambda *a: calls.append(a) or 0)}))
    monkeypatch.setattr(K_, "_raw_stream", lambda dev: 0); monkeypatch.setattr(K_, "_device", lambda: 0)
    for R, n in ((3, 17408), (6, 248320), (1, 65537)):
        made.clear()
        ids, vals = K_.argmax(torch.zeros((R, n)))
        scratch, need = calls[-1][6], L.hp_argmax_scratch_bytes(R, n)
        bufs = {t.data_ptr(): t.numel() * t.element_size() for t in made if t is not ids and t is not vals}
        assert (scratch is None and not bufs) if need == 0 else bufs[scratch] >= need
