"""CPU tests of the C-ABI library: it loads without a GPU, exports every symbol the header declares, and its
host-only entry points (rotation generator, sizing, argument checks) behave.  No kernel is launched here."""
import ctypes as C
import os
import re
import subprocess
import sys

import numpy as np
import pytest
import torch

import triebwerk_b200 as tq
from triebwerk_b200._lib import ModelShape
from oracle import tqo

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def header_functions():
    text = open(os.path.join(ROOT, "include", "triebwerk_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    names = re.findall(r"\b((?:launch|tq)_[a-z0-9_]+)\s*\(", text)
    return sorted(set(names))


def test_library_exports_every_declared_symbol():
    L = tq.lib()
    declared = header_functions()
    assert len(declared) >= 35
    for name in declared:
        assert hasattr(L, name), f"{name} is declared in include/triebwerk_b200.h but not exported"
    assert sorted(tq.SYMBOLS) == declared, "the loader's symbol list and the header disagree"


def test_reference_launcher_names_present():
    # the nine launcher symbols the reference's engine.cpp declares for this path (engine/engine.cpp:128-140,164)
    L = tq.lib()
    for name in ["launch_turbo_kv_quantize", "launch_turbo_kv_quantize_batch", "launch_turbo_gqa_attention_batch",
                 "launch_turbo_gqa_attention", "launch_turbo_gqa_prefill_attention", "launch_kv_cache_write_batch",
                 "launch_gqa_attention_batch", "launch_gqa_attention"]:
        assert hasattr(L, name)


def test_rotation_bytes_equal_oracle_generator():
    r = tq.ops.rotation_matrix(42).numpy()
    rh, _ = tqo.rotation(42)
    assert (r.view(np.uint16) == rh.view(np.uint16)).all()
    r7 = tq.ops.rotation_matrix(7).numpy()
    rh7, _ = tqo.rotation(7)
    assert (r7.view(np.uint16) == rh7.view(np.uint16)).all()


def test_status_strings_and_version():
    L = tq.lib()
    assert L.tq_version() >= 100
    assert L.tq_status_string(0) == b"ok"
    for code in range(-7, 0):
        assert L.tq_status_string(code) not in (None, b"", b"ok")


def test_workspace_bytes_grow_with_batch():
    L = tq.lib()
    a = L.tq_workspace_bytes(4, 16)
    b = L.tq_workspace_bytes(64, 16)
    c = L.tq_workspace_bytes(64, 32)
    assert 0 < a < b < c
    assert L.tq_workspace_bytes(0, 16) == 0


def _engine(kv_bits, layers=2, H=16, Hkv=8, D=128, msl=64):
    h = C.c_void_p()
    shape = ModelShape(layers, H, Hkv, D)
    st = tq.lib().tq_engine_create(C.byref(shape), msl, kv_bits, C.byref(h))
    return st, h


def test_engine_create_argument_checks():
    L = tq.lib()
    st, h = _engine(4)
    assert st == 0 and L.tq_engine_kv_bits(h) == 4
    L.tq_engine_destroy(h)
    st, h = _engine(3)  # unsupported kv_bits falls back to fp16 like the reference constructor
    assert st == 0 and L.tq_engine_kv_bits(h) == 0
    L.tq_engine_destroy(h)
    st, _ = _engine(4, D=64)
    assert st == -4
    st, _ = _engine(4, H=15)
    assert st == -1
    st, _ = _engine(4, msl=0)
    assert st == -1


def test_arena_sizing_matches_layout():
    L = tq.lib()
    G, msl, layers, Hkv, D = 4, 256, 3, 8, 128
    for bits, row_bytes, norm_bytes in ((4, 512, 16), (2, 256, 16), (0, 2048, 0)):
        st, h = _engine(bits, layers=layers)
        assert st == 0
        total = L.tq_engine_arena_bytes(h, G, msl, None)
        cache = layers * 2 * G * msl * (row_bytes + norm_bytes)
        assert total >= cache
        # what is not cache (positions, workspace, staging) does not scale with the context length
        total2 = L.tq_engine_arena_bytes(h, G, 2 * msl, None)
        grow = total2 - total
        assert cache <= grow <= cache + (1 << 20) + (4 * G * 16 * 4 * 132 if bits == 0 else 0)
        # ragged capacities: rounded up to 32 rows each
        caps = (C.c_int * G)(1, 33, 64, 250)
        ragged = L.tq_engine_arena_bytes(h, G, msl, caps)
        assert ragged < total
        L.tq_engine_destroy(h)


def test_calls_before_alloc_report_state_errors():
    L = tq.lib()
    st, h = _engine(4)
    assert L.tq_engine_advance(h, None) == -5
    assert L.tq_engine_layer_ptrs(h, 0, None, None, None, None, None) == -5
    assert L.tq_engine_layer_ptrs(h, 99, None, None, None, None, None) == -1
    assert L.tq_engine_set_arena(h, None, 0) == -1
    assert L.tq_engine_set_arena(h, 0x1001, 4096) == -1  # arena must be 256-byte aligned
    L.tq_engine_destroy(h)


def test_reference_engine_links_against_this_library_for_the_path():
    """The reference's engine.cpp, compiled to an object where it lies (headers only, nothing is run), leaves a set of
    launch_* symbols undefined.  Every one of them that belongs to this path must be exported by libtriebwerk_b200.so,
    and the header's prototype must have the parameter list of the reference's own declaration (half* <-> void*,
    cudaStream_t <-> tq_stream_t).  Symbol tables and declaration text only."""
    import re
    import subprocess
    import tempfile
    ref = os.path.join(os.path.dirname(ROOT), "reference", "engine", "engine.cpp")
    if not os.path.exists(ref):
        pytest.skip("the reference tree is not present on this machine")
    with tempfile.TemporaryDirectory() as tmp:
        obj = os.path.join(tmp, "engine_ref.o")
        r = subprocess.run(["g++", "-std=c++17", "-c", "-I/usr/local/cuda/include", "-I" + os.path.dirname(ref), ref, "-o", obj],
                           capture_output=True, text=True)
        if r.returncode != 0:
            pytest.skip("the reference engine.cpp does not compile here: " + r.stderr[-200:])
        undefined = {ln.split()[-1] for ln in subprocess.check_output(["nm", "-u", obj], text=True).splitlines() if " launch_" in ln}
    path = {s for s in undefined if "turbo" in s} | (undefined & {
        "launch_gqa_attention", "launch_gqa_attention_batch", "launch_gqa_prefill_attention", "launch_kv_cache_write_batch"})
    assert len(path) == 9, sorted(path)
    import triebwerk_b200
    exported = {ln.split()[-1] for ln in subprocess.check_output(["nm", "-D", "--defined-only", triebwerk_b200._lib.LIB_PATH], text=True).splitlines()}
    assert path <= exported, f"not exported: {sorted(path - exported)}"

    def params(text, name):
        m = re.search(r"void\s+" + name + r"\s*\(([^;{]*?)\)\s*[;{]", text, re.S)
        assert m, name
        out = []
        for prm in m.group(1).split(","):
            prm = re.sub(r"=.*", "", prm).strip()
            ptr = "*" in prm
            base = "int" if re.search(r"\bint\b", prm) and not ptr else ("float*" if "float" in prm else ("int*" if re.search(r"\bint\b", prm) else
                   ("stream" if "tream" in prm and not ptr else ("ptr" if ptr else prm.split()[0]))))
            out.append(base)
        return out

    ref_text = open(ref).read()
    hdr_text = open(os.path.join(ROOT, "include", "triebwerk_b200.h")).read()
    for name in sorted(path):
        assert params(ref_text, name) == params(hdr_text, name), name


@pytest.mark.skipif(torch.cuda.is_available(), reason="what a machine without a GPU does")
@pytest.mark.parametrize("call", [
    "tq.ops.launch_kv_cache_write_batch(None, None, None, None, None, 1, 1, 128)",  # there is no current stream
    "with FakeTensorMode():\n    t = torch.empty(1, 128, dtype=torch.float16, device='cuda')\n"
    "    tq.ops.launch_kv_cache_write_batch(t, t, t, t, t, 1, 1, 128)",             # there is no data pointer
])
def test_what_torch_throws_is_a_python_error(call):
    """... and not the end of the process: in a child, which would be gone."""
    src = ("import torch, triebwerk_b200 as tq\nfrom torch._subclasses.fake_tensor import FakeTensorMode\n"
           "try:\n" + "".join(f"    {line}\n" for line in call.split("\n")) + "except RuntimeError as e:\n    print('caught', type(e).__name__)")
    r = subprocess.run([sys.executable, "-c", src], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "caught" in r.stdout, f"{r.returncode}: {r.stderr[-600:]}"


def test_positions_are_taken_as_any_number():
    """The single-sequence launchers take the position as Python, numpy and torch make it, as int() does."""
    for name in ("launch_turbo_gqa_attention", "launch_gqa_attention"):
        seen = []
        old = tq._lib.hostcall.__dict__.get(name)
        tq._lib.hostcall.__dict__[name] = lambda *a: seen.append(a) or 0
        try:
            n = 14 if name == "launch_turbo_gqa_attention" else 10
            at = 8 if name == "launch_turbo_gqa_attention" else 5
            for pos in (3, 3.0, np.int64(3), np.float32(3), torch.tensor(3), torch.tensor(3.0)):
                args = [None] * n
                args[at] = pos
                getattr(tq.ops, name)(*args)
        finally:
            if old is None:
                del tq._lib.hostcall.__dict__[name]
            else:
                tq._lib.hostcall.__dict__[name] = old
        assert [type(a[at]) for a in seen] == [int] * 6 and {a[at] for a in seen} == {3}


def test_engine_calls_that_launch_kernels_check_the_device():
    """An engine's pointers belong to one device: with another one current its kernels would read memory that is not theirs.  There is
    one device at most to test on, so the source is read: every call with a stream that does more than copy begins with the check,
    or hands over to one that does."""
    src = open(os.path.join(ROOT, "triebwerk_b200", "csrc", "tq_capi.cu")).read()
    copies = {"tq_engine_reset", "tq_engine_status", "tq_engine_set_positions", "tq_engine_set_rotation", "tq_engine_read_output_f32"}
    bodies = {m.group(1): m.group(2) for m in re.finditer(r"^(?:static )?int (\w+)\([^{;]*?\) \{\n(.*?)^\}", src, re.S | re.M)}
    calls = [n for n in re.findall(r"^int (tq_engine_\w+)\([^)]*tq_stream_t[^)]*\) \{", src, re.M) if n not in copies]
    assert len(calls) >= 16

    def checks(name):
        first = re.search(r"engine_on_its_device|((?:tq_)?engine_\w+)\(e,", bodies[name])  # whichever comes first
        return first and (first.group(1) is None or first.group(1) in bodies and checks(first.group(1)))

    assert not [n for n in calls if not checks(n)]


@pytest.mark.parametrize("G,msl", [(1, 512), (1, 1536), (4, 256)])
def test_arena_of_a_small_engine_stays_in_proportion(G, msl):
    """The 64 MiB for prompts as fp16 rows are for batches that can use them; an engine whose slots fit 16 MiB takes those."""
    arena = {n: tq.Engine(msl, 4, num_layers=n, num_heads=16, num_kv_heads=8, head_dim=128).arena_bytes(G, msl) for n in (1, 2)}
    one_layer = arena[2] - arena[1]  # cache, partial results, staging of a layer
    assert arena[1] - one_layer <= (17 << 20) + (10 << 20)  # (10 MiB: the decode workspace)


def test_arena_holds_slots_longer_than_the_given_length():
    """Slots of capacities beyond max_seq_len (rounded up to 32 rows, or given so): what arena_bytes says is what alloc_batch carves."""
    e = tq.Engine(100, 4, num_layers=2, num_heads=16, num_kv_heads=8, head_dim=128)
    assert e.arena_bytes(2, 100, [100, 4000]) == e.arena_bytes(2, 4000, [100, 4000])
