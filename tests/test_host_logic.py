"""CPU tests of the host-side logic and of the C-ABI library as a binary (no compute calls)."""
import ctypes
import os
import re

import numpy as np
import pytest

import motifcl_b200 as mb
from motifcl_b200 import codec, synth
from motifcl_b200.counter import initial_ternary


def test_library_builds_loads_and_exports_every_declared_symbol():
    if not os.path.isfile(mb.LIB_PATH):
        mb.build_library()
    L = mb.lib()
    names = mb.declared_symbols()
    assert len(names) >= 20
    missing = [n for n in names if not hasattr(L, n)]
    assert not missing, missing


def test_header_cites_a_reference_interface_for_every_entry_point():
    text = open(mb._lib.HEADER_PATH).read()
    assert "extern \"C\"" in text and "torch" not in text.lower()
    for cite in ("vulkan_backend.hpp", "compact_counter.cpp", "compact_counter.cl", "matmul.cpp"):
        assert cite in text


def test_no_device_is_reported_not_crashed():
    """Without a GPU, context creation is refused with a message -- the analogue of the
    reference's probe_vulkan_runtime().available() == false."""
    L = mb.lib()
    if L.mcl_cuda_device_count() > 0:
        pytest.skip("a CUDA device is present")
    ctx = ctypes.c_void_p()
    rc = L.mcl_cuda_create(0, ctypes.byref(ctx))
    assert rc == 5 and not ctx.value
    assert b"no CUDA device" in L.mcl_cuda_last_error(None)
    with pytest.raises(mb.MotifclCudaError):
        mb.Context(0)


def test_pack_unpack_roundtrip_and_oracle_agreement(orc):
    rng = np.random.default_rng(0)
    codes = rng.integers(0, 64, size=(7, 36)).astype(np.uint8)
    st = codec.pack_codes(codes)
    assert st.shape == (7, 27)
    assert np.array_equal(codec.unpack_codes(st, 36), codes)
    assert np.array_equal(orc.pack_codes(codes.reshape(-1)), st.reshape(-1))
    t, c = codec.decode(codes, 11)
    assert np.array_equal(codec.encode(t, c, 11), codes)


def test_initial_state_matches_libstdcxx_stream():
    """First digits std::uniform_int_distribution<int>(-1,1) draws from std::mt19937(777),
    generated with g++ 13 / libstdc++ (the reference constructor's stream)."""
    assert initial_ternary(777, 8).tolist() == [-1, 0, -1, -1, -1, 0, 0, -1]


def test_synthetic_shapes_and_weight_counts():
    ls = synth.stories15m_linears()
    assert len(ls) == 42
    assert sum(l.out_features * l.in_features for l in ls) == 5_971_968
    assert sum(l.out_features for l in ls) == 17_856
    big = synth.llama_linears(2048, 5632, 22)
    assert sum(l.out_features * l.in_features for l in big) == 1_130_364_928
    st = synth.counters(1, 0, 288, 288)
    codes = codec.unpack_codes(st, 288)
    assert codes.min() == 0 and codes.max() == 63
    assert synth.seed_for(2, 3, 1) == 20261125 + 2000 + 30 + 1


@pytest.mark.parametrize("rows,cols", [(8192, 288), (4096, 32000), (16384, 2048), (777, 1000), (1024, 512), (65536, 256)])
def test_magnitude_sample_covers_rows_and_columns(tmp_path, rows, cols):
    """The sampled units of a tensor stay inside it, one to a run, and see its columns evenly, also where a run is whole rows."""
    import subprocess
    units = rows * cols // 4
    step = max(1, units // 4096)
    src = tmp_path / "s.cpp"
    src.write_text('#include <cstdio>\n#include "sample_rule.h"\nint main() { for (long long u = 0; u < %d; ++u) '
                   'std::printf("%%lld\\n", mcl::sample_unit(u, %d)); }\n' % (units // step, step))
    exe = str(tmp_path / "s")
    subprocess.check_call(["g++", "-std=c++17", "-I", os.path.join(os.path.dirname(mb._lib.HEADER_PATH), os.pardir, "motifcl_b200", "csrc"), str(src), "-o", exe])
    at = np.array(subprocess.check_output([exe]).split(), dtype=np.int64)
    assert at.size >= 4096 and at.max() < units and np.array_equal(at // step, np.arange(at.size))
    groups = cols // 4
    seen = np.bincount(at % groups, minlength=groups)
    assert seen.max() <= 3 * -(-at.size // groups) + 2                          # no column is favoured
    assert np.count_nonzero(seen) >= 0.35 * min(groups, at.size)                 # chance would give 1 - e^(-samples / groups)
    assert np.count_nonzero(np.bincount(at // groups, minlength=rows)) >= 0.35 * min(rows, at.size)


def test_overlapping_kernels_read_by_ordinary_loads():
    """A kernel that starts before the one in front of it has ended (grid_wait) must not read through the read-only path: __ldg,
    ld.global.nc or const __restrict__.  The 2-bit words of a decode GEMV, which no such launch writes, are the exception."""
    csrc = os.path.join(os.path.dirname(mb._lib.HEADER_PATH), os.pardir, "motifcl_b200", "csrc")
    kernels = 0
    for name in sorted(os.listdir(csrc)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(csrc, name)).read())
        text = re.sub(r"uint4 mv_load\(.*?\n}", "", text, flags=re.S)
        head, *parts = re.split(r"(?=__global__)", text)
        waiting = [p for p in parts if "grid_wait();" in p]
        kernels += len(waiting)
        if name == "counter_update_body.cuh" or waiting:           # and the helpers in front of the kernels
            waiting.append(head)
        for p in waiting:
            assert not re.search(r"__ldg\s*\(|ld\.global\.nc", p), (name, p[:120])
            assert "__restrict__" not in p[:p.find("{")] or p is head, (name, p[:120])
    assert kernels >= 15


def test_decode_epilogue_passes_its_barriers_whatever_a_warp_has_seen():
    """A wait that runs out is seen by the four epilogue warps of the decode kernel at different times: what leads to their common
    barriers may depend on the parts of the list alone, not on the warp's own state (`ok`)."""
    csrc = os.path.join(os.path.dirname(mb._lib.HEADER_PATH), os.pardir, "motifcl_b200", "csrc")
    text = re.sub(r"//[^\n]*", "", open(os.path.join(csrc, "gemv_tc.cu")).read())
    at = text.index("for (GvParts", text.index("int n_local = 0, x = -1;"))
    end = depth = 0
    for i in range(at, len(text)):                               # the loop over the parts
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0 and text[i] == "}":
            end = i
            break
    loop = text[at:end]
    assert loop.count("bar.sync 1, 128") == 4
    code = loop[:loop.rindex("bar.sync 1, 128")]
    inner = code.index("for (int h = 0; h < RT && ok; ++h) {")   # leaves by itself; no barrier inside
    depth = 0
    for i in range(inner, len(code)):
        depth += {"{": 1, "}": -1}.get(code[i], 0)
        if depth == 0 and code[i] == "}":
            break
    assert "bar.sync" not in code[inner:i]
    for line in (code[:inner] + code[i:]).splitlines():
        if re.search(r"\bok\b|\babort_flag\b", line):
            assert not re.search(r"\bif \((?!threadIdx)|\bfor\b|\bwhile\b|\bcontinue\b|\bbreak\b|\breturn\b", line), line
