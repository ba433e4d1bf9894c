"""The C-ABI library: it loads, exports every symbol the public header declares,
and refuses to compute without a GPU (no CPU fallback)."""
import ctypes as C
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib():
    from ornithology_b200 import _lib, build
    build.build()
    return _lib.load()


def declared_symbols():
    text = open(os.path.join(ROOT, "include", "ornith_cuda.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    names = set(re.findall(r"\b(ornith_[a-z0-9_]+)\s*\(", text))
    return sorted(names)


def test_header_symbols_are_exported(lib):
    names = declared_symbols()
    assert len(names) >= 40
    missing = [n for n in names if not hasattr(lib, n)]
    assert not missing, f"declared in include/ornith_cuda.h but not exported: {missing}"


def test_binding_table_matches_header(lib):
    from ornithology_b200 import _lib
    assert sorted(_lib.SYMBOLS) == declared_symbols()


def test_struct_layouts_match_the_engine(lib):
    from ornithology_b200 import _lib
    # reference: src/ornith_attn.h:57-69 -> 6 pointers + 5 ints on LP64
    assert C.sizeof(_lib.KvCache) == 6 * 8 + 5 * 4 + 4
    assert _lib.KvCache.quantized.offset == 48 and _lib.KvCache.len.offset == 56
    assert C.sizeof(_lib.DeltaState) == 16 and C.sizeof(_lib.ConvState) == 16
    assert lib.ornith_kv_bytes_per_token(2, 256, 0) == 4096
    assert lib.ornith_kv_bytes_per_token(2, 256, 1) == 1040


def test_no_cpu_fallback_without_a_gpu(lib):
    import torch
    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    assert lib.ornith_backend_cuda_available() == 0
    p = C.c_void_p()
    assert lib.ornith_cuda_malloc(C.byref(p), 64) == 6          # ORNITH_ERR_BACKEND
    assert b"no CPU fallback" in lib.ornith_cuda_last_error()
    from ornithology_b200 import attn
    import numpy as np
    # tier 1 keeps struct handling alive but computes nothing: outputs stay untouched
    c = attn.kv_init(4, 1, 8)
    out = np.full(8, 7.0, np.float32)
    z = np.ones(8, np.float32)
    attn.gqa_step(c, z, z, z, 1, out=out)
    assert (out == 7.0).all() and c.len == 0
    attn.kv_free(c)


def test_stream_of_a_torch_build_without_the_private_functions(monkeypatch):
    """The stream handed to the library comes from two private functions of torch where they exist, else from the public call."""
    import importlib.util
    import types
    import torch
    import ornithology_b200
    for name in ("_cuda_getCurrentRawStream", "_cuda_getDevice"):
        monkeypatch.delattr(torch._C, name, raising=False)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: types.SimpleNamespace(cuda_stream=1234))
    spec = importlib.util.spec_from_file_location("ornithology_b200._device_again", os.path.join(ornithology_b200.__path__[0], "device.py"))
    again = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(again)
    assert again._stream() == 1234


def test_decode_scratch_follows_the_batch(lib):
    """Host-side sizing only (no GPU work).  The size query does not see the cache, so it covers both schedules:
    the grid of splits (finer splits, hence more partials per head, when the batch is too small to fill the GPU;
    the CUDA-core kernel's 512-token splits as a floor) and the balanced ranges of the Q8_0 raw-fragment kernel
    (one partial slot per head for each of at most 592 / head-group-columns ranges plus one per sequence)."""
    from ornithology_b200._lib import CudaFullLayer
    layer = CudaFullLayer(16, 2, 256, 64, 1, 1e-6, 0.0, None, None, None)

    def rows(n_seq, max_len):
        total = lib.ornith_cuda_full_attn_step_scratch(C.byref(layer), n_seq, max_len)
        fixed = (n_seq * 16 * 256 * 4 + 255) // 256 * 256 + (n_seq * 16 * 4 + 255) // 256 * 256
        return (total - fixed) / (16 * 258 * 4)                          # partial rows per head

    def balanced(n_seq, max_len):
        tiles = -(-max_len // 16)
        floor_w = max(16, -(-tiles // 32))
        return min(592 // 2, -(-n_seq * tiles // floor_w)) + n_seq

    # 64 sequences of up to 32k tokens: the 512-token splits of the CUDA-core path (65 per sequence) bound it
    assert abs(rows(64, 32832) - 64 * 65) < 0.1 and balanced(64, 32832) == 296 + 64
    # 4 sequences x 8k: 320-token splits -> 26 partials per (sequence, head) = 104 rows; balanced: 122 ranges + 4
    assert abs(rows(4, 8256) - max(4 * 26, balanced(4, 8256))) < 0.1 and balanced(4, 8256) == 126
    # 8 sequences x 16k: 576-token splits -> 29, below the CUDA-core path's 33 -> 264 rows; balanced: 249 + 8
    assert abs(rows(8, 16448) - max(8 * 33, balanced(8, 16448))) < 0.1
    assert lib.ornith_cuda_full_attn_step_scratch(C.byref(layer), 0, 100) == 0
    # the short ranges (8 tiles and up, at most 16 per sequence) of a batch whose 16-tile ranges give fewer than 100 CTAs
    # (two head-group columns), and the 16-tile ranges of one that reaches them
    for n_seq, max_len, floor_w in ((12, 864, 8), (64, 180, 8), (33, 180, 8), (33, 564, 16), (16, 1564, 16), (20, 3064, 16)):
        ranges = lambda w: -(-n_seq * -(-max_len // 16) // w)
        assert (2 * ranges(16) < 100) == (floor_w == 8)
        assert abs(rows(n_seq, max_len) - (ranges(floor_w) + n_seq)) < 0.1, (n_seq, max_len)


def test_product_does_not_touch_the_oracle():
    """Nothing under the package or include/ may reference oracle/."""
    pkg = os.path.join(ROOT, "ornithology_b200")
    for dirpath, _, files in os.walk(pkg):
        if "build" in dirpath.split(os.sep)[-1:]:
            continue
        for f in files:
            if f.endswith((".py", ".cu", ".cuh", ".c", ".h")):
                text = open(os.path.join(dirpath, f), errors="replace").read()
                assert "oracle" not in text.lower(), f"{f} mentions the oracle"


def test_projection_sizing_and_no_gpu_behaviour(lib):
    """Host-side: the scratch of the integer projections is the Q8_K image of the activations (one 2336-byte image
    per 8 tokens x 256 inputs, the same for the three weight types), nothing for a type without an integer path or
    a width that is not a multiple of 256; without a GPU the products fail with a status."""
    import torch
    from ornithology_b200 import _lib
    img = lambda T, n_in: -(-(-(-T // 8) * (n_in // 256) * 2336) // 256) * 256
    for wt in (8, 12, 14):
        assert lib.ornith_cuda_matmul_q_scratch(wt, 1, 2048) == img(1, 2048)
        assert lib.ornith_cuda_matmul_q_scratch(wt, 70, 4096) == img(70, 4096)
    assert lib.ornith_cuda_matmul_q_scratch(13, 8, 2048) == 0          # Q5_K: the engine dequantises it
    assert lib.ornith_cuda_matmul_q_scratch(8, 8, 300) == 0
    assert lib.ornith_cuda_matmul_q_scratch(8, 0, 2048) == 0
    assert C.sizeof(_lib.CudaQproj) == 32 and _lib.CudaQproj.n_out.offset == 16 and _lib.CudaQproj.y.offset == 24
    # the dispatch of prompts, host only: the tile of every case that the GPU tests send to the tcgen05 kernels, each instantiation
    # of them among these, and shapes that stay with the other kernels
    from tests.test_gpu_qproj import TC5_CASES, tile_tokens
    for wtype, T, n_in, n_outs, tile in TC5_CASES:
        assert tile_tokens(wtype, n_in, n_outs, T) == tile, (wtype, T, n_in, n_outs)
    for wtype, tiles in (("q4_k", {64, 128, 192, 256}), ("q6_k", {128, 256}), ("q8_0", {64, 128})):
        assert {c[4] for c in TC5_CASES if c[0] == wtype} == tiles == {c[4] for c in TC5_CASES if c[0] == wtype and len(c[3]) > 1}
    for wtype, T, n_in, n_outs in (("q4_k", 64, 512, [16000]), ("q6_k", 300, 2304, [12300]), ("q6_k", 100, 4096, [2048]), ("q8_0", 64, 2048, [8192]),
                                   ("q6_k", 300, 2048, [512]), ("q6_k", 129, 2048, [1024]), ("q8_0", 128, 256, [8192]), ("q8_0", 80, 2048, [8192])):
        assert tile_tokens(wtype, n_in, n_outs, T) == 0
    assert tile_tokens("q8_0", 300, [64], 100) == -1 and tile_tokens("q8_0", 512, [64, 0], 100) == -1
    if not torch.cuda.is_available():
        p = _lib.CudaQproj(8, None, 64, None)
        assert lib.ornith_cuda_matmul_q_group(C.byref(p), 1, 2048, None, 4, 0, None) != 0
        assert lib.ornith_cuda_matmul_q(8, None, 2048, 64, None, 0, 4, None, 0, None, 0, None) != 0


@pytest.mark.parametrize("module", [True, False])
def test_fast_calls_pass_what_ctypes_passes(lib, monkeypatch, module):
    """The callables of _lib.fast(), with the _fastcall module and without it, against ctypes, on host-only entry points: sizes
    beyond 32 bits, null pointers, packed structs, whole numbers of every kind (as values, never as addresses), errors."""
    import struct
    import sys
    import numpy as np
    import torch
    from ornithology_b200 import _lib
    monkeypatch.setattr(_lib, "_fast", None)
    if not module:
        import ornithology_b200
        monkeypatch.delattr(ornithology_b200, "_fastcall", raising=False)
        monkeypatch.setitem(sys.modules, "ornithology_b200._fastcall", None)      # importing it raises ImportError
    f = _lib.fast()
    assert type(f.matmul_q_scratch).__name__ == ("Function" if module else "function")
    for args in ((8, 64, 4096), (14, 1 << 20, 8192), (3, 1, 256)):
        assert f.matmul_q_scratch(*args) == lib.ornith_cuda_matmul_q_scratch(*args)
    want = lib.ornith_cuda_matmul_q_scratch(8, 64, 4096)
    for whole in (np.int64, np.int32, torch.tensor, lambda n: torch.tensor([n])):
        assert f.matmul_q_scratch(8, 64, whole(4096)) == lib.ornith_cuda_matmul_q_scratch(8, 64, whole(4096)) == want > 0
    rows = struct.pack("@3i", 4096, 512, 512)
    arr = (C.c_int * 3)(4096, 512, 512)
    assert f.matmul_q_tile_tokens(14, 2048, rows, 3, 777) == lib.ornith_cuda_matmul_q_tile_tokens(14, 2048, C.addressof(arr), 3, 777)
    assert f.matmul_q_tile_tokens(14, 2048, torch.tensor([4096, 512, 512], dtype=torch.int32), 3, 777) == f.matmul_q_tile_tokens(14, 2048, rows, 3, 777)
    assert f.matmul_q_tile_tokens(14, 2048, None, 3, 777) == -1
    for bad in (1.5, None, "6", b"6"):
        with pytest.raises((TypeError, C.ArgumentError)):
            f.matmul_q_scratch(8, 64, bad)
    for n in (0, 2, 4, 17):
        with pytest.raises(TypeError):
            f.matmul_q_scratch(*range(n))
    assert not hasattr(f, "rope_inv_freq")                 # takes a float: ctypes only
