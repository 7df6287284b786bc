"""The host side of a kernel call: the built-in form of the entry points (csrc/binding.cc) beside ctypes', and the room of a layer's intermediates (ops/scratch.py).
What is called here computes on the host; nothing needs a GPU."""
import ctypes as C
import os
import shutil
import subprocess
import sys
import threading

import pytest
import torch

from jax_llama_b200.ops import _lib, build
from jax_llama_b200.models.feedforward import DenseFeedForward, MoeFeedForward
from jax_llama_b200.models.mixers import GlaMixer, LatentAttentionMixer
from jax_llama_b200.ops.scratch import ALIGN, CHUNK, LARGEST, Array, Scratch, empty, room_of


@pytest.fixture(scope="module")
def pair():
    """(the library with built-in entry points, the same library through ctypes alone)"""
    fast = _lib.lib()
    if build.build_binding() is None:
        pytest.skip("no interpreter headers: ctypes is what runs")
    slow = C.CDLL(fast._name)
    for name, (res, args) in {**_lib._SIGNATURES, **_lib._HYBRID}.items():
        getattr(slow, name).restype, getattr(slow, name).argtypes = res, args
    return fast, slow


def test_the_hot_entry_points_are_built_in(pair):
    fast, _ = pair
    for name in ("jl_gemm", "jl_linear_resident", "jl_gla_scan", "jl_attn_step", "jl_moe_combine", "jl_delta_head_scan", "jl_sample_full", "jl_decode_attn_fused"):
        assert type(getattr(fast, name)).__name__ == "builtin_function_or_method"


@pytest.mark.parametrize("name,args", [("jl_attn_generic_splits", (1, 16, 4, 4096)), ("jl_gla_scan_ws_floats", (3, 700, 16, 64, 128)),
                                       ("jl_gla_scan_ws_floats", (1, 2048, 4, 200, 64)), ("jl_delta_head_scan_ws_floats", (2, 1000, 16, 16, 64, 128)),
                                       ("jl_linear_f32_pair_ws", (4096, 2048, 8192, 200, 5464, 2048, 148)), ("jl_linear_f32_pair_ws", (4100, 2048, 8192, 200, 5464, 2048, 148)),
                                       ("jl_linear_f32_pair_ws", (None, 2048, 8192, 64, 64, 64, 148)), ("jl_attn_generic_splits", (True, 2, 1, 2 ** 31 - 1))])
def test_same_answers(pair, name, args):
    fast, slow = pair
    assert getattr(fast, name)(*args) == getattr(slow, name)(*args)


@pytest.mark.parametrize("M,N,K,pairs,slots,rows", [(300, 256, 256, 0, 0, 0), (65, 3000, 1024, 48, 2, 128), (2048, 6176, 1024, 74, 2, 256), (200, 10928, 2048, 74, 3, 224),
                                                    (2000, 256, 4096, 74, 2, 128), (18944, 256, 4096, 74, 1, 256)])
def test_workspace_of_the_float32_pairs(pair, M, N, K, pairs, slots, rows):
    """Two partial tiles a pair where runs end inside tiles, a further one only where a pair adds more blocks than it may in a row (148 SMs)."""
    assert pair[0].jl_linear_f32_pair_ws(4096, K, 8192, M, N, K, 148) == pairs * slots * rows * 256 * 4


def test_refusals_and_messages_are_the_same(pair):
    fast, slow = pair
    bad = (16, 16, 16, 16, 0, 8, 8, 0, 0, 148, 0)               # M = 0: refused before anything is launched
    assert fast.jl_gemm(*bad) == slow.jl_gemm(*bad) == 1
    assert b"M=0" in fast.jl_last_error()
    for call in ((), (1, 2), ("1", 2, 3, 4), (1.5, 2, 3, 4)):
        with pytest.raises((TypeError, C.ArgumentError)) as a:
            slow.jl_attn_generic_splits(*call)
        with pytest.raises(type(a.value)):
            fast.jl_attn_generic_splits(*call)
    assert fast.jl_attn_generic_splits(2 ** 32 + 1, 2, 1, 64) == slow.jl_attn_generic_splits(2 ** 32 + 1, 2, 1, 64)      # ctypes takes the low bits


def test_numbers_arrive_as_declared(pair):
    """Whole numbers for a float, None and 0 for an address: through the checks of a call that refuses its shape last."""
    fast, slow = pair
    args = lambda eps: (0, None, 0, 0, None, 0, 5, eps, 0)       # noqa: E731  jl_rmsnorm with M = 0 rows
    for eps in (1, 1e-5, True):
        assert fast.jl_rmsnorm(*args(eps)) == slow.jl_rmsnorm(*args(eps))


def _loaded(folder, **env):
    """What a new process that finds the package in `folder` says of an entry point's form."""
    code = "from jax_llama_b200.ops import _lib; f = _lib.lib(); print(type(f.jl_gemm).__name__, f.jl_attn_generic_splits(1, 16, 4, 4096))"
    kept = {k: v for k, v in os.environ.items() if not k.startswith("JLLAMA_")}
    r = subprocess.run([sys.executable, "-c", code], cwd=folder, env={**kept, "PYTHONPATH": str(folder), **env}, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return r.stdout.split()


@pytest.fixture
def installed(tmp_path, pair):
    """The package as an installation has it: its folder with the libraries (no stamps), neither csrc nor include."""
    shutil.copytree(build.ROOT / "jax_llama_b200", tmp_path / "jax_llama_b200", ignore=shutil.ignore_patterns("_C", "__pycache__"))
    libs = tmp_path / "jax_llama_b200" / "ops" / "_C"
    libs.mkdir()
    for so in (build.LIB_PATH, build.binding_path()):
        (libs / so.name).symlink_to(so)
    return tmp_path


def test_an_installed_package_without_sources_loads(installed, pair):
    splits = str(pair[1].jl_attn_generic_splits(1, 16, 4, 4096))
    assert _loaded(installed, JLLAMA_NO_AUTOBUILD="1") == ["builtin_function_or_method", splits]      # the binding that came with the library
    lib = installed / "jax_llama_b200" / "ops" / "_C" / build.LIB_PATH.name
    (installed / "another.so").symlink_to(build.LIB_PATH)
    assert _loaded(installed, JLLAMA_LIB=str(installed / "another.so")) == ["builtin_function_or_method", splits]
    (lib.parent / build.binding_path().name).unlink()
    assert _loaded(installed, JLLAMA_NO_AUTOBUILD="1") == ["_FuncPtr", splits]
    (lib.parent / build.binding_path().name).write_bytes(b"not a library")
    assert _loaded(installed, JLLAMA_NO_AUTOBUILD="1") == ["_FuncPtr", splits]


def test_a_binding_that_cannot_be_built_is_not_an_error(tmp_path, monkeypatch, caplog):
    ran = tmp_path / "ran"
    compiler = tmp_path / "cxx"
    compiler.write_text(f"#!/bin/sh\ntouch {ran}\nexit 1\n")
    compiler.chmod(0o755)
    monkeypatch.setenv("CXX", str(compiler))
    monkeypatch.setattr(build, "OUT_DIR", tmp_path / "out")
    monkeypatch.setenv("JLLAMA_NO_AUTOBUILD", "1")
    assert build.build_binding() is None and not ran.exists()                 # nothing is compiled where that is switched off
    monkeypatch.delenv("JLLAMA_NO_AUTOBUILD")
    assert build.build_binding() is None and ran.exists() and "ctypes" in caplog.text
    monkeypatch.setenv("CXX", str(tmp_path / "none"))
    assert build.build_binding() is None                                      # no compiler
    (tmp_path / "file").write_text("")
    monkeypatch.setattr(build, "OUT_DIR", tmp_path / "file" / "out")
    assert build.build_binding() is None                                      # no folder to write to


CPU = torch.device("cpu")


def test_outside_a_block_arrays_are_tensors():
    t = empty((3, 5), dtype=torch.float32, device=CPU)
    assert isinstance(t, torch.Tensor) and t.shape == (3, 5)


def test_arrays_of_a_block():
    with Scratch() as s:
        a, b, c = empty((3, 5), dtype=torch.float32, device=CPU), empty(7, dtype=torch.int32, device=CPU), empty((4, 6), dtype=torch.bfloat16, device=CPU)
        room = s.room
        assert all(isinstance(x, Array) for x in (a, b, c))
        assert a.data_ptr() == room.data_ptr() and b.data_ptr() - a.data_ptr() == ALIGN and c.data_ptr() - b.data_ptr() == ALIGN
        big = empty((LARGEST // 4 + 1, 1), dtype=torch.float32, device=CPU)
        none = empty((0, 4), dtype=torch.float32, device=CPU)
        assert isinstance(big, torch.Tensor) and isinstance(none, torch.Tensor)
        with Scratch() as inner:
            d = empty(3, dtype=torch.uint8, device=CPU)
            assert d.room is inner.room and d.room is not room
        assert empty(1, dtype=torch.uint8, device=CPU).room is room
        other = []
        th = threading.Thread(target=lambda: other.append(empty((2, 2), dtype=torch.float32, device=CPU)))
        th.start()
        th.join()
        assert isinstance(other[0], torch.Tensor)               # the block is its thread's
        first = s.room
        for _ in range(CHUNK // LARGEST + 1):                   # a full room: another one, the arrays keep theirs
            e = empty(LARGEST, dtype=torch.uint8, device=CPU)
        assert s.room is not first and e.room is s.room and a.room is first
    assert isinstance(empty(2, dtype=torch.uint8, device=CPU), torch.Tensor)


def test_an_array_answers_as_the_tensor_it_stands_for():
    t = torch.empty((6, 10), dtype=torch.bfloat16)
    a = Array(t.data_ptr(), (6, 10), 10, t.dtype, CPU, t)
    pairs = [(a, t), (a[:, 2:7], t[:, 2:7]), (a[:, :4], t[:, :4]), (a[:, 3:], t[:, 3:]), (a[:, 3:][:, 1:2], t[:, 3:][:, 1:2]), (a.view(60), t.view(60)),
             (a.view(4, 15), t.view(4, 15)), (a.view(-1), t.view(-1)), (a.view(-1, 5), t.view(-1, 5)), (a[:, :-4], t[:, :-4])]
    for x, y in pairs:
        assert x.data_ptr() == y.data_ptr() and tuple(x.shape) == tuple(y.shape) and x.numel() == y.numel() and x.dim() == y.dim()
        assert x.is_contiguous() == y.is_contiguous() and x.stride(0) == y.stride(0) and x.dtype == y.dtype and x.device == y.device
    for wrong in (lambda: a.view(7, 9), lambda: a[:, 1:3].view(-1), lambda: a[1:, :], lambda: a[:, ::2]):
        with pytest.raises((ValueError, IndexError)):
            wrong()


def test_an_array_says_what_it_is_not():
    t = torch.empty(4, 4)
    with pytest.raises(AttributeError, match="not a torch tensor"):
        Array(t.data_ptr(), (4, 4), 4, t.dtype, CPU, t).float()


@pytest.mark.parametrize("base", [GlaMixer, LatentAttentionMixer, DenseFeedForward, MoeFeedForward])
def test_a_layer_derived_elsewhere_has_tensors(base):
    class Own(base):
        pass

    for cls, kind in ((base, Array), (Own, torch.Tensor)):
        with room_of(object.__new__(cls)):
            assert type(empty((2, 2), dtype=torch.float32, device=CPU)) is kind
