"""The C-ABI library loads and exports every entry point include/roxy.h declares
(no device needed; nothing here launches a kernel)."""
import ctypes
import os
import re
import subprocess

import pytest

import roxy_native as nat

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared():
    src = open(os.path.join(ROOT, "include", "roxy.h")).read()
    return sorted(set(re.findall(r"^\s*(?:int|void\*|const char\*)\s+(rx_\w+)\s*\(", src, re.M)))


def test_header_declares_the_api():
    names = _declared()
    for n in ("rx_ctx_create", "rx_scene_set_triangles", "rx_bvh_build", "rx_trace_closest", "rx_render",
              "rx_accum_denoise", "rx_denoise"):
        assert n in names


@pytest.fixture(scope="module")
def L():
    if not os.path.exists(nat.LIB_PATH):
        nat.build()
    return nat.load_library()


def test_library_exports_every_declared_symbol(L):
    for name in _declared():
        assert hasattr(L, name), name


def test_binding_declares_every_symbol():
    assert set(_declared()) == set(nat._SIGS)


def test_binding_argument_counts_match_header():
    src = open(os.path.join(ROOT, "include", "roxy.h")).read()
    decls = re.findall(r"^\s*(?:int|void\*|const char\*)\s+(rx_\w+)\s*\(([^;]*?)\)\s*;", src, re.M | re.S)
    assert decls
    for name, params in decls:
        params = params.strip()
        n = 0 if params in ("", "void") else params.count(",") + 1
        assert len(nat._SIGS[name][0]) == n, f"{name}: header {n} args, binding {len(nat._SIGS[name][0])}"


def test_errors_without_device_are_reported_not_raised(L):
    import ctypes
    n = ctypes.c_int(-1)
    L.rx_device_count(ctypes.byref(n))
    assert n.value >= 0
    assert L.rx_version() >= 1


def _chained_kernels():
    """(kernel, pointers it only reads, what its chain_wait ties) of every
    kernel that may come up while the one before it runs."""
    csrc = os.path.join(os.path.dirname(nat.LIB_PATH), "csrc")
    for f in sorted(os.listdir(csrc)):
        if not f.endswith(".cu"):
            continue
        src = re.sub(r"//[^\n]*", "", open(os.path.join(csrc, f)).read())
        for part in re.split(r"\b__global__\b", src)[1:]:
            m = re.match(r"[^{;]*?\b(k_\w+)\s*\(((?:[^(){}]|\([^()]*\))*)\)\s*\{", part, re.S)
            assert m, part[:200]
            body = part[m.end():]
            end = re.search(r"^\}", body, re.M)
            w = re.search(r"\bchain_wait\(([^()]*)\)", body[:end.start()])
            if w:
                reads = re.findall(r"\bconst\s+\w+\s*\*\s*(?:__restrict__\s*)?(\w+)", m.group(2))
                yield m.group(1), reads, [a.strip() for a in w.group(1).split(",")]


def test_chained_kernels_tie_what_they_read_to_the_wait():
    """A load through a const pointer that did not pass through chain_wait may
    be moved before it, ahead of the kernel that writes the memory."""
    found = list(_chained_kernels())
    assert len(found) >= 20
    assert {"k_conv_fwd_ws", "k_conv_fwd_res", "k_atrous_r1", "k_lbvh_bottom_up"} <= {k for k, _, _ in found}
    loose = {k: sorted(set(reads) - set(tied)) for k, reads, tied in found}
    assert not {k: v for k, v in loose.items() if v}


_WAVE_CPP = """
#include "rx_wave.h"
extern "C" long long wave(long long frames, long long P, long long cap, long long shadow_cap, long long per_shadow,
                          long long free_bytes, int* asked) {
  return rx::default_wave_paths(frames, P, cap, shadow_cap, per_shadow, [&] { ++*asked; return free_bytes; });
}
"""


def test_free_memory_is_asked_for_only_while_the_buffers_do_not_hold_the_wave(tmp_path):
    """Images that do and do not divide the largest wave, one call after
    another: once the buffers hold the wave that a call takes, no later call
    like it asks (the question can stall for tens of milliseconds)."""
    (tmp_path / "wave.cpp").write_text(_WAVE_CPP)
    so = tmp_path / "wave.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I",
                    os.path.join(os.path.dirname(nat.LIB_PATH), "csrc"), "-o", so, tmp_path / "wave.cpp"], check=True)
    f = ctypes.CDLL(str(so)).wave
    f.restype, f.argtypes = ctypes.c_longlong, [ctypes.c_longlong] * 6 + [ctypes.POINTER(ctypes.c_int)]
    big = 180 << 30

    def call(frames, P, held, per, free):
        asked = ctypes.c_int(0)
        target = f(frames, P, held, held * per, per, free, ctypes.byref(asked))
        return target, max(1, min(frames, target // P)) * P, asked.value

    for P in (64 * 64, 1024 * 1024, 1920 * 1080, 1917 * 1081, 3840 * 2160, 7680 * 4320, 12000 * 12000):
        for frames in (1, 7, 64, 65, 100, 4096):
            for per in (1, 5):
                target, wave, asked = call(frames, P, 0, per, big)
                assert target == 1 << 27 and asked == (wave > 1 << 25)
                assert call(frames, P, wave, per, big) == (target, wave, 0), (P, frames)
                # held for a smaller wave than this call's: asked again
                if wave > 1 << 25:
                    assert call(frames, P, wave - 1, per, big)[2] == 1
    # a quarter of the free memory decides between 32 M and 128 M paths
    need = lambda paths: 4 * paths * (120 + 48)  # noqa: E731
    for free, want in ((need(1 << 27), 27), (need(1 << 27) - 4, 26), (need(1 << 26) - 4, 25), (0, 25)):
        assert call(4096, 1920 * 1080, 0, 1, free)[0] == 1 << want


def test_no_device_size_is_written_into_the_code():
    """The number of SMs comes from the device (Ctx::num_sms), so that rules
    that fill it hold on a part of one, too."""
    csrc = os.path.join(os.path.dirname(nat.LIB_PATH), "csrc")
    for f in sorted(os.listdir(csrc)):
        code = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(os.path.join(csrc, f)).read(), flags=re.S)
        assert not re.search(r"\b148(?:LL|u|U)?\b", code), f
