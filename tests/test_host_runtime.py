"""Host code of the library on a CUDA runtime without a GPU
(tests/cpp/fake_cudart.cpp): what is launched, copied and allocated when."""
import ctypes as C
import os
import shutil
import subprocess
import threading
import time

import numpy as np
import pytest

from nr_gpu_ldpc_gb300 import _lib, build
from nr_gpu_ldpc_gb300.batch import make_jobs

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not present")


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    objs = [os.path.join(build.BUILD, s.replace(".cu", ".o")) for s in build.SOURCES]
    build.build(force=not all(map(os.path.exists, objs)))
    so = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I",
                    os.path.join(CUDA, "include"), os.path.join(HERE, "cpp", "fake_cudart.cpp"), *objs, "-o", so],
                   check=True, capture_output=True, text=True)
    lib = C.CDLL(so)
    for name, (res, args) in _lib.SIGNATURES.items():
        fn = getattr(lib, name)
        fn.restype, fn.argtypes = res, args
    lib.fake_last_launch.restype = C.c_char_p
    lib.fake_unfinished.restype = lib.fake_uploaded.restype = C.c_long
    lib.fake_stream_full.argtypes = [C.c_void_p]
    for f in ("fake_stream_busy", "fake_stream_capturing"):
        getattr(lib, f).argtypes = [C.c_void_p, C.c_int]
    return lib


@pytest.fixture
def rt(fake):
    fake.fake_reset()
    return fake


class Handle:
    """A decoder handle and buffers for n codewords."""

    def __init__(self, rt, bg=1, z=384, n=64, device=0):
        cfg = _lib.ConfigC(bg=bg, z=z, max_batch=n, alpha=0.75, device=device, cw_per_cta=0)
        self.rt, self.h = rt, C.c_void_p()
        assert rt.nrldpc_init(C.byref(cfg), C.byref(self.h)) == 0
        cols = 68 if bg == 1 else 52
        self.buf = np.zeros(n * cols * z + 4, np.float32)
        self.llr = (self.buf.ctypes.data + 15) // 16 * 16
        self.out = np.zeros(n * (cols * z + 7) // 8 + 8, np.uint8)

    def decode(self, n, stream, early=0):
        assert self.rt.nrldpc_decode(self.h, self.llr, self.out.ctypes.data, n, 5, early, None, None, stream) == 0
        return b"split" in self.rt.fake_last_launch()

    def decode_host_q(self, n, stream):
        assert self.rt.nrldpc_decode_host_async_q(self.h, self.llr, 2, 0.5, self.out.ctypes.data, n, 5, 0, stream) == 0

    def close(self):
        self.rt.nrldpc_destroy(self.h)


class List:
    """A job list handle."""

    def __init__(self, rt, max_jobs=512):
        self.rt, self.h = rt, C.c_void_p()
        assert rt.nrldpc_batch_create(0, max_jobs, 0.75, C.byref(self.h)) == 0

    def set_jobs(self, bg, z):
        self.jobs, n_llr, _, n_out = make_jobs(np.broadcast_to(bg, np.shape(z)), np.asarray(z))
        self.buf = np.zeros(n_llr + 4, np.float32)
        self.llr = (self.buf.ctypes.data + 15) // 16 * 16
        self.out = np.zeros(n_out, np.uint8)
        return self.rt.nrldpc_batch_set_jobs(self.h, self.jobs.ctypes.data, self.jobs.size)

    def decode(self, stream):
        assert self.rt.nrldpc_batch_decode(self.h, self.llr, self.out.ctypes.data, 5, 0, None, stream) == 0
        return b"split" in self.rt.fake_last_launch()

    def close(self):
        self.rt.nrldpc_batch_destroy(self.h)


STREAM = [0x100, 0x200, 0x300, 0x400, 0x500, 0x600]  # non-blocking streams, made up


def test_nothing_runs_before_its_tables_and_lists_have_landed(rt):
    # work on a non-blocking stream is not ordered after a pageable copy or a
    # memset, which only the legacy stream waits for
    d = Handle(rt)
    assert rt.fake_unfinished() == 0
    b = List(rt)
    assert rt.fake_unfinished() == 0
    e = np.zeros(1 << 24, np.uint8)
    for z in ([384] * 5, [384] * 5 + [40] * 20, [64] * 400):
        for call in (lambda: b.decode(STREAM[0]),
                     lambda: rt.nrldpc_batch_derate(b.h, e.ctypes.data, b.llr, STREAM[0]),
                     lambda: rt.nrldpc_batch_gen(b.h, 1, 0, e.ctypes.data, None, STREAM[0]),
                     lambda: rt.nrldpc_batch_count_errors(b.h, b.out.ctypes.data, b.out.ctypes.data, e.ctypes.data,
                                                          STREAM[0])):
            assert b.set_jobs(1, z) == 0
            before = rt.fake_launches()
            call()
            assert rt.fake_launches() == before + 1 and rt.fake_early_launches() == 0
    d.close()
    b.close()


@pytest.mark.parametrize("bg,z", [(1, [384] * 400), ([1, 2] * 5, [2, 7, 16, 40, 64, 128, 208, 256, 320, 384])])
def test_list_that_could_not_be_loaded_is_not_run(rt, bg, z):
    for after in range(8):  # the allocation that fails
        b = List(rt)
        assert b.set_jobs(1, [384] * 2) == 0 and b.decode(STREAM[0])
        rt.fake_fail_malloc(after)
        rc = b.set_jobs(bg, z)
        rt.fake_fail_malloc(-1)
        before = rt.fake_launches()
        b.decode(STREAM[0])
        assert rt.fake_launches() == (before if rc else before + 1)
        assert b.set_jobs(1, [384] * 2) == 0 and b.decode(STREAM[0])
        b.close()
        if rc == 0:
            break
    assert rc == 0 and after > 0


# BG1 Z=384, 40 codewords: alone on clusters, beside others on decode_kernel


def test_busy_neighbours_are_counted_per_device(rt):
    far = [Handle(rt, device=1) for _ in range(3)]
    d = Handle(rt)
    for k, f in enumerate(far):
        f.decode(40, STREAM[k])
        rt.fake_stream_busy(STREAM[k], 1)
    records = rt.fake_records()
    assert d.decode(40, STREAM[3])  # no neighbour on its own device
    assert rt.fake_records() == records  # nor anything to note for one
    near = [Handle(rt) for _ in range(2)]
    for k, f in enumerate(near):
        f.decode(40, STREAM[4 + k])
        rt.fake_stream_busy(STREAM[4 + k], 1)
    assert not d.decode(40, STREAM[3])
    for h in (*far, *near, d):
        h.close()


def test_staged_host_calls_are_busy_neighbours(rt):
    small, big = Handle(rt), [Handle(rt, n=3000) for _ in range(2)]
    assert small.decode(40, STREAM[0])
    for k, h in enumerate(big):
        h.decode_host_q(3000, STREAM[1 + k])
        rt.fake_stream_busy(STREAM[1 + k], 1)
    assert not small.decode(40, STREAM[0])
    for h in (small, *big):
        h.close()


def test_lone_caller_is_back_on_clusters_after_a_burst(rt):
    hs = [Handle(rt) for _ in range(6)]
    for k, h in enumerate(hs):
        h.decode(40, STREAM[k])
        rt.fake_stream_busy(STREAM[k], 1)
    assert not hs[0].decode(40, 0x700)
    for s in STREAM:
        rt.fake_stream_busy(s, 0)
    hs[0].decode(40, STREAM[0])
    assert hs[0].decode(40, STREAM[0])
    for h in hs:
        h.close()


def test_captured_calls_presume_the_other_decoders_beside_them(rt):
    # what runs beside a replay is not known when the call is captured
    hs = [Handle(rt)]
    rt.fake_stream_capturing(STREAM[0], 1)
    assert hs[0].decode(40, STREAM[0])  # the only decoder
    hs += [Handle(rt) for _ in range(5)]
    assert not hs[0].decode(40, STREAM[0])
    lists = List(rt)
    assert lists.set_jobs(1, [384] * 40) == 0
    assert not lists.decode(STREAM[0])
    for h, close in ((hs[0], rt.nrldpc_set_neighbours), (lists, rt.nrldpc_batch_set_neighbours)):
        assert close(h.h, 0) == 0  # the caller knows better
    assert hs[0].decode(40, STREAM[0]) and lists.decode(STREAM[0])
    rt.fake_stream_capturing(STREAM[0], 0)
    assert rt.nrldpc_set_neighbours(hs[0].h, 5) == 0 and not hs[0].decode(40, STREAM[0])
    assert rt.nrldpc_set_neighbours(hs[0].h, -1) == 0 and hs[0].decode(40, STREAM[0])
    assert rt.nrldpc_set_neighbours(hs[0].h, -2) == -1  # NRLDPC_ERR_INVALID_ARG
    lists.close()
    for h in hs:
        h.close()


def test_error_of_the_caller_survives_a_decode(rt):
    hs = [Handle(rt) for _ in range(6)]
    for k, h in enumerate(hs):
        h.decode(40, STREAM[k])
        rt.fake_stream_busy(STREAM[k], 1)
    rt.fake_set_error(1)  # cudaErrorInvalidValue of an earlier call
    hs[0].decode(40, 0x700)
    assert rt.fake_peek_error() == 1
    rt.fake_set_error(0)
    hs[0].decode(40, 0x700)
    assert rt.fake_peek_error() == 0  # and none of the decoder's own
    for h in hs:
        h.close()


def test_job_lists_of_new_codes_allocate_nothing(rt):
    b = List(rt)
    assert b.set_jobs(1, [384] * 152) == 0  # the check-node state of a full round
    before = rt.fake_mallocs(), rt.fake_frees()
    for z in ([2], [40] * 20, [64, 128, 208, 352], [7, 13, 36, 72, 144, 288, 384] * 3):
        for bg in (1, 2):
            assert b.set_jobs(bg, z) == 0
            b.decode(None)
    assert (rt.fake_mallocs(), rt.fake_frees()) == before
    b.close()


@pytest.mark.parametrize("bg,z", [(1, 384), (2, 208), (1, 96), (2, 40)])
def test_handles_hold_the_cluster_sizes_that_they_can_pick(rt, bg, z):
    def upload(n):
        before = rt.fake_uploaded()
        h = Handle(rt, bg, z, n)
        return h, rt.fake_uploaded() - before
    big, most = upload(400)
    small, least = upload(1)
    assert least < most
    small.close()
    for n in (1, 2, 7, 8, 20, 36, 60, 100, 152, 300):  # the same choice whatever the largest batch
        picked = big.decode(n, None), rt.fake_last_cluster()
        h, _ = upload(n)
        assert (h.decode(n, None), rt.fake_last_cluster()) == picked
        h.close()
    big.close()


@pytest.mark.parametrize("offset,launches", [(0, 2), (1 << 16, 1)])  # in place; apart
def test_block_taken_apart_in_place_is_checked_first(rt, offset, launches):
    info = _lib.SegmentInfoC(C=1, L=24, k_prime=1029)
    buf, rem = np.zeros(1 << 17, np.uint8), np.zeros(1, np.uint32)
    at = buf.ctypes.data
    assert rt.nrldpc_cb_desegment(at, 256, C.byref(info), at + offset, rem.ctypes.data, None) == 0
    assert rt.fake_launches() == launches


def test_decoder_that_waits_for_its_stream_does_not_hold_up_others(rt):
    a, b = Handle(rt), Handle(rt)
    rt.fake_stream_full(STREAM[0])
    t = threading.Thread(target=a.decode, args=(40, STREAM[0]))
    t.start()
    while not rt.fake_blocked():
        time.sleep(0.001)
    b.decode(40, STREAM[1])
    assert rt.fake_blocked() == 1  # the first call still waits
    rt.fake_stream_full(None)
    t.join()
    a.close()
    b.close()


def test_handle_destroyed_while_the_program_exits(rt, tmp_path):
    # by a static object older than the library, so after the library's own
    src = tmp_path / "late.cpp"
    src.write_text("""
#include <dlfcn.h>
#include "nr_gpu_ldpc_gb300.h"
static int (*destroy)(nrldpc_handle*);
struct Late { nrldpc_handle* h[3] = {}; ~Late() { for (auto* x : h) destroy(x); } } late;
int main(int, char** argv) {
    void* so = dlopen(argv[1], RTLD_NOW);
    auto init = reinterpret_cast<int (*)(const nrldpc_config*, nrldpc_handle**)>(dlsym(so, "nrldpc_init"));
    destroy = reinterpret_cast<int (*)(nrldpc_handle*)>(dlsym(so, "nrldpc_destroy"));
    nrldpc_config c{1, 64, 4, 0.75f, 0, 0};
    for (auto& x : late.h) if (init(&c, &x)) return 2;
    return 0;
}
""")
    exe = str(tmp_path / "late")
    subprocess.run(["g++", "-std=c++17", str(src), "-I", os.path.join(HERE, "..", "include"), "-ldl", "-o", exe],
                   check=True, capture_output=True, text=True)
    junk = {"MALLOC_PERTURB_": "165", "GLIBC_TUNABLES": "glibc.malloc.tcache_count=0"}  # in freed memory
    assert subprocess.run([exe, rt._name], env={**os.environ, **junk}, timeout=60).returncode == 0
