"""The status word's host side (status_begin / status_end in runtime.cpp) compiled with a pretend stream:
a call never reports what an earlier call's kernel left behind, also when that call returned early with
its kernels still queued, and a failing call is always reported, its own code once."""
import ctypes as ct
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HOST = r"""
#include <functional>
#include <vector>
typedef int cudaStream_t;
enum { cudaMemcpyDeviceToHost };
static std::vector<std::function<void()>> queue;  // one stream's pending work
static int copies = 0;
static void drain() { for (auto& f : queue) f(); queue.clear(); }
static void cudaMemsetAsync(int* p, int v, size_t, cudaStream_t) { ++copies; queue.push_back([=] { *p = v; }); }
static void cudaMemcpy(int* d, const int* s, size_t, int) { ++copies; drain(); *d = *s; }
static int dev_word = 0, host_word = 0;
struct Runtime {
    int* d_status = &dev_word;
    int* h_status = &host_word;
    bool status_clean = true, status_open = false, status_ordered = false, async_seen = false;
};
static Runtime& runtime() { static Runtime r; return r; }
static void record(int code) { if (dev_word == 0) { dev_word = code; host_word = code; } }  // record_status
"""
DRIVER = r"""
extern "C" {
void begin(int sync) { status_begin(0, sync != 0); }
void kernel(int code) { queue.push_back([=] { if (code) record(code); }); }
int end() { drain(); return status_end(); }
void reset() { queue.clear(); dev_word = host_word = 0; copies = 0; runtime() = Runtime(); }
int stream_ops() { return copies; }
}
"""


@pytest.fixture(scope="module")
def S(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host C++ compiler")
    with open(os.path.join(ROOT, "blaze_gb300", "csrc", "runtime.cpp")) as f:
        src = f.read()
    body = src[src.index("void status_begin("):src.index("std::atomic<int64_t> g_pool_bytes")]
    d = tmp_path_factory.mktemp("status")
    (d / "s.cpp").write_text(HOST + body + DRIVER)
    subprocess.run([gxx, "-std=c++17", "-shared", "-fPIC", "-o", str(d / "s.so"), str(d / "s.cpp")], check=True)
    return ct.CDLL(str(d / "s.so"))


def _call(S, *codes, sync=1, abandon=False):
    S.begin(sync)
    for c in codes:
        S.kernel(c)
    return None if abandon or not sync else S.end()


def test_good_calls_cost_the_stream_nothing(S):
    S.reset()
    assert [_call(S, 0, 0) for _ in range(4)] == [0] * 4 and S.stream_ops() == 0


def test_a_failing_call_is_reported_once(S):
    S.reset()
    assert [_call(S, 0), _call(S, 3, 4), _call(S, 0), _call(S, 0)] == [0, 3, 0, 0]


@pytest.mark.parametrize("left_behind", [(), (0,), (5,), (5, 6)])
def test_an_abandoned_call_is_not_reported_by_the_next(S, left_behind):
    S.reset()
    assert _call(S, 0) == 0
    _call(S, *left_behind, abandon=True)  # returned early, its kernels still queued
    assert _call(S, 0) == 0
    assert _call(S, 0) == 0
    _call(S, *left_behind, abandon=True)
    assert _call(S, 7) == 7
    assert _call(S, 0) == 0


def test_calls_after_an_asynchronous_one(S):
    S.reset()
    _call(S, 9, sync=0)
    assert [_call(S, 0), _call(S, 2), _call(S, 0)] == [0, 2, 0]
