"""The process's pool of query stagings (session_query.cpp) against a CUDA runtime whose calls fail on
demand, on the CPU; and sessions of several threads that call at once, on the GPU."""
import os
import subprocess
import threading

import numpy as np
import pytest

import pathed
from _util import seeded_rays

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

DRIVER = r"""
#include "session_query.cpp"

#include <cstdio>
#include <cstdlib>

static int g_host = 0, g_dev = 0, g_streams = 0, g_stream_calls = 0, g_fail_stream = -1;
extern "C" {
cudaError_t cudaMallocHost(void** p, size_t n) { *p = std::malloc(n); g_host++; return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); g_host--; return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = std::malloc(n); g_dev++; return cudaSuccess; }
cudaError_t cudaFree(void* p) { std::free(p); g_dev--; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    if (g_stream_calls++ == g_fail_stream) return cudaErrorMemoryAllocation;
    *s = reinterpret_cast<cudaStream_t>(std::malloc(1));
    g_streams++;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { std::free(s); g_streams--; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
}

#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
using namespace pt;

int main() {
    QueryPool& pool = QueryPool::get();
    const size_t each = chunk_bytes(kChunkRays);
    {  // a stream that cannot be made leaves no null stream behind
        QueryStaging s(0);
        g_fail_stream = 2;
        CHECK(s.ensure(4, 256) != cudaSuccess);
        for (cudaStream_t st : s.streams) CHECK(st != nullptr);
        CHECK(s.ensure(4, 256) == cudaSuccess);
        CHECK(s.streams.size() == 4);
        for (cudaStream_t st : s.streams) CHECK(st != nullptr);
    }
    CHECK(g_host == 0 && g_dev == 0 && g_streams == 0);
    auto filled = [&](int device, size_t bytes) {
        std::unique_ptr<QueryStaging> s = pool.take(device);
        s->ensure(1, bytes);
        return s;
    };
    // no session: nothing is kept
    pool.give(filled(0, 256));
    CHECK(g_host == 0);
    // each device keeps its own, as many as the pool allows
    pool.attach(0);
    pool.attach(0);
    pool.attach(1);
    std::vector<std::unique_ptr<QueryStaging>> out;
    for (int k = 0; k < kQueryStagings + 1; k++) out.push_back(filled(0, each));
    out.push_back(filled(1, each));
    for (auto& s : out) pool.give(std::move(s));
    CHECK(g_host == kQueryStagings + 1);
    QueryStaging* one = nullptr;
    {
        std::unique_ptr<QueryStaging> s = pool.take(1);
        CHECK(s->device == 1 && s->host_bytes == each);
        one = s.get();
        pool.give(std::move(s));
        CHECK(pool.take(1).get() == one);  // freed here
    }
    CHECK(g_host == kQueryStagings);
    // a staging larger than the pool's bound is not kept
    pool.give(filled(1, kQueryWorkers * each + 256));
    CHECK(g_host == kQueryStagings);
    pool.give(filled(1, kQueryWorkers * each));
    CHECK(g_host == kQueryStagings + 1);
    // the last session of a device frees that device's, and no other's
    pool.detach(0);
    CHECK(g_host == kQueryStagings + 1);
    pool.detach(0);
    CHECK(g_host == 1);
    CHECK(pool.take(1)->host_bytes == kQueryWorkers * each);
    pool.detach(1);
    CHECK(g_host == 0 && g_dev == 0 && g_streams == 0);
    std::printf("ok\n");
    return 0;
}
"""


def test_pool_against_failing_calls(tmp_path):
    src, exe = tmp_path / "pool.cpp", tmp_path / "pool"
    src.write_text(DRIVER)
    csrc = os.path.join(ROOT, "gpu-pathed_b200", "csrc")
    # the rest of the library is never called: its symbols stay unresolved
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", csrc, "-I", os.path.join(CUDA, "include"), str(src), "-o",
                        str(exe), "-Wl,--unresolved-symbols=ignore-all"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.stdout, r.stderr)


@pytest.mark.gpu
def test_sessions_of_several_threads_call_at_once():
    """Sessions made, called and closed by four threads at once, of sizes that take every route, give the hits
    of the same calls made one after the other."""
    sizes = [1, 3000, 20000, 70001, 150000]
    jobs, errors = {}, []
    s = pathed.Session(32, 32)
    s.load_config(0)
    sc = s.export_scene()
    for n in sizes:
        o, d, tmin, tmax = (a[:n] for a in seeded_rays(sc, n + 2, seed=n))
        jobs[n] = (o, d, tmin, tmax, s.trace_rays(o, d, tmin, tmax, with_bary=True), s.occluded(o, d, tmin, tmax))
    s.close()

    def work(k):
        try:
            for rep in range(3):
                t = pathed.Session(32, 32)
                t.load_config(0)
                for j in range(len(sizes)):
                    o, d, tmin, tmax, ref, occ = jobs[sizes[(j + k) % len(sizes)]]
                    got = t.trace_rays(o, d, tmin, tmax, with_bary=True)
                    for key in ref:
                        assert np.array_equal(got[key], ref[key]), key
                    assert np.array_equal(t.occluded(o, d, tmin, tmax), occ)
                t.close()
        except Exception as e:  # noqa: BLE001 (reported by the test)
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
