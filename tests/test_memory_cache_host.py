"""The cache of destroyed contexts' memory (csrc/cp_pool.cuh) on the CPU, over a
fake of the CUDA calls that it makes: a device of 1000 MB that counts its blocks,
and a current context that the test switches."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

FAKE = r'''
#include <cstdio>
#include <cstdlib>
#include <map>
#include "cp_pool.cuh"

static size_t used = 0, calls = 0;
static const size_t capacity = size_t(1000) << 20;
static unsigned long long context = 1;
static std::map<void*, size_t> live;
static char* next_address = reinterpret_cast<char*>(1 << 20);

static cudaError_t last = cudaSuccess;
static cudaError_t fake_alloc(void** p, size_t bytes) {
    ++calls;
    if (used + bytes > capacity) return last = cudaErrorMemoryAllocation;
    *p = next_address;
    next_address += bytes;
    live[*p] = bytes;
    used += bytes;
    return cudaSuccess;
}
static cudaError_t fake_free(void* p) {
    if (!p) return cudaSuccess;
    if (!live.count(p)) { printf("free of an unknown block\n"); exit(2); }
    used -= live[p];
    live.erase(p);
    return cudaSuccess;
}
static CUresult current(CUcontext* c) { *c = reinterpret_cast<CUcontext>(context); return CUDA_SUCCESS; }
static CUresult id(CUcontext, unsigned long long* out) { *out = context; return CUDA_SUCCESS; }
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { return fake_alloc(p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) { return fake_alloc(p, n); }
cudaError_t cudaFree(void* p) { return fake_free(p); }
cudaError_t cudaFreeHost(void* p) { return fake_free(p); }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaGetDriverEntryPoint(const char* name, void** f, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    *f = name[5] == 'G' && name[8] == 'C' ? reinterpret_cast<void*>(current) : reinterpret_cast<void*>(id);
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
}

#define CHECK(c) do { if (!(c)) { printf("line %d: %s (used %zu MB, %zu calls)\n", __LINE__, #c, used >> 20, calls); return 1; } } while (0)
static const size_t MB = size_t(1) << 20;

// an object of one array of mb MB (at least 16: a block of its own)
static cudaError_t take(cp::Arena& a, size_t mb) { void* p; return a.take(mb * MB, &p); }

int main(int argc, char** argv) {
    const std::string what = argv[1];
    cp::BlockCache& cache = cp::device_cache();
    if (what == "reuse") {
        cp::Arena a, b;
        void* p = nullptr;
        CHECK(take(a, 100) == cudaSuccess && a.take(1000, &p) == cudaSuccess && a.take(1000, &p) == cudaSuccess);
        const size_t before = calls, held = used;
        CHECK(before == 2);                       // the small ones share a block
        a.give_back();
        CHECK(used == held);
        CHECK(take(b, 90) == cudaSuccess && b.take(5000, &p) == cudaSuccess);
        CHECK(calls == before);                   // both from the cache
        cp::Arena c;
        CHECK(take(c, 50) == cudaSuccess && calls == before + 1);
        CHECK(take(c, 90) == cudaSuccess && calls == before + 2);   // the cached one is taken
    } else if (what == "bound") {
        cache.set_limit(250 * MB);
        for (int n = 0; n < 5; ++n) {
            cp::Arena a[3];
            for (auto& x : a) CHECK(take(x, 100 + 20 * n) == cudaSuccess);
            for (auto& x : a) x.give_back();
            CHECK(used <= 250 * MB && used > 0);
        }
        cache.set_limit(0);
        CHECK(used == 0);
        cp::Arena a;
        CHECK(take(a, 100) == cudaSuccess);
        a.give_back();
        CHECK(used == 0);                         // no cache at all
    } else if (what == "retry") {
        cp::Arena a, b, c;
        CHECK(take(a, 400) == cudaSuccess && take(b, 400) == cudaSuccess);
        a.give_back();
        b.give_back();
        CHECK(used == 800 * MB);
        CHECK(take(c, 900) == cudaSuccess);       // does not fit beside the cache
        CHECK(used == 900 * MB);
        cp::Arena d;
        CHECK(take(d, 200) == cudaErrorMemoryAllocation);
        CHECK(used == 900 * MB);
        CHECK(cudaGetLastError() == cudaSuccess);   // nothing left for the next launch's check
    } else if (what == "context") {
        cp::Arena a, b;
        CHECK(take(a, 100) == cudaSuccess);
        a.give_back();
        context = 2;
        const size_t before = calls;
        CHECK(take(b, 100) == cudaSuccess && calls == before + 1);   // not the other context's
        cache.release_all();
        CHECK(used == 200 * MB);                  // nor is it freed from here
        context = 1;
        cache.release_all();
        CHECK(used == 100 * MB);
        b.give_back();                            // its context is not the current one: freed, not kept
        CHECK(used == 0);
    }
    printf("ok\n");
    return 0;
}
'''


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    d = tmp_path_factory.mktemp("pool")
    src = d / "fake.cpp"
    src.write_text("#include <string>\n" + FAKE)
    exe = d / "fake"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", os.path.join(ROOT, "coldplate-solver_b200", "csrc"), "-I",
                    os.path.join(CUDA, "include"), str(src), "-o", str(exe), "-lpthread"], check=True)
    return exe


@pytest.mark.parametrize("what", ["reuse", "bound", "retry", "context"])
def test_cache(fake, what):
    r = subprocess.run([str(fake), what], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr


def test_every_allocation_goes_through_the_cache():
    """No device or pinned memory is allocated past it: an allocation that fails
    gives the cache back first."""
    csrc = os.path.join(ROOT, "coldplate-solver_b200", "csrc")
    for name in sorted(os.listdir(csrc)):
        if name == "cp_pool.cuh":
            continue
        for n, line in enumerate(open(os.path.join(csrc, name)), 1):
            code = line.split("//")[0]
            assert "cudaMallocHost(" not in code and "cudaHostAlloc(" not in code, f"{name}:{n}"
            assert "cudaMalloc(" not in code, f"{name}:{n}"
