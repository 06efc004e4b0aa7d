// The engine's host-side memory classes against a runtime of this file's own
// whose allocations fail on demand (no GPU, no CUDA library). Each check names
// what it found wrong; the exit status is the number of them.
#include <cstdio>
#include <cstdlib>
#include <set>

#include "common.cuh"

static int g_allocs_left = -1; // allocations that still succeed; -1: all
static cudaError_t g_last = cudaSuccess;
static std::set<void*> g_live;

extern "C" {
cudaError_t cudaMalloc(void** p, size_t bytes)
{
    if (g_allocs_left == 0)
        return g_last = cudaErrorMemoryAllocation;
    if (g_allocs_left > 0)
        --g_allocs_left;
    *p = std::malloc(bytes);
    g_live.insert(*p);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p)
{
    if (p && !g_live.erase(p))
        return g_last = cudaErrorInvalidValue;
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void)
{
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "stub error"; }
}

using namespace reyn;

static int failures = 0;

static void expect(bool ok, const char* what)
{
    if (!ok) {
        std::printf("FAILED: %s\n", what);
        ++failures;
    }
}

template <class F> static bool throws(F&& f)
{
    try {
        f();
    } catch (const Error&) {
        return true;
    }
    return false;
}

// an error that was thrown is not met again by the check after the next launch
static void reported_once()
{
    g_allocs_left = 0;
    DevArray<float> a;
    expect(throws([&] { a.resize(10); }), "a failed allocation throws");
    expect(!throws([] { REYN_LAUNCHED("next launch"); }), "the next launch's check is clean");
    g_allocs_left = -1;
}

// the arrays of a reorder, some of which an earlier step already holds: a call
// that runs out of memory is refused, and so is the next one, until every array
// has its memory
static void reorder_arrays()
{
    for (int ok = 0; ok < 7; ++ok) {
        std::array<DevArray<float>, 7> alt;
        DevArray<float4> pm, vel;
        Slab slab;
        pm.resize(100);
        vel.resize(100);
        g_allocs_left = ok;
        auto reserve = [&] { reserve_together(100, alt, pm, vel, slab); };
        expect(throws(reserve), "out of memory is reported");
        expect(throws(reserve), "and reported again while it lasts");
        g_allocs_left = -1;
        expect(!throws(reserve), "memory again");
        for (auto& a : alt)
            expect(a.get() != nullptr && a.size() == 100, "every array has its memory");
    }
    // fresh: one allocation for all, none kept of a failed one
    std::array<DevArray<float>, 7> alt;
    DevArray<float4> pm, vel;
    Slab slab;
    g_allocs_left = 0;
    expect(throws([&] { reserve_together(100, alt, pm, vel, slab); }), "nothing fits");
    g_allocs_left = 1;
    expect(!throws([&] { reserve_together(100, alt, pm, vel, slab); }), "one allocation");
    reserve_together(100, alt, pm, vel, slab);
    for (auto& a : alt)
        expect(a.get() != nullptr && a.size() == 100, "every array has its memory");
    expect(pm.get() && vel.get(), "the packed copies too");
    g_allocs_left = -1;
}

int main()
{
    reported_once();
    reorder_arrays();
    expect(g_live.empty(), "every allocation was freed");
    return failures;
}
