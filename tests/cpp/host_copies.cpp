// Reads grids of a 128^3 handle into fresh host pages while this program's own pthread_create counts
// the threads that a copy starts: no more than the CPUs that the caller may run on, itself among them,
// and the values that were set whatever their number.  Prints "ok" and exits 0 when all hold.
#include <dlfcn.h>
#include <pthread.h>
#include <sched.h>
#include <sys/mman.h>

#include <atomic>
#include <cstdio>
#include <cstring>
#include <vector>

#include "ariel.h"

static std::atomic<int> g_started{0};

extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg) {
    using Fn = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
    static const Fn next = (Fn)dlsym(RTLD_NEXT, "pthread_create");
    ++g_started;
    return next(t, a, f, arg);
}

static ariel_sim* g_sim;

// The grid into fresh pages; the status, and whether it is `want`.
static ariel_status read_grid(int which, const void* want, size_t bytes, bool* same) {
    void* p = mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (p == MAP_FAILED) return ARIEL_ERR_OOM;
    const ariel_status st = ariel_get_grid(g_sim, 0, which, p, (int64_t)bytes);
    *same = std::memcmp(p, want, bytes) == 0;
    munmap(p, bytes);
    return st;
}

int main() {
    const int n = 128;
    const size_t cells = (size_t)n * n * n;
    AsimSceneDesc d;
    AsimParams prm;
    ariel_scene_dambreak(&d, n);
    d.n_liquid = 0;
    ariel_params_default(&prm);
    std::vector<double> p64(cells);
    std::vector<int32_t> a(cells);
    for (size_t i = 0; i < cells; ++i) {
        p64[i] = 0.25 * (double)i;
        a[i] = (int32_t)(i % 3);
    }
    if (ariel_create(&d, &prm, &g_sim) != ARIEL_OK || ariel_init(g_sim) != ARIEL_OK ||
        ariel_set_grid(g_sim, 0, ARIEL_GRID_P64, p64.data(), (int64_t)(8 * cells)) != ARIEL_OK ||
        ariel_set_grid(g_sim, 0, ARIEL_GRID_A, a.data(), (int64_t)(4 * cells)) != ARIEL_OK)
        return 2;
    struct {
        int which;
        const void* want;
        size_t bytes;
    } grids[] = {{ARIEL_GRID_P64, p64.data(), 8 * cells}, {ARIEL_GRID_A, a.data(), 4 * cells}};
    bool same = false;
    for (const auto& g : grids)
        if (read_grid(g.which, g.want, g.bytes, &same) != ARIEL_OK || !same) return 3;

    cpu_set_t all;
    if (sched_getaffinity(0, sizeof(all), &all) != 0) return 4;
    for (int cpus = 1; cpus <= 3; ++cpus) {
        cpu_set_t some;
        CPU_ZERO(&some);
        for (int c = 0; c < CPU_SETSIZE && CPU_COUNT(&some) < cpus; ++c)
            if (CPU_ISSET(c, &all)) CPU_SET(c, &some);
        if (CPU_COUNT(&some) < cpus) break;
        if (sched_setaffinity(0, sizeof(some), &some) != 0) return 5;
        for (const auto& g : grids) {
            // a copy of cell types maps the pages of two buffers in turn
            const int turns = g.which == ARIEL_GRID_A ? 2 : 1;
            g_started = 0;
            if (read_grid(g.which, g.want, g.bytes, &same) != ARIEL_OK || !same || g_started > turns * (cpus - 1)) {
                std::printf("grid %d on %d CPUs: %d threads started, values %s\n", g.which, cpus, g_started.load(),
                            same ? "right" : "wrong");
                return 1;
            }
        }
    }
    ariel_destroy(g_sim);
    std::printf("ok\n");
    return 0;
}
