// Copies to host buffers while the n-th allocation of host memory in the call fails, n = 1, 2, ...: every
// call of this C interface returns a status, and where that is ARIEL_OK the values are right.
// Prints "ok" and exits 0 when all hold.
#include <sys/mman.h>

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <vector>

#include "ariel.h"

static std::atomic<int> g_left{0};  // the allocation to fail, 0: none

void* operator new(size_t n) {
    if (g_left.load() > 0 && --g_left == 0) throw std::bad_alloc();
    void* p = std::malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

static void* fresh(size_t bytes) {
    return mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
}

int main() {
    const int n = 80;
    const size_t cells = (size_t)n * n * n;
    AsimSceneDesc d;
    AsimParams prm;
    ariel_scene_dambreak(&d, n);
    ariel_params_default(&prm);
    ariel_sim* sim = nullptr;
    if (ariel_create(&d, &prm, &sim) != ARIEL_OK || ariel_init(sim) != ARIEL_OK) return 2;
    std::vector<double> p64(cells);
    for (size_t i = 0; i < cells; ++i) p64[i] = 0.5 * (double)i;
    std::vector<int32_t> a(cells), got_a(cells);
    int64_t m = 0;
    if (ariel_set_grid(sim, 0, ARIEL_GRID_P64, p64.data(), (int64_t)(8 * cells)) != ARIEL_OK ||
        ariel_get_grid(sim, 0, ARIEL_GRID_A, a.data(), (int64_t)(4 * cells)) != ARIEL_OK ||
        ariel_particle_count(sim, 0, &m) != ARIEL_OK)
        return 2;
    std::vector<float> pos(3 * m), mass(m);
    if (ariel_get_particles(sim, 0, pos.data(), nullptr, nullptr, mass.data(), nullptr) != ARIEL_OK) return 2;
    for (int k = 1; k <= 12; ++k) {
        double* g = (double*)fresh(8 * cells);
        float* q = (float*)fresh(16 * m);
        int32_t* f = (int32_t*)fresh(4 * cells);
        ariel_status st[3];
        try {
            g_left = k;
            st[0] = ariel_get_grid(sim, 0, ARIEL_GRID_P64, g, (int64_t)(8 * cells));
            g_left = k;
            st[1] = ariel_get_grid(sim, 0, ARIEL_GRID_A, f, (int64_t)(4 * cells));
            g_left = k;
            st[2] = ariel_get_particles(sim, 0, q, nullptr, nullptr, q + 3 * m, nullptr);
            g_left = 0;
        } catch (...) {
            std::printf("allocation %d: an exception left a C function\n", k);
            return 1;
        }
        const bool same[3] = {std::memcmp(g, p64.data(), 8 * cells) == 0, std::memcmp(f, a.data(), 4 * cells) == 0,
                              std::memcmp(q, pos.data(), 12 * m) == 0 && std::memcmp(q + 3 * m, mass.data(), 4 * m) == 0};
        for (int i = 0; i < 3; ++i)
            if (!(st[i] == ARIEL_OK ? same[i] : st[i] == ARIEL_ERR_OOM)) {
                std::printf("allocation %d, call %d: status %d, values %s\n", k, i, (int)st[i],
                            same[i] ? "right" : "wrong");
                return 1;
            }
        munmap(g, 8 * cells);
        munmap(q, 16 * m);
        munmap(f, 4 * cells);
    }
    ariel_destroy(sim);
    std::printf("ok\n");
    return 0;
}
