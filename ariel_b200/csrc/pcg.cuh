// pcg.cuh -- pressure-solve data shared by pcg.cu and host.cu.
#pragma once

#include <algorithm>

#include "state.cuh"

namespace ariel {

enum PcgMode { kRef32 = 0, kFp64 = 1, kMixed = 2 };

// Per-scene solver scalars, written by the leader block of each grid barrier.
struct PcgScene {
    double bb;        // |b|^2 over FLUID cells
    double rr;        // r.r of the working (inner) residual
    double rho;       // z.r
    double alpha, beta;
    double rr_out;    // |b - A x|^2 at the last outer residual (FP64/MIXED true residual)
    double target;    // stop threshold on rr of the current (inner) solve
    float alpha32, beta32, rho32, pad32;
    int iters;        // CG iterations (summed over inner solves)
    int outer;        // refinement sweeps
    int done;         // whole solve finished
    int inner_done;   // current inner solve finished
    int converged;
    int ordered;      // preconditioner needs the ordered (wavefront) path
    int ones;         // FLUID cells whose order-free REF preconditioner value is exactly 1
    int nf;           // FLUID cells
    int csize;        // this scene's chunk size (FLUID cells per chunk)
    int pad;
};
static_assert(sizeof(PcgScene) % 16 == 0, "PcgScene is copied as 16-byte words");

// Accumulated over solves (reset by the host); written by the leader when a scene finishes.
struct PcgTotals {
    long long solves, iterations, outer;
    double cell_iterations, cell_outer;
    long long not_converged, pad;
};

struct PcgCtl {
    int all_done;
    int all_inner_done;
    int any_ordered;
    int nvirt[5];  // block positions of the resident solve's classes (whole groups of gridDim.x)
    int nstream;   // scenes left to the streaming kernel
    int pad[3];
};

struct Barrier {
    unsigned count;
    unsigned gen;
    int error;
    unsigned beat;  // exchanges completed by the resident solve (its waits' sign of progress)
};

struct PcgArgs {
    DevState S;
    int mode;
    int fast;            // k_pcg_fast handles launches without an ordered preconditioner
    int may_be_ordered;  // the general kernel must also be launched (see launch_pcg_solve)
    int precond;
    int stop_rule;
    int max_iters;     // <=0: n^3 per scene
    int max_outer;
    double tol;
    double inner_tol;
    double tau, sigma;
    unsigned long long timeout_ns;
    // FLUID list
    const uint32_t* fl;        // packed FLUID cells, scene by scene, in list_order
    uint4* rec;                // per FLUID-list entry: (cell, neighbour mask, diagonal bits)
    const long long* fl_pref;  // k+1
    const long long* ch_pref;  // k+1 chunk begins (scenes of the resident solve have none)
    uint32_t* hlist;           // resident solve, largest class: halo positions, 6 per FLUID-list entry
    const uint32_t* flscan;    // packed cell in list_order -> FLUID-list position
    // resident solve: per scene (first block position, positions, chunks, first partial), or
    // position kNotResident; one arrival counter per scene, 128 bytes apart, with a word that a
    // block sets when its halo does not fit
    int4* res;
    unsigned* res_count;
    int res_blocks;            // its blocks (one per SM)
    int all_resident;          // every scene fits the resident solve whatever its FLUID cells are
    int classes;               // bit c: some scene may be of class c (res_class_mask)
    // per-cell operator data (dense over packed cells)
    uint8_t* mask;   // bit d set: neighbour d (-x,+x,-y,+y,-z,+z) is FLUID
    double* diag;    // ADiag (fp32 value for REF32, fp64 otherwise)
    double* pc64;    // preconditioner values
    float* pc32;
    // vectors (dense over packed cells); element type per mode
    void* r;
    void* z;
    void* s0;
    void* s1;
    void* q;
    void* ordq;      // forward-sweep scratch of the ordered preconditioner
    void* u;         // single-reduction PCG: preconditioned residual
    void* p;         // single-reduction PCG: search direction
    void* va0;       // fast single-reduction PCG: packed (r, w, s, pc), two parities
    void* va1;
    void* vb;        // fast single-reduction PCG: packed (p, x)
    double* r64;     // MIXED outer residual
    float* d32;      // MIXED inner correction
    double* partial; // two sets of 3 * max chunks (three dot products per reduction)
    long long max_chunks;
    // ordered wavefront sweeps: bricks of every scene sorted by level I+J+K (then scene, I, J,
    // K), each scene's brick grid starting at brick_base[s], one progress flag per brick
    const int4* bricks;
    const int* brick_base;
    unsigned* bflag;
    int nbricks;
    int bx, by, bz;
    PcgScene* sc;
    PcgTotals* totals;
    PcgCtl* ctl;
    Barrier* bar;
};

// Build the FLUID list, per-cell operator data and chunk table; zero non-FLUID pressure.
cudaError_t launch_pcg_prepare(const PcgArgs& A, uint32_t* pred, uint32_t* scan, void* scan_tmp, cudaStream_t st);
// The cooperative persistent PCG kernel.
cudaError_t launch_pcg_solve(const PcgArgs& A, int nblocks, cudaStream_t st);
// Blocks of the persistent kernel that fit on the device at once; the resident solve's.
int pcg_max_blocks(int device, int mode, int per_sm_cap);
int pcg_res_blocks(int device, int mode, int classes);
// Self tests of the bounded waits (one arrival missing): err[0] for the grid barrier's, err[1] for the
// resident solve's, 1 where it gave up as it should; err[2] is theirs.
cudaError_t launch_barrier_selftest(Barrier* bar, int* err, unsigned long long timeout_ns, cudaStream_t st);

constexpr int kPcgThreads = 256;
// Chunks of the FLUID list, the unit of every reduction's partial sums.  Each scene's chunk size
// is the FLUID count split kChunkTarget ways (the persistent solve's resident blocks on a B200: 2
// per SM x 148 SMs), rounded up to a multiple of kChunkAlign and kept within [kChunkMin,
// kChunkMax]: a large scene then gives every resident block one chunk and every SM about the same
// number of cells (with power-of-two sizes a 128^3 dam break left 79 SMs with twice the cells of
// the others), a small one still spreads over as many blocks as 512-cell chunks allow, and a huge
// one keeps chunks that fit the shared-memory record cache.  The size depends on the scene alone,
// so a scene's bits do not depend on the batch it is solved in or on the grid.
constexpr int kChunkMin = 512;
constexpr int kChunkMax = 2048;
constexpr int kChunkAlign = 64;
constexpr long long kChunkTarget = 296;
__host__ __device__ inline int chunk_size(long long nf) {
    long long c = (nf + kChunkTarget - 1) / kChunkTarget;
    c = (c + kChunkAlign - 1) / kChunkAlign * kChunkAlign;
    return (int)(c < kChunkMin ? kChunkMin : (c > kChunkMax ? kChunkMax : c));
}
// Most chunks a scene of `cells` cells can have (its FLUID count is at most `cells`).
inline long long chunk_bound(long long cells) {
    const long long lo = (cells + kChunkMin - 1) / kChunkMin;
    const long long hi = (cells + kChunkMax - 1) / kChunkMax;
    return std::min(lo, std::max(kChunkTarget, hi));
}
// Whether a counter of arrivals has come to `want`.  Both wrap around in a solve of more than 2^32 arrivals
// (a tolerance out of reach, n^3 iterations, 296 blocks: from 245^3 on); they are never 2^31 apart.
__host__ __device__ constexpr bool arrived(unsigned count, unsigned want) { return count - want < 0x80000000u; }
static_assert(arrived(5u, 5u) && arrived(6u, 5u) && !arrived(4u, 5u), "plain counts");
static_assert(arrived(3u, 0xfffffff0u) && !arrived(0xfffffff0u, 3u), "counts on both sides of 2^32");
// The resident solve: scenes of one chunk or more per block (one block per SM) whose cells fit its
// shared memory together with slots for neighbours in other blocks.
constexpr int kResMaxChunks = 320;   // what the reduction of a scene's partials reads in one go:
constexpr int kResBigChunks = 608;   // up to two full-size chunks per block, and up to four
constexpr int kResMaxScenes = 128;   // as the streaming fast kernel
constexpr size_t kResSmem = 225 * 1024;  // all of an SM's but 2 KB for the static part
// Slots for neighbours in other blocks beside a block's `cells` cells (positions fit 14 bits).
__host__ __device__ constexpr int res_halo_slots(int mode, int cells, bool big) {
    const long long tb = mode == kFp64 ? 8 : 4;
    const long long left = ((long long)kResSmem - 64 - cells * ((big ? 3 : 5) * tb + 12)) / (tb + (big ? 0 : 4));
    const long long most = 16380 - cells;
    return (int)(left < most ? left : most);
}
// Classes of resident scenes, one kernel each, by the rounds of one cell per thread that a chunk
// takes and the chunks of a half block: a scene alone spreads over as many SMs as it can (one
// chunk per half); with other scenes small chunks share a block, up to 4,096 cells, so that all
// scenes iterate side by side (six 32^3-64^3 scenes: one group of blocks instead of four one
// after another).  The last class takes scenes of more than two full-size chunks per SM, up to four
// (MIXED): 0.6-1.2 M FLUID cells, whose (p, x) no longer fit beside the rest.
constexpr int kNotResident = -(1 << 30);
constexpr int kResClasses = 5;
constexpr int kResBig = 4;
__host__ __device__ constexpr int res_rounds(int c) { return c == 0 || c == 1 ? 2 : (c == 2 ? 4 : 8); }
__host__ __device__ constexpr int res_chunks(int c) { return c == 1 ? 4 : (c == 2 || c == kResBig ? 2 : 1); }
__host__ __device__ constexpr int res_class(int scenes, int csize, int chunks) {
    return chunks > kChunkTarget ? kResBig
           : csize <= 512        ? (scenes == 1 ? 0 : 1)
                                 : (csize <= 1024 && scenes > 1 ? 2 : 3);
}
// Whether any cells of a chunk of this class find a slot for each neighbour (at most six).
__host__ __device__ constexpr bool res_never_over(int mode, int csize, int cpb) {
    return cpb > 0 && res_halo_slots(mode, cpb * csize, false) >= 6 * cpb * csize;
}
// Slots enough for the usual halo: about 0.6 neighbours in other blocks per cell, or in the grid
// order of the FP64 list 2.1.
__host__ __device__ constexpr bool res_fits(int mode, int cells, bool big) {
    return 10 * res_halo_slots(mode, cells, big) >= (mode == kFp64 ? 21 : 8) * cells;
}
// Most chunks of `csize` cells that a block takes of a scene of `chunks` (0: none fits).
__host__ __device__ constexpr int res_max_cpb(int mode, int scenes, int csize, int chunks) {
    const int cls = res_class(scenes, csize, chunks);
    if (cls == kResBig && mode != kMixed) return 0;
    int c = 2 * res_chunks(cls);
    while (c > 0 && !res_fits(mode, c * csize, cls == kResBig)) c >>= 1;
    return c;
}
// The classes (bit c: class c) that a scene on a grid of `cells` cells may be of, over the FLUID
// counts that the grid allows: what a handle loads and launches.  A kernel that no scene of the
// handle can reach is not looked at, since the first look loads it (a process's first handle, MIXED:
// 32^3 6.7 -> 5.8 ms, 64^3 12.5 -> 11.9).  FP64 scenes are resident only alone (pcg_tables).
inline int res_class_mask(int mode, int scenes, long long cells) {
    if (mode == kRef32 || (mode == kFp64 && scenes > 1)) return 0;
    const int chunks = (int)std::min(chunk_bound(cells), kChunkTarget);
    int mask = mode == kMixed && chunk_bound(cells) > kChunkTarget ? 1 << kResBig : 0;
    for (int c = kChunkMin; c <= chunk_size(cells); c += kChunkAlign)
        if (res_max_cpb(mode, scenes, c, chunks) > 0) mask |= 1 << res_class(scenes, c, chunks);
    return mask;
}
constexpr int kBrickMaxCells = 2048;
constexpr int kBrickMaxExt = 2744;
constexpr int kBrickMaxLevels = 128;
// Dynamic shared memory of the general solve kernel (the ordered wavefront sweeps' boxes).
size_t brick_dyn_smem();
bool brick_shape_ok(int bx, int by, int bz);

}  // namespace ariel
