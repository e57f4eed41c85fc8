// rows.cu -- hit rows from one warp per grid cell, and the gather passes over them.
//
// k_cell_rows gives a warp the particles of one cell (up to a group of them).  Its lanes
// hold the candidates of the cell's 27 neighbour cells, in the reference's order (z, y, x
// ascending, each cell in sorted order: oclsph_kernel.h:155-183), a few in a row each, and
// test them all at once against each of the particles; a running sum over the lanes places
// those within range, and they go to the particle's hit row as sorted indices, in order.
// The candidates are loaded once for all particles of the group and no lane waits for
// another's longer list.
//
// The test runs on pairs of candidates in 16 bits, relative to the group's first particle,
// with a margin that covers its rounding (kHalfMargin): rows hold all that 32 bits would
// find and about 1 % more, which the passes drop.  A step's first search executes 159 warp
// instructions a particle (262 k cube; in 32 bits with a ballot for every 32 candidates it
// took 222) and is bound by the L1 data pipe (83 % at 1 M): the candidates' scattered 16-byte
// loads.  The first lambda stage (search and sums) of the 1 M dam break at steps 5, 30 and
// 100: 357, 387 and 357 us in 32 bits, 316, 328 and 319 now.
//
// Rows that last.  The step's first search keeps every candidate within h plus a skin of
// the grid positions.  Such a row holds every neighbour within h, in order, while no
// particle of the cell and no candidate have together moved further than the skin since
// (r_now <= h implies r_grid <= h + moved_a + moved_b).  The delta passes keep each cell's
// largest movement, and a later search only goes through the cells whose bound fails.  In
// a violent flow it fails nearly everywhere and the longer rows are wasted: the step before
// tells, per scene, whether they are worth keeping (RowPolicy).
//
// The passes (k_row_*) run one thread per particle over its row, two neighbours at a time,
// the neighbours' data through L1.  Every pass tests its range
// again, so the sums are those of the 27-cell walk of pbf.cu, bit for bit.
#include <algorithm>
#include <cstdint>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "fgb_internal.h"
#include "pbf_sums.cuh"

namespace fgb {
namespace {

struct RowArgs {
    const SceneDev *scenes;
    const TriDev *tris;
    Phys ph;
    uint32_t n, mbits;
    const uint32_t *keys;
    const uint2 *cells;
    const int32_t *type;
    const uint32_t *groups;      // first particle of every group, in no particular order
    const uint32_t *group_count;
    uint32_t group_mask;         // group_end's
    uint4 *hrows;                // hit rows, see row_of
    uint16_t *hcount;
    uint32_t hcap;               // entries a hit row has room for (a multiple of four)
    uint32_t none;               // the index that fills a row's last quad: the far entry past the particles
    int fetch;                   // the passes ask for their rows ahead (fetch_rows)
    uint32_t sparse;             // groups in 100 particles above which searches go by particles (0: never)
    const uint32_t *mass_range;
    uint32_t *over;              // hit rows that overflowed (null: not counted)
    const float4 *ps_grid;       // the grid positions
    uint32_t *moved;             // largest movement in a cell since then (float bits), at its first particle
    uint8_t *lasting;            // per group: its rows are the first search's, with the skin
    uint32_t *stale;             // first particles of the groups that a later search goes through
    uint32_t *stale_count;
    uint32_t *taken;             // groups that the search's warps took beyond their first
    float inv_h;
    float skin, skin_r2;         // the skin, and (h + skin)^2
    const RowPolicy *policy;     // per scene, of the step before; policy_next of this one
    RowPolicy *policy_next;
};

// A particle's hit row: its i-th four entries at [32 i].  Rows of 32 consecutive particles
// interleave.
__device__ __forceinline__ uint4 *row_of(const RowArgs &A, uint32_t a) {
    return A.hrows + (size_t)(a >> 5) * (A.hcap >> 2) * 32 + (a & 31u);
}

constexpr uint32_t kCellBlock = 128, kCellWarps = kCellBlock / 32;
constexpr uint32_t kFetchFrom = 400000;   // particles from which the passes ask for their rows ahead
constexpr uint32_t kListFrom = 100000;    // particles from which stale groups are listed first
constexpr uint32_t kQuadsTo = 24000, kQuadsToRef = 45000;  // particles below which one has four lanes
constexpr float kRowSkin = 0.1f;          // the skin of rows that last, in h
constexpr uint32_t kHeldAll = 256;        // candidates a warp holds at a time
constexpr uint32_t kList = 4;             // particles whose hits are collected before they are written
constexpr uint32_t kPitch = kHeldAll + 8;  // room to fill the last quad; the four lists in different banks

struct CellShared {
    alignas(16) uint32_t map[kHeldAll];         // sorted indices of the candidates held
    alignas(16) uint32_t hits[kList * kPitch];  // hits of four of the group's particles among them, in order
    uint4 own[32];                              // the group's particles: x, y and z twice in 16 bits, all bits if it has sums
};

// The lane's neighbour cell of the cell with Morton code m: its table index, or false
// outside the grid.  dx, dy, dz: the lane's step along each axis (-1, 0, 1).
__device__ __forceinline__ bool neighbour_cell(const SceneDev &S, uint32_t m, int dx, int dy, int dz, uint32_t &cell) {
    constexpr uint32_t kMX = 0x09249249u, kMY = kMX << 1, kMZ = kMX << 2;
    // one axis: a step of -1 adds all of its bits, +1 its lowest; carries run through the
    // other axes' bits, which are set
    auto axis = [&](uint32_t mask, int d, uint32_t ext, bool &ok) {
        const uint32_t own = m & mask;
        ok = ok && (d >= 0 || own != 0) && (d <= 0 || own < ext);
        return ((m | ~mask) + (d < 0 ? mask : d > 0 ? mask & (0u - mask) : 0u)) & mask;
    };
    bool ok = true;
    const uint32_t x = axis(kMX, dx, S.ext_code[0], ok), y = axis(kMY, dy, S.ext_code[1], ok),
                   z = axis(kMZ, dz, S.ext_code[2], ok);
    cell = S.table_base + (x | y | z);
    return ok;
}

// If `hits` has the bit: store b at shared address `to`, which moves on.  Written out so that
// both are predicated.
__device__ __forceinline__ void append_if(uint32_t hits, uint32_t bit, uint32_t b, uint32_t &to) {
    asm volatile(
        "{\n\t"
        ".reg .pred hit;\n\t"
        ".reg .b32 in;\n\t"
        "and.b32 in, %1, %2;\n\t"
        "setp.ne.u32 hit, in, 0;\n\t"
        "@hit st.shared.u32 [%0], %3;\n\t"
        "@hit add.u32 %0, %0, 4;\n\t"
        "}"
        : "+r"(to)
        : "r"(hits), "r"(bit), "r"(b)
        : "memory");
}

// Sums of the lanes up to and including this one.
__device__ __forceinline__ uint32_t running_sum(uint32_t v) {
#define FGB_ADD_FROM(d)                                            \
    asm("{\n\t.reg .pred in;\n\t.reg .b32 t;\n\t"                  \
        "shfl.sync.up.b32 t|in, %0, " #d ", 0, 0xffffffff;\n\t"    \
        "@in add.u32 %0, %0, t;\n\t}"                              \
        : "+r"(v))
    FGB_ADD_FROM(1);
    FGB_ADD_FROM(2);
    FGB_ADD_FROM(4);
    FGB_ADD_FROM(8);
    FGB_ADD_FROM(16);
#undef FGB_ADD_FROM
    return v;
}

__device__ __forceinline__ uint32_t bits_of(__half2 v) { return *reinterpret_cast<uint32_t *>(&v); }
__device__ __forceinline__ __half2 half2_of(uint32_t v) { return *reinterpret_cast<__half2 *>(&v); }

__device__ __forceinline__ void fill(uint32_t at, uint32_t b) {
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(at), "r"(b) : "memory");
}

// Whether this step's first search keeps the skin for a scene: it did in the step before
// and at least a fifth of the particles used their rows in its second search, or it did
// not for eight steps.  (The skin lengthens the rows, and so every pass, by a quarter; a
// search that a cell is spared costs as much as three passes over its rows.)
__device__ __forceinline__ RowPolicy decide(const RowPolicy &p) {
    RowPolicy n{0, 0, 0, 0};
    if (p.keep) {
        n.keep = p.asked == 0 || 5ull * p.used >= p.asked ? 1u : 0u;
    } else {
        n.without = p.without + 1;
        n.keep = n.without >= 8 ? 1u : 0u;
    }
    return n;
}

template <uint32_t P>
struct Pairs {
    static constexpr uint32_t value = P;
};

// The largest distance, in h, of a particle from the group's origin along an axis at which
// the 16-bit test holds, and the test's margin on (reach / h)^2.  Rounded to 16 bits, such a
// particle is off by at most 2^-11, a candidate in reach of it (below 3.2) by 2^-10 and their
// difference (below 2) by 2^-11: 2^-9 along an axis.  At a distance up to 1.11 the square is
// over by 2 * 2^-9 * sqrt(3) * 1.11 + 3 * 2^-18 < 0.00753, and the two roundings of the sum
// before its sign is settled add 2 * 2^-11 (it stays within 2): below 0.0086 in all.
constexpr float kHalfReach = 2.f, kHalfMargin = 0.0087f;

// Whether the step's searches go by particles: a thread builds the row of one by itself.  With
// hardly more than a particle a cell a warp that takes a cell has one particle to share its
// setup, and waits for the chain of loads to its candidates (sparse_above).  The rows carry no
// skin then: a search goes through all of them again.
__device__ __forceinline__ bool sparse(const RowArgs &A) {
    return A.sparse && 100ull * *A.group_count > (uint64_t)A.sparse * A.n;
}

// The rows of positions ps, by a thread each.
__device__ __forceinline__ void rows_by_particles(const RowArgs &A, const float4 *__restrict__ ps, float r2max) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t base = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; base < A.n; base += gridDim.x * blockDim.x) {
        const uint32_t a = base + lane;
        uint32_t found = 0;
        if (a < A.n) {
            const uint32_t key = A.keys[a], m = morton_of(key, A.mbits);
            const SceneDev &S = A.scenes[scene_of(key, A.mbits)];
            if (!(S.obstacles && A.type[a] == FGB_TYPE_OBSTACLE)) {  // no sums: an empty row
                const float4 pa = __ldg(&ps[a]);
                uint4 *row = row_of(A, a);
                uint4 quad = make_uint4(A.none, A.none, A.none, A.none);
#pragma unroll 1
                for (int dz = -1; dz <= 1; ++dz) {
                    uint2 range[9];
#pragma unroll
                    for (int k = 0; k < 9; ++k) {
                        uint32_t cell;
                        range[k] = make_uint2(0, 0);
                        if (neighbour_cell(S, m, k % 3 - 1, k / 3 - 1, dz, cell)) range[k] = __ldg(&A.cells[cell]);
                    }
#pragma unroll
                    for (int k = 0; k < 9; ++k)
                        for (uint32_t b = range[k].x; b < range[k].y; ++b) {
                            const float4 p = __ldg(&ps[b]);
                            if (!(dist2(p.x - pa.x, p.y - pa.y, p.z - pa.z) < r2max)) continue;
                            const uint32_t at = found++ & 3u;
                            if (at == 0) quad = make_uint4(b, A.none, A.none, A.none);
                            else if (at == 1) quad.y = b;
                            else if (at == 2) quad.z = b;
                            else quad.w = b;
                            if (at == 3 && found <= A.hcap) row[(found - 4) * 8] = quad;
                        }
                }
                if ((found & 3u) && found <= A.hcap) row[(found >> 2) * 32] = quad;
            }
            A.hcount[a] = found > A.hcap ? kListOverflow : (uint16_t)found;
        }
        if (A.over) {
            const unsigned full = __ballot_sync(0xffffffffu, found > A.hcap);
            if (full && lane == 0) atomicAdd(A.over, (uint32_t)__popc(full));
        }
    }
}

enum Search {
    kFirstSearch,  // the step's first one (the grid positions): all groups
    kLaterSearch,  // leaves the groups whose rows still last
    kStaleSearch,  // goes through the groups that k_stale_groups listed
};

// The groups whose rows do not last for the next search, by a thread each.
//
// Where most rows last a search comes down to this question, and a warp that asks it of one
// group at a time mostly waits.  A calm search of 1 M particles takes 34 us with this list
// and 60 without (steps of 1.43 and 1.54 ms; at step 100, where no row lasts, 2.12 and
// 2.13); 262 k 461 and 484 us a step, 110 k 271 and 276, 64 k 228 and 219, 14 k 181 and 162:
// hence kListFrom.  With the ref profile's constants hardly any row lasts (262 k 1480 and
// 1466): its searches ask as they go.  L1 lookups bound it, 54 scattered ones a group.
__global__ void __launch_bounds__(128, 8) k_stale_groups(RowArgs A, int count_use) {
    if (sparse(A)) return;
    const uint32_t groups = *A.group_count, lane = threadIdx.x & 31u;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t c0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); c0 < groups; c0 += stride) {
        const uint32_t c = c0 + lane;
        bool stale = false, lasts = false;
        uint32_t first = 0, scene = 0, own = 0;
        if (c < groups) {
            first = A.groups[c];
            lasts = A.lasting[c] != 0;
            stale = !lasts;
        }
        if (lasts || (count_use && c < groups)) {
            const uint32_t key = A.keys[first], m = morton_of(key, A.mbits);
            scene = scene_of(key, A.mbits);
            const SceneDev &S = A.scenes[scene];
            const uint32_t end = group_end(first, __ldg(&A.cells[S.table_base + m]).y, A.group_mask);
            own = end > first ? end - first : 0u;
            if (lasts) {
                uint32_t most = 0, mine = 0;
#pragma unroll 1
                for (int dz = -1; dz <= 1; ++dz) {
                    uint2 range[9];
#pragma unroll
                    for (int k = 0; k < 9; ++k) {
                        uint32_t cell;
                        range[k] = make_uint2(0, 0);
                        if (neighbour_cell(S, m, k % 3 - 1, k / 3 - 1, dz, cell)) range[k] = __ldg(&A.cells[cell]);
                    }
#pragma unroll
                    for (int k = 0; k < 9; ++k) {
                        const uint32_t moved = range[k].y > range[k].x ? __ldg(&A.moved[range[k].x]) : 0u;
                        most = max(most, moved);
                        if (k == 4 && dz == 0) mine = moved;
                    }
                }
                stale = !(__uint_as_float(mine) + __uint_as_float(most) <= A.skin);
                if (stale) A.lasting[c] = 0;
            }
        }
        const unsigned list = __ballot_sync(0xffffffffu, stale);
        if (list) {
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(A.stale_count, (uint32_t)__popc(list));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(list & lanemask_lt());
            if (stale) A.stale[at] = first;
        }
        if (count_use) {  // particles asked and those that use their rows, a scene at a time
            unsigned rest = __ballot_sync(0xffffffffu, own != 0);
            while (rest) {
                const uint32_t s0 = __shfl_sync(0xffffffffu, scene, __ffs(rest) - 1);
                const bool in = own != 0 && scene == s0;
                const uint32_t asked = __reduce_add_sync(0xffffffffu, in ? own : 0u),
                               used = __reduce_add_sync(0xffffffffu, in && !stale ? own : 0u);
                if (lane == 0) {
                    atomicAdd(&A.policy_next[s0].asked, asked);
                    if (used) atomicAdd(&A.policy_next[s0].used, used);
                }
                rest &= ~__ballot_sync(0xffffffffu, in);
            }
        }
    }
}

template <Search kSearch>
__global__ void __launch_bounds__(kCellBlock, 7)
    k_cell_rows(RowArgs A, const float4 *__restrict__ ps, float r2max, uint32_t n_scenes, int count_use) {
    constexpr bool kFirst = kSearch == kFirstSearch;
    __shared__ CellShared s_warp[kCellWarps];
    const uint32_t lane = threadIdx.x & 31u;
    CellShared &sh = s_warp[threadIdx.x >> 5];
    const uint32_t lists = (uint32_t)__cvta_generic_to_shared(sh.hits);
    const uint32_t *list = kSearch == kStaleSearch ? A.stale : A.groups;
    const uint32_t warps = gridDim.x * kCellWarps, groups = kSearch == kStaleSearch ? *A.stale_count : *A.group_count;
    if (kFirst && blockIdx.x == 0)
        for (uint32_t k = threadIdx.x; k < n_scenes; k += kCellBlock) A.policy_next[k] = decide(A.policy[k]);
    if (sparse(A)) return rows_by_particles(A, ps, r2max);  // all of them, at every search of the step
    // the lane's neighbour cell: x fastest; lanes 27 to 31 have none
    const int dz = (int)lane / 9 - 1, dy = (int)lane / 3 % 3 - 1, dx = (int)lane % 3 - 1;
    // particles of one scene that this warp asked and that used their rows
    uint32_t seen_scene = 0xffffffffu, asked = 0, used = 0;
    auto report = [&]() {
        if (lane == 0 && asked) {
            atomicAdd(&A.policy_next[seen_scene].asked, asked);
            if (used) atomicAdd(&A.policy_next[seen_scene].used, used);
        }
        asked = used = 0;
    };
    // The group after this one, asked for before this one is worked on: by turns where there are
    // few, else whichever is left, as groups' work differs with the flow (and by an order of
    // magnitude where the ref profile's fluid clumps).  By turns / by demand: 262 k ref 1.46 /
    // 1.41 ms a step, later 2.17 / 2.07; 1 M 2.05 / 2.02 and 2.09 / 2.06; for a few groups a warp
    // the counter costs a small scene 2 us a search.
    const bool by_demand = groups > 2 * warps;
    auto after = [&](uint32_t c) {
        if (!by_demand) return c + warps;
        uint32_t k = 0;
        if (lane == 0) k = atomicAdd(A.taken, 1u);
        return warps + k;  // in lane 0
    };
    uint32_t next;
    for (uint32_t c = blockIdx.x * kCellWarps + (threadIdx.x >> 5); c < groups;
         c = __shfl_sync(0xffffffffu, next, 0)) {
        next = after(c);
        const uint32_t first = list[c], key = A.keys[first], scene = scene_of(key, A.mbits);
        const SceneDev &S = A.scenes[scene];
        uint32_t cell;
        uint2 range = make_uint2(0, 0);
        if (neighbour_cell(S, morton_of(key, A.mbits), dx, dy, dz, cell) && lane < 27) range = __ldg(&A.cells[cell]);
        const uint32_t count = range.y > range.x ? range.y - range.x : 0u, from = range.x;
        const uint32_t end = group_end(first, __shfl_sync(0xffffffffu, range.y, 13), A.group_mask);
        float reach2 = r2max;
        if (kFirst) {
            const bool keep = decide(A.policy[scene]).keep != 0;
            if (keep) reach2 = A.skin_r2;
            if (lane == 0) A.lasting[c] = keep ? 1 : 0;
        } else if (kSearch == kLaterSearch) {
            const bool lasts = A.lasting[c] != 0;
            const uint32_t m = count ? __ldg(&A.moved[from]) : 0u;
            const float bound = __uint_as_float(__shfl_sync(0xffffffffu, m, 13)) +
                                __uint_as_float(__reduce_max_sync(0xffffffffu, m));
            const bool skip = lasts && bound <= A.skin;
            if (count_use) {
                if (scene != seen_scene) {
                    report();
                    seen_scene = scene;
                }
                const uint32_t group = end > first ? end - first : 0u;
                asked += group;
                if (skip) used += group;
            }
            if (skip) continue;
            if (lasts && lane == 0) A.lasting[c] = 0;
        }
        const uint32_t upto = running_sum(count);  // candidates up to and including the lane's cell
        const uint32_t total = __shfl_sync(0xffffffffu, upto, 31), before = upto - count;
        const bool obstacles = S.obstacles != 0;
        // 16-bit positions are taken from the group's first particle, in units of h
        const float inv_h = A.inv_h;
        const float4 origin = __ldg(&ps[first]);
        const float ox = -origin.x * inv_h, oy = -origin.y * inv_h, oz = -origin.z * inv_h;
        const __half2 less = __half2half2(__hneg(__float2half_ru(reach2 * inv_h * inv_h + kHalfMargin)));
        for (uint32_t base = first; base < end; base += 32) {
            const uint32_t own = min(end - base, 32u);
            uint32_t found = 0;  // lane j: the hits of the j-th particle
            bool far = false;
            __syncwarp();
            if (lane < own) {
                const float4 p = __ldg(&ps[base + lane]);
                const float x = __fmaf_rn(p.x, inv_h, ox), y = __fmaf_rn(p.y, inv_h, oy), z = __fmaf_rn(p.z, inv_h, oz);
                const bool none = obstacles && A.type[base + lane] == FGB_TYPE_OBSTACLE;  // no sums: an empty row
                far = !none && !(fabsf(x) <= kHalfReach && fabsf(y) <= kHalfReach && fabsf(z) <= kHalfReach);
                sh.own[lane] = make_uint4(bits_of(__floats2half2_rn(x, x)), bits_of(__floats2half2_rn(y, y)),
                                          bits_of(__floats2half2_rn(z, z)), none || far ? 0u : 0xffffffffu);
            }
            const unsigned fars = __ballot_sync(0xffffffffu, far);
            for (uint32_t seg = 0; seg < total; seg += kHeldAll) {
                // candidates [seg, seg + 256): the lanes list their cells' indices
                __syncwarp();
                {
                    const uint32_t lo = max(before, seg), hi = min(upto, seg + kHeldAll);
                    uint32_t b = from + (lo - before);
                    uint32_t *to = sh.map + (lo - seg);
                    for (uint32_t k = lo; k < hi; k += 4, to += 4, b += 4) {
                        to[0] = b;
                        if (k + 1 < hi) to[1] = b + 1;
                        if (k + 2 < hi) to[2] = b + 2;
                        if (k + 3 < hi) to[3] = b + 3;
                    }
                }
                __syncwarp();
                const uint32_t here = min(total - seg, kHeldAll);
                auto segment = [&](auto pairs) {
                    constexpr uint32_t P = decltype(pairs)::value;  // the lane's 2 P candidates in a row
                    __half2 X[P], Y[P], Z[P];
                    uint32_t idx[2 * P];
#pragma unroll
                    for (uint32_t k = 0; k < P; ++k) {
                        const uint2 i = reinterpret_cast<const uint2 *>(sh.map)[lane * P + k];
                        idx[2 * k] = i.x, idx[2 * k + 1] = i.y;
                    }
#pragma unroll
                    for (uint32_t k = 0; k < P; ++k) {
                        float4 p = make_float4(INFINITY, INFINITY, INFINITY, 0.f), q = p;
                        if (2 * (lane * P + k) < here) p = __ldg(&ps[idx[2 * k]]);
                        if (2 * (lane * P + k) + 1 < here) q = __ldg(&ps[idx[2 * k + 1]]);
                        X[k] = __floats2half2_rn(__fmaf_rn(p.x, inv_h, ox), __fmaf_rn(q.x, inv_h, ox));
                        Y[k] = __floats2half2_rn(__fmaf_rn(p.y, inv_h, oy), __fmaf_rn(q.y, inv_h, oy));
                        Z[k] = __floats2half2_rn(__fmaf_rn(p.z, inv_h, oz), __fmaf_rn(q.z, inv_h, oz));
                    }
                    // the lane's candidates within reach of the j-th particle: 2 k and 2 k + 1 at
                    // bits 16 - P + k and 32 - P + k
                    auto hits_of = [&](uint32_t j) {
                        const uint4 o = sh.own[j];
                        const __half2 x = half2_of(o.x), y = half2_of(o.y), z = half2_of(o.z);
                        uint32_t hits = 0;
#pragma unroll
                        for (uint32_t k = 0; k < P; ++k) {
                            const __half2 ex = __hsub2(X[k], x), ey = __hsub2(Y[k], y), ez = __hsub2(Z[k], z);
                            const __half2 r2 = __hfma2(ex, ex, __hfma2(ey, ey, __hfma2(ez, ez, less)));
                            hits = hits >> 1 | (bits_of(r2) & 0x80008000u);
                        }
                        return hits & o.w;
                    };
                    auto append = [&](uint32_t hits, uint32_t to) {
#pragma unroll
                        for (uint32_t k = 0; k < P; ++k) {
                            append_if(hits, 1u << (16 - P + k), idx[2 * k], to);
                            append_if(hits, 1u << (32 - P + k), idx[2 * k + 1], to);
                        }
                    };
#pragma unroll 1
                    for (uint32_t four = 0; four < own; four += kList) {
                        const uint32_t earlier = found;  // hits of earlier segments
                        const uint32_t last = min(four + kList, own);
                        __syncwarp();
#pragma unroll 1
                        for (uint32_t j = four; j < last; j += 2) {
                            const bool two = j + 1 < last;
                            const uint32_t h0 = hits_of(j), h1 = two ? hits_of(j + 1) : 0u;
                            const uint32_t n = __popc(h0) | __popc(h1) << 16;
                            const uint32_t sum = running_sum(n), at = sum - n;
                            const uint32_t all = __shfl_sync(0xffffffffu, sum, 31);
                            const uint32_t list = lists + 4 * (j - four) * kPitch;
                            append(h0, list + 4 * (at & 0xffffu));
                            if (lane < 3) fill(list + 4 * ((all & 0xffffu) + lane), A.none);
                            if (lane == j) found += all & 0xffffu;
                            if (two) {
                                append(h1, list + 4 * kPitch + 4 * (at >> 16));
                                if (lane < 3) fill(list + 4 * kPitch + 4 * ((all >> 16) + lane), A.none);
                                if (lane == j + 1) found += all >> 16;
                            }
                        }
                        __syncwarp();
                        // the four's hits to their rows: lane 4 p + j takes quad p of the j-th
                        const uint32_t j = four + (lane & 3u);
                        const uint32_t lo = __shfl_sync(0xffffffffu, earlier, j),
                                       hi = min(__shfl_sync(0xffffffffu, found, j), A.hcap);
                        if (j >= own) continue;
                        const uint32_t *have = sh.hits + (lane & 3u) * kPitch;
                        uint4 *row = row_of(A, base + j);
                        if (lo == 0) {
                            for (uint32_t e = 4 * (lane >> 2); e < hi; e += 32)
                                row[(e >> 2) * 32] = *reinterpret_cast<const uint4 *>(have + e);
                        } else {  // a later segment, which starts within a quad
                            for (uint32_t e = lo + (lane >> 2); e < ((hi + 3u) & ~3u); e += 8)
                                reinterpret_cast<uint32_t *>(row + (e >> 2) * 32)[e & 3u] = have[e - lo];
                        }
                    }
                };
                if (here <= 128)
                    segment(Pairs<2>{});
                else if (here <= 192)
                    segment(Pairs<3>{});
                else
                    segment(Pairs<4>{});
                // particles too far from the group's origin for 16 bits
                if (fars) __syncwarp();
                for (unsigned rest = fars; rest; rest &= rest - 1) {
                    const uint32_t j = __ffs(rest) - 1;
                    const float4 pa = __ldg(&ps[base + j]);
                    uint32_t *row = reinterpret_cast<uint32_t *>(row_of(A, base + j));
                    uint32_t at = __shfl_sync(0xffffffffu, found, j);
                    for (uint32_t k = 0; k < here; k += 32) {
                        bool hit = false;
                        uint32_t b = 0;
                        if (k + lane < here) {
                            b = sh.map[k + lane];
                            const float4 p = __ldg(&ps[b]);
                            hit = dist2(p.x - pa.x, p.y - pa.y, p.z - pa.z) < reach2;
                        }
                        const unsigned in = __ballot_sync(0xffffffffu, hit);
                        const uint32_t e = at + __popc(in & lanemask_lt());
                        if (hit && e < A.hcap) row[(e >> 2) * 128 + (e & 3u)] = b;
                        at += __popc(in);
                    }
                    if (lane < 3 && at + lane < ((at + 3u) & ~3u) && at + lane < A.hcap)
                        row[((at + lane) >> 2) * 128 + ((at + lane) & 3u)] = A.none;
                    if (lane == j) found = at;
                    __syncwarp();
                }
            }
            if (lane < own) A.hcount[base + lane] = found > A.hcap ? kListOverflow : (uint16_t)found;
            if (A.over) {
                const unsigned full = __ballot_sync(0xffffffffu, lane < own && found > A.hcap);
                if (full && lane == 0) atomicAdd(A.over, (uint32_t)__popc(full));
            }
        }
    }
    if (kSearch == kLaterSearch && count_use) report();
}

// The 27-cell walk, for rows that overflowed.
template <class F>
__device__ __forceinline__ void walk_cells(const RowArgs &A, const SceneDev &S, uint32_t key, F &&add) {
    const uint32_t m = morton_of(key, A.mbits);
    for_neighbour_cells(S, A.cells, (int)compact10(m), (int)compact10(m >> 1), (int)compact10(m >> 2), add);
}

// A hit row's neighbours two at a time as add(b0, b1, p0, p1), p their entries of `packed`:
// four entries' loads together, the next four's indices in flight.  What fills the last
// quad lies at infinity, where every pass's range test drops it, so the loop has no other
// conditions.  (Two pairs at a time, each tested for the row's end, took the delta pass of
// the 1 M dam break 111 us; quads take 96, and 92 to 78 deep in the flow.)
template <class F>
__device__ __forceinline__ void for_pairs(const uint4 *__restrict__ row, uint32_t count,
                                          const float4 *__restrict__ packed, F &&add) {
    const uint32_t quads = (count + 3) >> 2;
    uint4 next = quads ? __ldg(row) : make_uint4(0, 0, 0, 0);
    for (uint32_t i = 1; i <= quads; ++i) {
        const uint4 b = next;
        const float4 p = __ldg(&packed[b.x]), q = __ldg(&packed[b.y]), u = __ldg(&packed[b.z]), w = __ldg(&packed[b.w]);
        row += 32;
        if (i < quads) next = __ldg(row);
        add(b.x, b.y, p, q);
        add(b.z, b.w, u, w);
    }
}

// 32 aligned bytes by one load
__device__ __forceinline__ void load_two(const float4 *p, float4 &a, float4 &b) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}

// The warp's rows into L2 by one bulk request before its lanes go through them, where all
// rows together are more than L2 holds (kFetchFrom): a step of 1 M particles takes 1.70 ms
// with it and 1.75 without, one of 262 k, whose rows stay in L2, 0.521 and 0.514.
__device__ __forceinline__ void fetch_rows(const RowArgs &A, uint32_t a) {
    if (!A.fetch) return;
    const uint32_t count = a < A.n ? A.hcount[a] : 0u;
    const uint32_t most = __reduce_max_sync(0xffffffffu, count == kListOverflow ? 0u : count);
    if ((a & 31u) == 0 && most)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(row_of(A, a)), "r"(((most + 3) >> 2) * 512)
                     : "memory");
}

template <int PROFILE, bool kFast>
__global__ void __launch_bounds__(128, 8)
    k_row_lambda(RowArgs A, const float4 *__restrict__ ps, float *__restrict__ lambda, float *__restrict__ density,
                 float4 *__restrict__ plam) {
    const uint32_t a = blockIdx.x * blockDim.x + threadIdx.x;
    fetch_rows(A, a);
    if (a >= A.n) return;
    const float4 pa = ps[a];
    float lam = 0.f, dens = 0.f;
    if (A.type[a] != FGB_TYPE_OBSTACLE) {
        const Phys &ph = A.ph;
        const uint32_t count = A.hcount[a];
        LambdaSum<PROFILE> sum;
        if (count != kListOverflow)
            for_pairs(row_of(A, a), count, ps, [&](uint32_t, uint32_t, const float4 &p, const float4 &q) {
                sum.template add2<kFast>(ph, pa, Two(p.x, q.x), Two(p.y, q.y), Two(p.z, q.z), Two(p.w, q.w));
            });
        else
            walk_cells(A, A.scenes[scene_of(A.keys[a], A.mbits)], A.keys[a], [&](uint32_t b) {
                const float4 p = __ldg(&ps[b]);
                sum.add(ph, pa, p.x, p.y, p.z, p.w);
            });
        lam = sum.finish(ph, &dens);
    }
    lambda[a] = lam;
    density[a] = dens;
    plam[a] = make_float4(pa.x, pa.y, pa.z, lam);
    A.moved[a] = 0;  // before the delta pass that follows
}

// Keep the cell's largest movement since the grid was built: lanes of one cell (their
// particles are consecutive, every kStride lanes) settle theirs first.  All lanes take part.
template <int kStride>
__device__ __forceinline__ void keep_moved(const RowArgs &A, bool have, uint32_t cell_start, float moved) {
    uint32_t m = have ? __float_as_uint(moved) : 0u;
    if (have && !(moved == moved)) m = 0x7f800000u;  // not a number: the bound has to fail
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t where = have ? cell_start : 0xffffffffu;
#pragma unroll
    for (int d = kStride; d < 32; d <<= 1) {
        const uint32_t o = __shfl_down_sync(0xffffffffu, m, d), w = __shfl_down_sync(0xffffffffu, where, d);
        if (lane + d < 32 && w == where) m = max(m, o);
    }
    const uint32_t left = __shfl_up_sync(0xffffffffu, where, kStride);
    if (have && (lane < kStride || left != where) && m) atomicMax(&A.moved[where], m);
}

// The end of a particle's delta pass: its new position, after the step's last correction also
// its velocity; how far it is from its grid position, and where its cell begins.
template <int PROFILE>
__device__ __forceinline__ float finish_delta(const RowArgs &A, const SceneDev &S, const DeltaSum<PROFILE> &sum,
                                              uint32_t a, uint32_t key, const float4 &pa, float4 *__restrict__ ps_out,
                                              float4 *__restrict__ x, float4 *__restrict__ v, int last,
                                              float4 *__restrict__ pv, const HostParticlesOut *__restrict__ hout,
                                              uint32_t &cell_start) {
    const Phys &ph = A.ph;
    float4 va;
    float q[3], vel[3];
    sum.move(ph, S, A.tris, pa, a, v, q, va, vel);
    ps_out[a] = make_float4(q[0], q[1], q[2], pa.w);
    if (last) {
        const float4 now = finalise<PROFILE>(ph, S, a, q, va, vel, x, v, hout);
        if (PROFILE != kRef) {
            pv[2 * (size_t)a] = make_float4(q[0], q[1], q[2], pa.w);
            pv[2 * (size_t)a + 1] = now;
        }
    }
    const float4 g = __ldg(&A.ps_grid[a]);
    const float ex = q[0] - g.x, ey = q[1] - g.y, ez = q[2] - g.z;
    cell_start = __ldg(&A.cells[S.table_base + morton_of(key, A.mbits)]).x;
    return sqrtf(ex * ex + ey * ey + ez * ez);
}

template <int PROFILE, bool kFast>
__global__ void __launch_bounds__(128, 8)
    k_row_delta(RowArgs A, const float4 *__restrict__ ps_in, const float4 *__restrict__ plam,
                float4 *__restrict__ ps_out, float4 *__restrict__ x, float4 *__restrict__ v, int last,
                float4 *__restrict__ pv, const HostParticlesOut *__restrict__ hout) {
    const uint32_t a = blockIdx.x * blockDim.x + threadIdx.x;
    fetch_rows(A, a);
    const bool own = a < A.n;
    const bool fluid = own && A.type[a] != FGB_TYPE_OBSTACLE;
    uint32_t cell_start = 0;
    float moved = 0.f;
    if (own && !fluid) {
        ps_out[a] = ps_in[a];
        if (PROFILE != kRef && last) pv[2 * (size_t)a] = ps_in[a], pv[2 * (size_t)a + 1] = v[a];
        if (PROFILE == kRef && last) store_host_motion(hout, a, x[a], v[a]);
    }
    if (fluid) {
        const bool equal = PROFILE == kRef || A.mass_range[0] == ~A.mass_range[1];
        const float mass = __uint_as_float(A.mass_range[0]);
        const Phys &ph = A.ph;
        const float4 pa = ps_in[a];
        const uint32_t key = A.keys[a];
        const SceneDev &S = A.scenes[scene_of(key, A.mbits)];
        const float la = __ldg(&plam[a]).w;
        const uint32_t count = A.hcount[a];
        DeltaSum<PROFILE> sum;
        if (count != kListOverflow)
            for_pairs(row_of(A, a), count, plam, [&](uint32_t b0, uint32_t b1, const float4 &p, const float4 &q) {
                Two m(mass);
                if (!equal) m = Two(__ldg(&ps_in[b0]).w, __ldg(&ps_in[b1]).w);
                sum.template add2<kFast>(ph, pa, la, Two(p.x, q.x), Two(p.y, q.y), Two(p.z, q.z), Two(p.w, q.w), m);
            });
        else
            walk_cells(A, S, key, [&](uint32_t b) {
                const float4 p = __ldg(&plam[b]);
                sum.add(ph, pa, la, p.x, p.y, p.z, [&] { return p.w; }, __ldg(&ps_in[b]).w);
            });
        moved = finish_delta<PROFILE>(A, S, sum, a, key, pa, ps_out, x, v, last, pv, hout, cell_start);
    }
    if (PROFILE != kRef || !last) keep_moved<1>(A, fluid, cell_start, moved);  // a search follows
}

// Pass A of the velocity terms: fluid neighbours only, which rows do not tell apart.  The
// neighbours' positions and velocities come from one record of 32 bytes each (pv, by the
// last delta pass) by one load: 32 lanes' records cost the L1 a third less than a position
// and a velocity apart.  158 to 146 us at 1 M, 2 of it given back by the delta pass.
template <bool kFast>
__global__ void __launch_bounds__(128, 6)
    k_row_vorticity(RowArgs A, const float4 *__restrict__ pv, float4 *__restrict__ omega, float4 *__restrict__ pom,
                    float4 *__restrict__ vx) {
    const uint32_t a = blockIdx.x * blockDim.x + threadIdx.x;
    fetch_rows(A, a);
    if (a >= A.n) return;
    float4 pa, va;
    load_two(pv + 2 * (size_t)a, pa, va);
    if (A.type[a] == FGB_TYPE_OBSTACLE) {
        omega[a] = make_float4(0.f, 0.f, 0.f, 0.f);
        vx[a] = va;
        pom[a] = make_float4(pa.x, pa.y, pa.z, 0.f);
        return;
    }
    const Phys &ph = A.ph;
    const uint32_t key = A.keys[a];
    const SceneDev &S = A.scenes[scene_of(key, A.mbits)];
    const bool obstacles = S.obstacles != 0;
    const uint32_t count = A.hcount[a];
    VorticitySum sum;
    auto two = [&](uint32_t b0, uint32_t b1, float4 p, const float4 &u, float4 q, const float4 &w) {
        if (obstacles) {
            if (__ldg(&A.type[b0]) == FGB_TYPE_OBSTACLE) p.x = INFINITY;
            if (__ldg(&A.type[b1]) == FGB_TYPE_OBSTACLE) q.x = INFINITY;
        }
        sum.template add2<kFast>(ph, pa, va, Two(p.x, q.x), Two(p.y, q.y), Two(p.z, q.z), Two(p.w, q.w),
                                 Two(u.x, w.x), Two(u.y, w.y), Two(u.z, w.z));
    };
    if (count != kListOverflow) {
        const uint4 *row = row_of(A, a);
        const uint32_t quads = (count + 3) >> 2;
        uint4 next = quads ? __ldg(row) : make_uint4(0, 0, 0, 0);
        for (uint32_t i = 1; i <= quads; ++i) {
            const uint4 b = next;
            float4 p[4], u[4];
            load_two(pv + 2 * (size_t)b.x, p[0], u[0]);
            load_two(pv + 2 * (size_t)b.y, p[1], u[1]);
            load_two(pv + 2 * (size_t)b.z, p[2], u[2]);
            load_two(pv + 2 * (size_t)b.w, p[3], u[3]);
            row += 32;
            if (i < quads) next = __ldg(row);
            two(b.x, b.y, p[0], u[0], p[1], u[1]);
            two(b.z, b.w, p[2], u[2], p[3], u[3]);
        }
    } else
        walk_cells(A, S, key, [&](uint32_t b) {
            if (obstacles && __ldg(&A.type[b]) == FGB_TYPE_OBSTACLE) return;
            const float4 p = __ldg(&pv[2 * (size_t)b]);
            sum.add(ph, pa, va, p.x, p.y, p.z, p.w, [&] { return __ldg(&pv[2 * (size_t)b + 1]); });
        });
    sum.finish(ph, a, pa, va, omega, pom, vx);
}

template <bool kFast>
__global__ void __launch_bounds__(128, 8)
    k_row_apply(RowArgs A, const float4 *__restrict__ ps, const float4 *__restrict__ omega,
                const float4 *__restrict__ pom, const float4 *__restrict__ vx, float4 *__restrict__ v,
                float4 *__restrict__ x, const HostParticlesOut *__restrict__ hout) {
    const uint32_t a = blockIdx.x * blockDim.x + threadIdx.x;
    fetch_rows(A, a);
    if (a >= A.n) return;
    if (A.type[a] == FGB_TYPE_OBSTACLE) {
        store_host_motion(hout, a, x[a], v[a]);
        return;
    }
    const bool equal = A.mass_range[0] == ~A.mass_range[1];
    const float mass = __uint_as_float(A.mass_range[0]);
    const Phys &ph = A.ph;
    const uint32_t key = A.keys[a];
    const SceneDev &S = A.scenes[scene_of(key, A.mbits)];
    const float4 pa = ps[a], oa = omega[a];
    const uint32_t count = A.hcount[a];
    ApplySum sum;
    if (count != kListOverflow)
        for_pairs(row_of(A, a), count, pom, [&](uint32_t b0, uint32_t b1, float4 p, float4 q) {
            Two m(mass);
            if (S.obstacles) {
                if (__ldg(&A.type[b0]) == FGB_TYPE_OBSTACLE) p.x = INFINITY;
                if (__ldg(&A.type[b1]) == FGB_TYPE_OBSTACLE) q.x = INFINITY;
            }
            if (!equal) m = Two(__ldg(&ps[b0]).w, __ldg(&ps[b1]).w);
            sum.template add2<kFast>(ph, pa, oa.w, Two(p.x, q.x), Two(p.y, q.y), Two(p.z, q.z), Two(p.w, q.w), m);
        });
    else
        walk_cells(A, S, key, [&](uint32_t b) {
            if (S.obstacles && __ldg(&A.type[b]) == FGB_TYPE_OBSTACLE) return;
            const float4 p = __ldg(&pom[b]);
            sum.add(ph, pa, oa.w, p.x, p.y, p.z, [&] { return p.w; }, __ldg(&ps[b]).w);
        });
    sum.finish(ph, S, a, pa, oa, vx, v, x, hout);
}

// ---------------------------------------------------------------- four lanes a particle
//
// The same passes for small scenes.  A thread that goes through a row
// alone waits for one operation after another where a scheduler holds a warp or two, and a
// warp of 32 particles for its longest row; with four lanes a particle there are four times
// the warps, each lane forms the terms of every fourth entry, and they meet in shared memory,
// where lane 0 to 2 adds up one component, in the row's order, and lane 3 what remains.
// A step with a thread a particle / four lanes: baseline 4 k 133 / 115 us, 14 k 150 / 135,
// 33 k 179 / 183, 64 k 211 / 260; ref profile 14 k 430 / 342, 33 k 605 / 565, 64 k 578 / 616:
// a warp of lanes adds 68 instructions for four entries of eight particles where 160 did for
// those of 32, so it only pays where warps are few (kQuadsTo, kQuadsToRef).

constexpr uint32_t kQuadPitch = 40;  // floats: eight lanes' reads of four values touch all banks once

template <int kValues>
struct QuadBuffer {
    float v[2][kValues][kQuadPitch];  // by turns: one barrier an iteration
};

// A particle's row by its four lanes: fetch(b) gives an entry's data, terms(b, data, v, in, near)
// its terms and whether it is within range and not on top of the particle, add(v, at, in, near)
// takes four entries' terms: those of value k at v[k][at ..], bit e of in and near for the e-th.
// All lanes of a warp take part; count is 0 for those without a row.
template <int kValues, class Fetch, class Terms, class Add>
__device__ __forceinline__ void for_quads(const RowArgs &A, QuadBuffer<kValues> &buffer, uint32_t a, uint32_t count,
                                          Fetch &&fetch, Terms &&terms, Add &&add) {
    const uint32_t lane = threadIdx.x & 31u, at = lane & 28u, quads = (count + 3) >> 2;
    const uint32_t most = __reduce_max_sync(0xffffffffu, quads);
    const uint32_t *row = reinterpret_cast<const uint32_t *>(row_of(A, a)) + (lane & 3u);
    auto entry = [&](uint32_t i) { return i < quads ? __ldg(row + i * 128) : A.none; };
    uint32_t b = entry(0), next = entry(1);
    auto data = fetch(b);
    for (uint32_t i = 0; i < most; ++i) {
        const uint32_t this_b = b;
        const auto this_data = data;
        b = next;
        data = fetch(b);
        next = entry(i + 2);
        float v[kValues];
        bool in, near;
        terms(this_b, this_data, v, in, near);
        float(&to)[kValues][kQuadPitch] = buffer.v[i & 1u];
#pragma unroll
        for (int k = 0; k < kValues; ++k) to[k][lane] = v[k];
        const unsigned ins = __ballot_sync(0xffffffffu, in) >> at, nears = __ballot_sync(0xffffffffu, near) >> at;
        __syncwarp();
        add(to, at, ins, nears);
    }
}

// acc += f x for the entries whose bit is set, in order
__device__ __forceinline__ void add_four(float &acc, const float4 &f, const float4 &x, unsigned bits) {
    if (bits & 1u) acc = __fmaf_rn(f.x, x.x, acc);
    if (bits & 2u) acc = __fmaf_rn(f.y, x.y, acc);
    if (bits & 4u) acc = __fmaf_rn(f.z, x.z, acc);
    if (bits & 8u) acc = __fmaf_rn(f.w, x.w, acc);
}
__device__ __forceinline__ float4 four(const float (&v)[kQuadPitch], uint32_t at) {
    return *reinterpret_cast<const float4 *>(&v[at]);
}
// the value of the quad's lane k
__device__ __forceinline__ float of_lane(float v, int k) { return __shfl_sync(0xffffffffu, v, k, 4); }

template <int PROFILE, bool kFast>
__global__ void __launch_bounds__(128)
    k_quad_lambda(RowArgs A, const float4 *__restrict__ ps, float *__restrict__ lambda, float *__restrict__ density,
                  float4 *__restrict__ plam) {
    constexpr bool kR = PROFILE == kRef;
    __shared__ alignas(16) QuadBuffer<kR ? 4 : 8> s_buffer[4];
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, part = threadIdx.x & 3u;
    const bool own = (t >> 2) < A.n;
    const uint32_t a = own ? t >> 2 : A.n - 1;
    const Phys &ph = A.ph;
    const float4 pa = ps[a];
    const bool fluid = own && A.type[a] != FGB_TYPE_OBSTACLE;
    const uint32_t count = fluid ? A.hcount[a] : 0u;
    float first = 0.f, second = 0.f;  // the lane's sums
    const float hh = kR ? ph.hh_le : ph.hh;
    for_quads(
        A, s_buffer[threadIdx.x >> 5], a, count == kListOverflow ? 0u : count, [&](uint32_t b) { return __ldg(&ps[b]); },
        [&](uint32_t, const float4 &p, float *v, bool &in, bool &near) {
            const auto o = LambdaSum<PROFILE>::template terms<kFast>(ph, pa, p.x, p.y, p.z, p.w);
            in = o.q2 <= hh;
            near = o.q2 >= ph.eps_r2;
            v[0] = o.x, v[1] = o.y, v[2] = o.z, v[3] = o.w;
            if (kR) {
                if (kFast && !near) v[3] = LambdaSum<PROFILE>::on_top(ph);
            } else {
                v[4] = o.s, v[5] = p.w, v[6] = o.ss, v[7] = o.q2;
            }
        },
        [&](const auto &v, uint32_t at, unsigned in, unsigned near) {
            near &= in;
            const float4 x = four(v[part], at);
            if constexpr (kR) {
                const float f = part < 3 ? ph.inv_rho0 : pa.w;
                add_four(first, make_float4(f, f, f, f), x, part < 3 ? near : in);
            } else {
                add_four(first, four(v[part < 3 ? 4 : 5], at), x, part < 3 ? near : in);
                add_four(second, four(v[6], at), four(v[7], at), near);
            }
        });
    LambdaSum<PROFILE> sum;
    sum.gx = of_lane(first, 0), sum.gy = of_lane(first, 1), sum.gz = of_lane(first, 2);
    sum.rho = of_lane(first, 3), sum.g2 = second;  // second is the same in all four
    if (!own || part) return;
    float lam = 0.f, dens = 0.f;
    if (fluid) {
        if (count == kListOverflow)
            walk_cells(A, A.scenes[scene_of(A.keys[a], A.mbits)], A.keys[a], [&](uint32_t b) {
                const float4 p = __ldg(&ps[b]);
                sum.add(ph, pa, p.x, p.y, p.z, p.w);
            });
        lam = sum.finish(ph, &dens);
    }
    lambda[a] = lam;
    density[a] = dens;
    plam[a] = make_float4(pa.x, pa.y, pa.z, lam);
    A.moved[a] = 0;  // before the delta pass that follows
}

template <int PROFILE, bool kFast>
__global__ void __launch_bounds__(128)
    k_quad_delta(RowArgs A, const float4 *__restrict__ ps_in, const float4 *__restrict__ plam,
                 float4 *__restrict__ ps_out, float4 *__restrict__ x, float4 *__restrict__ v, int last,
                 float4 *__restrict__ pv, const HostParticlesOut *__restrict__ hout) {
    __shared__ alignas(16) QuadBuffer<4> s_buffer[4];
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, part = threadIdx.x & 3u;
    const bool own = (t >> 2) < A.n;
    const uint32_t a = own ? t >> 2 : A.n - 1;
    const Phys &ph = A.ph;
    const bool equal = PROFILE == kRef || A.mass_range[0] == ~A.mass_range[1];
    const float mass = __uint_as_float(A.mass_range[0]);
    const float4 pa = ps_in[a];
    const float la = __ldg(&plam[a]).w;
    const bool fluid = own && A.type[a] != FGB_TYPE_OBSTACLE;
    const uint32_t count = fluid ? A.hcount[a] : 0u;
    float first = 0.f;
    for_quads(
        A, s_buffer[threadIdx.x >> 5], a, count == kListOverflow ? 0u : count,
        [&](uint32_t b) { return __ldg(&plam[b]); },
        [&](uint32_t b, const float4 &p, float *o, bool &in, bool &near) {
            const float m = equal ? mass : __ldg(&ps_in[b]).w;
            const auto terms = DeltaSum<PROFILE>::template terms<kFast>(ph, pa, la, p.x, p.y, p.z, p.w, m);
            in = near = DeltaSum<PROFILE>::in_range(ph, terms.q2);
            o[0] = terms.x, o[1] = terms.y, o[2] = terms.z, o[3] = terms.f;
        },
        [&](const auto &o, uint32_t at, unsigned in, unsigned) {
            add_four(first, four(o[part < 3 ? part : 2], at), four(o[3], at), in);
        });
    DeltaSum<PROFILE> sum;
    sum.px = of_lane(first, 0), sum.py = of_lane(first, 1), sum.pz = of_lane(first, 2);
    const bool leads = own && part == 0;
    uint32_t cell_start = 0;
    float moved = 0.f;
    if (leads && !fluid) {
        ps_out[a] = ps_in[a];
        if (PROFILE != kRef && last) pv[2 * (size_t)a] = ps_in[a], pv[2 * (size_t)a + 1] = v[a];
        if (PROFILE == kRef && last) store_host_motion(hout, a, x[a], v[a]);
    }
    if (leads && fluid) {
        const uint32_t key = A.keys[a];
        const SceneDev &S = A.scenes[scene_of(key, A.mbits)];
        if (count == kListOverflow)
            walk_cells(A, S, key, [&](uint32_t b) {
                const float4 p = __ldg(&plam[b]);
                sum.add(ph, pa, la, p.x, p.y, p.z, [&] { return p.w; }, __ldg(&ps_in[b]).w);
            });
        moved = finish_delta<PROFILE>(A, S, sum, a, key, pa, ps_out, x, v, last, pv, hout, cell_start);
    }
    if (PROFILE != kRef || !last) keep_moved<4>(A, leads && fluid, cell_start, moved);  // a search follows
}

template <bool kFast>
__global__ void __launch_bounds__(128)
    k_quad_vorticity(RowArgs A, const float4 *__restrict__ pv, float4 *__restrict__ omega, float4 *__restrict__ pom,
                     float4 *__restrict__ vx) {
    __shared__ alignas(16) QuadBuffer<8> s_buffer[4];
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, part = threadIdx.x & 3u;
    const bool own = (t >> 2) < A.n;
    const uint32_t a = own ? t >> 2 : A.n - 1;
    const Phys &ph = A.ph;
    float4 pa, va;
    load_two(pv + 2 * (size_t)a, pa, va);
    const bool fluid = own && A.type[a] != FGB_TYPE_OBSTACLE;
    const uint32_t key = A.keys[a], count = fluid ? A.hcount[a] : 0u;
    const SceneDev &S = A.scenes[scene_of(key, A.mbits)];
    const bool obstacles = S.obstacles != 0;
    float first = 0.f, second = 0.f;
    struct Both {
        float4 p, u;
    };
    for_quads(
        A, s_buffer[threadIdx.x >> 5], a, count == kListOverflow ? 0u : count,
        [&](uint32_t b) {
            Both o;
            load_two(pv + 2 * (size_t)b, o.p, o.u);
            return o;
        },
        [&](uint32_t b, const Both &n, float *o, bool &in, bool &near) {
            const auto terms = VorticitySum::terms<kFast>(ph, pa, va, n.p.x, n.p.y, n.p.z, n.p.w, n.u.x, n.u.y, n.u.z);
            in = terms.q2 <= ph.hh && !(obstacles && __ldg(&A.type[b]) == FGB_TYPE_OBSTACLE);
            near = terms.q2 >= ph.eps_r2;
            o[0] = terms.vx, o[1] = terms.vy, o[2] = terms.vz, o[3] = terms.mw;
            o[4] = terms.cx, o[5] = terms.cy, o[6] = terms.cz, o[7] = terms.s;
        },
        [&](const auto &o, uint32_t at, unsigned in, unsigned near) {
            const uint32_t k = part < 3 ? part : 2;
            add_four(first, four(o[3], at), four(o[k], at), in);
            add_four(second, four(o[7], at), four(o[4 + k], at), in & near);
        });
    VorticitySum sum;
    for (int k = 0; k < 3; ++k) sum.xs[k] = of_lane(first, k), sum.o[k] = of_lane(second, k);
    if (!own || part) return;
    if (!fluid) {
        omega[a] = make_float4(0.f, 0.f, 0.f, 0.f);
        vx[a] = va;
        pom[a] = make_float4(pa.x, pa.y, pa.z, 0.f);
        return;
    }
    if (count == kListOverflow)
        walk_cells(A, S, key, [&](uint32_t b) {
            if (obstacles && __ldg(&A.type[b]) == FGB_TYPE_OBSTACLE) return;
            const float4 p = __ldg(&pv[2 * (size_t)b]);
            sum.add(ph, pa, va, p.x, p.y, p.z, p.w, [&] { return __ldg(&pv[2 * (size_t)b + 1]); });
        });
    sum.finish(ph, a, pa, va, omega, pom, vx);
}

template <bool kFast>
__global__ void __launch_bounds__(128)
    k_quad_apply(RowArgs A, const float4 *__restrict__ ps, const float4 *__restrict__ omega,
                 const float4 *__restrict__ pom, const float4 *__restrict__ vx, float4 *__restrict__ v,
                 float4 *__restrict__ x, const HostParticlesOut *__restrict__ hout) {
    __shared__ alignas(16) QuadBuffer<4> s_buffer[4];
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, part = threadIdx.x & 3u;
    const bool own = (t >> 2) < A.n;
    const uint32_t a = own ? t >> 2 : A.n - 1;
    const Phys &ph = A.ph;
    const bool equal = A.mass_range[0] == ~A.mass_range[1];
    const float mass = __uint_as_float(A.mass_range[0]);
    const uint32_t key = A.keys[a];
    const SceneDev &S = A.scenes[scene_of(key, A.mbits)];
    const bool obstacles = S.obstacles != 0;
    const float4 pa = ps[a], oa = omega[a];
    const bool fluid = own && A.type[a] != FGB_TYPE_OBSTACLE;
    const uint32_t count = fluid ? A.hcount[a] : 0u;
    float first = 0.f;
    for_quads(
        A, s_buffer[threadIdx.x >> 5], a, count == kListOverflow ? 0u : count,
        [&](uint32_t b) { return __ldg(&pom[b]); },
        [&](uint32_t b, const float4 &p, float *o, bool &in, bool &near) {
            const float m = equal ? mass : __ldg(&ps[b]).w;
            const auto terms = ApplySum::terms<kFast>(ph, pa, oa.w, p.x, p.y, p.z, p.w, m);
            in = near = ApplySum::in_range(ph, terms.q2) && !(obstacles && __ldg(&A.type[b]) == FGB_TYPE_OBSTACLE);
            o[0] = terms.x, o[1] = terms.y, o[2] = terms.z, o[3] = terms.f;
        },
        [&](const auto &o, uint32_t at, unsigned in, unsigned) {
            add_four(first, four(o[3], at), four(o[part < 3 ? part : 2], at), in);
        });
    ApplySum sum;
    for (int k = 0; k < 3; ++k) sum.e[k] = of_lane(first, k);
    if (!own || part) return;
    if (!fluid) {
        store_host_motion(hout, a, x[a], v[a]);
        return;
    }
    if (count == kListOverflow)
        walk_cells(A, S, key, [&](uint32_t b) {
            if (obstacles && __ldg(&A.type[b]) == FGB_TYPE_OBSTACLE) return;
            const float4 p = __ldg(&pom[b]);
            sum.add(ph, pa, oa.w, p.x, p.y, p.z, [&] { return p.w; }, __ldg(&ps[b]).w);
        });
    sum.finish(ph, S, a, pa, oa, vx, v, x, hout);
}

// How far the step's corrections moved each particle from its grid position (a probe).
__global__ void k_displacement(const float4 *__restrict__ ps_grid, const float4 *__restrict__ ps, uint32_t n,
                               float *__restrict__ out) {
    for (uint32_t a = blockIdx.x * blockDim.x + threadIdx.x; a < n; a += gridDim.x * blockDim.x) {
        const float ex = ps[a].x - ps_grid[a].x, ey = ps[a].y - ps_grid[a].y, ez = ps[a].z - ps_grid[a].z;
        out[a] = sqrtf(ex * ex + ey * ey + ez * ez);
    }
}

// RowArgs::sparse for n particles.  us a step by warps / by particles, of clouds of 0.1, 0.25, 0.5,
// 1, 1.5, 2 and 3 particles a cell (99, 88, 79, 63, 52, 43 and 32 groups in 100 particles), baseline
// profile: 10 k 119 / 109, 114 / 132, 105 / 153; 30 k 186 / 121, 185 / 144, 180 / 168, 175 / 219;
// 50 k 266 / 141, 255 / 160, 247 / 188, 232 / 225, 221 / 261; 100 k 308 / 168, 413 / 190, 386 / 223,
// 349 / 272, 333 / 313, 313 / 345; 1 M 2469 / 911, 3453 / 1029, 3123 / 1246, 2701 / 1593, 2424 /
// 1877, 2222 / 2175, 1971 / 2602.  With the ref profile, whose fluid gathers, the lines would lie a
// little higher: 30 k at 0.5 a cell 164 / 180, 1 M at 1.5 1830 / 1979.
uint32_t sparse_above(uint64_t n) {
    return n < 30000 ? 0u : n < 45000 ? 80u : n < 75000 ? 60u : n < 400000 ? 48u : 38u;
}

RowArgs row_args(const StepView &s) {
    RowArgs A;
    A.scenes = s.scenes;
    A.tris = s.tris;
    A.ph = s.ph;
    A.n = s.n;
    A.mbits = s.mbits;
    A.keys = s.keys_sorted;
    A.cells = s.cells;
    A.type = s.type1;
    A.groups = s.groups;
    A.group_count = s.group_count;
    A.group_mask = s.group_mask;
    A.hrows = reinterpret_cast<uint4 *>(s.hlist);
    A.hcount = s.hcount;
    A.hcap = s.hcap;
    A.none = s.none;
    A.fetch = s.n >= kFetchFrom;
    A.sparse = sparse_above(s.n);
    A.mass_range = s.mass_range;
    A.over = nullptr;
    A.ps_grid = s.ps_grid;
    A.moved = s.moved;
    A.lasting = s.lasting;
    A.stale = s.stale;
    A.stale_count = nullptr;
    A.taken = nullptr;
    A.inv_h = 1.f / s.ph.h;
    A.skin = kRowSkin * s.ph.h;
    const float reach = (s.ph.h + A.skin) * 1.00001f;
    A.skin_r2 = reach * reach;
    A.policy = s.row_policy;
    A.policy_next = s.row_policy_next;
    return A;
}

// As many CTAs as the GPU holds at once.
template <class K>
cudaError_t resident_grid(K kernel, const StepView &s, uint32_t block, unsigned *grid) {
    int resident = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kernel, (int)block, 0);
    const uint64_t most = (uint64_t)(s.sm_count > 0 ? s.sm_count : 152) * (uint64_t)std::max(resident, 1);
    *grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(most, s.n));
    return e;
}

// The hit rows of positions ps for the step's pass-th search.
cudaError_t rows_of(const StepView &s, const float4 *ps, uint32_t pass, cudaStream_t st) {
    RowArgs A = row_args(s);
    // membership only (the passes test again): the test's rounding is within 3 ulp of r^2,
    // below the margin
    const float r2max = (s.ph.profile == FGB_PROFILE_REF ? s.ph.hh_le : s.ph.hh) * 1.000002f;
    unsigned grid = 1;
    cudaError_t e;
    A.taken = s.group_count + 2 + s.iterations + pass;
    if (pass == 0) {
        if (s.over) A.over = s.over + 1;  // counted once a step
        e = resident_grid(k_cell_rows<kFirstSearch>, s, kCellBlock, &grid);
        if (e != cudaSuccess) return e;
        k_cell_rows<kFirstSearch><<<grid, kCellBlock, 0, st>>>(A, ps, r2max, s.n_scenes, 0);
    } else if (row_later_search_launches(s.ph.profile, s.n) == 1) {
        e = resident_grid(k_cell_rows<kLaterSearch>, s, kCellBlock, &grid);
        if (e != cudaSuccess) return e;
        k_cell_rows<kLaterSearch><<<grid, kCellBlock, 0, st>>>(A, ps, r2max, s.n_scenes, pass == 1);
    } else {
        A.stale_count = s.group_count + pass;  // one a pass, zeroed with the groups' number
        e = resident_grid(k_stale_groups, s, 128, &grid);
        if (e != cudaSuccess) return e;
        k_stale_groups<<<grid, 128, 0, st>>>(A, pass == 1);
        e = resident_grid(k_cell_rows<kStaleSearch>, s, kCellBlock, &grid);
        if (e != cudaSuccess) return e;
        k_cell_rows<kStaleSearch><<<grid, kCellBlock, 0, st>>>(A, ps, r2max, s.n_scenes, 0);
    }
    return cudaGetLastError();
}

inline unsigned row_grid(const StepView &s) { return (s.n + 127) / 128; }
inline unsigned quad_grid(const StepView &s) { return (unsigned)(((uint64_t)s.n + 31) / 32); }

// Whether the passes give a particle four lanes.
inline bool by_quads(const StepView &s) { return s.n < (s.ph.profile == FGB_PROFILE_REF ? kQuadsToRef : kQuadsTo); }

template <int PROFILE, bool kFast>
cudaError_t lambda_as(const StepView &s, const float4 *ps, int iteration, cudaStream_t st) {
    cudaError_t e = rows_of(s, ps, (uint32_t)iteration, st);
    if (e != cudaSuccess) return e;
    if (by_quads(s))
        k_quad_lambda<PROFILE, kFast><<<quad_grid(s), 128, 0, st>>>(row_args(s), ps, s.lambda, s.density, s.plam);
    else
        k_row_lambda<PROFILE, kFast><<<row_grid(s), 128, 0, st>>>(row_args(s), ps, s.lambda, s.density, s.plam);
    return cudaGetLastError();
}

template <int PROFILE, bool kFast>
cudaError_t delta_as(const StepView &s, const float4 *ps_in, float4 *ps_out, bool last, cudaStream_t st) {
    if (by_quads(s))
        k_quad_delta<PROFILE, kFast><<<quad_grid(s), 128, 0, st>>>(row_args(s), ps_in, s.plam, ps_out, s.x1, s.v1,
                                                                   last ? 1 : 0, s.pv, s.hout);
    else
        k_row_delta<PROFILE, kFast><<<row_grid(s), 128, 0, st>>>(row_args(s), ps_in, s.plam, ps_out, s.x1, s.v1,
                                                                 last ? 1 : 0, s.pv, s.hout);
    return cudaGetLastError();
}

template <bool kFast>
cudaError_t velocity_as(const StepView &s, const float4 *ps, cudaStream_t st, const std::function<void()> &between) {
    cudaError_t e = rows_of(s, ps, s.iterations, st);
    if (e != cudaSuccess) return e;
    const RowArgs A = row_args(s);
    const bool quads = by_quads(s);
    if (quads)
        k_quad_vorticity<kFast><<<quad_grid(s), 128, 0, st>>>(A, s.pv, s.omega, s.pom, s.vx);
    else
        k_row_vorticity<kFast><<<row_grid(s), 128, 0, st>>>(A, s.pv, s.omega, s.pom, s.vx);
    if (between) between();
    if (quads)
        k_quad_apply<kFast><<<quad_grid(s), 128, 0, st>>>(A, ps, s.omega, s.pom, s.vx, s.v1, s.x1, s.hout);
    else
        k_row_apply<kFast><<<row_grid(s), 128, 0, st>>>(A, ps, s.omega, s.pom, s.vx, s.v1, s.x1, s.hout);
    return cudaGetLastError();
}

}  // namespace

// A batch without particles (scenes that are yet to be filled, or drained) has nothing to launch.

cudaError_t launch_row_lambda(const StepView &s, const float4 *ps, int iteration, cudaStream_t st) {
    if (!s.n) return cudaSuccess;
    if (s.ph.profile == FGB_PROFILE_REF)
        return s.ph.fast_root ? lambda_as<FGB_PROFILE_REF, true>(s, ps, iteration, st)
                              : lambda_as<FGB_PROFILE_REF, false>(s, ps, iteration, st);
    return s.ph.fast_root ? lambda_as<FGB_PROFILE_BASELINE, true>(s, ps, iteration, st)
                          : lambda_as<FGB_PROFILE_BASELINE, false>(s, ps, iteration, st);
}

cudaError_t launch_row_delta(const StepView &s, const float4 *ps_in, float4 *ps_out, bool last, cudaStream_t st) {
    if (!s.n) return cudaSuccess;
    if (s.ph.profile == FGB_PROFILE_REF)
        return s.ph.fast_root ? delta_as<FGB_PROFILE_REF, true>(s, ps_in, ps_out, last, st)
                              : delta_as<FGB_PROFILE_REF, false>(s, ps_in, ps_out, last, st);
    return s.ph.fast_root ? delta_as<FGB_PROFILE_BASELINE, true>(s, ps_in, ps_out, last, st)
                          : delta_as<FGB_PROFILE_BASELINE, false>(s, ps_in, ps_out, last, st);
}

cudaError_t launch_row_velocity_terms(const StepView &s, const float4 *ps, cudaStream_t st,
                                       const std::function<void()> &between) {
    if (!s.n) {
        if (between) between();
        return cudaSuccess;
    }
    return s.ph.fast_root ? velocity_as<true>(s, ps, st, between) : velocity_as<false>(s, ps, st, between);
}

void launch_displacement(const StepView &s, float *out, cudaStream_t st) {
    const float4 *last = (s.iterations & 1) ? s.ps_a : s.ps_b;
    k_displacement<<<(unsigned)std::min<uint64_t>(((uint64_t)s.n + 255) / 256, 1216), 256, 0, st>>>(s.ps_grid, last,
                                                                                                  s.n, out);
}

uint32_t row_later_search_launches(int profile, uint64_t n) {
    return profile == FGB_PROFILE_REF || n < kListFrom ? 1u : 2u;
}

// Particles of a group.  A cell's setup is shared by the particles of its group, but small
// scenes have too few cells to fill the GPU, and the ref profile's constants clump the fluid
// into few crowded ones, so a cell's particles go to several warps.  us a step (cubes at rest,
// steps 10 to 30), groups that end at multiples of 4 / 8 / 16 / 32 / 256: baseline 4 k 107 / 111
// / 113 / 113 / 115, 14 k 126 / 120 / 122 / 122 / 121, 64 k 248 / 229 / 221 / 217 / 212, 110 k
// 272 / 266 / 264 / 260 / 258; ref 14 k 319 / 323 / 355 / 427 / 581, 33 k 640 / 614 / 620 / 676
// / 821, 64 k 969 / 931 / 937 / 1004 / 1099, 123 k 1349 / 1261 / 1258 / 1303 / 1429, 250 k
// 2182 / 1996 / 1933 / 1957 / 2068, 1 M 6412 / 5664 / 5312 / 5190 / 5202.
//
// In crowds of the baseline profile groups of up to 256 leave a few warps with nearly all the
// work, hence group_end's last rule: 100 k particles in 8^3 cells, up to 3400 of them in one,
// take 38.6 instead of 95.7 ms a step, 8 k in one cell 14.2 instead of 20.1.  Where no cell has
// 32 particles it costs nothing, at step 100 of the 1 M dam break 2.062 instead of 2.053 ms.
uint32_t row_group_mask(int profile, uint64_t n) {
    if (profile == FGB_PROFILE_REF) return n < 65536 ? 7u : 15u;
    return n < 8000 ? 3u : 255u;
}

}  // namespace fgb
