// rows.cu -- hit rows from one warp per grid cell, and the gather passes over them.
//
// k_cell_rows gives a warp the particles of one cell (up to a group of them): its lanes
// hold the candidates of the cell's 27 neighbour cells, in the reference's order (z, y, x
// ascending, each cell in sorted order: oclsph_kernel.h:155-183), in registers, and test
// them all at once against each of the particles; a ballot ranks those within range, and
// they go to the particle's hit row as sorted indices, in order.  The candidates are loaded
// once for all particles of the group, every lane tests 32 different ones, and no lane
// waits for another's longer list.
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
    uint32_t group_mask;         // a group ends with its cell or where index & mask wraps
    uint4 *hrows;                // hit rows, see row_of
    uint16_t *hcount;
    uint32_t hcap;               // entries a hit row has room for (a multiple of four)
    uint32_t none;               // the index that fills a row's last quad: the far entry past the particles
    int fetch;                   // the passes ask for their rows ahead (fetch_rows)
    const uint32_t *mass_range;
    uint32_t *over;              // hit rows that overflowed (null: not counted)
    const float4 *ps_grid;       // the grid positions
    uint32_t *moved;             // largest movement in a cell since then (float bits), at its first particle
    uint8_t *lasting;            // per group: its rows are the first search's, with the skin
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
constexpr float kRowSkin = 0.1f;          // the skin of rows that last, in h
constexpr uint32_t kHeld = 8;             // candidates a lane holds at a time
constexpr uint32_t kHeldAll = 32 * kHeld;  // candidates a warp holds
constexpr uint32_t kGroup = 4;            // particles whose hits are collected before they are written
constexpr uint32_t kPitch = kHeldAll + 8;  // room to fill the last quad; the four lists in different banks

struct CellShared {
    uint32_t map[kHeldAll];                         // sorted indices of the candidates held
    alignas(16) uint32_t hits[kGroup * kPitch];  // hits of a group's particles among them, in order
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

// Where r2 is negative: store b to the warp's list at shared address `to`, in lane order;
// `to` moves past the entries.  Written out so that the store is predicated: as a branch it
// cost more instructions than the test.
__device__ __forceinline__ void append_hits(float r2, uint32_t b, uint32_t before, uint32_t &to) {
    asm volatile(
        "{\n\t"
        ".reg .pred hit;\n\t"
        ".reg .b32 in, at;\n\t"
        "setp.lt.f32 hit, %1, 0f00000000;\n\t"
        "vote.sync.ballot.b32 in, hit, 0xffffffff;\n\t"
        "and.b32 at, in, %3;\n\t"
        "popc.b32 at, at;\n\t"
        "mad.lo.u32 at, at, 4, %0;\n\t"
        "@hit st.shared.u32 [at], %2;\n\t"
        "popc.b32 in, in;\n\t"
        "mad.lo.u32 %0, in, 4, %0;\n\t"
        "}"
        : "+r"(to)
        : "f"(r2), "r"(b), "r"(before)
        : "memory");
}

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

template <int R>
struct Rounds {
    static constexpr int value = R;
};

// kFirst: the step's first search (the grid positions); else a later one, which leaves the
// groups whose rows still last.
template <bool kFirst>
__global__ void __launch_bounds__(kCellBlock, 7)
    k_cell_rows(RowArgs A, const float4 *__restrict__ ps, float r2max, uint32_t n_scenes, int count_use) {
    __shared__ CellShared s_warp[kCellWarps];
    const uint32_t lane = threadIdx.x & 31u, before = lanemask_lt();
    CellShared &sh = s_warp[threadIdx.x >> 5];
    const uint32_t lists = (uint32_t)__cvta_generic_to_shared(sh.hits);
    const uint32_t warps = gridDim.x * kCellWarps, groups = *A.group_count;
    if (kFirst && blockIdx.x == 0)
        for (uint32_t k = threadIdx.x; k < n_scenes; k += kCellBlock) A.policy_next[k] = decide(A.policy[k]);
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
    for (uint32_t c = blockIdx.x * kCellWarps + (threadIdx.x >> 5); c < groups; c += warps) {
        const uint32_t first = A.groups[c], key = A.keys[first], scene = scene_of(key, A.mbits);
        const SceneDev &S = A.scenes[scene];
        uint32_t cell;
        uint2 range = make_uint2(0, 0);
        if (neighbour_cell(S, morton_of(key, A.mbits), dx, dy, dz, cell) && lane < 27) range = __ldg(&A.cells[cell]);
        const uint32_t count = range.y > range.x ? range.y - range.x : 0u;
        const uint32_t end = min(__shfl_sync(0xffffffffu, range.y, 13), (first | A.group_mask) + 1);
        const uint32_t own = end > first ? end - first : 0u;  // at most 32
        float reach2 = r2max;
        if (kFirst) {
            const bool keep = decide(A.policy[scene]).keep != 0;
            if (keep) reach2 = A.skin_r2;
            if (lane == 0) A.lasting[c] = keep ? 1 : 0;
        } else {
            const bool lasts = A.lasting[c] != 0;
            const uint32_t m = count ? __ldg(&A.moved[range.x]) : 0u;
            const float bound = __uint_as_float(__shfl_sync(0xffffffffu, m, 13)) +
                                __uint_as_float(__reduce_max_sync(0xffffffffu, m));
            const bool skip = lasts && bound <= A.skin;
            if (count_use) {
                if (scene != seen_scene) {
                    report();
                    seen_scene = scene;
                }
                asked += own;
                if (skip) used += own;
            }
            if (skip) continue;
            if (lasts && lane == 0) A.lasting[c] = 0;
        }
        uint32_t upto = count;  // candidates up to and including the lane's cell
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, upto, d);
            if ((int)lane >= d) upto += v;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, upto, 31), from = upto - count;
        const bool obstacles = S.obstacles != 0;
        uint32_t found = 0;  // lane j: hits of the group's j-th particle
        for (uint32_t seg = 0; seg < total; seg += kHeldAll) {
            // candidates [seg, seg + 256): the lanes list their cells' indices, then each
            // takes every 32nd candidate
            __syncwarp();
            {
                const uint32_t lo = max(from, seg), hi = min(upto, seg + kHeldAll);
                uint32_t b = range.x + (lo - from);
                for (uint32_t k = lo; k < hi; ++k) sh.map[k - seg] = b++;
            }
            __syncwarp();
            uint32_t idx[kHeld];
            float X[kHeld], Y[kHeld], Z[kHeld];
#pragma unroll
            for (uint32_t q = 0; q < kHeld; ++q) {
                const uint32_t at = 32 * q + lane;
                X[q] = INFINITY, Y[q] = Z[q] = 0.f, idx[q] = 0;
                if (seg + at < total) {
                    idx[q] = sh.map[at];
                    const float4 p = __ldg(&ps[idx[q]]);
                    X[q] = p.x, Y[q] = p.y, Z[q] = p.z;
                }
            }
            // particle a against the first R candidates of every lane; the shared address
            // past its list
            auto test = [&](auto rounds, uint32_t a, uint32_t to) {
                const float4 pa = __ldg(&ps[a]);
#pragma unroll
                for (int q = 0; q < decltype(rounds)::value; ++q) {
                    const float ex = X[q] - pa.x, ey = Y[q] - pa.y, ez = Z[q] - pa.z;
                    append_hits(__fmaf_rn(ex, ex, __fmaf_rn(ey, ey, __fmaf_rn(ez, ez, -reach2))), idx[q], before, to);
                }
                return to;
            };
            const uint32_t held = min((total - seg + 31) >> 5, kHeld);
            for (uint32_t four = 0; four < own; four += kGroup) {
                const uint32_t earlier = found;  // hits of earlier segments
                const uint32_t last = min(four + kGroup, own);
                __syncwarp();
                auto each = [&](auto rounds) {
#pragma unroll 1
                    for (uint32_t j = four; j < last; ++j) {
                        if (obstacles && A.type[first + j] == FGB_TYPE_OBSTACLE) continue;  // no sums: an empty row
                        const uint32_t list = lists + 4 * (j - four) * kPitch, to = test(rounds, first + j, list);
                        if (lane < 3) fill(to + 4 * lane, A.none);
                        if (lane == j) found += (to - list) >> 2;
                    }
                };
                switch (held) {
                case 8: each(Rounds<8>{}); break;
                case 7: each(Rounds<7>{}); break;
                case 6: each(Rounds<6>{}); break;
                case 5: each(Rounds<5>{}); break;
                default: each(Rounds<4>{}); break;
                }
                __syncwarp();
                // the four's hits to their rows: lane 4 p + j takes quad p of the j-th
                const uint32_t j = four + (lane & 3u);
                const uint32_t lo = __shfl_sync(0xffffffffu, earlier, j),
                               hi = min(__shfl_sync(0xffffffffu, found, j), A.hcap);
                if (j >= own) continue;
                const uint32_t *have = sh.hits + (lane & 3u) * kPitch;
                uint4 *row = row_of(A, first + j);
                if (lo == 0) {
                    for (uint32_t e = 4 * (lane >> 2); e < hi; e += 32)
                        row[(e >> 2) * 32] = *reinterpret_cast<const uint4 *>(have + e);
                } else {  // a later segment, which starts within a quad
                    for (uint32_t e = lo + (lane >> 2); e < ((hi + 3u) & ~3u); e += 8)
                        reinterpret_cast<uint32_t *>(row + (e >> 2) * 32)[e & 3u] = have[e - lo];
                }
            }
        }
        if (lane < own) A.hcount[first + lane] = found > A.hcap ? kListOverflow : (uint16_t)found;
        if (A.over) {
            const unsigned full = __ballot_sync(0xffffffffu, lane < own && found > A.hcap);
            if (full && lane == 0) atomicAdd(A.over, (uint32_t)__popc(full));
        }
    }
    if (!kFirst && count_use) report();
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
// particles are consecutive) settle theirs first.  All lanes take part.
__device__ __forceinline__ void keep_moved(const RowArgs &A, bool have, uint32_t cell_start, float moved) {
    uint32_t m = have ? __float_as_uint(moved) : 0u;
    if (have && !(moved == moved)) m = 0x7f800000u;  // not a number: the bound has to fail
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t where = have ? cell_start : 0xffffffffu;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_down_sync(0xffffffffu, m, d), w = __shfl_down_sync(0xffffffffu, where, d);
        if (lane + d < 32 && w == where) m = max(m, o);
    }
    const uint32_t left = __shfl_up_sync(0xffffffffu, where, 1);
    if (have && (lane == 0 || left != where) && m) atomicMax(&A.moved[where], m);
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
        moved = sqrtf(ex * ex + ey * ey + ez * ez);
        cell_start = __ldg(&A.cells[S.table_base + morton_of(key, A.mbits)]).x;
    }
    if (PROFILE != kRef || !last) keep_moved(A, fluid, cell_start, moved);  // a search follows
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
    A.mass_range = s.mass_range;
    A.over = nullptr;
    A.ps_grid = s.ps_grid;
    A.moved = s.moved;
    A.lasting = s.lasting;
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
    if (pass == 0) {
        if (s.over) A.over = s.over + 1;  // counted once a step
        e = resident_grid(k_cell_rows<true>, s, kCellBlock, &grid);
        if (e != cudaSuccess) return e;
        k_cell_rows<true><<<grid, kCellBlock, 0, st>>>(A, ps, r2max, s.n_scenes, 0);
    } else {
        e = resident_grid(k_cell_rows<false>, s, kCellBlock, &grid);
        if (e != cudaSuccess) return e;
        k_cell_rows<false><<<grid, kCellBlock, 0, st>>>(A, ps, r2max, s.n_scenes, pass == 1);
    }
    return cudaGetLastError();
}

inline unsigned row_grid(const StepView &s) { return (s.n + 127) / 128; }

template <int PROFILE, bool kFast>
cudaError_t lambda_as(const StepView &s, const float4 *ps, int iteration, cudaStream_t st) {
    cudaError_t e = rows_of(s, ps, (uint32_t)iteration, st);
    if (e != cudaSuccess) return e;
    k_row_lambda<PROFILE, kFast><<<row_grid(s), 128, 0, st>>>(row_args(s), ps, s.lambda, s.density, s.plam);
    return cudaGetLastError();
}

template <int PROFILE, bool kFast>
cudaError_t delta_as(const StepView &s, const float4 *ps_in, float4 *ps_out, bool last, cudaStream_t st) {
    k_row_delta<PROFILE, kFast><<<row_grid(s), 128, 0, st>>>(row_args(s), ps_in, s.plam, ps_out, s.x1, s.v1,
                                                                  last ? 1 : 0, s.pv, s.hout);
    return cudaGetLastError();
}

template <bool kFast>
cudaError_t velocity_as(const StepView &s, const float4 *ps, cudaStream_t st, const std::function<void()> &between) {
    cudaError_t e = rows_of(s, ps, s.iterations, st);
    if (e != cudaSuccess) return e;
    const RowArgs A = row_args(s);
    k_row_vorticity<kFast><<<row_grid(s), 128, 0, st>>>(A, s.pv, s.omega, s.pom, s.vx);
    if (between) between();
    k_row_apply<kFast><<<row_grid(s), 128, 0, st>>>(A, ps, s.omega, s.pom, s.vx, s.v1, s.x1, s.hout);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_row_lambda(const StepView &s, const float4 *ps, int iteration, cudaStream_t st) {
    if (s.ph.profile == FGB_PROFILE_REF)
        return s.ph.fast_root ? lambda_as<FGB_PROFILE_REF, true>(s, ps, iteration, st)
                              : lambda_as<FGB_PROFILE_REF, false>(s, ps, iteration, st);
    return s.ph.fast_root ? lambda_as<FGB_PROFILE_BASELINE, true>(s, ps, iteration, st)
                          : lambda_as<FGB_PROFILE_BASELINE, false>(s, ps, iteration, st);
}

cudaError_t launch_row_delta(const StepView &s, const float4 *ps_in, float4 *ps_out, bool last, cudaStream_t st) {
    if (s.ph.profile == FGB_PROFILE_REF)
        return s.ph.fast_root ? delta_as<FGB_PROFILE_REF, true>(s, ps_in, ps_out, last, st)
                              : delta_as<FGB_PROFILE_REF, false>(s, ps_in, ps_out, last, st);
    return s.ph.fast_root ? delta_as<FGB_PROFILE_BASELINE, true>(s, ps_in, ps_out, last, st)
                          : delta_as<FGB_PROFILE_BASELINE, false>(s, ps_in, ps_out, last, st);
}

cudaError_t launch_row_velocity_terms(const StepView &s, const float4 *ps, cudaStream_t st,
                                       const std::function<void()> &between) {
    return s.ph.fast_root ? velocity_as<true>(s, ps, st, between) : velocity_as<false>(s, ps, st, between);
}

// Particles of a group: small scenes have too few cells to fill the GPU, and the ref
// profile's constants clump the fluid into few crowded ones, so a cell's particles go to
// several warps.
uint32_t row_group_mask(int profile, uint64_t n) {
    return n < 24000 ? 3u : profile == FGB_PROFILE_REF ? 7u : 31u;
}

}  // namespace fgb
