// weld.cu -- vertex welding of a triangle soup (an index buffer for rendering).
//
// Reference: geometry::indexVBO2 (include/fluid/geometry.hpp:152-166, unused by the
// solver): the vertices v0, v1, v2 of each triangle in order; a vertex whose
// position is byte-identical to an earlier one (PackedVertex compares with memcmp,
// geometry.hpp:81-88) takes that one's index, otherwise it is appended.  So the
// output is the distinct positions in order of first appearance, and every input
// vertex's index is the rank of its position's first appearance.
//
// On the device, order-free and deterministic:
//   k_weld_insert  each vertex i inserts its 12-byte position into an open-
//                  addressing table (a slot holds the index of the vertex that
//                  claimed it; keys are compared through the input positions) and
//                  lowers the slot's `first` to i with atomicMin
//   k_weld_first   first[i] = the minimum index of i's position; flag[i] = first == i
//   scan           rank of each flagged vertex (scan.cu)
//   k_weld_emit    index[i] = rank[first[i]], vertices[rank[i]] = position i if flagged
// The reference stores indices as unsigned short, which wraps after 65 535 distinct
// vertices; these are 32-bit.
#include <cstring>
#include <cuda_runtime.h>
#include <map>
#include <mutex>

#include "fgb_internal.h"

namespace fgb {
namespace {

constexpr uint32_t kEmpty = 0xffffffffu;

// Position of vertex i: triangle i / 3, corner i % 3, in the 21-word triangle record.
__device__ __forceinline__ uint3 vertex_bits(const float *tris, uint64_t i) {
    const float *p = tris + 21 * (i / 3) + 3 * (i % 3);
    return make_uint3(__float_as_uint(p[0]), __float_as_uint(p[1]), __float_as_uint(p[2]));
}

__device__ __forceinline__ uint32_t hash3(uint3 k) {
    uint32_t h = k.x * 0x9E3779B1u;
    h ^= (k.y + 0x7F4A7C15u + (h << 6) + (h >> 2)) * 0x85EBCA77u;
    h ^= (k.z + 0x165667B1u + (h << 6) + (h >> 2)) * 0xC2B2AE3Du;
    return h ^ (h >> 15);
}

__global__ void k_weld_insert(const float *__restrict__ tris, uint64_t nv, uint32_t mask, uint32_t *owner,
                              uint32_t *first, uint32_t *slot_of, uint32_t *err) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint3 key = vertex_bits(tris, i);
        uint32_t h = hash3(key) & mask;
        bool placed = false;
        // the table has at least twice as many slots as vertices, so a free or
        // matching slot is found within mask + 1 probes
        for (uint32_t probe = 0; probe <= mask; ++probe, h = (h + 1) & mask) {
            uint32_t o = atomicCAS(&owner[h], kEmpty, (uint32_t)i);
            if (o != kEmpty) {
                const uint3 other = vertex_bits(tris, o);
                if (other.x != key.x || other.y != key.y || other.z != key.z) continue;
            }
            atomicMin(&first[h], (uint32_t)i);
            slot_of[i] = h;
            placed = true;
            break;
        }
        if (!placed) {  // unreachable at load <= 1/2; keeps later passes in bounds
            slot_of[i] = 0;
            raise_error(err, ERR_WELD_TABLE);
        }
    }
}

__global__ void k_weld_first(uint64_t nv, const uint32_t *__restrict__ first, const uint32_t *__restrict__ slot_of,
                             uint32_t *__restrict__ first_of, uint32_t *__restrict__ flag) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t f = first[slot_of[i]];
        if (f > (uint32_t)i) f = (uint32_t)i;  // only after a table error: keep indices in range
        first_of[i] = f;
        flag[i] = f == (uint32_t)i ? 1u : 0u;
    }
}

__global__ void k_weld_emit(const float *__restrict__ tris, uint64_t nv, const uint32_t *__restrict__ first_of,
                            const uint32_t *__restrict__ flag, const uint32_t *__restrict__ rank,
                            uint32_t *__restrict__ index, float *__restrict__ vertices) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += (uint64_t)gridDim.x * blockDim.x) {
        index[i] = rank[first_of[i]];
        if (flag[i]) {
            const float *p = tris + 21 * (i / 3) + 3 * (i % 3);
            float *o = vertices + 3 * (uint64_t)rank[i];
            o[0] = p[0];
            o[1] = p[1];
            o[2] = p[2];
        }
    }
}

// Device memory of the welds: a pool of the driver's stream-ordered allocator per device, which
// keeps at most kKeep bytes between welds until the next solver is destroyed.  (Twelve
// cudaMalloc and cudaFree took 340 us of a weld of 36 k triangles, 600 us; its kernels take
// 35.)
constexpr uint64_t kKeep = 64ull << 20;

struct Pools {
    std::mutex mutex;
    std::map<int, cudaMemPool_t> of_device;
};
Pools &pools() {
    static Pools *p = new Pools;  // never destroyed: solvers may be at exit
    return *p;
}

// The current device's pool (null: it has none).
cudaMemPool_t device_pool() {
    int dev = 0, supported = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    Pools &ps = pools();
    std::lock_guard<std::mutex> lock(ps.mutex);
    const auto it = ps.of_device.find(dev);
    if (it != ps.of_device.end()) return it->second;
    cudaMemPool_t pool = nullptr;
    if (cudaDeviceGetAttribute(&supported, cudaDevAttrMemoryPoolsSupported, dev) == cudaSuccess && supported) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        uint64_t keep = kKeep;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess ||
            cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess)
            pool = nullptr;
    }
    return ps.of_device[dev] = pool;
}

// Memory for several arrays, given back in the stream's order.
class Workspace {
public:
    explicit Workspace(cudaStream_t st) : st_(st), pool_(device_pool()) {}
    Workspace(const Workspace &) = delete;
    ~Workspace() {
        if (!base_) return;
        if (pool_) cudaFreeAsync(base_, st_);
        else cudaFree(base_);
    }
    template <class T>
    void want(T *&p, uint64_t n) {
        parts_[count_++] = Part{(void **)&p, size_};
        size_ += ((n ? n : 1) * sizeof(T) + 255) & ~255ull;
    }
    cudaError_t alloc() {
        const cudaError_t e =
            pool_ ? cudaMallocFromPoolAsync((void **)&base_, size_, pool_, st_) : cudaMalloc((void **)&base_, size_);
        for (int i = 0; e == cudaSuccess && i < count_; ++i) *parts_[i].p = base_ + parts_[i].at;
        return e;
    }

private:
    struct Part {
        void **p;
        uint64_t at;
    };
    cudaStream_t st_;
    cudaMemPool_t pool_;
    char *base_ = nullptr;
    uint64_t size_ = 0;
    Part parts_[12];
    int count_ = 0;
};

unsigned grid_of(uint64_t n) {
    uint64_t g = (n + 255) / 256;
    if (g > 152u * 8u) g = 152u * 8u;
    return g ? (unsigned)g : 1u;
}

}  // namespace

// Weld the triangles at device address d_tris (21-word records).  Indices (3 per
// triangle) and the distinct vertices (3 floats each, at most 3 n) go to device
// memory; the vertex count to *n_vertices.
int weld_device(const fgb_mesh_triangle *d_tris, uint64_t n_tris, uint32_t *d_index, float *d_vertices,
                uint64_t *n_vertices, cudaStream_t st) {
    const uint64_t nv = 3 * n_tris;
    *n_vertices = 0;
    if (!nv) return FGB_OK;
    if (nv > 0x7fffffffull) return fail(FGB_ERR_CAPACITY, "weld: more than 2^31 vertices");
    uint64_t slots = 1;
    while (slots < 2 * nv) slots <<= 1;
    const float *tris = reinterpret_cast<const float *>(d_tris);
    uint32_t *owner, *first, *slot_of, *first_of, *flag, *rank, *total;  // total: and the error flags
    char *scratch;
    const uint64_t sb = scan_u32_scratch_bytes(nv);
    Workspace space(st);
    space.want(owner, slots);
    space.want(first, slots);
    space.want(slot_of, nv);
    space.want(first_of, nv);
    space.want(flag, nv);
    space.want(rank, nv);
    space.want(total, 2);
    space.want(scratch, sb);
    cudaError_t e = space.alloc();
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(FGB_ERR_OOM, "weld: scratch allocation failed");
    }
    uint32_t *err = total + 1;
    e = cudaMemsetAsync(owner, 0xff, slots * sizeof(uint32_t), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(first, 0xff, slots * sizeof(uint32_t), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(err, 0, sizeof(uint32_t), st);
    if (e != cudaSuccess) return fail_cuda(e, "weld: clear");
    k_weld_insert<<<grid_of(nv), 256, 0, st>>>(tris, nv, (uint32_t)(slots - 1), owner, first, slot_of, err);
    k_weld_first<<<grid_of(nv), 256, 0, st>>>(nv, first, slot_of, first_of, flag);
    e = scan_u32(flag, rank, total, nv, scratch, sb, st, err, nullptr);
    if (e == cudaSuccess) {
        k_weld_emit<<<grid_of(nv), 256, 0, st>>>(tris, nv, first_of, flag, rank, d_index, d_vertices);
        e = cudaGetLastError();
    }
    uint32_t result[2] = {0, 0};
    if (e == cudaSuccess) e = cudaMemcpyAsync(result, total, sizeof result, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail_cuda(e, "weld");
    const uint32_t t = result[0], flags = result[1];
    if (flags) return fail(FGB_ERR_TIMEOUT, "weld: a device-side bound was hit (error flag set)");
    *n_vertices = t;
    return FGB_OK;
}

// What the welds' pools keep, back to the device (a solver is being destroyed).
void weld_release() {
    Pools &ps = pools();
    std::lock_guard<std::mutex> lock(ps.mutex);
    for (auto &p : ps.of_device)
        if (p.second) cudaMemPoolTrimTo(p.second, 0);
}

}  // namespace fgb

using fgb::fail;

extern "C" {

int fgb_weld_mesh(const fgb_mesh *mesh, uint32_t *indices, float *vertices, uint64_t *n_vertices) {
    if (!mesh || !n_vertices) return fail(FGB_ERR_INVALID, "weld_mesh: null argument");
    *n_vertices = 0;
    const uint64_t n = mesh->n, nv = 3 * n;
    if (!n) return FGB_OK;
    if (!mesh->triangles || !indices || !vertices) return fail(FGB_ERR_INVALID, "weld_mesh: null array");
    cudaStream_t st = nullptr;
    cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e != cudaSuccess) return fgb::fail_cuda(e, "weld_mesh: stream");
    int rc = FGB_OK;
    uint64_t count = 0;
    {
        fgb_mesh_triangle *tris = nullptr;
        uint32_t *idx = nullptr;
        float *verts = nullptr;
        fgb::Workspace space(st);
        space.want(tris, n);
        space.want(idx, nv);
        space.want(verts, 3 * nv);
        if (space.alloc() != cudaSuccess) {
            cudaGetLastError();
            rc = fail(FGB_ERR_OOM, "weld_mesh: allocation failed");
        }
        if (!rc) {
            e = cudaMemcpyAsync(tris, mesh->triangles, n * sizeof(fgb_mesh_triangle), cudaMemcpyHostToDevice, st);
            if (e != cudaSuccess) rc = fgb::fail_cuda(e, "weld_mesh: upload");
        }
        if (!rc) rc = fgb::weld_device(tris, n, idx, verts, &count, st);
        if (!rc) {
            fgb::ready_output(indices, nv * sizeof(uint32_t));
            fgb::ready_output(vertices, 3 * count * sizeof(float));
            e = cudaMemcpyAsync(indices, idx, nv * sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess && count)
                e = cudaMemcpyAsync(vertices, verts, 3 * count * sizeof(float), cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
            if (e != cudaSuccess) rc = fgb::fail_cuda(e, "weld_mesh: download");
        }
    }
    cudaStreamSynchronize(st);
    cudaStreamDestroy(st);
    if (!rc) *n_vertices = count;
    return rc;
}

int fgb_batch_weld_surface(fgb_batch *b, uint32_t scene, uint32_t *indices, float *vertices, uint64_t *n_vertices) {
    if (!n_vertices) return fail(FGB_ERR_INVALID, "weld_surface: null count");
    *n_vertices = 0;
    fgb::ResidentScene r;
    int rc = fgb::batch_resident(b, scene, &r);
    if (rc) return rc;
    if (!r.tris) return fail(FGB_ERR_INVALID, "weld_surface: call fgb_batch_surface_all first");
    const uint64_t nv = 3 * r.tri_count;
    if (!nv) return FGB_OK;
    if (!indices || !vertices) return fail(FGB_ERR_INVALID, "weld_surface: null array");
    uint32_t *idx = nullptr;
    float *verts = nullptr;
    fgb::Workspace space(r.stream);
    space.want(idx, nv);
    space.want(verts, 3 * nv);
    if (space.alloc() != cudaSuccess) {
        cudaGetLastError();
        return fail(FGB_ERR_OOM, "weld_surface: allocation failed");
    }
    uint64_t count = 0;
    rc = fgb::weld_device(r.tris, r.tri_count, idx, verts, &count, r.stream);
    if (rc) return rc;
    fgb::ready_output(indices, nv * sizeof(uint32_t));
    fgb::ready_output(vertices, 3 * count * sizeof(float));
    cudaError_t e = cudaMemcpyAsync(indices, idx, nv * sizeof(uint32_t), cudaMemcpyDeviceToHost, r.stream);
    if (e == cudaSuccess && count)
        e = cudaMemcpyAsync(vertices, verts, 3 * count * sizeof(float), cudaMemcpyDeviceToHost, r.stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(r.stream);
    if (e != cudaSuccess) return fgb::fail_cuda(e, "weld_surface: download");
    *n_vertices = count;
    return FGB_OK;
}

}  // extern "C"
