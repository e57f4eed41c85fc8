// pbf_sums.cuh -- the pair sums of the gather passes and what each particle does with
// them, shared by the row kernels (rows.cu) and the list kernels (pbf.cu).
//
// Every sum adds its neighbours in the order it is given them, with the reference's
// formulas; both kernel families visit the same neighbours in the same order, so they
// compute the same bits.
#pragma once

#include "fgb_internal.h"

namespace fgb {

constexpr int kRef = FGB_PROFILE_REF;

// Squared distance of a pair in the baseline profile's gathers: two fused
// multiply-adds, as the oracle's baseline restatement computes it (the ref profile
// keeps the reference's sum of three products).
__device__ __forceinline__ float dist2(float dx, float dy, float dz) {
    return __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
}

__device__ __forceinline__ float corr_pow(float ratio, float n) {
    if (n == 4.f) {
        const float r2 = ratio * ratio;
        return r2 * r2;
    }
    return powf(ratio, n);
}

__device__ __forceinline__ float dot3(const float *a, const float *b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }

// oclsph_collision.h:7-58 (first containing triangle within 40 world units wins).
__device__ inline void collide_triangles(const TriDev *__restrict__ tris, uint32_t first, uint32_t count, float *pos,
                                  float *vel) {
    for (uint32_t i = 0; i < count; ++i) {
        const TriDev t = tris[first + i];
        float e1[3], e2[3], nrm[3];
        for (int a = 0; a < 3; ++a) {
            e1[a] = t.b[a] - t.a[a];
            e2[a] = t.c[a] - t.a[a];
        }
        nrm[0] = e1[1] * e2[2] - e1[2] * e2[1];
        nrm[1] = e1[2] * e2[0] - e1[0] * e2[2];
        nrm[2] = e1[0] * e2[1] - e1[1] * e2[0];
        const float len = sqrtf(dot3(nrm, nrm));
        const float nn[3] = {nrm[0] / len, nrm[1] / len, nrm[2] / len};
        const float dist = dot3(nn, t.a) - dot3(nn, pos);
        if (-40.f <= dist && dist <= 40.f) {
            const float p0[3] = {pos[0] + nn[0] * dist, pos[1] + nn[1] * dist, pos[2] + nn[2] * dist};
            float v0[3], v1[3], v2[3];
            for (int a = 0; a < 3; ++a) {
                v0[a] = t.c[a] - t.a[a];
                v1[a] = t.b[a] - t.a[a];
                v2[a] = p0[a] - t.a[a];
            }
            const float d00 = dot3(v0, v0), d01 = dot3(v0, v1), d02 = dot3(v0, v2);
            const float d11 = dot3(v1, v1), d12 = dot3(v1, v2);
            const float inv = 1.f / (d00 * d11 - d01 * d01);
            const float u = (d11 * d02 - d01 * d12) * inv;
            const float w = (d00 * d12 - d01 * d02) * inv;
            if ((u >= 0.f) && (w >= 0.f) && (u + w < 1.f)) {
                const float vn = dot3(vel, nn);
                for (int a = 0; a < 3; ++a) {
                    vel[a] = vel[a] - (nn[a] * 2.f) * vn;
                    pos[a] = p0[a];
                }
                return;
            }
        }
    }
}

__device__ __forceinline__ void collide_sphere(const SceneDev &S, float *pos) {
    if (!S.sphere_enabled) return;
    const float d[3] = {pos[0] - S.sphere[0], pos[1] - S.sphere[1], pos[2] - S.sphere[2]};
    const float r = S.sphere[3];
    const float d2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
    if (!(d2 < r * r)) return;
    const float dist = sqrtf(d2);
    if (dist > 0.f) {
        const float s = r / dist;
        for (int a = 0; a < 3; ++a) pos[a] = S.sphere[a] + d[a] * s;
    } else {
        pos[0] = S.sphere[0];
        pos[1] = S.sphere[1] + r;
        pos[2] = S.sphere[2];
    }
}


// Final position and velocity of particle a into the caller's arrays (fgb_advance
// with direct host I/O): the step's last kernel stores them beside its own writes.
__device__ __forceinline__ void store_host_motion(const HostParticlesOut *__restrict__ hout, uint32_t a,
                                                  const float4 &xa, const float4 &va) {
    if (!hout) return;
    const uint32_t stride = hout->stride;  // 0: packed arrays, else the caller's records
    float *pp = hout->position, *pv = hout->velocity;
    if (pp) {
        float *q = stride ? (float *)((char *)pp + (size_t)a * stride) : pp + 3 * (size_t)a;
        q[0] = xa.x;
        q[1] = xa.y;
        q[2] = xa.z;
    }
    if (pv) {
        float *q = stride ? (float *)((char *)pv + (size_t)a * stride) : pv + 3 * (size_t)a;
        q[0] = va.x;
        q[1] = va.y;
        q[2] = va.z;
    }
}

__device__ __forceinline__ void cross3(const float *a, const float *b, float *o) {
    o[0] = a[1] * b[2] - a[2] * b[1];
    o[1] = a[2] * b[0] - a[0] * b[2];
    o[2] = a[0] * b[1] - a[1] * b[0];
}


// A value for each of two neighbours.  The pair form lets their roots and quotients run
// beside each other.  (The packed add, mul and fma of two floats issue at half the rate of
// the scalar ones here, 1.65 against 3.73 a clock and SM, and their register pairs cost
// moves: the delta pass takes 112 us with scalar operations and 117 with packed ones, and
// ptxas fuses a packed product with the sum that follows, which changes its bits.)
struct Two {
    float a, b;
    __device__ __forceinline__ Two() {}
    __device__ __forceinline__ Two(float a_, float b_) : a(a_), b(b_) {}
    __device__ __forceinline__ explicit Two(float v) : a(v), b(v) {}
    __device__ __forceinline__ float lo() const { return a; }
    __device__ __forceinline__ float hi() const { return b; }
};
__device__ __forceinline__ Two operator-(const Two &x, const Two &y) { return Two(x.a - y.a, x.b - y.b); }
__device__ __forceinline__ Two operator+(const Two &x, const Two &y) { return Two(x.a + y.a, x.b + y.b); }
__device__ __forceinline__ Two operator*(const Two &x, const Two &y) { return Two(x.a * y.a, x.b * y.b); }
__device__ __forceinline__ Two operator-(const Two &x) { return Two(-x.a, -x.b); }
__device__ __forceinline__ Two fma(const Two &x, const Two &y, const Two &z) {
    return Two(__fmaf_rn(x.a, y.a, z.a), __fmaf_rn(x.b, y.b, z.b));
}
__device__ __forceinline__ float fma(float x, float y, float z) { return __fmaf_rn(x, y, z); }
// r^2 of a pair of neighbours, as dist2
__device__ __forceinline__ Two dist2(const Two &dx, const Two &dy, const Two &dz) {
    return fma(dx, dx, fma(dy, dy, dz * dz));
}

__device__ __forceinline__ float rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ Two rsqrt_approx(const Two &x) { return Two(rsqrt_approx(x.a), rsqrt_approx(x.b)); }
__device__ __forceinline__ float ieee_root(float x) { return sqrtf(x); }
__device__ __forceinline__ Two ieee_root(const Two &x) { return Two(sqrtf(x.a), sqrtf(x.b)); }
__device__ __forceinline__ float ieee_div(float x, float y) { return x / y; }
__device__ __forceinline__ Two ieee_div(const Two &x, const Two &y) { return Two(x.a / y.a, x.b / y.b); }

// Of a neighbour, or a pair of them (T: float or Two), at squared distances q2 <= h^2: r = sqrt(q2) and
// s = (h - r)^2 / r, both correctly rounded -- the bits of sqrtf and of the division.
//
// kFast (Phys::fast_root): one approximate reciprocal square root y serves both.  A
// Newton step on q2 y gives the root, a Newton step on y the reciprocal of r, and the
// quotient is corrected by its exact remainder (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990: with the correctly rounded
// reciprocal and a faithful quotient the corrected quotient is correctly rounded).  The
// reciprocal's error is below 2^-43 before its rounding, so it can be misrounded only for
// the few mantissas whose reciprocals lie that near the midpoint of two floats; the host
// checks the quotients of those for the solver's h (fast_root.h) and
// clears fast_root if one fails.  17 operations a neighbour, where the compiler's
// root and quotient take about 30 with their range checks.
// Below q2 = 1e-30 (only there does the approximation leave the normal range) r is
// meaningless; its users drop s below eps_r2.
template <bool kFast, class T>
__device__ __forceinline__ void root_and_spiky(const Phys &ph, const T &q2, T &r, T &s) {
    if constexpr (kFast) {
        const T y = rsqrt_approx(q2);
        const T g = q2 * y;
        r = fma(fma(-g, g, q2), y * T(0.5f), g);
        const T hr = T(ph.h) - r, a = hr * hr, nr = -r;
        const T inv = fma(fma(nr, y, T(1.f)), y, y);
        const T w = a * inv;
        s = fma(fma(nr, w, a), inv, w);
    } else {
        r = ieee_root(q2);
        const T hr = T(ph.h) - r;
        s = ieee_div(hr * hr, r);
    }
}

// a / c of a pair, correctly rounded, for a constant c with inv_c = 1 / c correctly rounded.
// kFast: Markstein's correction again; a is zero or within 2^+-90 (else the division).
template <bool kFast, class T>
__device__ __forceinline__ T over_const(const T &a, float c, float inv_c) {
    if constexpr (kFast) {
        const T w = a * T(inv_c);
        return fma(fma(T(-c), w, a), T(inv_c), w);
    }
    return ieee_div(a, T(c));
}

// The sums add their neighbours' terms with `add2`, two neighbours a thread, or from where
// `terms` of one neighbour each have left them (rows.cu: a particle's four lanes).

// Density and constraint gradients of one particle (oclsph_kernel.h:305-346).
template <int PROFILE>
struct LambdaSum {
    float rho = 0.f, gx = 0.f, gy = 0.f, gz = 0.f, g2 = 0.f;

    __device__ __forceinline__ void add(const Phys &ph, const float4 &pa, float bx, float by, float bz, float mb) {
        const float dx = pa.x - bx, dy = pa.y - by, dz = pa.z - bz;
        if (PROFILE == kRef) {
            const float r2 = dx * dx + dy * dy + dz * dz;
            if (!(r2 <= ph.hh_le)) return;  // sqrtf(r2) > h: no contribution
            const float r = sqrtf(r2);
            if (r <= ph.h) {
                const float t = ph.hh - r * r;
                rho = __fmaf_rn(pa.w, ph.poly6f * (t * t * t), rho);
                if (r >= kKernelEpsilon) {
                    const float hr = ph.h - r;
                    const float sc = ph.spikyf * ((hr * hr) / r);
                    gx = __fmaf_rn(dx * sc, ph.inv_rho0, gx);
                    gy = __fmaf_rn(dy * sc, ph.inv_rho0, gy);
                    gz = __fmaf_rn(dz * sc, ph.inv_rho0, gz);
                }
            }
        } else {
            const float q2 = dist2(dx, dy, dz);
            if (q2 <= ph.hh) {
                const float t = ph.hh - q2;
                rho = __fmaf_rn(mb, t * t * t, rho);
                const float r = sqrtf(q2);
                if (r >= kKernelEpsilon) {
                    const float hr = ph.h - r;
                    const float sc = mb * ((hr * hr) / r);
                    gx = __fmaf_rn(sc, dx, gx);
                    gy = __fmaf_rn(sc, dy, gy);
                    gz = __fmaf_rn(sc, dz, gz);
                    g2 = __fmaf_rn(sc * sc, q2, g2);
                }
            }
        }
    }

    // a neighbour's (or two neighbours') share.  baseline: w = t^3, s = m (h - r)^2 / r, ss = s^2
    // and the difference; ref: w its density, x, y, z the gradient's share but for 1 / rho0
    template <class T>
    struct Terms {
        T q2, w, s, ss, x, y, z;
    };
    template <bool kFast, class T>
    static __device__ __forceinline__ Terms<T> terms(const Phys &ph, const float4 &pa, const T &bx, const T &by,
                                                     const T &bz, const T &mb) {
        Terms<T> o;
        const T dx = T(pa.x) - bx, dy = T(pa.y) - by, dz = T(pa.z) - bz;
        T r, s;
        if (PROFILE == kRef) {
            o.q2 = (dx * dx + dy * dy) + dz * dz;
            root_and_spiky<kFast>(ph, o.q2, r, s);
            const T t = T(ph.hh) - r * r, sc = T(ph.spikyf) * s;
            o.w = T(ph.poly6f) * (t * t * t);
            o.x = dx * sc, o.y = dy * sc, o.z = dz * sc;
        } else {
            o.q2 = dist2(dx, dy, dz);
            root_and_spiky<kFast>(ph, o.q2, r, s);
            const T t = T(ph.hh) - o.q2;
            o.w = t * t * t;
            o.s = mb * s;
            o.ss = o.s * o.s;
            o.x = dx, o.y = dy, o.z = dz;
        }
        return o;
    }

    // two neighbours in order; r^2 above h^2 (a point at infinity) adds nothing
    template <bool kFast>
    __device__ __forceinline__ void add2(const Phys &ph, const float4 &pa, const Two &bx, const Two &by, const Two &bz,
                                         const Two &mb) {
        const Terms<Two> t = terms<kFast>(ph, pa, bx, by, bz, mb);
        if (PROFILE == kRef) {
            one<kFast>(ph, pa, t.q2.lo(), t.w.lo(), t.x.lo(), t.y.lo(), t.z.lo());
            one<kFast>(ph, pa, t.q2.hi(), t.w.hi(), t.x.hi(), t.y.hi(), t.z.hi());
        } else {
            one(ph, t.q2.lo(), mb.lo(), t.w.lo(), t.s.lo(), t.ss.lo(), t.x.lo(), t.y.lo(), t.z.lo());
            one(ph, t.q2.hi(), mb.hi(), t.w.hi(), t.s.hi(), t.ss.hi(), t.x.hi(), t.y.hi(), t.z.hi());
        }
    }
    __device__ __forceinline__ void one(const Phys &ph, float q2, float m, float w, float sc, float ss, float dx,
                                        float dy, float dz) {
        if (q2 <= ph.hh) {
            rho = __fmaf_rn(m, w, rho);
            if (q2 >= ph.eps_r2) {
                gx = __fmaf_rn(sc, dx, gx);
                gy = __fmaf_rn(sc, dy, gy);
                gz = __fmaf_rn(sc, dz, gz);
                g2 = __fmaf_rn(ss, q2, g2);
            }
        }
    }
    template <bool kFast>
    __device__ __forceinline__ void one(const Phys &ph, const float4 &pa, float q2, float w, float kx, float ky,
                                        float kz) {
        if (!(q2 <= ph.hh_le)) return;
        if (kFast && q2 < ph.eps_r2) w = on_top(ph);
        rho = __fmaf_rn(pa.w, w, rho);
        if (q2 >= ph.eps_r2) {
            gx = __fmaf_rn(kx, ph.inv_rho0, gx);
            gy = __fmaf_rn(ky, ph.inv_rho0, gy);
            gz = __fmaf_rn(kz, ph.inv_rho0, gz);
        }
    }

    // the density of two particles on top of each other, at fast_root's h: r^2 vanishes beside
    // h^2 (and the fast root of r^2 below 1e-30 is meaningless)
    static __device__ __forceinline__ float on_top(const Phys &ph) { return ph.poly6f * (ph.hh * ph.hh * ph.hh); }

    // lambda, and the density in *dens
    __device__ __forceinline__ float finish(const Phys &ph, float *dens) const {
        if (PROFILE == kRef) {
            *dens = rho;
            const float norm2 = gx * gx + gy * gy + gz * gz;
            const float C = rho / ph.rho0 - 1.f;
            return -C / (norm2 + ph.cfm);
        }
        *dens = rho * ph.poly6f;
        const float gs = ph.spikyf * ph.inv_rho0;
        const float sx = gx * gs, sy = gy * gs, sz = gz * gs;
        const float denom = (sx * sx + sy * sy + sz * sz) + g2 * (gs * gs);
        const float C = *dens * ph.inv_rho0 - 1.f;
        return -C / (denom + ph.cfm);
    }
};

// Position correction of one particle (oclsph_kernel.h:348-384).
template <int PROFILE>
struct DeltaSum {
    float px = 0.f, py = 0.f, pz = 0.f;

    // la: the particle's lambda; lam_b(): the neighbour's
    template <class L>
    __device__ __forceinline__ void add(const Phys &ph, const float4 &pa, float la, float bx, float by, float bz,
                                        L &&lam_b, float mb) {
        const float dx = pa.x - bx, dy = pa.y - by, dz = pa.z - bz;
        if (PROFILE == kRef) {
            const float r2 = dx * dx + dy * dy + dz * dz;
            if (!(r2 <= ph.hh_le)) return;  // sqrtf(r2) > h: no contribution
            const float r = sqrtf(r2);
            float w = 0.f;
            if (r <= ph.h) {
                const float t = ph.hh - r * r;
                w = ph.poly6f * (t * t * t);
            }
            const float corr = -ph.corr_k * corr_pow(w / ph.corr_ref, ph.corr_n);
            const float factor = (la + lam_b() + corr) / ph.rho0;
            if (r >= kKernelEpsilon && r <= ph.h) {
                const float hr = ph.h - r;
                const float sc = ph.spikyf * ((hr * hr) / r);
                px = __fmaf_rn(dx * sc, factor, px);
                py = __fmaf_rn(dy * sc, factor, py);
                pz = __fmaf_rn(dz * sc, factor, pz);
            }
        } else {
            const float q2 = dist2(dx, dy, dz);
            if (q2 <= ph.hh) {
                const float r = sqrtf(q2);
                if (r >= kKernelEpsilon) {
                    const float t = ph.hh - q2;
                    const float corr = -ph.corr_k * corr_pow((t * t * t) * ph.inv_corr_wdq, ph.corr_n);
                    const float hr = ph.h - r;
                    const float sc = mb * ((hr * hr) / r) * (la + lam_b() + corr);
                    px = __fmaf_rn(sc, dx, px);
                    py = __fmaf_rn(sc, dy, py);
                    pz = __fmaf_rn(sc, dz, pz);
                }
            }
        }
    }

    // a neighbour's (or two neighbours') share: f times (x, y, z)
    template <class T>
    struct Terms {
        T q2, f, x, y, z;
    };
    template <bool kFast, class T>
    static __device__ __forceinline__ Terms<T> terms(const Phys &ph, const float4 &pa, float la, const T &bx,
                                                     const T &by, const T &bz, const T &lb, const T &mb) {
        Terms<T> o;
        const T dx = T(pa.x) - bx, dy = T(pa.y) - by, dz = T(pa.z) - bz;
        T r, s;
        if (PROFILE == kRef) {
            o.q2 = (dx * dx + dy * dy) + dz * dz;
            root_and_spiky<kFast>(ph, o.q2, r, s);
            const T t = T(ph.hh) - r * r, w = T(ph.poly6f) * (t * t * t);
            const T c = T(-ph.corr_k) * corr<kFast>(ph, over_const<kFast>(w, ph.corr_ref, ph.inv_corr_ref));
            const T sum = (T(la) + lb) + c;
            o.f = over_const<kFast>(sum, ph.rho0, ph.inv_rho0);
            // outside over_const's range (a sum that cancelled, or one that ran away)
            if (kFast && out_of_range(ph, o.q2, sum)) o.f = ieee_div(sum, T(ph.rho0));
            const T sc = T(ph.spikyf) * s;
            o.x = dx * sc, o.y = dy * sc, o.z = dz * sc;
        } else {
            o.q2 = dist2(dx, dy, dz);
            root_and_spiky<kFast>(ph, o.q2, r, s);
            const T t = T(ph.hh) - o.q2;
            const T c = T(-ph.corr_k) * corr<kFast>(ph, (t * t * t) * T(ph.inv_corr_wdq));
            o.f = mb * s * ((T(la) + lb) + c);
            o.x = dx, o.y = dy, o.z = dz;
        }
        return o;
    }
    static __device__ __forceinline__ bool in_range(const Phys &ph, float q2) {
        return q2 <= (PROFILE == kRef ? ph.hh_le : ph.hh) && q2 >= ph.eps_r2;
    }
    static __device__ __forceinline__ bool out_of_range(const Phys &ph, float q2, float sum) {
        return q2 <= ph.hh_le && !(fabsf(sum) > 1e-27f && fabsf(sum) < 1e27f);
    }
    static __device__ __forceinline__ bool out_of_range(const Phys &ph, const Two &q2, const Two &sum) {
        return out_of_range(ph, q2.lo(), sum.lo()) || out_of_range(ph, q2.hi(), sum.hi());
    }

    // two neighbours in order, their lambdas in lb
    template <bool kFast>
    __device__ __forceinline__ void add2(const Phys &ph, const float4 &pa, float la, const Two &bx, const Two &by,
                                         const Two &bz, const Two &lb, const Two &mb) {
        const Terms<Two> t = terms<kFast>(ph, pa, la, bx, by, bz, lb, mb);
        if (in_range(ph, t.q2.lo())) move_by(t.f.lo(), t.x.lo(), t.y.lo(), t.z.lo());
        if (in_range(ph, t.q2.hi())) move_by(t.f.hi(), t.x.hi(), t.y.hi(), t.z.hi());
    }
    __device__ __forceinline__ void move_by(float f, float kx, float ky, float kz) {
        px = __fmaf_rn(kx, f, px);
        py = __fmaf_rn(ky, f, py);
        pz = __fmaf_rn(kz, f, pz);
    }
    // corr_pow (fast_root asks for the fourth power)
    template <bool kFast, class T>
    static __device__ __forceinline__ T corr(const Phys &ph, const T &ratio) {
        if constexpr (kFast) {
            const T r2 = ratio * ratio;
            return r2 * r2;
        }
        return power(ratio, ph.corr_n);
    }
    static __device__ __forceinline__ float power(float ratio, float n) { return corr_pow(ratio, n); }
    static __device__ __forceinline__ Two power(const Two &ratio, float n) {
        return Two(corr_pow(ratio.lo(), n), corr_pow(ratio.hi(), n));
    }

    // The corrected p* after the colliders and the bounds (solver units) in q[3], and
    // the particle's velocity as they leave it (va: as stored, vel: after a triangle).
    __device__ __forceinline__ void move(const Phys &ph, const SceneDev &S, const TriDev *tris, const float4 &pa,
                                         uint32_t a, float4 *__restrict__ v, float *q, float4 &va, float *vel) const {
        float world[3];
        if (PROFILE == kRef) {
            world[0] = (pa.x + px) * S.scale;
            world[1] = (pa.y + py) * S.scale;
            world[2] = (pa.z + pz) * S.scale;
        } else {
            const float gs = ph.spikyf * ph.inv_rho0;
            world[0] = (pa.x + px * gs) * S.scale;
            world[1] = (pa.y + py * gs) * S.scale;
            world[2] = (pa.z + pz * gs) * S.scale;
            collide_sphere(S, world);
        }
        va = v[a];
        vel[0] = va.x;
        vel[1] = va.y;
        vel[2] = va.z;
        if (S.tri_count) {
            collide_triangles(tris, S.tri_first, S.tri_count, world, vel);
            v[a] = make_float4(vel[0], vel[1], vel[2], va.w);
        }
        for (int d = 0; d < 3; ++d) {
            float w = world[d];
            w = fmaxf(S.min_b[d], w);
            w = fminf(S.max_b[d], w);
            q[d] = w / S.scale;
        }
    }
};

// Final velocity (returned, too; in the ref profile also position) after the step's last correction
// (oclsph_kernel.h:404-416).
template <int PROFILE>
__device__ __forceinline__ float4 finalise(const Phys &ph, const SceneDev &S, uint32_t a, const float *q,
                                         const float4 &va, const float *vel, float4 *__restrict__ x,
                                         float4 *__restrict__ v, const HostParticlesOut *__restrict__ hout) {
    const float4 xa = x[a];
    const float xo[3] = {xa.x, xa.y, xa.z};
    float nv[3], nx[3];
    for (int d = 0; d < 3; ++d) {
        const float dd = q[d] - xo[d] / S.scale;
        if (PROFILE == kRef) {
            nx[d] = q[d] * S.scale;
            nv[d] = __fmaf_rn(dd, S.inv_dt, vel[d]) * ph.damping;
        } else {
            nv[d] = dd * S.inv_dt;
        }
    }
    const float4 now = make_float4(nv[0], nv[1], nv[2], va.w);
    v[a] = now;
    if (PROFILE == kRef) {
        x[a] = make_float4(nx[0], nx[1], nx[2], xa.w);
        store_host_motion(hout, a, x[a], now);
    }
    return now;
}

// Vorticity and the XSPH sum of one particle over its fluid neighbours.
struct VorticitySum {
    float o[3] = {0.f, 0.f, 0.f}, xs[3] = {0.f, 0.f, 0.f};

    // vel_b(): the neighbour's velocity
    template <class V>
    __device__ __forceinline__ void add(const Phys &ph, const float4 &pa, const float4 &va, float bx, float by,
                                        float bz, float mb, V &&vel_b) {
        const float d[3] = {pa.x - bx, pa.y - by, pa.z - bz};
        const float r2 = dist2(d[0], d[1], d[2]);
        if (!(r2 <= ph.hh)) return;
        const float4 vb = vel_b();
        const float vab[3] = {vb.x - va.x, vb.y - va.y, vb.z - va.z};
        const float t = ph.hh - r2;
        const float mw = mb * (t * t * t);
        xs[0] = __fmaf_rn(mw, vab[0], xs[0]);
        xs[1] = __fmaf_rn(mw, vab[1], xs[1]);
        xs[2] = __fmaf_rn(mw, vab[2], xs[2]);
        const float r = sqrtf(r2);
        if (r >= kKernelEpsilon) {
            const float hr = ph.h - r;
            const float sc = mb * ((hr * hr) / r);
            float cr[3];
            cross3(vab, d, cr);
            o[0] = __fmaf_rn(sc, cr[0], o[0]);
            o[1] = __fmaf_rn(sc, cr[1], o[1]);
            o[2] = __fmaf_rn(sc, cr[2], o[2]);
        }
    }

    // a neighbour's (or two neighbours') share, at velocities (ux, uy, uz): mw times (vx, vy, vz)
    // and s times (cx, cy, cz)
    template <class T>
    struct Terms {
        T q2, mw, vx, vy, vz, s, cx, cy, cz;
    };
    template <bool kFast, class T>
    static __device__ __forceinline__ Terms<T> terms(const Phys &ph, const float4 &pa, const float4 &va, const T &bx,
                                                     const T &by, const T &bz, const T &mb, const T &ux, const T &uy,
                                                     const T &uz) {
        Terms<T> o;
        const T dx = T(pa.x) - bx, dy = T(pa.y) - by, dz = T(pa.z) - bz;
        o.q2 = dist2(dx, dy, dz);
        T r, s;
        root_and_spiky<kFast>(ph, o.q2, r, s);
        o.vx = ux - T(va.x), o.vy = uy - T(va.y), o.vz = uz - T(va.z);
        const T t = T(ph.hh) - o.q2;
        o.mw = mb * (t * t * t);
        o.s = mb * s;
        o.cx = o.vy * dz - o.vz * dy, o.cy = o.vz * dx - o.vx * dz, o.cz = o.vx * dy - o.vy * dx;
        return o;
    }

    // two neighbours in order
    template <bool kFast>
    __device__ __forceinline__ void add2(const Phys &ph, const float4 &pa, const float4 &va, const Two &bx,
                                         const Two &by, const Two &bz, const Two &mb, const Two &ux, const Two &uy,
                                         const Two &uz) {
        const Terms<Two> t = terms<kFast>(ph, pa, va, bx, by, bz, mb, ux, uy, uz);
        one(ph, t.q2.lo(), t.mw.lo(), t.vx.lo(), t.vy.lo(), t.vz.lo(), t.s.lo(), t.cx.lo(), t.cy.lo(), t.cz.lo());
        one(ph, t.q2.hi(), t.mw.hi(), t.vx.hi(), t.vy.hi(), t.vz.hi(), t.s.hi(), t.cx.hi(), t.cy.hi(), t.cz.hi());
    }
    __device__ __forceinline__ void one(const Phys &ph, float q2, float mw, float vx, float vy, float vz, float sc,
                                        float cx, float cy, float cz) {
        if (!(q2 <= ph.hh)) return;
        xs[0] = __fmaf_rn(mw, vx, xs[0]);
        xs[1] = __fmaf_rn(mw, vy, xs[1]);
        xs[2] = __fmaf_rn(mw, vz, xs[2]);
        if (q2 >= ph.eps_r2) {
            o[0] = __fmaf_rn(sc, cx, o[0]);
            o[1] = __fmaf_rn(sc, cy, o[1]);
            o[2] = __fmaf_rn(sc, cz, o[2]);
        }
    }

    // omega with |omega| in w, pom (p* with |omega| in w; null: not kept) and vx
    __device__ __forceinline__ void finish(const Phys &ph, uint32_t a, const float4 &pa, const float4 &va,
                                           float4 *__restrict__ omega, float4 *__restrict__ pom,
                                           float4 *__restrict__ vx) const {
        const float gs = ph.spikyf * ph.inv_rho0;
        const float ws = ph.poly6f * ph.inv_rho0;
        // omega = sum_b m_b / rho0 (v_b - v_a) x grad_b W(x_a - x_b), and grad_b W = -grad_a W
        // = -spikyf (h - r)^2 d / r: the sum o carries grad_a's factor, so its sign flips
        const float ox = -(o[0] * gs), oy = -(o[1] * gs), oz = -(o[2] * gs);
        const float om = sqrtf(ox * ox + oy * oy + oz * oz);
        omega[a] = make_float4(ox, oy, oz, om);
        if (pom) pom[a] = make_float4(pa.x, pa.y, pa.z, om);
        vx[a] = make_float4(__fmaf_rn(ph.xsph_c, xs[0] * ws, va.x), __fmaf_rn(ph.xsph_c, xs[1] * ws, va.y),
                            __fmaf_rn(ph.xsph_c, xs[2] * ws, va.z), va.w);
    }
};

// eta = grad |omega| of one particle over its fluid neighbours, and the step's end:
// N = eta / |eta|, f = eps (N x omega), v = vx + dt f, x = p*.
struct ApplySum {
    float e[3] = {0.f, 0.f, 0.f};

    // oa: the particle's |omega|; om_b(): the neighbour's
    template <class O>
    __device__ __forceinline__ void add(const Phys &ph, const float4 &pa, float oa, float bx, float by, float bz,
                                        O &&om_b, float mb) {
        const float d[3] = {pa.x - bx, pa.y - by, pa.z - bz};
        const float r2 = dist2(d[0], d[1], d[2]);
        if (!(r2 <= ph.hh)) return;
        const float r = sqrtf(r2);
        if (!(r >= kKernelEpsilon)) return;
        const float hr = ph.h - r;
        const float sc = mb * ((hr * hr) / r) * (om_b() - oa);
        e[0] = __fmaf_rn(sc, d[0], e[0]);
        e[1] = __fmaf_rn(sc, d[1], e[1]);
        e[2] = __fmaf_rn(sc, d[2], e[2]);
    }

    // a neighbour's (or two neighbours') share, |omega| in ob: f times (x, y, z)
    template <class T>
    struct Terms {
        T q2, f, x, y, z;
    };
    template <bool kFast, class T>
    static __device__ __forceinline__ Terms<T> terms(const Phys &ph, const float4 &pa, float oa, const T &bx,
                                                     const T &by, const T &bz, const T &ob, const T &mb) {
        Terms<T> o;
        o.x = T(pa.x) - bx, o.y = T(pa.y) - by, o.z = T(pa.z) - bz;
        o.q2 = dist2(o.x, o.y, o.z);
        T r, s;
        root_and_spiky<kFast>(ph, o.q2, r, s);
        o.f = mb * s * (ob - T(oa));
        return o;
    }
    static __device__ __forceinline__ bool in_range(const Phys &ph, float q2) { return q2 <= ph.hh && q2 >= ph.eps_r2; }

    // two neighbours in order
    template <bool kFast>
    __device__ __forceinline__ void add2(const Phys &ph, const float4 &pa, float oa, const Two &bx, const Two &by,
                                         const Two &bz, const Two &ob, const Two &mb) {
        const Terms<Two> t = terms<kFast>(ph, pa, oa, bx, by, bz, ob, mb);
        if (in_range(ph, t.q2.lo())) one(t.f.lo(), t.x.lo(), t.y.lo(), t.z.lo());
        if (in_range(ph, t.q2.hi())) one(t.f.hi(), t.x.hi(), t.y.hi(), t.z.hi());
    }
    __device__ __forceinline__ void one(float sc, float dx, float dy, float dz) {
        e[0] = __fmaf_rn(sc, dx, e[0]);
        e[1] = __fmaf_rn(sc, dy, e[1]);
        e[2] = __fmaf_rn(sc, dz, e[2]);
    }

    __device__ __forceinline__ void finish(const Phys &ph, const SceneDev &S, uint32_t a, const float4 &pa,
                                           const float4 &oa, const float4 *__restrict__ vx, float4 *__restrict__ v,
                                           float4 *__restrict__ x, const HostParticlesOut *__restrict__ hout) const {
        const float gs = ph.spikyf * ph.inv_rho0;
        const float ex = e[0] * gs, ey = e[1] * gs, ez = e[2] * gs;
        const float el = sqrtf(ex * ex + ey * ey + ez * ez);
        float N[3] = {0.f, 0.f, 0.f};
        if (el > 0.f) {
            N[0] = ex / el;
            N[1] = ey / el;
            N[2] = ez / el;
        }
        const float om[3] = {oa.x, oa.y, oa.z};
        float f[3];
        cross3(N, om, f);
        const float4 vxa = vx[a];
        const float ve = ph.vort_eps, dt = S.dt;
        const float4 vn = make_float4(__fmaf_rn(dt, f[0] * ve, vxa.x), __fmaf_rn(dt, f[1] * ve, vxa.y),
                                      __fmaf_rn(dt, f[2] * ve, vxa.z), vxa.w);
        v[a] = vn;
        const float4 xa = x[a];
        const float4 xn = make_float4(pa.x * S.scale, pa.y * S.scale, pa.z * S.scale, xa.w);
        x[a] = xn;
        store_host_motion(hout, a, xn, vn);
    }
};

}  // namespace fgb
