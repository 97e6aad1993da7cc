// aw_uniform.cuh — register-resident multigrid kernels of the finite-volume V-cycle.
//
// A block of R^3 cells takes R * R/2 lanes: a lane holds the x pair (2 xp, 2 xp + 1) of one y for every z,
// so z neighbours are the lane's own registers, x and y neighbours come by warp shuffles and only the
// block's halo comes from memory.  A warp serves one 8^3, 4 4^3, 16 2^3 or 32 1^3 blocks, without shared
// memory and without a CTA barrier.
//
// With one density (beta = 1/rho constant over a block) the conductances of a block are seven numbers: one
// for every face between two of its cells and one per side of the block (wall, same, coarser, finer or
// absent neighbour).  k_uni_check establishes this from the coefficient arrays themselves at the start of
// every solve, block by block; nothing is remembered from an earlier call.  Blocks that are not uniform
// (a two-phase interface) read each cell's six conductances where they need them.
//
// What bounded the staged form (one CTA per 8^3 block: block, halo and the three coefficient arrays
// in shared memory) was instruction issue: index splits of the staging loops, six shared-memory
// weight loads per update, and a CTA barrier per colour: 45.7M warp instructions and 60 us per colour
// of the 4.7M-cell poisson_256 level at 13% of the HBM rate.  Here the same launch takes 27 us (ncu,
// cold), the solve to 1e-6 2.71 instead of 5.92 ms; the small levels' launches 5 to 10 instead of 10 to 13
// us, and the dam_drop_128 step's solve 1.06 instead of 1.71 ms.  What bounds it now is the latency of a launch's
// loads (slot record, then cells and halo).  The arithmetic of a cell is that of the staged kernels,
// operation by operation, so both forms agree bit for bit.
#pragma once

#include "aw_internal.cuh"

namespace aw {

struct Coef3 {
    const float* w[3];
};

// Programmatic dependent launch: the V-cycle's kernels are launched so that each may start while its
// predecessor drains.  A kernel reads what its predecessor wrote only after pdl_wait() (which returns
// once the predecessor grid has completed and its memory is visible; at once for a kernel launched
// without the attribute), and lets its successor start with pdl_trigger() once its own main work is
// issued.  Descriptors and slot metadata (fixed at solver build) are staged before the wait, and so are
// k_uni_check's weights and masks: the launch after it is an ordinary one (launch_dep).
__device__ inline void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ inline void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" :::); }

constexpr int UNT = 128;              // threads per CTA: 4 independent warps
constexpr int UWARPS = UNT / 32;
constexpr int UREC = 8;               // int4 words of a slot record
constexpr int UNI_MAX_RES = 8;        // 16^3 blocks would take 128 cells per lane: they keep the staged form

// state of a slot, set by k_uni_check: no fluid cell (nothing to do), one conductance, several
enum { US_AIR = 0, US_UNIFORM = 1, US_GENERAL = 2 };

// The arrays of a level start on 16 bytes (the solver's own do, aw_solve sees to the caller's): a pair of cells
// at an even index is one access.
//
// One block-structured level as the kernels below see it.  Slots: the level's active blocks, colour 0
// then colour 1, resolutions descending.  Warp w serves desc[w] = {first slot, count | res << 8}.
//   rec: {cell offset, block, kinds, coarse cell offset}, neighbour cell offsets (6), neighbour blocks
//        (6), neighbour coarse cell offsets (6), face offsets (3)
//   kinds: 4 bits per face direction (NB_*), bit 24 + f: neighbour f is halved on the coarse level
//   wt:  {interior, -x, +x, -y}, {+y, -z, +z, state}
//   mask: fluid bit 2 z + i of the lane's cell (2 xp + i, y, z), 32 lanes per warp
struct UniView {
    const int2* desc;
    const int4* rec;
    const float4* wt;
    const uint16_t* mask;
    const uint8_t* general;  // per warp: some block of it is not uniform
    Coef3 W;           // the level's conductances (blocks that are not uniform)
    int first, nwarp;  // the warps of this launch
};

template <int R>
struct UG {
    static constexpr int XP = R >= 2 ? R / 2 : 1;  // x pairs per row
    static constexpr int LPB = XP * R;             // lanes per block
    static constexpr int BPW = 32 / LPB;           // blocks per warp
    static constexpr int NI = R >= 2 ? 2 : 1;
};
// Products and sums with their roundings spelt out: here a product is often shared between two cells,
// and the compiler then contracts other pairs than in the staged kernels.
__device__ __forceinline__ float ufma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double ufma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float umul(float a, float b) { return __fmul_rn(a, b); }
// The staged kernels divide with __fdividef, which is a multiplication by the approximate reciprocal (PTX
// div.approx.f32) for divisors within 2^-126 .. 2^126; here a cell's divisor is fixed for a launch, so its
// reciprocal is taken once.
__device__ __forceinline__ float urcp(float d) {
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(d));
    return r;
}
__device__ __forceinline__ double umul(double a, double b) { return __dmul_rn(a, b); }

inline int uni_blocks_per_warp(int r) { return r == 8 ? 1 : (r == 4 ? 4 : (r == 2 ? 16 : 32)); }

// x of a level: FP32, or FP16 with one FP32 scale per block
template <bool HALF>
struct UX {
    float* f;
    __half* h;
    float* scale;
    __device__ __forceinline__ float sc(int b) const { return HALF ? scale[b] : 1.f; }
    __device__ __forceinline__ float get(uint32_t i, float s) const { return HALF ? umul(__half2float(h[i]), s) : f[i]; }
    // two consecutive values; `even`: i is even
    __device__ __forceinline__ float2 get2(uint32_t i, float s, bool even) const {
        if (HALF) {
            if (even) {
                const float2 v = __half22float2(*reinterpret_cast<const __half2*>(h + i));
                return make_float2(umul(v.x, s), umul(v.y, s));
            }
            return make_float2(umul(__half2float(h[i]), s), umul(__half2float(h[i + 1]), s));
        }
        if (even) return *reinterpret_cast<const float2*>(f + i);
        return make_float2(f[i], f[i + 1]);
    }
};

template <class T>
__device__ __forceinline__ void uload2(const T* p, uint32_t i, bool even, T& a, T& b) {
    if (even) {
        if constexpr (sizeof(T) == 4) {
            const float2 v = *reinterpret_cast<const float2*>(p + i);
            a = v.x;
            b = v.y;
        } else {
            const double2 v = *reinterpret_cast<const double2*>(p + i);
            a = v.x;
            b = v.y;
        }
    } else {
        a = p[i];
        b = p[i + 1];
    }
}
template <class T>
__device__ __forceinline__ void ustore2(T* p, uint32_t i, bool even, T a, T b) {
    if (even) {
        if constexpr (sizeof(T) == 4) *reinterpret_cast<float2*>(p + i) = make_float2(a, b);
        else *reinterpret_cast<double2*>(p + i) = make_double2(a, b);
    } else {
        p[i] = a;
        p[i + 1] = b;
    }
}

// The lane's block, read from its slot record.
template <int R>
struct ULane {
    using G = UG<R>;
    int lane, y, xp;
    bool live, general;  // holds fluid; has no single conductance
    uint32_t off;      // cell offset of the block
    uint32_t at;       // ... of the lane's pair at z = 0
    bool even;         // pairs start at even indices
    int block, kinds;
    uint32_t coff;     // cell offset on the coarse level
    float wi, wx0, wx1, wy0, wy1, wz0, wz1;
    uint32_t mask;
    const int4* rec;
    // read before the wait: the record is fixed at solver build, and k_uni_check, which writes weights and mask,
    // has ended before the first launch after it begins
    __device__ __forceinline__ bool init(const UniView& V, int warp) {
        lane = threadIdx.x & 31;
        const int li = lane % G::LPB, s = lane / G::LPB;
        y = li / G::XP;
        xp = li % G::XP;
        const int2 d = V.desc[warp];
        const int cnt = d.y & 0xFF;
        const int slot = d.x + (s < cnt ? s : 0);
        rec = V.rec + (size_t)slot * UREC;
        const float4 wa = V.wt[2 * (size_t)slot], wb = V.wt[2 * (size_t)slot + 1];
        const int4 r0 = rec[0];
        mask = V.mask[(size_t)warp * 32 + lane];
        wi = wa.x;
        wx0 = wa.y;
        wx1 = wa.z;
        wy0 = wa.w;
        wy1 = wb.x;
        wz0 = wb.y;
        wz1 = wb.z;
        live = s < cnt && __float_as_int(wb.w) != US_AIR;
        general = live && __float_as_int(wb.w) == US_GENERAL;
        off = (uint32_t)r0.x;
        block = r0.y;
        kinds = r0.z;
        coff = (uint32_t)r0.w;
        at = off + (uint32_t)(G::NI * xp + R * y);
        even = (off & 1u) == 0;
        return __any_sync(0xffffffffu, live);
    }
    // the six conductances {W, E, S, N, B, T} of cell (2 xp + i, y, z)
    __device__ __forceinline__ void weights(const Coef3& W, int i, int z, float (&w)[6]) const {
        const int x = G::NI * xp + i;
        const float* a = W.w[0] + foff(0) + (x + (R + 1) * (y + R * z));
        const float* b = W.w[1] + foff(1) + (x + R * (y + (R + 1) * z));
        const float* c = W.w[2] + foff(2) + (x + R * (y + R * z));
        w[0] = a[0];
        w[1] = a[1];
        w[2] = b[0];
        w[3] = b[R];
        w[4] = c[0];
        w[5] = c[R * R];
    }
    __device__ __forceinline__ int word(int k) const { return reinterpret_cast<const int*>(rec)[k]; }
    __device__ __forceinline__ int kind(int f) const { return (kinds >> (4 * f)) & 15; }
    __device__ __forceinline__ uint32_t nboff(int f) const { return (uint32_t)word(4 + f); }
    __device__ __forceinline__ int nbblk(int f) const { return word(10 + f); }
    __device__ __forceinline__ uint32_t nbcoff(int f) const { return (uint32_t)word(16 + f); }
    __device__ __forceinline__ uint32_t foff(int a) const { return (uint32_t)word(22 + a); }
};

// One face of the block's halo: the neighbouring cell layer at (u, v) along the axes (a + 1, a + 2) mod
// 3: the cell of a same-resolution neighbour, the parent of a coarser one, the mean of the four touching
// cells of a finer one, 0 where there is none.  S reads one cell; with PROL the coarse correction of the
// cell's parent is added first (a coarse air cell holds 0).
//
// A row is read in two steps so that all rows of a block are in flight together (a branch on the kind
// around each load made them a chain of memory latencies: 21 us a launch instead of 9): issue() loads one
// cell per value whatever the kind, finish() completes the values, and only warps that touch a finer
// neighbour (any_fine) read its three other cells there.  Lanes that do not want a row read a cell of
// their own block and get 0.
template <int R, class S, bool PROL>
struct UHalo {
    using T = typename S::T;
    uint32_t base, cbase, off, coff;
    int su, sv, csu, csv, sh, csh, blk;
    bool ok, fine;
    typename S::Ctx ctx;
    __device__ __forceinline__ void init(const ULane<R>& L, int f, bool want) {  // before the wait: geometry only
        const int kind = L.kind(f);
        ok = L.live && want && kind != 0;
        fine = ok && kind == 4;
        sh = kind == 3 ? 1 : 0;
        const int a = f >> 1;
        const int rn = kind == 3 ? R / 2 : (kind == 4 ? 2 * R : R);
        const int qa = (f & 1) ? 0 : rn - 1;
        const int st1 = rn, st2 = rn * rn;
        su = a == 0 ? st1 : (a == 1 ? st2 : 1);
        sv = a == 0 ? st2 : (a == 1 ? 1 : st1);
        base = L.nboff(f) + (uint32_t)(qa * (a == 0 ? 1 : (a == 1 ? st1 : st2)));
        blk = ok ? L.nbblk(f) : L.block;
        off = L.off;
        coff = L.coff;
        if (PROL) {
            const int hv = (L.kinds >> (24 + f)) & 1;
            const int rc = hv ? rn / 2 : rn;
            const int c1 = rc, c2 = rc * rc;
            csh = hv + (kind == 3 ? 1 : 0) - (kind == 4 ? 1 : 0);
            csu = a == 0 ? c1 : (a == 1 ? c2 : 1);
            csv = a == 0 ? c2 : (a == 1 ? 1 : c1);
            cbase = L.nbcoff(f) + (uint32_t)((qa >> hv) * (a == 0 ? 1 : (a == 1 ? c1 : c2)));
        }
    }
    __device__ __forceinline__ uint32_t cell(int2 p) const {
        const int m = fine ? 2 : 1;
        return ok ? base + (uint32_t)(m * ((p.x >> sh) * su + (p.y >> sh) * sv)) : off;
    }
    template <int N, class F>
    __device__ __forceinline__ void issue(const S& src, F uv, T* r, T* c) const {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const int2 p = uv(k);
            r[k] = src.get(cell(p), ctx);
            if (PROL) c[k] = src.coarse(ok ? cbase + (uint32_t)((p.x >> csh) * csu + (p.y >> csh) * csv) : coff, ctx);
        }
    }
    template <int N, class F>
    __device__ __forceinline__ void finish(const S& src, bool any_fine, F uv, T* r, const T* c) const {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            if (PROL) r[k] += c[k];
            if (!ok) r[k] = T(0);
        }
        if (!any_fine) return;
        const uint32_t o1 = fine ? sv : 0, o2 = fine ? su : 0;
        T e[N][3];
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const uint32_t o = cell(uv(k));
            e[k][0] = src.get(o + o1, ctx);
            e[k][1] = src.get(o + o2, ctx);
            e[k][2] = src.get(o + o1 + o2, ctx);
        }
#pragma unroll
        for (int k = 0; k < N; ++k) {
            if (PROL) {
                e[k][0] += c[k];
                e[k][1] += c[k];
                e[k][2] += c[k];
            }
            T t = r[k];
            t += e[k][0];
            t += e[k][1];
            t += e[k][2];
            if (fine) r[k] = T(0.25) * t;
        }
    }
};

// The halo of a lane: the x side(s) its pair lies on, its y side, both z sides.  iy(k, z): x coordinate
// of the k-th y value at height z; iz(side, k): of the k-th value under / above the block.
template <int R, class S, bool PROL>
struct UHalos {
    using T = typename S::T;
    using G = UG<R>;
    UHalo<R, S, PROL> X, X1, Y, Z0, Z1;
    bool any_fine;
    T hx[R == 2 ? 2 * R : R], hy[2][R], hz[2][2];  // hx[R + z] (R = 2): the +x side
    __device__ __forceinline__ void init(const ULane<R>& L) {
        const bool ex = L.xp == 0 || L.xp == G::XP - 1, ey = L.y == 0 || L.y == R - 1;
        X.init(L, R == 2 || L.xp == 0 ? 0 : 1, ex);
        if (R == 2) X1.init(L, 1, true);
        Y.init(L, L.y == 0 ? 2 : 3, ey);
        Z0.init(L, 4, true);
        Z1.init(L, 5, true);
        any_fine = __any_sync(0xffffffffu, X.fine || (R == 2 && X1.fine) || Y.fine || Z0.fine || Z1.fine);
    }
    template <class FY, class FZ>
    __device__ __forceinline__ void load(const ULane<R>& L, const S& src, FY iy, FZ iz) {
        X.ctx = src.ctx(X.blk);
        if (R == 2) X1.ctx = src.ctx(X1.blk);
        Y.ctx = src.ctx(Y.blk);
        Z0.ctx = src.ctx(Z0.blk);
        Z1.ctx = src.ctx(Z1.blk);
        T cx[R], cx1[R], cy0[R], cy1[R], cz0[2], cz1[2];
        const auto ux = [&](int z) { return make_int2(L.y, z); };
        const auto u0 = [&](int z) { return make_int2(z, iy(0, z)); };
        const auto u1 = [&](int z) { return make_int2(z, iy(1, z)); };
        const auto w0 = [&](int k) { return make_int2(iz(0, k), L.y); };
        const auto w1 = [&](int k) { return make_int2(iz(1, k), L.y); };
        X.template issue<R>(src, ux, hx, cx);
        if (R == 2) X1.template issue<R>(src, ux, hx + (R == 2 ? R : 0), cx1);
        Y.template issue<R>(src, u0, hy[0], cy0);
        Y.template issue<R>(src, u1, hy[1], cy1);
        Z0.template issue<2>(src, w0, hz[0], cz0);
        Z1.template issue<2>(src, w1, hz[1], cz1);
        if (any_fine) {
            finish_all(src, true, ux, u0, u1, w0, w1, cx, cx1, cy0, cy1, cz0, cz1);
        } else {
            finish_all(src, false, ux, u0, u1, w0, w1, cx, cx1, cy0, cy1, cz0, cz1);
        }
    }
    template <class A, class B, class C, class D, class E>
    __device__ __forceinline__ void finish_all(const S& src, bool f, A ux, B u0, C u1, D w0, E w1, const T* cx, const T* cx1,
                                               const T* cy0, const T* cy1, const T* cz0, const T* cz1) {
        X.template finish<R>(src, f, ux, hx, cx);
        if (R == 2) X1.template finish<R>(src, f, ux, hx + (R == 2 ? R : 0), cx1);
        Y.template finish<R>(src, f, u0, hy[0], cy0);
        Y.template finish<R>(src, f, u1, hy[1], cy1);
        Z0.template finish<2>(src, f, w0, hz[0], cz0);
        Z1.template finish<2>(src, f, w1, hz[1], cz1);
    }
};

// Cell sources of the halo: x of a V-cycle level (with the coarse level for PROL), FP64 vectors.
template <bool HALF, bool HC>
struct USrcX {
    using T = float;
    struct Ctx {
        float s, sc;
    };
    UX<HALF> x;
    UX<HC> c;
    bool prol;
    __device__ __forceinline__ Ctx ctx(int b) const {
        Ctx k;
        k.s = x.sc(b);
        k.sc = HC && prol ? c.scale[b] : 1.f;
        return k;
    }
    __device__ __forceinline__ float get(uint32_t i, const Ctx& k) const { return x.get(i, k.s); }
    __device__ __forceinline__ float coarse(uint32_t i, const Ctx& k) const { return c.get(i, k.sc); }
};
struct USrcD {
    using T = double;
    struct Ctx {};
    const double* p;
    __device__ __forceinline__ Ctx ctx(int) const { return Ctx{}; }
    __device__ __forceinline__ double get(uint32_t i, const Ctx&) const { return p[i]; }
    __device__ __forceinline__ double coarse(uint32_t, const Ctx&) const { return 0.0; }
    __device__ __forceinline__ void get2(uint32_t i, bool even, double& a, double& b) const { uload2(p, i, even, a, b); }
};
// the search direction z + beta d of a conjugate-gradient step, formed where it is read
struct USrcDir {
    using T = double;
    struct Ctx {};
    const float* z;
    const double* d;
    double beta;
    bool first;
    __device__ __forceinline__ Ctx ctx(int) const { return Ctx{}; }
    __device__ __forceinline__ double get(uint32_t i, const Ctx&) const {
        return first ? (double)z[i] : (double)z[i] + beta * d[i];
    }
    __device__ __forceinline__ double coarse(uint32_t, const Ctx&) const { return 0.0; }
    __device__ __forceinline__ void get2(uint32_t i, bool even, double& a, double& b) const {
        float za, zb;
        uload2(z, i, even, za, zb);
        if (first) {
            a = za;
            b = zb;
            return;
        }
        uload2(d, i, even, a, b);
        a = (double)za + beta * a;
        b = (double)zb + beta * b;
    }
};

// Store the block: FP32, or FP16 with a fresh per-block scale.  v0/v1: the pair at every z.
template <int R, bool HALF, bool KEEP = false>  // KEEP: v0, v1 become the values as read back
__device__ __forceinline__ void uni_store(const ULane<R>& L, const UX<HALF>& x, float* v0, float* v1) {
    using G = UG<R>;
    if (!HALF) {
        if (!L.live) return;
#pragma unroll
        for (int z = 0; z < R; ++z) {
            if (R == 1) x.f[L.at] = v0[z];
            else ustore2(x.f, L.at + (uint32_t)(R * R * z), L.even, v0[z], v1[z]);
        }
        return;
    }
    float m = 0.f;
#pragma unroll
    for (int z = 0; z < R; ++z) {
        m = fmaxf(m, fabsf(v0[z]));
        if (G::NI == 2) m = fmaxf(m, fabsf(v1[z]));
    }
#pragma unroll
    for (int o = 1; o < G::LPB; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (!L.live) return;
    const float inv = m > 0.f ? 32768.f / m : 0.f, scale = m > 0.f ? m * (1.f / 32768.f) : 0.f;
#pragma unroll
    for (int z = 0; z < R; ++z) {
        const uint32_t i = L.at + (uint32_t)(R * R * z);
        const __half a = __float2half_rn(v0[z] * inv);
        if (KEEP) v0[z] = umul(__half2float(a), scale);
        if (G::NI == 1) {
            x.h[i] = a;
            continue;
        }
        const __half b = __float2half_rn(v1[z] * inv);
        if (KEEP) v1[z] = umul(__half2float(b), scale);
        if (L.even) *reinterpret_cast<__half2*>(x.h + i) = __halves2half2(a, b);
        else {
            x.h[i] = a;
            x.h[i + 1] = b;
        }
    }
    if (L.lane % G::LPB == 0) x.scale[L.block] = scale;
}

// How a smoothing launch meets its input:
//   PLAIN        x from memory
//   ZERO_ALL     x = 0 everywhere (first colour of a level's first sweep): nothing of x is read
//   ZERO_OWN     the block's own x = 0, the halo (the other colour, just smoothed) from memory
//   PROLONG_ALL  x + P xc for the block and its halo (first colour after the coarse-grid correction)
//   PROLONG_OWN  x + P xc for the block, the halo (already corrected and smoothed) as stored
// so that zeroing a level and prolongating into it take no pass of their own.
enum { UM_PLAIN = 0, UM_ZERO_ALL = 1, UM_ZERO_OWN = 2, UM_PROLONG_ALL = 3, UM_PROLONG_OWN = 4 };

// One colour of one sweep: cells A (updated) from cells B (the other colour).  At height z the lane's
// cell of colour class CLS is i = (q ^ z ^ CLS) & 1, so its z and y neighbours of the other colour sit
// in B[z -+ 1] and in B[z] of the lanes one row up and down, and the outer x neighbour in B[z] of the
// next lane on its side.
template <int R>
struct UCoef {
    const float* face[3];  // the first faces of the pair's first cell at z = 0 (general blocks)
    bool one[2], edge[2];
    int src[2];
    float cW[2], cE[2], wS, wN, diag[2][3], rcp[2][3];
};

template <int R, int CLS, bool GEN>
__device__ __forceinline__ void uni_sweep(const ULane<R>& L, const UCoef<R>& C, float (&A)[R], const float (&B)[R],
                                          const float (&b)[R], const float* hx, const float (&hy)[R], float zlo, float zhi,
                                          uint32_t fl, float omega) {
    using G = UG<R>;
    float An[R];
#pragma unroll
    for (int z = 0; z < R; ++z) {
        const int par = (z ^ CLS) & 1;
        float outer = __shfl_sync(0xffffffffu, B[z], C.src[par]);
        if (C.edge[par]) outer = hx[R == 2 ? 2 * z + CLS : z];
        float vS = __shfl_sync(0xffffffffu, B[z], L.lane - G::XP);
        float vN = __shfl_sync(0xffffffffu, B[z], L.lane + G::XP);
        if (L.y == 0) vS = hy[z];
        if (L.y == R - 1) vN = hy[z];
        const float vW = C.one[par] ? B[z] : outer, vE = C.one[par] ? outer : B[z];
        const float vB = z > 0 ? B[z > 0 ? z - 1 : 0] : zlo;
        const float vT = z < R - 1 ? B[z < R - 1 ? z + 1 : 0] : zhi;
        const int zk = z == 0 ? 0 : (z == R - 1 ? 2 : 1);
        float w[6] = {C.cW[par], C.cE[par], C.wS, C.wN, z == 0 ? L.wz0 : L.wi, z == R - 1 ? L.wz1 : L.wi};
        float diag = C.diag[par][zk], rcp = C.rcp[par][zk];
        bool on = (fl >> (2 * z + CLS)) & 1u;
        if (GEN) {
            asm volatile("" ::: "memory");  // one height's weights at a time: all at once would spill
            const float *fx = C.face[0] + C.one[par], *fy = C.face[1] + C.one[par], *fz = C.face[2] + C.one[par];
            w[0] = fx[(R + 1) * R * z];
            w[1] = fx[(R + 1) * R * z + 1];
            w[2] = fy[R * (R + 1) * z];
            w[3] = fy[R * (R + 1) * z + R];
            w[4] = fz[R * R * z];
            w[5] = fz[R * R * z + R * R];
            diag = -(w[0] + w[1] + w[2] + w[3] + w[4] + w[5]);
            rcp = urcp(diag);
            on = on && !(fabsf(diag) < 1e-9f);
        }
        float Ax = ufma(w[0], vW, umul(w[1], vE));
        Ax = ufma(w[2], vS, Ax);
        Ax = ufma(w[3], vN, Ax);
        Ax = ufma(w[4], vB, Ax);
        Ax = ufma(w[5], vT, Ax);
        Ax = ufma(diag, A[z], Ax);
        const float v = ufma(omega, umul(b[z] - Ax, rcp), A[z]);
        An[z] = on ? v : A[z];
    }
#pragma unroll
    for (int z = 0; z < R; ++z) A[z] = An[z];
}

// The halo of a block by colour class: hx by height (R = 2: by height and class, the pair being the whole
// row), hy and hz by class.
template <int R, class HS, class S>
__device__ __forceinline__ void uni_halo(const ULane<R>& L, HS& H, const S& src, int q, float (&hx)[R == 2 ? 4 : R]) {
    // R - 1 is odd, so the classes of the plane above the block are swapped
    H.load(L, src, [&](int k, int z) { return 2 * L.xp + ((q ^ z ^ k) & 1); },
           [&](int side, int k) { return 2 * L.xp + ((q ^ k ^ side) & 1); });
#pragma unroll
    for (int z = 0; z < R; ++z) {
        if (R == 2) {
            const bool one = ((q ^ z) & 1) != 0;
            const float lo = H.hx[z], hi = H.hx[R == 2 ? R + z : z];
            hx[R == 2 ? 2 * z : z] = one ? hi : lo;
            hx[R == 2 ? 2 * z + 1 : z] = one ? lo : hi;
        } else {
            hx[z] = H.hx[z];
        }
    }
}
// The lane's weights and the fluid bits by class (those of cells cut off from every neighbour cleared).
template <int R>
__device__ __forceinline__ void uni_coef(const ULane<R>& L, int q, UCoef<R>& C, uint32_t& fl) {
    using G = UG<R>;
    // swap the two bits of every height whose E cell is the pair's second
    const uint32_t sw = ((L.mask & 0x5555u) << 1) | ((L.mask >> 1) & 0x5555u);
    const uint32_t selm = q ? 0x3333u : 0xCCCCu;
    fl = (L.mask & ~selm) | (sw & selm);
    C.wS = L.y == 0 ? L.wy0 : L.wi;
    C.wN = L.y == R - 1 ? L.wy1 : L.wi;
#pragma unroll
    for (int par = 0; par < 2; ++par) {
        const bool one = ((q ^ par) & 1) != 0;
        C.one[par] = one;
        C.edge[par] = one ? L.xp == G::XP - 1 : L.xp == 0;
        C.src[par] = one ? L.lane + 1 : L.lane - 1;
        C.cW[par] = !one && L.xp == 0 ? L.wx0 : L.wi;
        C.cE[par] = one && L.xp == G::XP - 1 ? L.wx1 : L.wi;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float wB = k == 0 ? L.wz0 : L.wi, wT = k == 2 ? L.wz1 : L.wi;
            const float d = -(C.cW[par] + C.cE[par] + C.wS + C.wN + wB + wT);
            C.diag[par][k] = d;
            C.rcp[par][k] = urcp(d);
            if (!L.general && fabsf(d) < 1e-9f) {  // never updated
                uint32_t bits = 0;
#pragma unroll
                for (int z = 0; z < R; ++z)
                    if ((z == 0 ? 0 : (z == R - 1 ? 2 : 1)) == k) bits |= 1u << (2 * z + ((z ^ par) & 1));
                fl &= ~bits;
            }
        }
    }
}
template <int R>
__device__ __forceinline__ void uni_faces(const ULane<R>& L, const Coef3& W, UCoef<R>& C) {
    C.face[0] = W.w[0] + L.foff(0) + (2 * L.xp + (R + 1) * L.y);
    C.face[1] = W.w[1] + L.foff(1) + (2 * L.xp + R * L.y);
    C.face[2] = W.w[2] + L.foff(2) + (2 * L.xp + R * L.y);
}
template <int R, bool GEN, class HS>
__device__ __forceinline__ void uni_iterate(const ULane<R>& L, const UCoef<R>& C, float (&E)[R], float (&O)[R],
                                            const float (&bE)[R], const float (&bO)[R], const float (&hx)[R == 2 ? 4 : R],
                                            const HS& H, uint32_t fl, float omega, int iters, bool general) {
    if (GEN && general) {
#pragma unroll 1
        for (int it = 0; it < iters; ++it) {
            uni_sweep<R, 0, GEN>(L, C, E, O, bE, hx, H.hy[0], H.hz[0][0], H.hz[1][0], fl, omega);
            uni_sweep<R, 1, GEN>(L, C, O, E, bO, hx, H.hy[1], H.hz[0][1], H.hz[1][1], fl, omega);
        }
    } else {
#pragma unroll 1
        for (int it = 0; it < iters; ++it) {
            uni_sweep<R, 0, false>(L, C, E, O, bE, hx, H.hy[0], H.hz[0][0], H.hz[1][0], fl, omega);
            uni_sweep<R, 1, false>(L, C, O, E, bO, hx, H.hy[1], H.hz[0][1], H.hz[1][1], fl, omega);
        }
    }
}

// the arguments of a smoothing launch
template <bool HALF, bool HC>
struct USmooth {
    UniView V;
    UX<HALF> x;
    UX<HC> xc;
    const float* b;
    float omega;
    int iters, rev;
};
template <int R, bool HALF, int MODE, bool HC, bool GEN>
__device__ __forceinline__ void uni_smooth_body(const USmooth<HALF, HC>& K, int warp) {
    using G = UG<R>;
    const UniView& V = K.V;
    const UX<HALF> x = K.x;
    const UX<HC> xc = K.xc;
    const float* bvec = K.b;
    const float omega = K.omega;
    const int iters = K.iters, rev = K.rev;
    constexpr bool PO = MODE == UM_PROLONG_ALL || MODE == UM_PROLONG_OWN, PH = MODE == UM_PROLONG_ALL;
    constexpr bool ZO = MODE == UM_ZERO_ALL || MODE == UM_ZERO_OWN, ZH = MODE == UM_ZERO_ALL;
    using S = USrcX<HALF, HC>;
    ULane<R> L;
    UHalos<R, S, PH> H;
    const bool any = L.init(V, warp);
    if (!ZH) H.init(L);
    pdl_wait();
    if (!any) return;
    const S src{x, xc, PO};
    const int q = (L.y & 1) ^ rev;
    // own cells by colour class: E is smoothed first, at height z it is cell i = (q ^ z) & 1 of the pair
    float E[R], O[R], bE[R], bO[R];
    const float sc = ZO ? 1.f : x.sc(L.block);
    const float scc = PO && HC ? xc.scale[L.block] : 1.f;
#pragma unroll
    for (int z = 0; z < R; ++z) {
        const uint32_t i = L.at + (uint32_t)(R * R * z);
        float2 v = make_float2(0.f, 0.f);
        float2 bv = make_float2(0.f, 0.f);
        if (L.live) {
            if (!ZO) v = x.get2(i, sc, L.even);
            uload2(bvec, i, L.even, bv.x, bv.y);
            if (PO) {
                // parent cells of the pair: one when the block is halved, else the block keeps its cell
                const float c = xc.get(L.coff + (uint32_t)(L.xp + (R / 2) * ((L.y >> 1) + (R / 2) * (z >> 1))), scc);
                if ((L.mask >> (2 * z)) & 1u) v.x += c;
                if ((L.mask >> (2 * z + 1)) & 1u) v.y += c;
            }
        }
        const bool one = ((q ^ z) & 1) != 0;
        E[z] = one ? v.y : v.x;
        O[z] = one ? v.x : v.y;
        bE[z] = one ? bv.y : bv.x;
        bO[z] = one ? bv.x : bv.y;
    }
    float hx[R == 2 ? 4 : R];
    if (ZH) {
#pragma unroll
        for (int z = 0; z < R; ++z) H.hy[0][z] = H.hy[1][z] = hx[z] = 0.f;
        if (R == 2) hx[R == 2 ? 2 : 0] = hx[R == 2 ? 3 : 0] = 0.f;
        H.hz[0][0] = H.hz[0][1] = H.hz[1][0] = H.hz[1][1] = 0.f;
    } else {
        uni_halo<R>(L, H, src, q, hx);
    }
    uint32_t fl;
    UCoef<R> C;
    uni_coef<R>(L, q, C, fl);
    const bool general = GEN && V.general[warp];
    if (general) uni_faces<R>(L, V.W, C);
    uni_iterate<R, GEN>(L, C, E, O, bE, bO, hx, H, fl, omega, iters, general);
    pdl_trigger();
    float v0[R], v1[R];
#pragma unroll
    for (int z = 0; z < R; ++z) {
        const bool one = ((q ^ z) & 1) != 0;
        v0[z] = one ? O[z] : E[z];
        v1[z] = one ? E[z] : O[z];
    }
    uni_store<R, HALF>(L, x, v0, v1);
}

// The six halo values of a one-cell block, the lanes' loads in flight together; only where some
// neighbour is finer (2^3 cells) its four touching cells are read.
template <class S, bool PROL>
struct UHaloOne {
    using T = typename S::T;
    UHalo<1, S, PROL> F[6];
    bool any_fine;
    T h[6];
    __device__ __forceinline__ void init(const ULane<1>& L) {
        bool f = false;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            F[k].init(L, k, true);
            f = f || F[k].fine;
        }
        any_fine = __any_sync(0xffffffffu, f);
    }
    __device__ __forceinline__ void load(const S& src) {
        const auto uv = [](int) { return make_int2(0, 0); };
        T c[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            F[k].ctx = src.ctx(F[k].blk);
            F[k].template issue<1>(src, uv, h + k, c + k);
        }
        if (any_fine) {
#pragma unroll
            for (int k = 0; k < 6; ++k) F[k].template finish<1>(src, true, uv, h + k, c + k);
        } else {
#pragma unroll
            for (int k = 0; k < 6; ++k) F[k].template finish<1>(src, false, uv, h + k, c + k);
        }
    }
};

// Blocks of one cell: a lane per block, six halo values.  The cell is black or red by its parity 0, so
// every sweep updates it once.
template <bool HALF, int MODE, bool HC>
__device__ __forceinline__ void uni_smooth_one(const USmooth<HALF, HC>& K, int warp) {
    const UniView& V = K.V;
    const UX<HALF> x = K.x;
    const UX<HC> xc = K.xc;
    const float* bvec = K.b;
    const float omega = K.omega;
    const int iters = K.iters;
    constexpr bool PO = MODE == UM_PROLONG_ALL || MODE == UM_PROLONG_OWN, PH = MODE == UM_PROLONG_ALL;
    constexpr bool ZO = MODE == UM_ZERO_ALL || MODE == UM_ZERO_OWN, ZH = MODE == UM_ZERO_ALL;
    using S = USrcX<HALF, HC>;
    ULane<1> L;
    UHaloOne<S, PH> H;
    const bool any = L.init(V, warp);
    if (!ZH) H.init(L);
    pdl_wait();
    if (!any) return;
    const S src{x, xc, PO};
    float v = 0.f, b = 0.f;
    if (L.live) {
        if (!ZO) v = x.get(L.at, x.sc(L.block));
        b = bvec[L.at];
        if (PO && (L.mask & 1u)) v += xc.get(L.coff, HC ? xc.scale[L.block] : 1.f);
    }
    if (!ZH) H.load(src);
    else H.h[0] = H.h[1] = H.h[2] = H.h[3] = H.h[4] = H.h[5] = 0.f;
    const float(&h)[6] = H.h;
    const float diag = -(L.wx0 + L.wx1 + L.wy0 + L.wy1 + L.wz0 + L.wz1);
    const float rcp = urcp(diag);
    if ((L.mask & 1u) && !(fabsf(diag) < 1e-9f))
#pragma unroll 1
        for (int it = 0; it < iters; ++it) {
            float Ax = ufma(L.wx0, h[0], umul(L.wx1, h[1]));
            Ax = ufma(L.wy0, h[2], Ax);
            Ax = ufma(L.wy1, h[3], Ax);
            Ax = ufma(L.wz0, h[4], Ax);
            Ax = ufma(L.wz1, h[5], Ax);
            Ax = ufma(diag, v, Ax);
            v = ufma(omega, umul(b - Ax, rcp), v);
        }
    pdl_trigger();
    uni_store<1, HALF>(L, x, &v, &v);
}

#define AW_UNI_RES(r, BODY, ONE)    \
    switch (r) {                    \
        case 8: BODY(8); break;     \
        case 4: BODY(4); break;     \
        case 2: BODY(2); break;     \
        default: ONE; break;        \
    }

// One block colour of the block red-black smoother (the arithmetic of k_smooth).
// GEN: the level has blocks that are not uniform; their warps (and the uniform blocks these share) read
// every weight from memory.  An instance of its own: in one kernel the second body's addresses and weights
// cost the common path registers (dam_drop_128 step 1.86 to 1.94 ms inlined, 1.92 ms as a call).
// 4 CTAs per SM (128 registers a thread): the 8^3 body holds 16 cells, 16 right-hand sides and 28 halo
// values per lane, and spills at 5 (96 registers; small-level launches 10 to 11 instead of 7.5 to 9.5 us).
template <bool HALF, int MODE, bool HC, bool GEN>
__global__ void __launch_bounds__(UNT, 4) k_uni_smooth(const __grid_constant__ USmooth<HALF, HC> K) {
    const int w = blockIdx.x * UWARPS + (threadIdx.x >> 5);
    if (w >= K.V.nwarp) {
        pdl_wait();
        return;
    }
    const int warp = K.V.first + w;
    const int r = K.V.desc[warp].y >> 8;
#define AW_UB(R) uni_smooth_body<R, HALF, MODE, HC, GEN>(K, warp)
    AW_UNI_RES(r, AW_UB, (uni_smooth_one<HALF, MODE, HC>(K, warp)))
#undef AW_UB
}

// x += P xc on fluid cells of an FP16 level (its re-encoding needs the whole block's maximum before
// any neighbour may read it, so it cannot ride on the first smoothing launch).
template <int R, bool HALF, bool HC>
__device__ __forceinline__ void uni_prolong_body(const UniView& V, int warp, const UX<HALF>& x, const UX<HC>& xc) {
    ULane<R> L;
    const bool any = L.init(V, warp);
    pdl_wait();
    if (!any) return;
    float v0[R], v1[R];
    const float sc = L.live ? x.sc(L.block) : 1.f, scc = HC && L.live ? xc.scale[L.block] : 1.f;
#pragma unroll
    for (int z = 0; z < R; ++z) {
        float2 v = make_float2(0.f, 0.f);
        if (L.live) {
            const uint32_t i = L.at + (uint32_t)(R * R * z);
            if (R == 1) v.x = x.get(i, sc);
            else v = x.get2(i, sc, L.even);
            const float c = xc.get(L.coff + (R == 1 ? 0u : (uint32_t)(L.xp + (R / 2) * ((L.y >> 1) + (R / 2) * (z >> 1)))), scc);
            if ((L.mask >> (2 * z)) & 1u) v.x += c;
            if (R > 1 && ((L.mask >> (2 * z + 1)) & 1u)) v.y += c;
        }
        v0[z] = v.x;
        v1[z] = v.y;
    }
    pdl_trigger();
    uni_store<R, HALF>(L, x, v0, v1);
}
template <bool HALF, bool HC>
__global__ void __launch_bounds__(UNT) k_uni_prolong(UniView V, UX<HALF> x, UX<HC> xc) {
    const int w = blockIdx.x * UWARPS + (threadIdx.x >> 5);
    if (w >= V.nwarp) {
        pdl_wait();
        return;
    }
    const int warp = V.first + w;
    const int r = V.desc[warp].y >> 8;
#define AW_UB(R) uni_prolong_body<R, HALF, HC>(V, warp, x, xc)
    AW_UNI_RES(r, AW_UB, AW_UB(1))
#undef AW_UB
}

// Where a residual goes: r (FP32), r64 and, restricted (8-child sum on the coarse level's fluid
// cells), the coarse right-hand side.  dsum: partial sums of r^2, or of d . r for DOT.
struct UOut {
    float* r;
    double* r64;
    float* bc;
    const uint8_t* fluid_c;
    double* dnew;  // the search direction, stored by its owner (USrcDir)
};

template <class T>
__device__ __forceinline__ T uni_Ax(T diag, T v, T w0, T x0, T w1, T x1, T w2, T x2, T w3, T x3, T w4, T x4, T w5, T x5) {
    T a = ufma(w0, x0, umul(diag, v));
    a = ufma(w1, x1, a);
    a = ufma(w2, x2, a);
    a = ufma(w3, x3, a);
    a = ufma(w4, x4, a);
    return ufma(w5, x5, a);
}

// r = b - A x of the lane's cells (bvec == nullptr: b = 0), 0 on air cells.  Returns the lane's partial
// sum.
template <int R, class S, bool DOT, bool GEN>
__device__ __forceinline__ double uni_residual_body(const ULane<R>& L, const Coef3& W, bool general,
                                                    UHalos<R, S, false>& H, const S& src, const float* bvec, const UOut& out, float sc) {
    using G = UG<R>;
    using T = typename S::T;
    double acc = 0.0;
    const T wi = L.wi;
    const T cW = L.xp == 0 ? (T)L.wx0 : wi, cE = L.xp == G::XP - 1 ? (T)L.wx1 : wi;
    const T wS = L.y == 0 ? (T)L.wy0 : wi, wN = L.y == R - 1 ? (T)L.wy1 : wi;
    T v0[R], v1[R];
    float bb0[R], bb1[R];
#pragma unroll
    for (int z = 0; z < R; ++z) {
        v0[z] = v1[z] = T(0);
        bb0[z] = bb1[z] = 0.f;
        if (L.live) {
            const uint32_t i = L.at + (uint32_t)(R * R * z);
            if (bvec) uload2(bvec, i, L.even, bb0[z], bb1[z]);
            if constexpr (sizeof(T) == 4) {
                const float2 v = src.x.get2(i, sc, L.even);
                v0[z] = v.x;
                v1[z] = v.y;
            } else {
                src.get2(i, L.even, v0[z], v1[z]);
            }
        }
    }
    H.load(L, src, [&](int k, int) { return 2 * L.xp + k; }, [&](int, int k) { return 2 * L.xp + k; });
    const T *hx = H.hx, *hy0 = H.hy[0], *hy1 = H.hy[1];
    const T zlo0 = H.hz[0][0], zlo1 = H.hz[0][1], zhi0 = H.hz[1][0], zhi1 = H.hz[1][1];
    T ra[2], rb[2];  // residuals of two heights, for the restriction
#pragma unroll
    for (int z = 0; z < R; ++z) {
        const uint32_t i = L.at + (uint32_t)(R * R * z);
        T xm = __shfl_sync(0xffffffffu, v1[z], L.lane - 1), xq = __shfl_sync(0xffffffffu, v0[z], L.lane + 1);
        T s0 = __shfl_sync(0xffffffffu, v0[z], L.lane - G::XP), s1 = __shfl_sync(0xffffffffu, v1[z], L.lane - G::XP);
        T n0 = __shfl_sync(0xffffffffu, v0[z], L.lane + G::XP), n1 = __shfl_sync(0xffffffffu, v1[z], L.lane + G::XP);
        if (R == 2) {
            xm = hx[z];
            xq = hx[z + (R == 2 ? R : 0)];
        } else {
            if (L.xp == 0) xm = hx[z];
            if (L.xp == G::XP - 1) xq = hx[z];
        }
        if (L.y == 0) {
            s0 = hy0[z];
            s1 = hy1[z];
        }
        if (L.y == R - 1) {
            n0 = hy0[z];
            n1 = hy1[z];
        }
        const T b0 = z > 0 ? v0[z > 0 ? z - 1 : 0] : zlo0, b1 = z > 0 ? v1[z > 0 ? z - 1 : 0] : zlo1;
        const T t0 = z < R - 1 ? v0[z < R - 1 ? z + 1 : 0] : zhi0, t1 = z < R - 1 ? v1[z < R - 1 ? z + 1 : 0] : zhi1;
        const T wB = z == 0 ? (T)L.wz0 : wi, wT = z == R - 1 ? (T)L.wz1 : wi;
        const float bv0 = bb0[z], bv1 = bb1[z];
        T r0 = T(0), r1 = T(0);
        T w0[6] = {cW, wi, wS, wN, wB, wT}, w1[6] = {wi, cE, wS, wN, wB, wT};
        if (GEN && general) {
            float g[6];
            L.weights(W, 0, z, g);
#pragma unroll
            for (int k = 0; k < 6; ++k) w0[k] = g[k];
            L.weights(W, 1, z, g);
#pragma unroll
            for (int k = 0; k < 6; ++k) w1[k] = g[k];
        }
        if ((L.mask >> (2 * z)) & 1u) {
            const T diag = -(w0[0] + w0[1] + w0[2] + w0[3] + w0[4] + w0[5]);
            r0 = (T)bv0 - uni_Ax(diag, v0[z], w0[0], xm, w0[1], v1[z], w0[2], s0, w0[3], n0, w0[4], b0, w0[5], t0);
        }
        if ((L.mask >> (2 * z + 1)) & 1u) {
            const T diag = -(w1[0] + w1[1] + w1[2] + w1[3] + w1[4] + w1[5]);
            r1 = (T)bv1 - uni_Ax(diag, v1[z], w1[0], v0[z], w1[1], xq, w1[2], s1, w1[3], n1, w1[4], b1, w1[5], t1);
        }
        if (L.live) {
            if (out.r) ustore2(out.r, i, L.even, (float)r0, (float)r1);
            if (out.r64) ustore2(out.r64, i, L.even, (double)r0, (double)r1);
            if (out.dnew) ustore2(out.dnew, i, L.even, (double)v0[z], (double)v1[z]);
            if (DOT) acc += (double)v0[z] * (double)r0 + (double)v1[z] * (double)r1;
            else acc += (double)r0 * (double)r0 + (double)r1 * (double)r1;
        }
        if (out.bc) {  // 8-child sum, children in x, y, z order
            ra[z & 1] = r0;
            rb[z & 1] = r1;
            if (z & 1) {
                const T p0 = __shfl_sync(0xffffffffu, ra[0], L.lane + G::XP), p1 = __shfl_sync(0xffffffffu, rb[0], L.lane + G::XP);
                const T p2 = __shfl_sync(0xffffffffu, ra[1], L.lane + G::XP), p3 = __shfl_sync(0xffffffffu, rb[1], L.lane + G::XP);
                if (L.live && !(L.y & 1)) {
                    T s = ra[0];
                    s += rb[0];
                    s += p0;
                    s += p1;
                    s += ra[1];
                    s += rb[1];
                    s += p2;
                    s += p3;
                    const uint32_t ci = L.coff + (uint32_t)(L.xp + (R / 2) * ((L.y >> 1) + (R / 2) * (z >> 1)));
                    out.bc[ci] = out.fluid_c[ci] ? (float)s : 0.f;
                }
            }
        }
    }
    return acc;
}
template <class S, bool DOT>
__device__ __forceinline__ double uni_residual_one(const ULane<1>& L, UHaloOne<S, false>& H, const S& src,
                                                   const float* bvec, const UOut& out) {
    using T = typename S::T;
    const T v = src.get(L.at, src.ctx(L.block));
    H.load(src);
    const T(&h)[6] = H.h;
    if (!L.live) return 0.0;
    const T w0 = L.wx0, w1 = L.wx1, w2 = L.wy0, w3 = L.wy1, w4 = L.wz0, w5 = L.wz1;
    T r = T(0);
    if (L.mask & 1u) {
        const T diag = -(w0 + w1 + w2 + w3 + w4 + w5);
        r = (T)(bvec ? bvec[L.at] : 0.f) - uni_Ax(diag, v, w0, h[0], w1, h[1], w2, h[2], w3, h[3], w4, h[4], w5, h[5]);
    }
    if (out.r) out.r[L.at] = (float)r;
    if (out.r64) out.r64[L.at] = (double)r;
    if (out.dnew) out.dnew[L.at] = (double)v;
    if (out.bc) out.bc[L.coff] = out.fluid_c[L.coff] ? (float)r : 0.f;
    return DOT ? (double)v * (double)r : (double)r * (double)r;
}

// The last CTA of a launch to finish adds the CTAs' partial sums, in index order, and `done` uses the
// total in its thread 0: a reduction without a launch of its own.  part[0, gridDim.x); ticket starts
// and ends at 0.
template <class F>
__device__ __forceinline__ void last_cta_sum(double v, double* part, unsigned* ticket, F done) {
    __shared__ double red[32];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    v = warp_sum(v);
    if (lane == 0) red[w] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int k = 0; k < nw; ++k) t += red[k];
        part[blockIdx.x] = t;
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double s = 0.0;
    for (unsigned i = threadIdx.x; i < gridDim.x; i += blockDim.x) s += __ldcg(part + i);
    s = warp_sum(s);
    __syncthreads();
    if (lane == 0) red[w] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int k = 0; k < nw; ++k) t += red[k];
        *ticket = 0u;
        done(t);
    }
}

// r = b - A x on a V-cycle level (FP32 or FP16 x): to r, or restricted into the coarse right-hand side,
// with an optional sum of r^2 into *sum.
template <bool HALF, bool GEN>
__global__ void __launch_bounds__(UNT, 4) k_uni_residual(const __grid_constant__ UniView V, UX<HALF> x,
                                                         const float* __restrict__ b, const __grid_constant__ UOut out,
                                                         double* part, unsigned* ticket, double* sum) {
    const int w = blockIdx.x * UWARPS + (threadIdx.x >> 5);
    double acc = 0.0;
    bool waited = false;
    if (w < V.nwarp) {
        const int warp = V.first + w;
        const int r = V.desc[warp].y >> 8;
        using S = USrcX<HALF, false>;
        const S src{x, UX<false>{nullptr, nullptr, nullptr}, false};
#define AW_UB(R)                                                                                      \
    {                                                                                                 \
        ULane<R> L;                                                                                   \
        UHalos<R, S, false> H;                                                                        \
        const bool any = L.init(V, warp);                                                             \
        H.init(L);                                                                                    \
        pdl_wait();                                                                                   \
        waited = true;                                                                                \
        if (any)                                                                                      \
            acc = uni_residual_body<R, S, false, GEN>(L, V.W, GEN && V.general[warp], H, src, b, out, x.sc(L.block)); \
    }
#define AW_UB1                                                                     \
    {                                                                              \
        ULane<1> L;                                                                \
        UHaloOne<S, false> H;                                                      \
        const bool any = L.init(V, warp);                                          \
        H.init(L);                                                                 \
        pdl_wait();                                                                \
        waited = true;                                                             \
        if (any) acc = uni_residual_one<S, false>(L, H, src, b, out);              \
    }
        AW_UNI_RES(r, AW_UB, AW_UB1)
#undef AW_UB
#undef AW_UB1
    }
    if (!waited) pdl_wait();
    pdl_trigger();
    if (sum) last_cta_sum(acc, part, ticket, [&](double t) { *sum = t; });
}

// The V-cycle's small block-structured levels as one launch: one CTA walks levels first .. last down
// (smoothing, restricted residual), applies the inverse of the coarsest operator where that is the next
// level and small, and walks back up (prolongation, smoothing).  down / up alone: the legs around a coarser
// part with launches of its own.  A warp keeps its blocks' cells, weights and addresses in registers for a
// leg of a level, keeps x in shared memory too (halos read from L1 or L2 after another warp's store took
// 0.5 us of a step), and meets the others at CTA barriers; a colour's step then reads the halo, updates and
// stores.  Every cell's arithmetic is that of the separate launches, bit for bit.
// A level of at most ULOW_WARPS warps leaves most of the chip idle either way, and as launches its steps were
// latency alone, 3.5 to 4 us a colour of 32 4^3 blocks, most of it the record, weight and halo-address chain
// and the fetch of straight-line code that runs once: the 64-block levels under a 32^3 grid and their coarsest
// solve took 79 us a cycle, 34.5 in this launch; the 16^3 FLIP step 982, now 831 us.  (A cluster of 2 to 8 CTAs
// for levels of 17 to 128 warps lost: 64^3 V-cycle 170 to 182 us, its barrier and halos through L2.)  What
// bounds it is the latency of one colour's update.
constexpr int UNI_MAX_LEVELS = 4;  // 8^3 blocks halve to one cell in three steps
constexpr int ULOW_THREADS = 512;
constexpr int ULOW_WARPS = ULOW_THREADS / 32;
constexpr int ULOW_CELLS = 512 * ULOW_WARPS;  // an 8^3 block a warp at most
constexpr int ULOW_EXACT = 128;  // cells of a coarsest level taken along (its inverse comes from L2: 128 KB)
struct ULowLevel {
    UniView v;   // both colours
    int n0;      // warps of colour 0
    float* xf;
    __half* xh;  // nullptr: FP32 storage
    float* scale;
    const float* b;
    UOut out;    // restricted residual
};
struct ULow {
    ULowLevel lv[UNI_MAX_LEVELS];  // lv[last + 1]: x of the level below
    int first, last, pre, post, iters;
    bool zero, down, up, exact;        // zero: level `first` starts from zero
    float omega;
    const int* idx;                    // the coarsest level's inverse
    const int* ex_n;
    const double* Minv;
    const uint32_t* cell;              // cell offset of a block of the coarsest level
    const float* xb;
};
// x of the walk's current level in shared memory, as the kernels read it back from its storage
struct UXS {
    float* s;
    __device__ __forceinline__ float2 get2(uint32_t i, float, bool even) const {
        if (even) return *reinterpret_cast<const float2*>(s + i);
        return make_float2(s[i], s[i + 1]);
    }
};
struct USrcS {
    using T = float;
    struct Ctx {};
    UXS x;
    __device__ __forceinline__ Ctx ctx(int) const { return Ctx{}; }
    __device__ __forceinline__ float get(uint32_t i, const Ctx&) const { return x.s[i]; }
    __device__ __forceinline__ float coarse(uint32_t, const Ctx&) const { return 0.f; }
};
// the block to shared memory (v0, v1 as stored)
template <int R>
__device__ __forceinline__ void uni_low_put(const ULane<R>& L, float* xs, const float* v0, const float* v1) {
#pragma unroll
    for (int z = 0; z < R; ++z) {
        if (R == 1) xs[L.at] = v0[z];
        else ustore2(xs, L.at + (uint32_t)(R * R * z), L.even, v0[z], v1[z]);
    }
}
// one warp's smoothing of one leg: 1 + ns barriers
template <int R, bool HALF, bool GEN>
__device__ __forceinline__ void uni_low_smooth(const ULow& K, const ULowLevel& l, const ULowLevel& c, int warp, int leg, bool zero, float* xs) {
    const int k = warp >= l.n0, ns = 2 * (leg ? K.post : K.pre);
    const UX<HALF> x{l.xf, l.xh, l.scale};
    using S = USrcS;
    const S src{UXS{xs}};
    ULane<R> L;
    UHalos<R, S, false> H;
    const bool any = L.init(l.v, warp);
    const bool in = L.lane / UG<R>::LPB < (l.v.desc[warp].y & 0xFF);  // a block's lane; air blocks are read too
    H.init(L);
    const int q = (L.y & 1) ^ leg;
    float E[R], O[R], bE[R], bO[R];
    {
        float v0[R], v1[R];
        const bool moved = zero || leg;  // x changes before the first step
        const float sc = zero || !in ? 1.f : x.sc(L.block);
        const float scc = leg && c.xh && L.live ? c.scale[L.block] : 1.f;
#pragma unroll
        for (int z = 0; z < R; ++z) {
            float2 v = make_float2(0.f, 0.f), bv = make_float2(0.f, 0.f);
            const uint32_t i = L.at + (uint32_t)(R * R * z);
            if (in && !zero) v = x.get2(i, sc, L.even);
            if (L.live) {
                uload2(l.b, i, L.even, bv.x, bv.y);
                if (leg) {
                    const uint32_t ci = L.coff + (uint32_t)(L.xp + (R / 2) * ((L.y >> 1) + (R / 2) * (z >> 1)));
                    const float d = c.xh ? umul(__half2float(c.xh[ci]), scc) : c.xf[ci];
                    if ((L.mask >> (2 * z)) & 1u) v.x += d;
                    if ((L.mask >> (2 * z + 1)) & 1u) v.y += d;
                }
            }
            v0[z] = v.x;
            v1[z] = v.y;
            const bool one = ((q ^ z) & 1) != 0;
            bE[z] = one ? bv.y : bv.x;
            bO[z] = one ? bv.x : bv.y;
        }
        if (moved && any) uni_store<R, HALF, true>(L, x, v0, v1);
        if (in) uni_low_put<R>(L, xs, v0, v1);
#pragma unroll
        for (int z = 0; z < R; ++z) {
            const bool one = ((q ^ z) & 1) != 0;
            E[z] = one ? v1[z] : v0[z];
            O[z] = one ? v0[z] : v1[z];
        }
    }
    uint32_t fl;
    UCoef<R> C;
    uni_coef<R>(L, q, C, fl);
    const bool general = GEN && l.v.general[warp];
    if (general) uni_faces<R>(L, l.v.W, C);
    __syncthreads();
#pragma unroll 1
    for (int st = 0; st < ns; ++st) {
        if (((st ^ leg) & 1) == k && any) {
            float hx[R == 2 ? 4 : R], v0[R], v1[R];
            uni_halo<R>(L, H, src, q, hx);
            uni_iterate<R, GEN>(L, C, E, O, bE, bO, hx, H, fl, K.omega, K.iters, general);
#pragma unroll
            for (int z = 0; z < R; ++z) {
                const bool one = ((q ^ z) & 1) != 0;
                v0[z] = one ? O[z] : E[z];
                v1[z] = one ? E[z] : O[z];
            }
            uni_store<R, HALF, true>(L, x, v0, v1);
            if (L.live) uni_low_put<R>(L, xs, v0, v1);
            if (HALF) {
#pragma unroll
                for (int z = 0; z < R; ++z) {
                    const bool one = ((q ^ z) & 1) != 0;
                    E[z] = one ? v1[z] : v0[z];
                    O[z] = one ? v0[z] : v1[z];
                }
            }
        }
        __syncthreads();
    }
}
template <bool HALF>
__device__ __forceinline__ void uni_low_smooth_one(const ULow& K, const ULowLevel& l, const ULowLevel& c, int warp, int leg, bool zero, float* xs) {
    const int k = warp >= l.n0, ns = 2 * (leg ? K.post : K.pre);
    const UX<HALF> x{l.xf, l.xh, l.scale};
    using S = USrcS;
    const S src{UXS{xs}};
    ULane<1> L;
    UHaloOne<S, false> H;
    const bool any = L.init(l.v, warp);
    const bool in = L.lane < (l.v.desc[warp].y & 0xFF);
    H.init(L);
    float v = 0.f, b = 0.f;
    if (in && !zero) v = x.get(L.at, x.sc(L.block));
    if (L.live) {
        b = l.b[L.at];
        if (leg && (L.mask & 1u)) v += c.xh ? umul(__half2float(c.xh[L.coff]), c.scale[L.block]) : c.xf[L.coff];
    }
    if ((zero || leg) && any) uni_store<1, HALF, true>(L, x, &v, &v);
    if (in) xs[L.at] = v;
    const float diag = -(L.wx0 + L.wx1 + L.wy0 + L.wy1 + L.wz0 + L.wz1);
    const float rcp = urcp(diag);
    const bool on = (L.mask & 1u) && !(fabsf(diag) < 1e-9f);
    __syncthreads();
#pragma unroll 1
    for (int st = 0; st < ns; ++st) {
        if (((st ^ leg) & 1) == k && any) {
            H.load(src);
            const float(&h)[6] = H.h;
            if (on)
#pragma unroll 1
                for (int it = 0; it < K.iters; ++it) {
                    float Ax = ufma(L.wx0, h[0], umul(L.wx1, h[1]));
                    Ax = ufma(L.wy0, h[2], Ax);
                    Ax = ufma(L.wy1, h[3], Ax);
                    Ax = ufma(L.wz0, h[4], Ax);
                    Ax = ufma(L.wz1, h[5], Ax);
                    Ax = ufma(diag, v, Ax);
                    v = ufma(K.omega, umul(b - Ax, rcp), v);
                }
            uni_store<1, HALF, true>(L, x, &v, &v);
            if (L.live) xs[L.at] = v;
        }
        __syncthreads();
    }
}
template <bool GEN>
__global__ void __launch_bounds__(ULOW_THREADS, 1) k_uni_low(const __grid_constant__ ULow K) {
    __shared__ __align__(16) float xs[ULOW_CELLS];
    const int wid = threadIdx.x >> 5;
    pdl_wait();
#pragma unroll 1
    for (int leg = K.down ? 0 : 1; leg < (K.up ? 2 : 1); ++leg) {
#pragma unroll 1
        for (int i = 0; i <= K.last - K.first; ++i) {
            const int m = leg ? K.last - i : K.first + i;
            const ULowLevel& l = K.lv[m];
            const ULowLevel& c = K.lv[m + 1];
            const bool zero = leg == 0 && (m > K.first || K.zero);
            const bool has = wid < l.v.nwarp;  // a warp per descriptor
            const int r = has ? l.v.desc[wid].y >> 8 : 0;
#define AW_UB(R) uni_low_smooth<R, false, GEN>(K, l, c, wid, leg, zero, xs)
            if (!has) {
                for (int st = 0; st <= 2 * (leg ? K.post : K.pre); ++st) __syncthreads();
            } else if (l.xh) {
                if (r == 4) uni_low_smooth<4, true, GEN>(K, l, c, wid, leg, zero, xs);
                else if (r == 2) uni_low_smooth<2, true, GEN>(K, l, c, wid, leg, zero, xs);
                else uni_low_smooth_one<true>(K, l, c, wid, leg, zero, xs);
            } else {
                AW_UNI_RES(r, AW_UB, (uni_low_smooth_one<false>(K, l, c, wid, leg, zero, xs)))
            }
#undef AW_UB
            if (leg == 0) {
                if (has) {
                    const USrcS src{UXS{xs}};
#define AW_UB(R)                                                                                                    \
    {                                                                                                               \
        ULane<R> L;                                                                                                 \
        UHalos<R, USrcS, false> E;                                                                                  \
        const bool any = L.init(l.v, wid);                                                                          \
        E.init(L);                                                                                                  \
        if (any)                                                                                                    \
            uni_residual_body<R, USrcS, false, GEN>(L, l.v.W, GEN && l.v.general[wid], E, src, l.b, l.out, 1.f);     \
    }
#define AW_UB1                                                         \
    {                                                                  \
        ULane<1> L;                                                    \
        UHaloOne<USrcS, false> E;                                      \
        const bool any = L.init(l.v, wid);                             \
        E.init(L);                                                     \
        if (any) uni_residual_one<USrcS, false>(L, E, src, l.b, l.out); \
    }
                    AW_UNI_RES(r, AW_UB, AW_UB1)
#undef AW_UB
#undef AW_UB1
                }
                __syncthreads();
            }
        }
        if (leg == 0 && K.exact) {  // x = Minv b, as k_coarse_apply
            const int n = K.ex_n[0], lane = threadIdx.x & 31;
            for (int i = wid; i < n; i += ULOW_WARPS) {
                double t = 0.0;
                for (int j = lane; j < n; j += 32) t += K.Minv[(size_t)i * n + j] * (double)K.xb[K.cell[K.idx[j]]];
                t = warp_sum(t);
                if (lane == 0) K.lv[K.last + 1].xf[K.cell[K.idx[i]]] = (float)t;
            }
            __syncthreads();
        }
    }
    pdl_trigger();
}

// FP64: r64 = b - A p with its FP32 copy r and |r|^2 (k_uni_residual64), or one step of the conjugate
// gradients: q = -A d with d = z + beta d_old formed where it is read (own cells and halo), stored as the
// new direction, and d . q (k_uni_apply).  The direction alternates between two buffers, since a
// neighbour's halo still reads the old one.
template <class S, bool DOT, bool GEN, class F>
__device__ __forceinline__ double uni_residual64(const UniView& V, S& src, const float* b, UOut& out, F begin) {
    const int w = blockIdx.x * UWARPS + (threadIdx.x >> 5);
    double acc = 0.0;
    if (w >= V.nwarp) {
        pdl_wait();
        return 0.0;
    }
    const int warp = V.first + w;
    const int r = V.desc[warp].y >> 8;
#define AW_UB(R)                                                          \
    {                                                                     \
        ULane<R> L;                                                       \
        UHalos<R, S, false> H;                                            \
        const bool any = L.init(V, warp);                                 \
        H.init(L);                                                        \
        pdl_wait();                                                       \
        begin();                                                          \
        if (any)                                                          \
            acc = uni_residual_body<R, S, DOT, GEN>(L, V.W, GEN && V.general[warp], H, src, b, out, 1.f); \
    }
#define AW_UB1                                                            \
    {                                                                     \
        ULane<1> L;                                                       \
        UHaloOne<S, false> H;                                             \
        const bool any = L.init(V, warp);                                 \
        H.init(L);                                                        \
        pdl_wait();                                                       \
        begin();                                                          \
        if (any) acc = uni_residual_one<S, DOT>(L, H, src, b, out);       \
    }
    AW_UNI_RES(r, AW_UB, AW_UB1)
#undef AW_UB
#undef AW_UB1
    return acc;
}
template <bool GEN>
__global__ void __launch_bounds__(UNT, 3) k_uni_residual64(const __grid_constant__ UniView V, USrcD src,
                                                           const float* __restrict__ b, UOut out,
                                                           double* part, unsigned* ticket, double* sum) {
    const double acc = uni_residual64<USrcD, false, GEN>(V, src, b, out, []() {});
    last_cta_sum(acc, part, ticket, [&](double t) { *sum = t; });
}
// sc = {rho, rho_old}, st = {iterations, restart}: d1 becomes the direction in even iterations, d0 in odd
template <bool GEN>
__global__ void __launch_bounds__(UNT, 3) k_uni_apply(const __grid_constant__ UniView V, const float* __restrict__ z, double* d0, double* d1,
                                                      UOut out, const double* __restrict__ sc, const int* __restrict__ st,
                                                      double* part, unsigned* ticket, double* sum) {
    USrcDir src{z, d0, 0.0, true};
    const double acc = uni_residual64<USrcDir, true, GEN>(V, src, nullptr, out, [&]() {
        const bool odd = (st[0] & 1) != 0;
        src.first = st[1] != 0;
        src.beta = src.first ? 0.0 : sc[0] / sc[1];
        src.d = odd ? d1 : d0;
        out.dnew = odd ? d0 : d1;
    });
    pdl_trigger();
    last_cta_sum(acc, part, ticket, [&](double t) { *sum = t; });
}

// ------------------------------------------------------------------------------------------------
// Per solve: which blocks are uniform, their weights, fluid masks and states
// ------------------------------------------------------------------------------------------------
// A block is uniform when every face between two of its cells has one conductance and every side of
// the block has one; a block without fluid takes no part (its x is set to 0, which its neighbours
// read, and so are its b and r, as the staged kernels leave them).
struct UCheck {
    const uint8_t* fluid;
    float* x;       // FP32 storage of the level's x to clear in air blocks (nullptr: keep)
    __half* xh;     // FP16 storage
    float* scale;
    float *b, *r, *q;  // cleared there too (nullptr: keep)
    double *d0, *d1;  // FP64 vectors to clear there too
    float4* wt;
    uint16_t* mask;
    uint8_t* general;
    int* count;     // += blocks that are not uniform
};
struct UCheckAll {
    UniView v[UNI_MAX_LEVELS];
    UCheck k[UNI_MAX_LEVELS];
};
template <int R>
__device__ __forceinline__ void uni_check_body(const UniView& V, const UCheck& K, int warp) {
    using G = UG<R>;
    const int lane = threadIdx.x & 31, s = lane / G::LPB, li = lane % G::LPB;
    const int y = li / G::XP, xp = li % G::XP;
    const int2 d = V.desc[warp];
    const bool valid = s < (d.y & 0xFF);
    const int slot = d.x + (valid ? s : 0);
    const int* rec = reinterpret_cast<const int*>(V.rec + (size_t)slot * UREC);
    const uint32_t off = (uint32_t)rec[0];
    // fluid bits
    uint32_t m = 0;
    if (valid)
#pragma unroll
        for (int z = 0; z < R; ++z)
#pragma unroll
            for (int i = 0; i < G::NI; ++i) {
                const uint32_t c = off + (uint32_t)(G::NI * xp + i + R * (y + R * z));
                if (K.fluid[c]) m |= 1u << (2 * z + i);
            }
    K.mask[(size_t)warp * 32 + lane] = (uint16_t)m;
    uint32_t any = m;
#pragma unroll
    for (int o = 1; o < G::LPB; o <<= 1) any |= __shfl_xor_sync(0xffffffffu, any, o);
    // weights
    constexpr int nf = (R + 1) * R * R;
    const uint32_t f0 = (uint32_t)rec[22], f1 = (uint32_t)rec[23], f2 = (uint32_t)rec[24];
    const float* w0 = V.W.w[0] + f0;
    const float* w1 = V.W.w[1] + f1;
    const float* w2 = V.W.w[2] + f2;
    const float wx0 = w0[0], wx1 = w0[R], wy0 = w1[0], wy1 = w1[R * R], wz0 = w2[0], wz1 = w2[R * R * R];
    const float wi = R >= 2 ? w0[1] : wx0;
    // UB values of each axis in flight per lane (one at a time, 54 dependent round trips of an 8^3 block took
    // 31 us a launch)
    constexpr int UB = 6;
    bool same = true;
#pragma unroll 1
    for (int i0 = li; i0 < nf; i0 += UB * G::LPB) {
        float a0[UB], a1[UB], a2[UB];
#pragma unroll
        for (int k = 0; k < UB; ++k) {
            const int i = min(i0 + k * G::LPB, nf - 1);
            a0[k] = w0[i];
            a1[k] = w1[i];
            a2[k] = w2[i];
        }
#pragma unroll
        for (int k = 0; k < UB; ++k) {
            const int i = min(i0 + k * G::LPB, nf - 1);
            const int fx = i % (R + 1), fy = (i / R) % (R + 1), fz = i / (R * R);
            same = same && a0[k] == (fx == 0 ? wx0 : (fx == R ? wx1 : wi));
            same = same && a1[k] == (fy == 0 ? wy0 : (fy == R ? wy1 : wi));
            same = same && a2[k] == (fz == 0 ? wz0 : (fz == R ? wz1 : wi));
        }
    }
    int ok = same;
#pragma unroll
    for (int o = 1; o < G::LPB; o <<= 1) ok &= __shfl_xor_sync(0xffffffffu, ok, o);
    const int state = any == 0 ? US_AIR : (ok ? US_UNIFORM : US_GENERAL);
    if (valid && state == US_AIR) {
        for (int z = 0; z < R; ++z)
            for (int i = 0; i < G::NI; ++i) {
                const uint32_t c = off + (uint32_t)(G::NI * xp + i + R * (y + R * z));
                if (K.x) K.x[c] = 0.f;
                if (K.xh) K.xh[c] = __float2half_rn(0.f);
                if (K.b) K.b[c] = 0.f;
                K.r[c] = 0.f;
                if (K.q) K.q[c] = 0.f;
                if (K.d0) K.d0[c] = K.d1[c] = 0.0;
            }
        if (K.xh && li == 0) K.scale[rec[1]] = 0.f;
    }
    // (the six faces of one cell are its six sides)
    const unsigned gen = __ballot_sync(0xffffffffu, R > 1 && valid && li == 0 && state == US_GENERAL);
    if (lane == 0) {
        K.general[warp] = gen != 0;
        if (gen) atomicAdd(K.count, __popc(gen));
    }
    if (valid && li == 0) {
        K.wt[2 * (size_t)slot] = make_float4(wi, wx0, wx1, wy0);
        K.wt[2 * (size_t)slot + 1] = make_float4(wy1, wz0, wz1, __int_as_float(state));
    }
}
// level = blockIdx.y
__global__ void __launch_bounds__(UNT) k_uni_check(const __grid_constant__ UCheckAll A) {
    const UniView& V = A.v[blockIdx.y];
    const UCheck& K = A.k[blockIdx.y];
    const int warp = blockIdx.x * UWARPS + (threadIdx.x >> 5);
    if (warp >= V.nwarp) return;
    const int r = V.desc[warp].y >> 8;
#define AW_UB(R) uni_check_body<R>(V, K, warp)
    AW_UNI_RES(r, AW_UB, AW_UB(1))
#undef AW_UB
}

// Slot records of one level (geometry only), one thread per slot.
struct MetaSrc {
    const int* res;
    const uint32_t* off[4];
};
__global__ void k_build_records(Geo geo, const int* __restrict__ blocks, int n, MetaSrc h, MetaSrc coarser, int* __restrict__ recs) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const int b = blocks[j];
    const int r = h.res[b];
    int* rec = recs + (size_t)j * 4 * UREC;
    int kinds = 0;
    int c[3];
    bcoord(geo, b, c);
    for (int f = 0; f < 6; ++f) {
        int nc[3] = {c[0], c[1], c[2]};
        nc[f >> 1] += (f & 1) ? 1 : -1;
        int o = 0, nbk = 0, oc = 0;
        if (inside(geo, nc)) {
            const int q = bidx(geo, nc[0], nc[1], nc[2]);
            const int rn = h.res[q];
            if (rn) {
                o = (int)h.off[0][q];
                nbk = q;
                kinds |= (rn == r ? 2 : (rn < r ? 3 : 4)) << (4 * f);
                if (coarser.res) {
                    oc = (int)coarser.off[0][q];
                    if (rn == 2 * coarser.res[q]) kinds |= 1 << (24 + f);
                }
            }
        }
        rec[4 + f] = o;
        rec[10 + f] = nbk;
        rec[16 + f] = oc;
    }
    rec[0] = (int)h.off[0][b];
    rec[1] = b;
    rec[2] = kinds;
    rec[3] = coarser.res ? (int)coarser.off[0][b] : 0;
    for (int a = 0; a < 3; ++a) rec[22 + a] = (int)h.off[1 + a][b];
    for (int k = 25; k < 4 * UREC; ++k) rec[k] = 0;
}

}  // namespace aw
