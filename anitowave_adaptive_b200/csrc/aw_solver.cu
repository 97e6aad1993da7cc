// aw_solver.cu — multigrid pressure solver on the MSBG: block red-black smoother, residual,
// restriction/prolongation, uniform coarse levels, FP64 coarsest solve, FP32 and mixed solves.
//
// Reference behaviour followed (paths within the reference project):
//   Smoother.cuh:23-94    ghost values across blocks (getPressureLevel; T-junction rule D8 fixed)
//   Smoother.cuh:105-202  smoothActiveBlocks: block parity colouring, <= MAX_BLOCK_ITER block-local
//                         red-black GS sweeps, early exit at TARGET_RESIDUAL_REDUCTION, activation
//   Smoother.cuh:249-291  solveLevel: active set per iteration (here device flags, no host sync)
//   VCycle.cuh:81-131     computeExplicitResidual
//   MultigridTransfer.cuh:9-102 restriction (8-child sum) / prolongation (injection add)
//   VCycle.cuh:177-304    init (coarse offsets, Galerkin) and recursive runCycle
//
// B200 design: finite-volume solves on blocks of up to 8^3 cells run out of registers, a group of lanes per
// block (aw_uniform.cuh), the smallest block-structured levels in one CTA (k_uni_low).  The staged kernels
// here serve the rest (larger blocks, residual tracking, deactivation, the reference's operator, the level
// calls): a CTA per batch of blocks with the blocks and a one-cell halo in shared memory; the smoother runs
// all its block-local sweeps there and touches HBM once per launch.  Uniform coarse levels continue below one
// cell per block (k_dense_tail from 4096 cells on) and end in an FP64 dense solve (Cholesky inverse built on
// the device each setup).
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <memory>

#include "aw_internal.cuh"
#include "aw_uniform.cuh"

namespace aw {

static inline unsigned nblk(size_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }
aw_status level_offsets(MsbgState& G, int m, int vanish, uint32_t* d_off4, int* d_res, uint32_t tot[4], cudaStream_t s);
__global__ void k_galerkin_ref(Geo g, const uint32_t* __restrict__ level, int axis, int dest,
                               const float* __restrict__ fine, float* __restrict__ coarse,
                               const uint32_t* __restrict__ foff, const uint32_t* __restrict__ coff);

constexpr int EXACT_CAP = 512;       // largest coarsest system factorised densely
constexpr int EXACT_POS_CAP = 32768; // largest coarsest grid scanned by the factor kernel

struct MGLevel {
    bool dense = false;
    int D[3] = {0, 0, 0};
    float H = 0.f;
    bool half = false;  // x stored as FP16 + per-block scale
    DBuf<int> res;
    std::vector<int> h_res;
    DBuf<uint32_t> off[4];
    uint32_t tot[4] = {0, 0, 0, 0};
    // CTA batches: [0]/[1] blocks of one colour, [2] all blocks; each entry {first, count, res, 0}, the
    // block of every slot and the slot metadata (NMETA fields x slots, field-major), in one allocation
    DBuf<int4> batches;
    int4* desc[3] = {};
    int* blk[3] = {};
    int* meta[3] = {};
    int nslots[3] = {0, 0, 0};
    int ndesc[3] = {0, 0, 0};
    // dynamic shared memory of the batched kernels on this level
    size_t smem_smooth = 0, smem_x64 = 0, smem_prolong = 0, smem_meta = 0;
    int maxres = 0;
    // the same blocks as warps of the uniform-coefficient kernels (aw_uniform.cuh): colour 0, colour 1
    int2* udesc = nullptr;  // these five lie in the solver's uslab
    int4* urec = nullptr;
    float4* uwt = nullptr;
    uint16_t* umask = nullptr;
    uint8_t* ugeneral = nullptr;
    int uwarps[2] = {0, 0};
    DBuf<float> W[3], bbar[3];
    DBuf<uint8_t> fluid;
    DBuf<float> x, b, r;
    DBuf<__half> xh;
    DBuf<float> xscale;
    DBuf<uint8_t> status[2];
    size_t ncell() const { return dense ? (size_t)D[0] * D[1] * D[2] : tot[0]; }
    size_t nface(int a) const {
        return dense ? (size_t)(D[0] + (a == 0)) * (D[1] + (a == 1)) * (D[2] + (a == 2)) : tot[1 + a];
    }
};

}  // namespace aw

struct aw_solver {
    aw_msbg* g = nullptr;
    aw_solver_desc d{};
    std::vector<aw::MGLevel> lv;
    int nmsbg = 0;
    // coarsest exact solve
    bool exact = false;
    aw::DBuf<double> M, Minv;
    aw::DBuf<int> ex_idx, ex_n, ex_pos;
    aw::DBuf<uint8_t> ex_prev;  // coarsest fluid flags of the last factorisation (per position)
    bool coef_dirty = true;     // coefficients changed since the last factorisation
    // level-0 bindings for the current solve
    float* x0 = nullptr;
    const float* b0 = nullptr;
    // the hierarchy runs the register-resident kernels of aw_uniform.cuh (FV mode, 8^3 blocks at most, no
    // activation or early exit)
    bool uni = false;
    unsigned gen = 0;  // bit m: level m has blocks without a single conductance (the current solve's check)
    bool keep_r = true;  // the cycles store every level's residual (not those that precondition a CG solve)
    aw::DBuf<int4> uslab;  // slot records, weights, masks and warp descriptors of every level
    // mixed precision: FP64 vectors of the conjugate-gradient outer loop (residual, direction (two
    // buffers: the uniform form reads the old one while it writes the new), -A d), its scalars
    // {rho, rho_old, d.(-A d)} and a zero right-hand side for applying A
    aw::DBuf<double> cg_r, cg_d, cg_d2, cg_q, cg_sc;
    // aligned copies of a caller's b and p that do not start on 16 bytes (aw_solve)
    aw::DBuf<float> b_copy;
    aw::DBuf<double> p_copy;
    aw::DBuf<unsigned> ticket;  // last_cta_sum: finished CTAs of the running launch (0 between launches)
    aw::DBuf<float> cg_zero;
    // FP32 conjugate gradients: direction, -A d, scalars {rho, rho_old, d.(-A d)}, partial sums
    aw::DBuf<float> cg32_d, cg32_q, cg32_sc, partials32;
    aw::DBuf<double> partials, norm;
    size_t smem_max = 0, smem_max64 = 0;
    // the whole V-cycle as a CUDA graph, captured once per (x0, b0) binding: aw_solve's and aw_vcycle_run's, so
    // that a program that calls both in turn captures neither again.  Of aw_solve's graphs the last two are kept:
    // a program may solve for one density and for a varying one, or for two pressure arrays, in turn.
    cudaStream_t cap = nullptr;
    struct Cycle {
        cudaGraphExec_t exec = nullptr;
        const void *x0 = nullptr, *b0 = nullptr;
        unsigned form = ~0u;  // 2 * gen + (level-0 x starts at zero)
        unsigned long long kernels = 0;
        void drop() {
            if (exec) cudaGraphExecDestroy(exec);
            exec = nullptr;
        }
    } solve_cycle[2], call_cycle;
    int solve_last = 0;          // the solve_cycle used last
    bool vcycle_called = false;  // aw_vcycle_run ran since the solver was built
    // the mixed-precision CG iterations as one graph with a device-side while loop, per pressure
    // array and gen (the last two); cgst = {iterations, restart flag, iteration limit}, cgprm = {||b||, tolerance}
    struct Loop {
        cudaGraphExec_t exec = nullptr;
        const void* p = nullptr;
        unsigned gen = 0;
        unsigned long long kernels = 0;
        void drop() {
            if (exec) cudaGraphExecDestroy(exec);
            exec = nullptr;
        }
    } cgloop[2];
    int cgloop_last = 0;  // the one used last
    bool use_devloop = true;
    aw::DBuf<int> cgst;
    aw::DBuf<double> cgprm;
    bool use_graph = true;
    bool use_pdl = true;  // V-cycle kernels as programmatic dependent launches
    bool full_next = false;  // the next of them starts after its predecessor has ended (launch_dep)
    int low = 1 << 30;    // first level of those that k_uni_low walks
    int tail = 0;         // first level of the uniform tail run as one k_dense_tail launch (0: none)
    double* h_norm = nullptr;  // pinned host words: a squared norm, uniform_check's counts
    double* h_cg = nullptr;    // pinned host words of the device-loop state
    ~aw_solver() {
        for (Cycle& c : solve_cycle) c.drop();
        call_cycle.drop();
        for (Loop& l : cgloop) l.drop();
        if (cap) cudaStreamDestroy(cap);
        if (h_norm) cudaFreeHost(h_norm);
        if (h_cg) cudaFreeHost(h_cg);
    }
};

namespace aw {

struct SmoothParams {
    float omega, target, theta;
    int iters;
    int check_fluid;
    int reverse;  // visit the cell colours black, red (the adjoint order of red, black)
};

__host__ __device__ inline int xi3(int x, int y, int z, int R2) { return (x + 1) + R2 * ((y + 1) + R2 * (z + 1)); }

__device__ inline float block_max(float v, float* red) {
    v = warp_max(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) red[w] = v;
    __syncthreads();
    if (w == 0) {
        float t = lane < (int)(blockDim.x >> 5) ? red[lane] : 0.f;
        t = warp_max(t);
        if (lane == 0) red[32] = t;
    }
    __syncthreads();
    float out = red[32];
    __syncthreads();
    return out;
}

__device__ inline double block_sum(double v, double* red) {
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) red[w] = v;
    __syncthreads();
    double out = 0.0;
    if (w == 0) {
        double t = lane < (int)(blockDim.x >> 5) ? red[lane] : 0.0;
        out = warp_sum(t);
    }
    __syncthreads();
    return out;  // valid in thread 0
}

// ------------------------------------------------------------------------------------------------
// Batched block kernels.  A CTA serves `count` blocks ("slots") of one resolution r, listed
// contiguously: 1 block of 8^3 or 16^3 cells, 4 of 4^3, 16 of 2^3, 64 of 1^3.  Every slot keeps
// its block and a one-cell halo in shared memory; slots never interact (same colour = no shared
// faces), so each slot's arithmetic, early exit and activation are exactly those of a CTA that
// owns one block.
// ------------------------------------------------------------------------------------------------
struct Batch {
    const int4* desc;  // {first slot, count, res, 0}
    const int* meta;   // batch-ordered slot metadata, NMETA fields x nslots (field-major)
    int nslots;
};

// Slot metadata fields.  The host lays them out in batch order when the solver is created, so a CTA
// reads its slots' block ids, offsets and face neighbours with one coalesced round trip after the
// descriptor instead of chasing block id -> offsets -> neighbour offsets.
enum {
    MF_BLOCK = 0,        // block id
    MF_OFF = 1,          // 4 fields: cells, faces x, y, z of this level
    MF_NB = 5,           // 6 directions (2a + (s > 0)) x {neighbour cell offset, kind, neighbour block}
    MF_FINE_OFF = 23,    // cell offset and resolution of the block on the next finer level
    MF_FINE_RES = 24,
    MF_COARSE_OFF = 25,  // ... and on the next coarser level
    MF_COARSE_RES = 26,
    NMETA = 27
};

// Face-neighbour kinds: 0 = outside the domain or absent (ghost 0), 2 = same resolution,
// 3 = coarser neighbour (parent cell), 4 = finer neighbour (mean of the 4 touching cells).
enum { NB_NONE = 0, NB_SAME = 2, NB_COARSE = 3, NB_FINE = 4 };

// Every thread of a batched CTA only ever touches cells of one slot (G * r^3 <= 256, or G == 1).
// Reduce a per-thread non-negative value over the threads of each slot: shuffle within aligned
// groups of min(r^3, 32) lanes, then one shared atomicMax per group.
__device__ inline void slot_max(int* dst, int n3, float v) {
    const int grp = n3 < 32 ? n3 : 32;
    int iv = __float_as_int(v);
    for (int o = 1; o < grp; o <<= 1) iv = max(iv, __shfl_xor_sync(0xffffffffu, iv, o));
    if ((threadIdx.x & (grp - 1)) == 0 && iv > 0) atomicMax(dst, iv);
}

// ---- asynchronous global -> shared copies (completion via cp.async.wait_all) ----
__device__ inline uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ inline void cp_async4(void* s, const void* g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(smem_addr(s)), "l"(g) : "memory");
}
__device__ inline void cp_async8(void* s, const void* g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(smem_addr(s)), "l"(g) : "memory");
}
__device__ inline void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
// Sources of x for staging: FP32 (copied asynchronously), FP16 + per-block scale (decoded in
// registers), FP64 (copied asynchronously).
struct SrcX {
    XStore x;
    using T = float;
    __device__ bool async() const { return x.f != nullptr; }
    __device__ float get(uint32_t i, int b) const { return x.get(i, b); }
    __device__ void copy(float* dst, uint32_t i) const { cp_async4(dst, x.f + i); }
};
struct SrcD {
    const double* p;
    using T = double;
    __device__ bool async() const { return true; }
    __device__ double get(uint32_t i, int) const { return p[i]; }
    __device__ void copy(double* dst, uint32_t i) const { cp_async8(dst, p + i); }
};

// (p0, p1, p2) given along the axes (a, a+1, a+2) mod 3 -> (x, y, z)
__device__ inline void rot3(int a, int p0, int p1, int p2, int& x, int& y, int& z) {
    x = a == 0 ? p0 : (a == 1 ? p2 : p1);
    y = a == 0 ? p1 : (a == 1 ? p0 : p2);
    z = a == 0 ? p2 : (a == 1 ? p1 : p0);
}

// Every batched CTA runs NT threads over G slots of one resolution R (a power of two, 1..16), so
// that G * R^3 <= NT or G == 1.  The kernels switch on R once per CTA and run a body compiled for
// that R: every index split is then a shift, a mask or a multiply by a constant, and every loop
// has a fixed trip count.
constexpr int NT = 256;
// CTAs per SM the batched block kernels are compiled for (registers per thread <= 64K / (NT x this))
#ifndef AW_BLOCK_CTAS_PER_SM
#define AW_BLOCK_CTAS_PER_SM 6
#endif
// loads in flight per thread when staging decoded or averaged halo values
#ifndef AW_STAGE_BATCH
#define AW_STAGE_BATCH 2
#endif

template <int R>
struct Geom {
    static constexpr int n3 = R * R * R, rr = R * R, nf = (R + 1) * R * R, R2 = R + 2, X3 = R2 * R2 * R2;
    static constexpr int FS = n3 + 3 * nf;  // b, then the three face-coefficient arrays
    static constexpr int FW = n3 / 4 + 2;   // 32-bit words that cover a block's fluid bytes
    static constexpr int GMAX = n3 >= NT ? 1 : NT / n3;
};

#define AW_SWITCH_RES(r, BODY) \
    switch (r) {               \
        case 1: BODY(1); break;  \
        case 2: BODY(2); break;  \
        case 4: BODY(4); break;  \
        case 8: BODY(8); break;  \
        default: BODY(16); break; \
    }

// Shared-memory image of a batched CTA: per slot x with a one-cell halo (xs, (R+2)^3 values of
// type T), b and the face coefficients (fs), the fluid words (fw) and the slot metadata.
template <class T, int R>
struct SlotImage {
    using Gm = Geom<R>;
    T* xs;
    int* meta;
    float* fs;
    uint32_t* fw;
    int G;
    __device__ SlotImage(void* base, int G_) : G(G_) {
        xs = (T*)base;
        meta = (int*)(xs + G * Gm::X3);
        fs = (float*)(meta + NMETA * G);
        fw = (uint32_t*)(fs + G * Gm::FS);
    }
    __device__ int m(int f, int sl) const { return meta[f * G + sl]; }
    __device__ uint32_t off(int k, int sl) const { return (uint32_t)meta[(MF_OFF + k) * G + sl]; }
    __device__ bool fluid(int sl, int i) const {
        return ((const uint8_t*)(fw + sl * Gm::FW))[(off(0, sl) & 3u) + i] != 0;
    }
};

__host__ __device__ inline size_t slot_image_bytes(int G, int r, size_t tsize) {
    const size_t n3 = (size_t)r * r * r, nf = (size_t)(r + 1) * r * r, X3 = (size_t)(r + 2) * (r + 2) * (r + 2);
    return (size_t)G * (X3 * tsize + NMETA * 4 + (n3 + 3 * nf) * 4 + (n3 / 4 + 2) * 4) + 16;
}

// Stage the metadata of a CTA's G slots into meta[NMETA * G] (one round trip); slots whose block is
// inactive (status[b] == 0) get block id -1.
template <int R>
__device__ inline void stage_meta(int* meta, int G, const Batch& B, int first, const uint8_t* __restrict__ status) {
    constexpr int GM = Geom<R>::GMAX;
    const int t = threadIdx.x % GM;
    if (t < G)
        for (int f = threadIdx.x / GM; f < NMETA; f += NT / GM)
            cp_async4(meta + f * G + t, B.meta + (size_t)f * B.nslots + first + t);
    cp_async_wait_all();
    __syncthreads();
    if (status) {
        for (int s = threadIdx.x; s < G; s += NT)
            if (!status[meta[s]]) meta[s] = -1;
        __syncthreads();
    }
}

struct MetaView {
    const int* p;
    int G;
    __device__ int m(int f, int sl) const { return p[f * G + sl]; }
    __device__ uint32_t off(int k, int sl) const { return (uint32_t)p[(MF_OFF + k) * G + sl]; }
};

// Register-batched staging of values that need a decode or a mean: the FP16 interior cells and the
// halo cells (0, 1 or 4 sources each).  K items per thread are addressed, then loaded, then
// stored, so that their loads are in flight together.
template <int R, class Src, bool HALO>
__device__ inline void stage_items(SlotImage<typename Src::T, R>& S, const Src& x) {
    using T = typename Src::T;
    using Gm = Geom<R>;
    constexpr int GM = Gm::GMAX, n3 = Gm::n3, rr = Gm::rr, K = AW_STAGE_BATCH;
    constexpr int NI = HALO ? GM * 6 * rr : GM * n3;
#pragma unroll
    for (int base = 0; base < NI; base += K * NT) {
        uint32_t src[K][4];
        int ns[K], blk[K], dst[K];
        T raw[K][4];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int t = base + k * NT + threadIdx.x;
            ns[k] = 0;
            dst[k] = -1;
            blk[k] = 0;
            if (t >= NI) continue;
            if (!HALO) {
                const int sl = t / n3, i = t % n3;
                if (sl >= S.G) continue;
                const int b = S.m(MF_BLOCK, sl);
                if (b < 0) continue;
                ns[k] = 1;
                src[k][0] = S.off(0, sl) + i;
                blk[k] = b;
                dst[k] = sl * Gm::X3 + xi3(i % R, (i / R) % R, i / rr, Gm::R2);
                continue;
            }
            const int sl = t / (6 * rr), rem0 = t % (6 * rr);
            if (sl >= S.G || S.m(MF_BLOCK, sl) < 0) continue;
            const int face = rem0 / rr, rem = rem0 % rr;
            const int a = face >> 1, sd = (face & 1) ? 1 : -1;
            const int u = rem % R, v = rem / R;  // coordinates along the axes a+1 and a+2
            const int kind = S.m(MF_NB + 3 * face + 1, sl);
            if (kind != NB_NONE) {
                const uint32_t o = (uint32_t)S.m(MF_NB + 3 * face, sl);
                blk[k] = S.m(MF_NB + 3 * face + 2, sl);
                const int rn = kind == NB_SAME ? R : (kind == NB_COARSE ? R / 2 : 2 * R);
                const int qa = sd > 0 ? 0 : rn - 1;
                int qx, qy, qz;
                if (kind != NB_FINE) {
                    const int sh = kind == NB_SAME ? 0 : 1;
                    rot3(a, qa, u >> sh, v >> sh, qx, qy, qz);
                    ns[k] = 1;
                    src[k][0] = o + cidx(qx, qy, qz, rn);
                } else {
                    ns[k] = 4;
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        rot3(a, qa, 2 * u + (e >> 1), 2 * v + (e & 1), qx, qy, qz);
                        src[k][e] = o + cidx(qx, qy, qz, rn);
                    }
                }
            }
            int hx, hy, hz;
            rot3(a, sd > 0 ? R : -1, u, v, hx, hy, hz);
            dst[k] = sl * Gm::X3 + xi3(hx, hy, hz, Gm::R2);
        }
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
            for (int e = 0; e < 4; ++e) raw[k][e] = e < ns[k] ? x.get(src[k][e], blk[k]) : T(0);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (dst[k] < 0) continue;
            T v;
            if (ns[k] == 4) {
                T sum = T(0);
#pragma unroll
                for (int e = 0; e < 4; ++e) sum += raw[k][e];
                v = T(0.25) * sum;
            } else {
                v = raw[k][0];
            }
            S.xs[dst[k]] = v;
        }
    }
}

// Stage x (interior + halo), b, the face coefficients and the fluid flags of every live slot.
// Every global load is issued before the first wait: plain copies go through cp.async, decoded
// and averaged values through register batches, so that a CTA pays about one memory round trip.
template <int R, class Src>
__device__ inline void stage_data(SlotImage<typename Src::T, R>& S, const Src& x, const float* __restrict__ bvec, Coef3 W,
                                  const uint8_t* __restrict__ fluid) {
    using Gm = Geom<R>;
    constexpr int GM = Gm::GMAX, n3 = Gm::n3, nf = Gm::nf;
    const bool xa = x.async();
#pragma unroll
    for (int t0 = 0; t0 < GM * n3; t0 += NT) {
        const int t = t0 + threadIdx.x, sl = t / n3, i = t % n3;
        if (sl >= S.G || S.m(MF_BLOCK, sl) < 0) continue;
        const uint32_t oc = S.off(0, sl);
        if (xa) x.copy(S.xs + sl * Gm::X3 + xi3(i % R, (i / R) % R, i / Gm::rr, Gm::R2), oc + i);
        cp_async4(S.fs + sl * Gm::FS + i, bvec + oc + i);
    }
#pragma unroll 4
    for (int t0 = 0; t0 < GM * 3 * nf; t0 += NT) {
        const int t = t0 + threadIdx.x;
        if (t >= GM * 3 * nf) break;
        const int sl = t / (3 * nf), j = t % (3 * nf);
        if (sl >= S.G || S.m(MF_BLOCK, sl) < 0) continue;
        const int a = j / nf;
        const float* wa = a == 0 ? W.w[0] : (a == 1 ? W.w[1] : W.w[2]);
        cp_async4(S.fs + sl * Gm::FS + n3 + j, wa + S.off(1 + a, sl) + (j - a * nf));
    }
    if (fluid) {
        const uint32_t* fwg = (const uint32_t*)fluid;
#pragma unroll
        for (int t0 = 0; t0 < GM * Gm::FW; t0 += NT) {
            const int t = t0 + threadIdx.x;
            if (t >= GM * Gm::FW) break;
            const int sl = t / Gm::FW, w = t % Gm::FW;
            if (sl >= S.G || S.m(MF_BLOCK, sl) < 0) continue;
            const uint32_t oc = S.off(0, sl);
            if (w * 4 < (int)(oc & 3u) + n3) cp_async4(S.fw + sl * Gm::FW + w, fwg + (oc >> 2) + w);
        }
    }
    if (!xa) stage_items<R, Src, false>(S, x);
    stage_items<R, Src, true>(S, x);
    cp_async_wait_all();
}

// Write every slot's x back: FP32, or FP16 with a fresh per-block scale.  sb/off0 are per-slot
// block ids (-1 = skip) and cell offsets in shared memory.
template <int R>
__device__ inline void store_slots(const XStore& x, const int* sb, const int* off0, int G, const float* xs, int* smax) {
    using Gm = Geom<R>;
    constexpr int GM = Gm::GMAX, n3 = Gm::n3;
    if (x.f) {
#pragma unroll
        for (int t0 = 0; t0 < GM * n3; t0 += NT) {
            const int t = t0 + threadIdx.x, sl = t / n3, i = t % n3;
            if (sl >= G || sb[sl] < 0) continue;
            x.f[(uint32_t)off0[sl] + i] = xs[sl * Gm::X3 + xi3(i % R, (i / R) % R, i / Gm::rr, Gm::R2)];
        }
        return;
    }
    for (int t = threadIdx.x; t < G; t += NT) smax[t] = 0;
    __syncthreads();
    {
        float m = 0.f;
#pragma unroll
        for (int t0 = 0; t0 < GM * n3; t0 += NT) {
            const int t = t0 + threadIdx.x, sl = t / n3, i = t % n3;
            if (sl >= G || sb[sl] < 0) continue;
            m = fmaxf(m, fabsf(xs[sl * Gm::X3 + xi3(i % R, (i / R) % R, i / Gm::rr, Gm::R2)]));
        }
        const int sl = GM == 1 ? 0 : min((int)threadIdx.x / n3, G - 1);
        slot_max(&smax[sl], n3, m);
    }
    __syncthreads();
#pragma unroll
    for (int t0 = 0; t0 < GM * n3; t0 += NT) {
        const int t = t0 + threadIdx.x, sl = t / n3, i = t % n3;
        if (sl >= G || sb[sl] < 0) continue;
        const float m = __int_as_float(smax[sl]);
        const float inv = m > 0.f ? 32768.f / m : 0.f;
        x.h[(uint32_t)off0[sl] + i] = __float2half_rn(xs[sl * Gm::X3 + xi3(i % R, (i / R) % R, i / Gm::rr, Gm::R2)] * inv);
    }
    for (int t = threadIdx.x; t < G; t += NT)
        if (sb[t] >= 0) {
            const float m = __int_as_float(smax[t]);
            x.scale[sb[t]] = m > 0.f ? m * (1.f / 32768.f) : 0.f;
        }
}

// Shared smoother state of one CTA (one entry per slot).
struct SmoothShared {
    int smr[NT], sdone[NT];
    float sinit[NT];
};

template <int R>
__device__ inline void smooth_body(int4 d, unsigned char* smraw, SmoothShared& Z, const LevelView& L, const XStore& x,
                                   const float* __restrict__ bvec, const Coef3& W, const uint8_t* __restrict__ fluid,
                                   const Batch& B, const uint8_t* __restrict__ status, uint8_t* __restrict__ status_next,
                                   const SmoothParams& P) {
    using Gm = Geom<R>;
    constexpr int GM = Gm::GMAX, n3 = Gm::n3, nf = Gm::nf, R2 = Gm::R2, sy = R2, sz = R2 * R2;
    SlotImage<float, R> S(smraw, d.y);
    const int G = S.G;
    if (status) pdl_wait();  // the activation flags come from the previous sweep
    stage_meta<R>(S.meta, G, B, d.x, status);
    const int* sb = S.meta + MF_BLOCK * G;
    if (!__syncthreads_or(threadIdx.x < G && sb[threadIdx.x] >= 0)) return;
    pdl_wait();
    for (int t = threadIdx.x; t < G; t += NT) {
        Z.smr[t] = 0;
        Z.sdone[t] = 0;
        Z.sinit[t] = -1.f;
    }
    stage_data<R>(S, SrcX{x}, bvec, W, P.check_fluid ? fluid : nullptr);
    __syncthreads();
    const int my_slot = GM == 1 ? 0 : min((int)threadIdx.x / n3, G - 1);
    // The per-slot residual maximum feeds the early exit and the activation of neighbours.  With no
    // activation output and no exit possible (at most two sweeps and a reduction target below 1:
    // the first sweep only records the initial residual), it is skipped with its two barriers.
    const bool track = status_next || (P.target > 0.f && (P.iters > 2 || (P.iters == 2 && P.target >= 1.f)));
    for (int bi = 0; bi < P.iters; ++bi) {
        float lmax = 0.f;
#pragma unroll
        for (int col = 0; col < 2; ++col) {
            // one slot per CTA (8^3 and 16^3 blocks): each thread visits only cells of this colour;
            // smaller blocks keep one thread per cell so that a slot's threads stay contiguous
            constexpr bool HALF = GM == 1 && R >= 2;
            constexpr int NC = HALF ? n3 / 2 : GM * n3;
            constexpr int RH = R >= 2 ? R / 2 : 1;  // cells of one colour per row (HALF only)
            const int cc = P.reverse ? 1 - col : col;
#pragma unroll
            for (int t0 = 0; t0 < NC; t0 += NT) {
                const int t = t0 + threadIdx.x;
                int sl, i, cx, cy, cz;
                if (HALF) {
                    if (t >= NC) continue;
                    sl = 0;
                    cy = (t / RH) % R;
                    cz = t / (RH * R);
                    cx = 2 * (t % RH) + ((cy + cz + cc) & 1);
                    i = cx + R * (cy + R * cz);
                } else {
                    sl = t / n3;
                    i = t % n3;
                    cx = i % R;
                    cy = (i / R) % R;
                    cz = i / Gm::rr;
                }
                if (sl >= G || sb[sl] < 0 || Z.sdone[sl]) continue;
                if (!HALF && ((cx + cy + cz) & 1) != cc) continue;
                if (P.check_fluid && !S.fluid(sl, i)) continue;
                float* xs = S.xs + sl * Gm::X3;
                const float* bs = S.fs + sl * Gm::FS;
                const float* Ws = bs + n3;
                const float wW = Ws[fidx(0, cx, cy, cz, R)];
                const float wE = Ws[fidx(0, cx + 1, cy, cz, R)];
                const float wS = Ws[nf + fidx(1, cx, cy, cz, R)];
                const float wN = Ws[nf + fidx(1, cx, cy + 1, cz, R)];
                const float wB = Ws[2 * nf + fidx(2, cx, cy, cz, R)];
                const float wT = Ws[2 * nf + fidx(2, cx, cy, cz + 1, R)];
                const float diag = -(wW + wE + wS + wN + wB + wT);
                if (fabsf(diag) < 1e-9f) continue;
                const int q = xi3(cx, cy, cz, R2);
                const float xc = xs[q];
                const float Ax = wW * xs[q - 1] + wE * xs[q + 1] + wS * xs[q - sy] + wN * xs[q + sy] + wB * xs[q - sz] +
                                 wT * xs[q + sz] + diag * xc;
                const float res = bs[i] - Ax;
                xs[q] = xc + P.omega * __fdividef(res, diag);  // a smoother tolerates the 2-ulp quotient
                lmax = fmaxf(lmax, fabsf(res));
            }
            __syncthreads();
        }
        if (!track) continue;
        slot_max(&Z.smr[my_slot], n3, lmax);
        __syncthreads();
        // per-slot early exit (block-uniform); smr keeps the last executed sweep's max
        int more = 0;
        for (int t = threadIdx.x; t < G; t += NT) {
            if (sb[t] < 0 || Z.sdone[t]) continue;
            const float mr = __int_as_float(Z.smr[t]);
            if (bi == 0) Z.sinit[t] = mr;
            if (Z.sinit[t] > 1e-9f && mr < Z.sinit[t] * P.target) Z.sdone[t] = 1;
            else if (bi + 1 < P.iters) {
                Z.smr[t] = 0;
                more = 1;
            }
        }
        if (!__syncthreads_or(more)) break;
    }
    __syncthreads();
    pdl_trigger();
    store_slots<R>(x, sb, S.meta + MF_OFF * G, G, S.xs, Z.sdone);  // sdone reused as per-slot |x| max
    if (!status_next) return;
    for (int t = threadIdx.x; t < G; t += NT) {
        const int b = sb[t];
        if (b < 0 || !(__int_as_float(Z.smr[t]) > P.theta)) continue;
        status_next[b] = 1;
        int cb[3];
        bcoord(L.g, b, cb);
        for (int a = 0; a < 3; ++a)
            for (int sd = -1; sd <= 1; sd += 2) {
                int nc[3] = {cb[0], cb[1], cb[2]};
                nc[a] += sd;
                if (inside(L.g, nc)) status_next[bidx(L.g, nc[0], nc[1], nc[2])] = 1;
            }
    }
}

// smoothActiveBlocks (Smoother.cuh:105-202) for one block colour, batched.  status == nullptr
// means every block is active (no residual-threshold deactivation) and no activation is written.
__global__ void __launch_bounds__(NT, AW_BLOCK_CTAS_PER_SM) k_smooth(LevelView L, XStore x, const float* __restrict__ bvec, Coef3 W,
                                               const uint8_t* __restrict__ fluid, Batch B,
                                               const uint8_t* __restrict__ status, uint8_t* __restrict__ status_next,
                                               SmoothParams P) {
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ SmoothShared Z;
    const int4 d = B.desc[blockIdx.x];
#define AW_SMOOTH(R) smooth_body<R>(d, smraw, Z, L, x, bvec, W, fluid, B, status, status_next, P)
    AW_SWITCH_RES(d.z, AW_SMOOTH)
#undef AW_SMOOTH
}

// r = b - A x of cell i of slot sl from the staged slot image (0 on air cells when check_fluid)
template <int R, class T>
__device__ __forceinline__ T residual_cell(const SlotImage<T, R>& S, int sl, int i, int check_fluid) {
    using Gm = Geom<R>;
    constexpr int n3 = Gm::n3, nf = Gm::nf, R2 = Gm::R2, sy = R2, sz = R2 * R2;
    T rv = T(0);
    const float* bs = S.fs + sl * Gm::FS;
    if (!check_fluid || S.fluid(sl, i)) {
        const int cx = i % R, cy = (i / R) % R, cz = i / Gm::rr;
        const float* Ws = bs + n3;
        const T wW = Ws[fidx(0, cx, cy, cz, R)];
        const T wE = Ws[fidx(0, cx + 1, cy, cz, R)];
        const T wS = Ws[nf + fidx(1, cx, cy, cz, R)];
        const T wN = Ws[nf + fidx(1, cx, cy + 1, cz, R)];
        const T wB = Ws[2 * nf + fidx(2, cx, cy, cz, R)];
        const T wT = Ws[2 * nf + fidx(2, cx, cy, cz + 1, R)];
        const T diag = -(wW + wE + wS + wN + wB + wT);
        const T* xs = S.xs + sl * Gm::X3;
        const int q = xi3(cx, cy, cz, R2);
        const T Ax = diag * xs[q] + wW * xs[q - 1] + wE * xs[q + 1] + wS * xs[q - sy] + wN * xs[q + sy] +
                     wB * xs[q - sz] + wT * xs[q + sz];
        rv = (T)bs[i] - Ax;
    }
    return rv;
}

// DOTX: the per-CTA partial sums are of x . r instead of r . r (with a zero right-hand side, the
// d . (-A d) of a conjugate-gradient step, taken while d is staged)
template <int R, class Src, bool DOTX = false>
__device__ inline void residual_body(int4 d, unsigned char* smraw, double* dred, const Src& x, const float* __restrict__ bvec,
                                     const Coef3& W, const uint8_t* __restrict__ fluid, const Batch& B, int check_fluid,
                                     float* __restrict__ rout, double* __restrict__ rout64, double* __restrict__ part) {
    using T = typename Src::T;
    using Gm = Geom<R>;
    constexpr int GM = Gm::GMAX, n3 = Gm::n3;
    SlotImage<T, R> S(smraw, d.y);
    const int G = S.G;
    stage_meta<R>(S.meta, G, B, d.x, nullptr);
    pdl_wait();
    stage_data<R>(S, x, bvec, W, check_fluid ? fluid : nullptr);
    __syncthreads();
    pdl_trigger();
    double acc = 0.0;
#pragma unroll
    for (int t0 = 0; t0 < GM * n3; t0 += NT) {
        const int t = t0 + threadIdx.x, sl = t / n3, i = t % n3;
        if (sl >= G) continue;
        const T rv = residual_cell<R>(S, sl, i, check_fluid);
        if (rout) rout[S.off(0, sl) + i] = (float)rv;
        if (rout64) rout64[S.off(0, sl) + i] = (double)rv;
        if (DOTX) acc += (double)S.xs[sl * Gm::X3 + xi3(i % R, (i / R) % R, i / Gm::rr, Gm::R2)] * (double)rv;
        else acc += (double)rv * (double)rv;
    }
    if (part) {
        double tsum = block_sum(acc, dred);
        if (threadIdx.x == 0) part[blockIdx.x] = tsum;
    }
}

// computeExplicitResidual (VCycle.cuh:81-131), batched: r = b - A x on every cell (0 on air cells
// in FV mode); optional per-CTA partial sums of r^2.  Src::T = float for the V-cycle's own
// residual, double for the FP64 residual of the outer defect correction (stored as FP32 into the
// V-cycle right-hand side).
template <class Src>
__global__ void __launch_bounds__(NT, AW_BLOCK_CTAS_PER_SM) k_residual(Src x, const float* __restrict__ bvec, Coef3 W,
                                                 const uint8_t* __restrict__ fluid, Batch B, int check_fluid,
                                                 float* __restrict__ rout, double* __restrict__ rout64,
                                                 double* __restrict__ part) {
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double dred[32];
    const int4 d = B.desc[blockIdx.x];
#define AW_RESID(R) residual_body<R>(d, smraw, dred, x, bvec, W, fluid, B, check_fluid, rout, rout64, part)
    AW_SWITCH_RES(d.z, AW_RESID)
#undef AW_RESID
}

// qn = -A d in FP64 and the per-CTA partial sums of d . qn (the mixed-precision CG step), in one pass
__global__ void __launch_bounds__(NT, AW_BLOCK_CTAS_PER_SM) k_apply_dot(SrcD x, const float* __restrict__ zero, Coef3 W,
                                                                  const uint8_t* __restrict__ fluid, Batch B,
                                                                  int check_fluid, double* __restrict__ qn,
                                                                  double* __restrict__ part) {
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double dred[32];
    const int4 d = B.desc[blockIdx.x];
#define AW_APPLY(R) residual_body<R, SrcD, true>(d, smraw, dred, x, zero, W, fluid, B, check_fluid, nullptr, qn, part)
    AW_SWITCH_RES(d.z, AW_APPLY)
#undef AW_APPLY
}

template <int R>
__device__ inline void restrict_body(int4 d, unsigned char* smraw, const float* __restrict__ r, float* __restrict__ bc,
                                     const uint8_t* __restrict__ fluid_c, int check_fluid, const Batch& B) {
    using Gm = Geom<R>;
    constexpr int GM = Gm::GMAX, n3 = Gm::n3, K = 2;
    const int G = d.y;
    int* meta = (int*)smraw;
    stage_meta<R>(meta, G, B, d.x, nullptr);
    pdl_wait();
    pdl_trigger();
    const MetaView S{meta, G};
#pragma unroll
    for (int base = 0; base < GM * n3; base += K * NT) {
        float v[K][8];
        uint8_t fl[K];
        uint32_t dst[K];
        bool ok[K], full[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int t = base + k * NT + threadIdx.x, sl = t / n3, i = t % n3;
            ok[k] = t < GM * n3 && sl < G;
            full[k] = false;
            dst[k] = 0;
            fl[k] = 1;
            if (!ok[k]) continue;
            const int rf = S.m(MF_FINE_RES, sl);
            const uint32_t of = (uint32_t)S.m(MF_FINE_OFF, sl);
            dst[k] = S.off(0, sl) + i;
            if (check_fluid) fl[k] = fluid_c[dst[k]];
            full[k] = rf == 2 * R;
            if (full[k]) {
                const int x = i % R, y = (i / R) % R, z = i / Gm::rr;
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    v[k][c] = r[of + cidx(2 * x + (c & 1), 2 * y + ((c >> 1) & 1), 2 * z + (c >> 2), 2 * R)];
            } else {
                v[k][0] = r[of + i];
            }
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (!ok[k]) continue;
            float s = v[k][0];
            if (full[k]) {
#pragma unroll
                for (int c = 1; c < 8; ++c) s += v[k][c];
            }
            bc[dst[k]] = fl[k] ? s : 0.f;
        }
    }
}

// restrictResidualsKernel (MultigridTransfer.cuh:9-59), batched over the coarse level's blocks:
// 8-child sum, or a copy for a block that keeps one cell.  Coarse air cells get 0.
__global__ void __launch_bounds__(NT) k_restrict(const float* __restrict__ r, float* __restrict__ bc,
                                                 const uint8_t* __restrict__ fluid_c, int check_fluid, Batch B) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const int4 d = B.desc[blockIdx.x];
#define AW_RESTR(R) restrict_body<R>(d, smraw, r, bc, fluid_c, check_fluid, B)
    AW_SWITCH_RES(d.z, AW_RESTR)
#undef AW_RESTR
}

template <int R>
__device__ inline void prolong_body(int4 d, unsigned char* smraw, int* smax, const XStore& xf, const XStore& xc,
                                    const uint8_t* __restrict__ fluid_f, int check_fluid, const Batch& B) {
    using Gm = Geom<R>;
    constexpr int GM = Gm::GMAX, n3 = Gm::n3, K = 2;
    const int G = d.y;
    // FP16 fine storage keeps the updated block in shared memory for the re-encode
    float* xs = (float*)smraw;
    int* meta = (int*)(xs + (xf.f ? 0 : G * Gm::X3));
    stage_meta<R>(meta, G, B, d.x, nullptr);
    pdl_wait();
    pdl_trigger();
    const MetaView S{meta, G};
#pragma unroll
    for (int base = 0; base < GM * n3; base += K * NT) {
        float add[K], cur[K];
        int sl_[K], i_[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int t = base + k * NT + threadIdx.x, sl = t / n3, i = t % n3;
            sl_[k] = -1;
            i_[k] = i;
            add[k] = 0.f;
            cur[k] = 0.f;
            if (t >= GM * n3 || sl >= G) continue;
            sl_[k] = sl;
            const int b = S.m(MF_BLOCK, sl);
            const int rc = S.m(MF_COARSE_RES, sl);
            const uint32_t of = S.off(0, sl), oc = (uint32_t)S.m(MF_COARSE_OFF, sl);
            if (rc && (!check_fluid || fluid_f[of + i])) {
                const uint32_t ci = (R == 2 * rc) ? cidx((i % R) >> 1, ((i / R) % R) >> 1, (i / Gm::rr) >> 1, R / 2)
                                                  : (uint32_t)i;
                add[k] = xc.get(oc + ci, b);
            }
            cur[k] = xf.get(of + i, b);
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int sl = sl_[k];
            if (sl < 0) continue;
            const int i = i_[k];
            if (xf.f) xf.f[S.off(0, sl) + i] = cur[k] + add[k];
            else xs[sl * Gm::X3 + xi3(i % R, (i / R) % R, i / Gm::rr, Gm::R2)] = cur[k] + add[k];
        }
    }
    if (xf.f) return;
    __syncthreads();
    store_slots<R>(xf, meta + MF_BLOCK * G, meta + MF_OFF * G, G, xs, smax);
}

// prolongateCorrection (MultigridTransfer.cuh:63-102), batched over the fine level's blocks:
// x_f += x_c[parent] on fluid cells (FP16 fine storage is decoded, updated and re-encoded).
__global__ void __launch_bounds__(NT) k_prolong(XStore xf, XStore xc, const uint8_t* __restrict__ fluid_f,
                                                int check_fluid, Batch B) {
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ int smax[NT];
    const int4 d = B.desc[blockIdx.x];
#define AW_PROL(R) prolong_body<R>(d, smraw, smax, xf, xc, fluid_f, check_fluid, B)
    AW_SWITCH_RES(d.z, AW_PROL)
#undef AW_PROL
}

// ---- conjugate-gradient outer loop of the mixed-precision solve (FP64 vectors) ----------------
// *out = dot(a, z) over fluid cells (a FP64, z FP32), two cells per thread and step
__global__ void __launch_bounds__(256) k_dot64(const double* __restrict__ a, const float* __restrict__ z,
                                               const uint8_t* __restrict__ fluid, size_t n, double* part,
                                               unsigned* ticket, double* out) {
    pdl_wait();
    double acc = 0.0;
    const size_t n2 = n / 2, step = (size_t)gridDim.x * blockDim.x, t0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (size_t i = t0; i < n2; i += step) {
        const double2 av = reinterpret_cast<const double2*>(a)[i];
        const float2 zv = reinterpret_cast<const float2*>(z)[i];
        const uchar2 f = reinterpret_cast<const uchar2*>(fluid)[i];
        if (f.x) acc += av.x * (double)zv.x;
        if (f.y) acc += av.y * (double)zv.y;
    }
    if (t0 == 0 && (n & 1) && fluid[n - 1]) acc += a[n - 1] * (double)z[n - 1];
    pdl_trigger();
    last_cta_sum(acc, part, ticket, [&](double t) { *out = t; });
}
// z (FP32 V-cycle output) -> search direction d = z + beta d, beta = rho / rho_old (0 when first)
// *first: the restart flag
__global__ void k_cg_direction(double* __restrict__ d, const float* __restrict__ z, const uint8_t* __restrict__ fluid,
                               const double* __restrict__ sc, const int* __restrict__ first, size_t n) {
    pdl_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double beta = *first ? 0.0 : sc[0] / sc[1];
    d[i] = fluid[i] ? (double)z[i] + beta * d[i] : 0.0;
}
// The end of one CG iteration.  qn = -A d; alpha = rho / (d . A d); on fluid cells p += alpha d,
// r += alpha qn (with `air` on every cell), and the FP32 copy of r for the next V-cycle; rho_old = rho for the next iteration's
// direction (sc[1] is read by no CTA of this kernel).  The last CTA to finish has |r|^2: it stores it,
// counts the iteration, clears the restart flag and, in the device-side loop (DEV), runs the loop body
// again while the residual is finite, at or above the tolerance and the iteration limit is not reached.
// st = {iterations, restart, limit}, prm = {||b||, tolerance}; the direction is d1 in even iterations,
// d0 in odd ones (the same buffer twice where it is updated in place).  One pass over the vectors:
// 32 bytes read and 20 written per cell; two cells per thread and step.
struct CgVec {
    double* p;
    double* r;
    float* rf;
    const double *d0, *d1, *qn;
    double* sc;
    const uint8_t* fluid;
    int air;  // the operator has rows on air cells (reference mode): r and its copy follow there too
    size_t n;
    double* norm2;
    const double* prm;
    int* st;
};
template <bool DEV>
__global__ void __launch_bounds__(256) k_cg_update(CgVec K, double* part, unsigned* ticket, cudaGraphConditionalHandle h) {
    pdl_wait();
    const double dq = -K.sc[2];
    const double alpha = dq != 0.0 ? K.sc[0] / dq : 0.0;
    const double* __restrict__ d = (K.st[0] & 1) ? K.d0 : K.d1;
    if (blockIdx.x == 0 && threadIdx.x == 0) K.sc[1] = K.sc[0];
    double acc = 0.0;
    const size_t n2 = K.n / 2, step = (size_t)gridDim.x * blockDim.x, t0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (size_t i = t0; i < n2; i += step) {
        const uchar2 f = reinterpret_cast<const uchar2*>(K.fluid)[i];
        if (!(f.x | f.y | K.air)) continue;
        const double2 dv = reinterpret_cast<const double2*>(d)[i], qv = reinterpret_cast<const double2*>(K.qn)[i];
        double2 rv = reinterpret_cast<const double2*>(K.r)[i];
        double2 pv = reinterpret_cast<const double2*>(K.p)[i];
        const bool rx = f.x || K.air, ry = f.y || K.air;
        if (rx) rv.x = rv.x + alpha * qv.x;
        if (ry) rv.y = rv.y + alpha * qv.y;
        if (f.x) {
            pv.x += alpha * dv.x;
            acc += rv.x * rv.x;
        }
        if (f.y) {
            pv.y += alpha * dv.y;
            acc += rv.y * rv.y;
        }
        reinterpret_cast<double2*>(K.p)[i] = pv;
        reinterpret_cast<double2*>(K.r)[i] = rv;
        reinterpret_cast<float2*>(K.rf)[i] = make_float2(rx ? (float)rv.x : 0.f, ry ? (float)rv.y : 0.f);
    }
    if (t0 == 0 && (K.n & 1) && (K.fluid[K.n - 1] || K.air)) {
        const size_t i = K.n - 1;
        const double rv = K.r[i] + alpha * K.qn[i];
        K.r[i] = rv;
        K.rf[i] = (float)rv;
        if (K.fluid[i]) {
            K.p[i] += alpha * d[i];
            acc += rv * rv;
        }
    }
    last_cta_sum(acc, part, ticket, [&](double t) {
        K.norm2[0] = t;
        const double rel = sqrt(t) / K.prm[0];
        const int it = K.st[0] + 1;
        K.st[0] = it;
        K.st[1] = 0;
        if constexpr (DEV) cudaGraphSetConditional(h, (rel == rel && rel >= K.prm[1] && it < K.st[2]) ? 1u : 0u);
    });
}

// ---- conjugate gradients with every vector and scalar in FP32 (AW_PRECISION_FP32_PCG) ----------
// The same V-cycle preconditioner as the mixed form, without its FP64 residual, direction and
// accumulation: the like-for-like baseline of the mixed precision.  Partial sums and scalars are
// FP32 as well.
__device__ inline float block_sum_f(float v, float* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) red[w] = v;
    __syncthreads();
    float t = 0.f;
    if (w == 0) {
        t = lane < (int)(blockDim.x >> 5) ? red[lane] : 0.f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    return t;  // valid in thread 0
}
__global__ void k_dot32(const float* __restrict__ a, const float* __restrict__ b, const uint8_t* __restrict__ fluid,
                        size_t n, float* __restrict__ part) {
    pdl_wait();
    __shared__ float red[32];
    float acc = 0.f;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        if (fluid[i]) acc += a[i] * b[i];
    const float t = block_sum_f(acc, red);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}
__global__ void k_reduce_sum32(const float* __restrict__ part, int n, float* out) {
    pdl_wait();
    __shared__ float red[32];
    float acc = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) acc += part[i];
    const float t = block_sum_f(acc, red);
    if (threadIdx.x == 0) *out = t;
}
__global__ void k_cg_direction32(float* __restrict__ d, const float* __restrict__ z, const uint8_t* __restrict__ fluid,
                                 const float* __restrict__ sc, int first, size_t n) {
    pdl_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float beta = first ? 0.f : sc[0] / sc[1];
    d[i] = fluid[i] ? z[i] + beta * d[i] : 0.f;
}
// p += alpha d; r += alpha qn (qn = -A d, alpha = rho / (d . A d)); per-CTA partial sums of |r|^2
__global__ void k_cg_update32(float* __restrict__ p, float* __restrict__ r, const float* __restrict__ d,
                              const float* __restrict__ qn, const float* __restrict__ sc,
                              const uint8_t* __restrict__ fluid, size_t n, float* __restrict__ part) {
    pdl_wait();
    __shared__ float red[32];
    const float dq = -sc[2];
    const float alpha = dq != 0.f ? sc[0] / dq : 0.f;
    float acc = 0.f;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        p[i] += alpha * d[i];
        const float rv = r[i] + alpha * qn[i];
        r[i] = rv;
        if (fluid[i]) acc += rv * rv;
    }
    const float t = block_sum_f(acc, red);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}
__global__ void k_copy_scalar32(float* __restrict__ sc, int dst, int src) {
    pdl_wait();
    sc[dst] = sc[src];
}

__global__ void k_reduce_sum(const double* __restrict__ part, int n, double* out) {
    pdl_wait();
    __shared__ double red[32];
    double acc = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) acc += part[i];
    double t = block_sum(acc, red);
    if (threadIdx.x == 0) *out = t;
}

// *out = sum of v^2 over fluid cells (or all cells)
__global__ void __launch_bounds__(256) k_sumsq(const float* __restrict__ v, const uint8_t* __restrict__ fluid, size_t n,
                                               int check_fluid, double* part, unsigned* ticket, double* out) {
    double acc = 0.0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        if (!check_fluid || fluid[i]) acc += (double)v[i] * (double)v[i];
    last_cta_sum(acc, part, ticket, [&](double t) { *out = t; });
}
// ---------------------------------- uniform (dense) levels ------------------------------------
struct DenseArgs {
    DenseView d;
    const float* W[3];
    const uint8_t* fluid;
};

__device__ inline float dense_nb(const DenseView& d, const float* x, int i, int j, int k, int a, int s) {
    int q[3] = {i, j, k};
    q[a] += s;
    if (q[a] < 0 || q[a] >= d.D[a]) return 0.f;
    return x[didx(d, q[0], q[1], q[2])];
}

__device__ inline float dense_Ax(const DenseArgs& A, const float* x, int i, int j, int k, float* diag_out) {
    const DenseView& d = A.d;
    float wW = A.W[0][dfidx(d, 0, i, j, k)], wE = A.W[0][dfidx(d, 0, i + 1, j, k)];
    float wS = A.W[1][dfidx(d, 1, i, j, k)], wN = A.W[1][dfidx(d, 1, i, j + 1, k)];
    float wB = A.W[2][dfidx(d, 2, i, j, k)], wT = A.W[2][dfidx(d, 2, i, j, k + 1)];
    float diag = -(wW + wE + wS + wN + wB + wT);
    *diag_out = diag;
    return wW * dense_nb(d, x, i, j, k, 0, -1) + wE * dense_nb(d, x, i, j, k, 0, 1) + wS * dense_nb(d, x, i, j, k, 1, -1) +
           wN * dense_nb(d, x, i, j, k, 1, 1) + wB * dense_nb(d, x, i, j, k, 2, -1) + wT * dense_nb(d, x, i, j, k, 2, 1) +
           diag * x[didx(d, i, j, k)];
}

// Per-cell values of the uniform-level kernels (the caller stores them), shared by the
// one-launch-per-step kernels below; k_dense_tail does the same arithmetic in
// the same order.  Each returns false where the kernel leaves the cell unchanged.
__device__ inline bool dense_smooth_value(const DenseArgs& A, const float* x, const float* __restrict__ b, int t,
                                          int col, float omega, float* out) {
    const DenseView& d = A.d;
    const int i = t % d.D[0], j = (t / d.D[0]) % d.D[1], k = t / (d.D[0] * d.D[1]);
    if (((i + j + k) & 1) != col || !A.fluid[t]) return false;
    float diag;
    const float ax = dense_Ax(A, x, i, j, k, &diag);
    if (fabsf(diag) < 1e-30f) return false;
    *out = x[t] + omega * __fdividef(b[t] - ax, diag);
    return true;
}
__device__ inline float dense_residual_value(const DenseArgs& A, const float* x, const float* __restrict__ b, int t) {
    const DenseView& d = A.d;
    const int i = t % d.D[0], j = (t / d.D[0]) % d.D[1], k = t / (d.D[0] * d.D[1]);
    float diag;
    return A.fluid[t] ? b[t] - dense_Ax(A, x, i, j, k, &diag) : 0.f;
}
// restriction into a dense level from the one-cell-per-block MSBG level (from_msbg) or a dense level
__device__ inline float dense_restrict_value(const DenseView& K, const uint8_t* __restrict__ fluid_c, int from_msbg,
                                             const LevelView& F, const DenseView& Fd, const float* rf, int t) {
    const int i = t % K.D[0], j = (t / K.D[0]) % K.D[1], k = t / (K.D[0] * K.D[1]);
    float s = 0.f;
    for (int dz = 0; dz < 2; ++dz)
        for (int dy = 0; dy < 2; ++dy)
            for (int dx = 0; dx < 2; ++dx) {
                int ci = 2 * i + dx, cj = 2 * j + dy, ck = 2 * k + dz;
                if (from_msbg) {
                    int b = bidx(F.g, ci, cj, ck);
                    if (F.res[b]) s += rf[F.off[0][b]];
                } else {
                    s += rf[didx(Fd, ci, cj, ck)];
                }
            }
    return fluid_c[t] ? s : 0.f;
}
// x_f + x_c[parent] on fluid cells: t is a block of the one-cell MSBG level (to_msbg, *at = its
// cell) or a dense cell (*at = t)
__device__ inline bool dense_prolong_value(const DenseView& K, const float* xc, int to_msbg, const LevelView& F,
                                           const float* xf_msbg, const DenseView& Fd, const float* xf,
                                           const uint8_t* __restrict__ fluid_f, int t, uint32_t* at, float* out) {
    if (to_msbg) {
        if (!F.res[t]) return false;
        const uint32_t ci = F.off[0][t];
        if (!fluid_f[ci]) return false;
        int c[3];
        bcoord(F.g, t, c);
        *at = ci;
        *out = xf_msbg[ci] + xc[didx(K, c[0] >> 1, c[1] >> 1, c[2] >> 1)];
        return true;
    }
    if (!fluid_f[t]) return false;
    const int i = t % Fd.D[0], j = (t / Fd.D[0]) % Fd.D[1], k = t / (Fd.D[0] * Fd.D[1]);
    *at = (uint32_t)t;
    *out = xf[t] + xc[didx(K, i >> 1, j >> 1, k >> 1)];
    return true;
}

__global__ void k_dense_smooth(DenseArgs A, float* x, const float* __restrict__ b, int col, float omega) {
    pdl_wait();
    const DenseView& d = A.d;
    const int n = d.D[0] * d.D[1] * d.D[2];
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    float v;
    if (t < n && dense_smooth_value(A, x, b, t, col, omega, &v)) x[t] = v;
}

__global__ void k_dense_residual(DenseArgs A, const float* __restrict__ x, const float* __restrict__ b, float* r) {
    pdl_wait();
    const DenseView& d = A.d;
    const int n = d.D[0] * d.D[1] * d.D[2];
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) r[t] = dense_residual_value(A, x, b, t);
}

__global__ void k_dense_restrict(DenseView K, const uint8_t* __restrict__ fluid_c, float* __restrict__ bc, int from_msbg,
                                 LevelView F, DenseView Fd, const float* __restrict__ rf) {
    pdl_wait();
    const int n = K.D[0] * K.D[1] * K.D[2];
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) bc[t] = dense_restrict_value(K, fluid_c, from_msbg, F, Fd, rf, t);
}

__global__ void k_dense_prolong(DenseView K, const float* __restrict__ xc, int to_msbg, LevelView F, XStore xf_msbg,
                                DenseView Fd, float* __restrict__ xf, const uint8_t* __restrict__ fluid_f) {
    pdl_wait();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = to_msbg ? F.g.nb : Fd.D[0] * Fd.D[1] * Fd.D[2];
    uint32_t at;
    float v;
    if (t < n && dense_prolong_value(K, xc, to_msbg, F, xf_msbg.f, Fd, xf, fluid_f, t, &at, &v))
        (to_msbg ? xf_msbg.f : xf)[at] = v;
}

// ------------------------------- hierarchy setup kernels --------------------------------------
// coarse fluid flags: a coarse cell is fluid iff all of its children are fluid (copy when the
// block keeps one cell)
__global__ void k_coarse_fluid(LevelView F, LevelView K, const uint8_t* __restrict__ ff, uint8_t* __restrict__ fc) {
    const int b = blockIdx.x;
    const int rc = K.res[b], rf = F.res[b];
    if (!rc) return;
    const bool halved = rf == 2 * rc;
    const uint32_t of = F.off[0][b], oc = K.off[0][b];
    const int n3 = rc * rc * rc;
    for (int i = threadIdx.x; i < n3; i += blockDim.x) {
        int x = i % rc, y = (i / rc) % rc, z = i / (rc * rc);
        uint8_t f = 1;
        if (halved) {
            for (int dz = 0; dz < 2; ++dz)
                for (int dy = 0; dy < 2; ++dy)
                    for (int dx = 0; dx < 2; ++dx) f &= ff[of + cidx(2 * x + dx, 2 * y + dy, 2 * z + dz, rf)];
        } else {
            f = ff[of + i];
        }
        fc[oc + i] = f;
    }
}

// coarse 1/rho per face: mean of the 4 fine faces (copy when the block keeps one cell)
// the three axes in one launch: axis = blockIdx.y
struct Face3 {
    float* p[3];
};

__global__ void k_coarse_bbar(LevelView F, LevelView K, Face3 bfs, Face3 bcvs) {
    const int a = blockIdx.y;
    const float* __restrict__ bf = bfs.p[a];
    float* __restrict__ bcv = bcvs.p[a];
    const int b = blockIdx.x;
    const int rc = K.res[b], rf = F.res[b];
    if (!rc) return;
    const bool halved = rf == 2 * rc;
    const int nf = (rc + 1) * rc * rc;
    const int t1 = (a + 1) % 3, t2 = (a + 2) % 3;
    for (int i = threadIdx.x; i < nf; i += blockDim.x) {
        int f[3];
        if (a == 0) { f[0] = i % (rc + 1); int rem = i / (rc + 1); f[1] = rem % rc; f[2] = rem / rc; }
        else if (a == 1) { f[0] = i % rc; int rem = i / rc; f[1] = rem % (rc + 1); f[2] = rem / (rc + 1); }
        else { f[0] = i % rc; int rem = i / rc; f[1] = rem % rc; f[2] = rem / rc; }
        float v;
        if (halved) {
            float s = 0.f;
            for (int d1 = 0; d1 < 2; ++d1)
                for (int d2 = 0; d2 < 2; ++d2) {
                    int q[3];
                    q[a] = 2 * f[a];
                    q[t1] = 2 * f[t1] + d1;
                    q[t2] = 2 * f[t2] + d2;
                    s += bf[F.off[1 + a][b] + fidx(a, q[0], q[1], q[2], rf)];
                }
            v = 0.25f * s;
        } else {
            v = bf[F.off[1 + a][b] + i];
        }
        bcv[K.off[1 + a][b] + i] = v;
    }
}

// finite-volume conductance W = geo * bbar: interior h, wall 0, absent neighbour h (Dirichlet),
// same level h, coarser neighbour (2/3) h, finer neighbour (4/3) h  (h = the block's cell size)
__global__ void k_conductance(LevelView L, Face3 bbars, Face3 Ws) {
    const int a = blockIdx.y;
    const float* __restrict__ bbar = bbars.p[a];
    float* __restrict__ W = Ws.p[a];
    const int b = blockIdx.x;
    const int r = L.res[b];
    if (!r) return;
    int cb[3];
    bcoord(L.g, b, cb);
    const float H = L.g.bs / (float)r;
    const int nf = (r + 1) * r * r;
    float gl = H, gh = H;
    for (int s = -1; s <= 1; s += 2) {
        int nc[3] = {cb[0], cb[1], cb[2]};
        nc[a] += s;
        float gv;
        if (!inside(L.g, nc)) gv = 0.f;
        else {
            int rn = L.res[bidx(L.g, nc[0], nc[1], nc[2])];
            if (rn == 0 || rn == r) gv = H;
            else if (2 * rn == r) gv = (2.f / 3.f) * H;
            else gv = (4.f / 3.f) * H;
        }
        if (s < 0) gl = gv;
        else gh = gv;
    }
    for (int i = threadIdx.x; i < nf; i += blockDim.x) {
        int fa;
        if (a == 0) fa = i % (r + 1);
        else if (a == 1) fa = (i / r) % (r + 1);
        else fa = i / (r * r);
        float geo = fa == 0 ? gl : (fa == r ? gh : H);
        W[L.off[1 + a][b] + i] = geo * bbar[L.off[1 + a][b] + i];
    }
}

__global__ void k_dense_fluid(DenseView K, int from_msbg, LevelView F, const uint8_t* __restrict__ ff, DenseView Fd,
                              uint8_t* __restrict__ fc) {
    int n = K.D[0] * K.D[1] * K.D[2];
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    int i = t % K.D[0], j = (t / K.D[0]) % K.D[1], k = t / (K.D[0] * K.D[1]);
    uint8_t f = 1;
    for (int dz = 0; dz < 2; ++dz)
        for (int dy = 0; dy < 2; ++dy)
            for (int dx = 0; dx < 2; ++dx) {
                int ci = 2 * i + dx, cj = 2 * j + dy, ck = 2 * k + dz;
                uint8_t c;
                if (from_msbg) {
                    int b = bidx(F.g, ci, cj, ck);
                    c = F.res[b] ? ff[F.off[0][b]] : 0;
                } else {
                    c = ff[didx(Fd, ci, cj, ck)];
                }
                f &= c;
            }
    fc[t] = f;
}

// 1/rho on the faces of axis a of a uniform level: the mean of the four faces it covers on the next
// finer level, either the last block-structured level (one cell per block; a face is read from the
// block above it along a, else from the block below, else taken as 1 when neither is active) or the
// previous uniform level.
__global__ void k_dense_bbar(DenseView K, int a, int from_msbg, LevelView F, const float* __restrict__ fb, DenseView Fd,
                             float* __restrict__ bc) {
    const int n = (K.D[0] + (a == 0)) * (K.D[1] + (a == 1)) * (K.D[2] + (a == 2));
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int dx = K.D[0] + (a == 0), dy = K.D[1] + (a == 1);
    const int f[3] = {t % dx, (t / dx) % dy, t / (dx * dy)};
    const int t1 = (a + 1) % 3, t2 = (a + 2) % 3;
    float sum = 0.f;
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        int q[3];
        q[a] = 2 * f[a];
        q[t1] = 2 * f[t1] + (d & 1);
        q[t2] = 2 * f[t2] + (d >> 1);
        float v = 1.f;
        if (from_msbg) {
            int lo[3] = {q[0], q[1], q[2]};
            lo[a] -= 1;
            const int bh = inside(F.g, q) ? bidx(F.g, q[0], q[1], q[2]) : -1;
            const int bl = inside(F.g, lo) ? bidx(F.g, lo[0], lo[1], lo[2]) : -1;
            if (bh >= 0 && F.res[bh]) v = fb[F.off[1 + a][bh]];           // its low face
            else if (bl >= 0 && F.res[bl]) v = fb[F.off[1 + a][bl] + 1];  // its high face
        } else {
            v = fb[dfidx(Fd, a, q[0], q[1], q[2])];
        }
        sum += v;
    }
    bc[t] = 0.25f * sum;
}

// conductance W = H * bbar on a uniform level, 0 on the domain walls
__global__ void k_dense_conductance(DenseView K, int a, float H, const float* __restrict__ bbar, float* W) {
    int n = (K.D[0] + (a == 0)) * (K.D[1] + (a == 1)) * (K.D[2] + (a == 2));
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    int dx = K.D[0] + (a == 0), dy = K.D[1] + (a == 1);
    int f[3] = {t % dx, (t / dx) % dy, t / (dx * dy)};
    W[t] = (f[a] == 0 || f[a] == K.D[a]) ? 0.f : H * bbar[t];
}

// ------------------------------- coarsest FP64 dense solve ------------------------------------
// The coarsest level is a uniform grid (dense level, or the one-cell-per-block MSBG level).
struct Uniform {
    int D[3];
    int msbg;
    LevelView L;       // msbg == 1
    DenseArgs A;       // msbg == 0
    const uint8_t* fluid;
};

__device__ inline int uni_cell(const Uniform& U, int p) {  // cell index of grid position p, or -1
    if (!U.msbg) return p;
    return U.L.res[p] ? (int)U.L.off[0][p] : -1;
}
__device__ inline float uni_W(const Uniform& U, int p, int a, int hi) {
    if (!U.msbg) {
        int c[3] = {p % U.D[0], (p / U.D[0]) % U.D[1], p / (U.D[0] * U.D[1])};
        c[a] += hi;
        return U.A.W[a][dfidx(U.A.d, a, c[0], c[1], c[2])];
    }
    return U.A.W[a][U.L.off[1 + a][p] + hi];
}

// One CTA: enumerate fluid cells, assemble -A, regularise Neumann components, Cholesky, and
// write Minv = -( -A + reg )^-1 so that x = Minv b.  ex_n[0] = n (or -1 when n > EXACT_CAP).
// When the fluid flags match those of the last factorisation (prev) and the coefficients did not
// change (force == 0), the factorisation in place is still exact and the kernel returns at once.
__global__ void __launch_bounds__(512) k_coarse_factor(Uniform U, int* pos_of, int* idx, int* ex_n, double* M,
                                                       double* Minv, uint8_t* prev, int force) {
    __shared__ int cnt, diff;
    {
        const int np0 = U.D[0] * U.D[1] * U.D[2];
        if (threadIdx.x == 0) diff = force;
        __syncthreads();
        for (int p = threadIdx.x; p < np0; p += blockDim.x) {
            const int ci = uni_cell(U, p);
            const uint8_t f = (ci >= 0 && U.fluid[ci]) ? 1 : 0;
            if (f != prev[p]) diff = 1;
        }
        __syncthreads();
        if (!diff) return;
        for (int p = threadIdx.x; p < np0; p += blockDim.x) {
            const int ci = uni_cell(U, p);
            prev[p] = (ci >= 0 && U.fluid[ci]) ? 1 : 0;
        }
    }
    __shared__ int lab[EXACT_CAP];
    __shared__ int dir[EXACT_CAP];
    __shared__ double dsum[EXACT_CAP];
    __shared__ int csz[EXACT_CAP];
    __shared__ int changed;
    __shared__ double piv;
    const int np = U.D[0] * U.D[1] * U.D[2];
    if (threadIdx.x == 0) cnt = 0;
    __syncthreads();
    // deterministic compaction: serial order by position (np <= EXACT_POS_CAP)
    if (threadIdx.x == 0) {
        int c = 0;
        for (int p = 0; p < np; ++p) {
            int ci = uni_cell(U, p);
            if (ci >= 0 && U.fluid[ci]) {
                if (c < EXACT_CAP) idx[c] = p;
                pos_of[p] = c;
                ++c;
            } else {
                pos_of[p] = -1;
            }
        }
        cnt = c;
    }
    __syncthreads();
    const int n = cnt;
    if (n > EXACT_CAP) {
        if (threadIdx.x == 0) ex_n[0] = -1;
        return;
    }
    for (int t = threadIdx.x; t < n * n; t += blockDim.x) M[t] = 0.0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        int p = idx[i];
        int c[3] = {p % U.D[0], (p / U.D[0]) % U.D[1], p / (U.D[0] * U.D[1])};
        double diag = 0.0, off = 0.0;
        for (int a = 0; a < 3; ++a)
            for (int s = 0; s < 2; ++s) {
                double w = uni_W(U, p, a, s);
                diag += w;
                int q[3] = {c[0], c[1], c[2]};
                q[a] += s ? 1 : -1;
                if (q[a] < 0 || q[a] >= U.D[a]) continue;
                int qp = q[0] + U.D[0] * (q[1] + U.D[1] * q[2]);
                int j = pos_of[qp];
                if (j >= 0) {
                    M[(size_t)i * n + j] -= w;
                    off += w;
                }
            }
        M[(size_t)i * n + i] += diag;
        dir[i] = (diag - off) > 1e-12 * diag ? 1 : 0;
        lab[i] = i;
    }
    __syncthreads();
    // connected components by min-label propagation
    for (int it = 0; it < n + 1; ++it) {
        if (threadIdx.x == 0) changed = 0;
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            int l = lab[i];
            for (int j = 0; j < n; ++j)
                if (M[(size_t)i * n + j] != 0.0 && j != i && lab[j] < l) l = lab[j];
            if (l < lab[i]) {
                lab[i] = l;
                changed = 1;
            }
        }
        __syncthreads();
        if (!changed) break;
        __syncthreads();
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        dsum[i] = 0.0;
        csz[i] = 0;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 0; i < n; ++i) {
            int l = lab[i];
            dsum[l] += M[(size_t)i * n + i];
            csz[l] += 1;
            if (dir[i]) dir[l] = 1;
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < n * n; t += blockDim.x) {
        int i = t / n, j = t % n;
        int l = lab[i];
        if (lab[j] == l && !dir[l]) M[t] += dsum[l] / ((double)csz[l] * csz[l]);
    }
    __syncthreads();
    // Cholesky (lower, in place)
    for (int j = 0; j < n; ++j) {
        if (threadIdx.x == 0) {
            double s = M[(size_t)j * n + j];
            for (int k = 0; k < j; ++k) s -= M[(size_t)j * n + k] * M[(size_t)j * n + k];
            piv = sqrt(fmax(s, 1e-300));
            M[(size_t)j * n + j] = piv;
        }
        __syncthreads();
        for (int i = j + 1 + threadIdx.x; i < n; i += blockDim.x) {
            double t = M[(size_t)i * n + j];
            for (int k = 0; k < j; ++k) t -= M[(size_t)i * n + k] * M[(size_t)j * n + k];
            M[(size_t)i * n + j] = t / piv;
        }
        __syncthreads();
    }
    // inverse, one column per thread
    for (int col = threadIdx.x; col < n; col += blockDim.x) {
        for (int i = 0; i < n; ++i) {
            double t = (i == col) ? 1.0 : 0.0;
            for (int k = 0; k < i; ++k) t -= M[(size_t)i * n + k] * Minv[(size_t)k * n + col];
            Minv[(size_t)i * n + col] = t / M[(size_t)i * n + i];
        }
        for (int i = n - 1; i >= 0; --i) {
            double t = Minv[(size_t)i * n + col];
            for (int k = i + 1; k < n; ++k) t -= M[(size_t)k * n + i] * Minv[(size_t)k * n + col];
            Minv[(size_t)i * n + col] = t / M[(size_t)i * n + i];
        }
        for (int i = 0; i < n; ++i) Minv[(size_t)i * n + col] = -Minv[(size_t)i * n + col];
    }
    if (threadIdx.x == 0) ex_n[0] = n;
}

// x = Minv b on the fluid cells of the coarsest level (FP64 accumulation), a warp per row (a thread per
// row walked 512 uncoalesced values one after the other)
__global__ void __launch_bounds__(256) k_coarse_apply(Uniform U, const int* __restrict__ idx, const int* __restrict__ ex_n,
                                                      const double* __restrict__ Minv, const float* __restrict__ b,
                                                      float* __restrict__ x) {
    pdl_wait();
    const int n = ex_n[0], lane = threadIdx.x & 31;
    for (int i = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); i < n; i += (int)(gridDim.x * blockDim.x) >> 5) {
        double s = 0.0;
        for (int j = lane; j < n; j += 32) s += Minv[(size_t)i * n + j] * (double)b[uni_cell(U, idx[j])];
        s = warp_sum(s);
        if (lane == 0) x[uni_cell(U, idx[i])] = (float)s;
    }
}

// The tail of an FV V-cycle in one CTA: from the first level of at most TAIL_TOP cells on a uniform
// lattice (the last MSBG level, one cell per block, or a uniform level) down to the coarsest solve and
// back up, from a zero guess.  As separate launches each of these steps costs a launch's latency rather
// than its work; here a step is a shared-memory pass and a barrier.
// - The top level's weights, right-hand side, flags and x sit in registers.  Its x extent is even, so its
//   cells split into x pairs of one cell of each colour: a thread owns 4 pairs and every lane works in
//   every colour pass.  The cells of a colour have a shared-memory array of their own for the neighbours'
//   reads (without bank conflicts), with a layer of ghost zeros around it (no neighbour tests).
// - The levels below (at most 512 cells, one per thread) sit in shared memory and are walked by just
//   enough warps, on a barrier of their own.
// - Weights, flags and the inverse of the coarsest operator are fixed during a solve, so they are read
//   before the wait for the preceding kernel, every load of a step issued before the first is used.
// Every cell's arithmetic is that of the separate kernels in the same order, so the results are
// bit-identical to the launch-per-step form up to the coarsest solve, whose FP64 row sums are taken by a
// warp.  What bounds it is instruction issue and barrier latency of one SM.
constexpr int TAIL_THREADS = 512;
constexpr int TAIL_TOP = 4096;        // cells of the top level
constexpr int TAIL_PAIRS = TAIL_TOP / (2 * TAIL_THREADS);
constexpr int TAIL_MAX = 4;           // uniform levels below the top
constexpr int TAIL_MAX_CELLS = 512;   // cells of each of them
constexpr int TAIL_INV = 64;          // inverses up to this size are kept in shared memory
struct DenseTail {
    DenseArgs top;            // lattice, weights and fluid flags of a uniform top level
    int from_msbg;            // the top is the one-cell MSBG level F (lattice in top.d)
    LevelView F;
    float* x;
    const float* b;
    float* r;                 // nullptr: residuals are not stored
    DenseArgs lv[TAIL_MAX];   // uniform levels below, lv[n - 1] the coarsest
    float *lx[TAIL_MAX], *lb[TAIL_MAX], *lr[TAIL_MAX];  // their x, b and r (the coarsest has none), stored on the way
    int low[TAIL_MAX];        // their places in shared memory, in floats behind the top's arrays
    int n;
    int pre, post, local;     // smoothing of the top: sweeps, updates of a cell per colour (MSBG)
    int sweeps, coarsest_iters, exact;
    float omega;
    const int* idx;
    const int* ex_n;
    const double* Minv;
};
__host__ __device__ inline int lattice_cells(const DenseView& d) { return d.D[0] * d.D[1] * d.D[2]; }
__host__ __device__ inline int lattice_padded(const DenseView& d) { return (d.D[0] + 2) * (d.D[1] + 2) * (d.D[2] + 2); }
// the pairs of a lattice of even x extent, one value per pair
__host__ __device__ inline DenseView lattice_pairs(const DenseView& d) { return DenseView{{d.D[0] / 2, d.D[1], d.D[2]}}; }
// padded index of a cell
__host__ __device__ inline int pad_index(const DenseView& d, int i, int j, int k) {
    return (i + 1) + (d.D[0] + 2) * ((j + 1) + (d.D[1] + 2) * (k + 1));
}
// shared memory: inverse, indices of the coarsest system, padded x of both colours and r of the top, then
// per level below
// padded x | b | r | six weights | fluid | two packed index words per cell (TAIL_CELL_WORDS)
constexpr int TAIL_CELL_WORDS = 11;
inline size_t tail_layout(DenseTail& T) {  // fills T.low, returns the bytes
    int f = 0;
    for (int l = 0; l < T.n; ++l) {
        T.low[l] = f;
        f += lattice_padded(T.lv[l].d) + TAIL_CELL_WORDS * lattice_cells(T.lv[l].d);
    }
    return ((size_t)f + 2 * lattice_padded(lattice_pairs(T.top.d)) + lattice_cells(T.top.d) + TAIL_MAX_CELLS) * sizeof(float) +
           (size_t)TAIL_INV * TAIL_INV * sizeof(double);
}
// A x at a cell, with the roundings of the separate kernels: the residual of the MSBG level starts with
// the diagonal, its smoother and the uniform levels end with it.  w, v: W, E, S, N, B, T
__device__ __forceinline__ float tail_sum(const float* w, const float* v, float a) {
    a = ufma(w[2], v[2], a);
    a = ufma(w[3], v[3], a);
    a = ufma(w[4], v[4], a);
    return ufma(w[5], v[5], a);
}
__device__ __forceinline__ float tail_uniform(const float* w, const float* v) {
    return tail_sum(w, v, ufma(w[1], v[1], umul(w[0], v[0])));
}
__device__ __forceinline__ float tail_block(const float* w, const float* v) {
    return tail_sum(w, v, ufma(w[0], v[0], umul(w[1], v[1])));
}
__device__ __forceinline__ float tail_block_resid(const float* w, const float* v, float diag, float x) {
    return tail_sum(w, v, ufma(w[1], v[1], ufma(w[0], v[0], umul(diag, x))));
}
__device__ __forceinline__ float tail_diag(const float* w) { return -(w[0] + w[1] + w[2] + w[3] + w[4] + w[5]); }
__device__ __forceinline__ void tail_nb(const float* x, int sy, int sz, float v[6]) {
    v[0] = x[-1];
    v[1] = x[1];
    v[2] = x[-sy];
    v[3] = x[sy];
    v[4] = x[-sz];
    v[5] = x[sz];
}
__device__ __forceinline__ void tail_bar(int threads) { asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); }

// this thread's cell of a level below the top
struct TailLow {
    float *x, *b, *r;     // x: the level's padded lattice; b, r: unpadded
    float* own;           // this cell in x
    float w[6], diag, rcp;
    int n, sy, sz, parent, child;  // parent: in the next level's padded x; child: its first child in r of the level above
    bool mine, fluid;
    int col;
};
__device__ __forceinline__ TailLow tail_low(const DenseTail& T, float* low, int l) {
    TailLow L;
    const DenseView& d = T.lv[l].d;
    float* f = low + T.low[l];
    L.n = lattice_cells(d);
    L.sy = d.D[0] + 2;
    L.sz = L.sy * (d.D[1] + 2);
    L.x = f;
    f += lattice_padded(d);
    L.b = f;
    L.r = f + L.n;
    const int t = threadIdx.x;
    L.mine = t < L.n;
    const int at = L.mine ? t : 0;
#pragma unroll
    for (int k = 0; k < 6; ++k) L.w[k] = f[(2 + k) * L.n + at];
    L.fluid = L.mine && f[8 * L.n + at] != 0.f;
    const int p0 = __float_as_int(f[9 * L.n + at]);
    L.child = __float_as_int(f[10 * L.n + at]);
    L.own = L.x + (p0 & 0x7FFF);
    L.col = (p0 >> 15) & 1;
    L.parent = p0 >> 16;
    L.diag = tail_diag(L.w);
    L.rcp = urcp(L.diag);
    return L;
}
__device__ __forceinline__ void tail_low_smooth(const TailLow& L, int iters, int rev, float omega, int threads) {
    const bool on = L.fluid && !(fabsf(L.diag) < 1e-30f);
    const float b = L.b[L.mine ? threadIdx.x : 0];
    for (int it = 0; it < iters; ++it)
        for (int k = 0; k < 2; ++k) {
            if (on && L.col == (rev ? 1 - k : k)) {
                float v[6];
                tail_nb(L.own, L.sy, L.sz, v);
                const float x = *L.own;
                *L.own = ufma(omega, umul(b - ufma(L.diag, x, tail_uniform(L.w, v)), L.rcp), x);
            }
            tail_bar(threads);
        }
}
// sum of the 8 fine values under a coarse cell (children in x, y, z order)
__device__ __forceinline__ float tail_restrict(const float* r, const DenseView& f) {
    const int sy = f.D[0], sz = f.D[0] * f.D[1];
    float s = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) s += r[(e & 1) + ((e >> 1) & 1) * sy + (e >> 2) * sz];
    return s;
}
__global__ void __launch_bounds__(TAIL_THREADS, 1) k_dense_tail(const __grid_constant__ DenseTail T) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const int tid = threadIdx.x;
    const DenseView& d0 = T.top.d;
    const DenseView dp = lattice_pairs(d0);
    const int n0 = lattice_cells(d0), np0 = lattice_padded(dp);
    const int sy0 = dp.D[0] + 2, sz0 = sy0 * (d0.D[1] + 2);
    double* inv = reinterpret_cast<double*>(smraw);
    int* idx = reinterpret_cast<int*>(inv + TAIL_INV * TAIL_INV);
    float* xs = reinterpret_cast<float*>(idx + TAIL_MAX_CELLS);
    float* rs = xs + 2 * np0;
    float* low = rs + n0;
    // ---- fixed data, before the wait
    const int nex = T.exact ? T.ex_n[0] : 0;
    // top level: pair p = tid + i * TAIL_THREADS is the cells 2 p, 2 p + 1; slot 2 i + c its cell of colour c
    float w[2 * TAIL_PAIRS][6], diag[2 * TAIL_PAIRS], rcp[2 * TAIL_PAIRS], b[2 * TAIL_PAIRS];
    float x[2 * TAIL_PAIRS];
    int cell[TAIL_PAIRS], odd[TAIL_PAIRS], parent[TAIL_PAIRS];  // padded index of the pair; colour of its first cell
    uint32_t at[2 * TAIL_PAIRS], act = 0, fl = 0;               // cell offsets; bit masks over the slots
    {
        int2 res[TAIL_PAIRS];
        uint2 oc[TAIL_PAIRS], of[TAIL_PAIRS][3];
        const int hx = d0.D[0] >> 1;
#pragma unroll
        for (int i = 0; i < TAIL_PAIRS; ++i) {
            const int pr = tid + i * TAIL_THREADS;
            const bool in = 2 * pr < n0;
            const int p = in ? pr : 0;
            const int x2 = p % hx, yz = p / hx, y = yz % d0.D[1], z = yz / d0.D[1];
            cell[i] = pad_index(dp, x2, y, z);
            odd[i] = (y + z) & 1;
            parent[i] = T.n ? pad_index(T.lv[0].d, x2, y >> 1, z >> 1) : 0;
            res[i] = make_int2(in, in);
            oc[i] = make_uint2(2 * p, 2 * p + 1);
            if (T.from_msbg) {
                const int2 r = reinterpret_cast<const int2*>(T.F.res)[p];
                res[i] = make_int2(in && r.x, in && r.y);
                oc[i] = reinterpret_cast<const uint2*>(T.F.off[0])[p];
#pragma unroll
                for (int a = 0; a < 3; ++a) of[i][a] = reinterpret_cast<const uint2*>(T.F.off[1 + a])[p];
            } else {
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    of[i][a].x = dfidx(d0, a, 2 * x2, y, z);
                    of[i][a].y = of[i][a].x + 1;
                }
            }
        }
        float lo[TAIL_PAIRS][2][3], hi[TAIL_PAIRS][2][3];
#pragma unroll
        for (int i = 0; i < TAIL_PAIRS; ++i) {
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                // an inactive block owns no face: its offset may lie at the array's end
                const uint32_t f0 = res[i].x ? of[i][a].x : 0, f1 = res[i].y ? of[i][a].y : 0;
                const uint32_t up = T.from_msbg || a == 0 ? 1u : (a == 1 ? (uint32_t)d0.D[0] : (uint32_t)(d0.D[0] * d0.D[1]));
                if (T.from_msbg && f1 == f0 + 2 && (f0 & 3u) == 0) {  // both blocks' two faces: 16 bytes
                    const float4 v = *reinterpret_cast<const float4*>(T.top.W[a] + f0);
                    lo[i][0][a] = v.x;
                    hi[i][0][a] = v.y;
                    lo[i][1][a] = v.z;
                    hi[i][1][a] = v.w;
                } else {
                    lo[i][0][a] = T.top.W[a][f0];
                    hi[i][0][a] = T.top.W[a][f0 + up];
                    lo[i][1][a] = T.top.W[a][f1];
                    hi[i][1][a] = T.top.W[a][f1 + up];
                }
            }
        }
        bool f[TAIL_PAIRS][2];
#pragma unroll
        for (int i = 0; i < TAIL_PAIRS; ++i) {
            if (!res[i].x) oc[i].x = 0;
            if (!res[i].y) oc[i].y = 0;
            f[i][0] = T.top.fluid[oc[i].x] != 0;
            f[i][1] = T.top.fluid[oc[i].y] != 0;
        }
#pragma unroll
        for (int i = 0; i < TAIL_PAIRS; ++i)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int j = 2 * i + c;
                const bool second = (odd[i] ^ c) != 0;  // the pair's cell of colour c
                at[j] = second ? oc[i].y : oc[i].x;
                const bool on = second ? res[i].y : res[i].x;
                act |= (on ? 1u : 0u) << j;
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    w[j][2 * a] = second ? lo[i][1][a] : lo[i][0][a];
                    w[j][2 * a + 1] = second ? hi[i][1][a] : hi[i][0][a];
                }
                diag[j] = tail_diag(w[j]);
                rcp[j] = urcp(diag[j]);
                const bool fluid = second ? f[i][1] : f[i][0];
                if (on && fluid) fl |= 1u << j;
            }
    }
    // update mask: fluid cells that are not cut off from every neighbour
    uint32_t upd = 0;
#pragma unroll
    for (int j = 0; j < 2 * TAIL_PAIRS; ++j)
        if (((fl >> j) & 1u) && !(fabsf(diag[j]) < (T.from_msbg ? 1e-9f : 1e-30f))) upd |= 1u << j;
    if (T.exact) {
        for (int i = tid; i < nex; i += TAIL_THREADS) idx[i] = T.idx[i];
        if (nex <= TAIL_INV)
            for (int i = tid; i < nex * nex; i += TAIL_THREADS) inv[i] = T.Minv[i];
    }
    for (int l = 0; l < T.n; ++l) {
        const DenseArgs& A = T.lv[l];
        const DenseView& d = A.d;
        const int n = lattice_cells(d), np = lattice_padded(d);
        float* f = low + T.low[l];
        for (int i = tid; i < np; i += TAIL_THREADS) f[i] = 0.f;
        f += np;
        if (tid >= n) continue;
        const int q0 = tid % d.D[0], q1 = (tid / d.D[0]) % d.D[1], q2 = tid / (d.D[0] * d.D[1]);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            f[(2 + 2 * a) * n + tid] = A.W[a][dfidx(d, a, q0, q1, q2)];
            f[(3 + 2 * a) * n + tid] = A.W[a][dfidx(d, a, q0 + (a == 0), q1 + (a == 1), q2 + (a == 2))];
        }
        f[8 * n + tid] = A.fluid[tid] ? 1.f : 0.f;
        const int par = l + 1 < T.n ? pad_index(T.lv[l + 1].d, q0 >> 1, q1 >> 1, q2 >> 1) : 0;
        f[9 * n + tid] = __int_as_float(pad_index(d, q0, q1, q2) | ((q0 + q1 + q2) & 1) << 15 | par << 16);
        const DenseView& u = l ? T.lv[l - 1].d : d0;
        f[10 * n + tid] = __int_as_float(2 * q0 + u.D[0] * (2 * q1 + u.D[1] * 2 * q2));
    }
    for (int t = tid; t < 2 * np0 + n0; t += TAIL_THREADS) xs[t] = 0.f;  // x and r
    pdl_wait();
#pragma unroll
    for (int j = 0; j < 2 * TAIL_PAIRS; ++j) {
        b[j] = T.b[at[j]];
        x[j] = 0.f;
    }
    __syncthreads();
    // neighbours of slot 2 i + c: the partner on one x side, the next pair's cell on the other
    auto neighbours = [&](int i, int c, float v[6]) {
        const bool second = (odd[i] ^ c) != 0;
        const float* o = xs + (1 - c) * np0 + cell[i];
        const float outer = o[second ? 1 : -1], partner = x[2 * i + (1 - c)];
        v[0] = second ? partner : outer;
        v[1] = second ? outer : partner;
        v[2] = o[-sy0];
        v[3] = o[sy0];
        v[4] = o[-sz0];
        v[5] = o[sz0];
    };
    const bool msbg = T.from_msbg != 0;
    const int local = msbg ? T.local : 1;
    auto pass = [&](int c) {
        float v[TAIL_PAIRS][6];
#pragma unroll
        for (int i = 0; i < TAIL_PAIRS; ++i) neighbours(i, c, v[i]);
        // (a uniform cell differs in the order of its x products and in being updated once)
        float y[TAIL_PAIRS], a[TAIL_PAIRS];
#pragma unroll
        for (int i = 0; i < TAIL_PAIRS; ++i) {
            const int j = 2 * i + c;
            y[i] = x[j];
            a[i] = msbg ? tail_block(w[j], v[i]) : tail_uniform(w[j], v[i]);
        }
        for (int u = 0; u < local; ++u)
#pragma unroll
            for (int i = 0; i < TAIL_PAIRS; ++i) {
                const int j = 2 * i + c;
                y[i] = ufma(T.omega, umul(b[j] - ufma(diag[j], y[i], a[i]), rcp[j]), y[i]);
            }
#pragma unroll
        for (int i = 0; i < TAIL_PAIRS; ++i)
            if ((upd >> (2 * i + c)) & 1u) {
                x[2 * i + c] = y[i];
                xs[c * np0 + cell[i]] = y[i];
            }
        __syncthreads();
    };
    // one loop over the passes, so that each colour's code exists (and is fetched) once: red, black, ...
    // before the coarse-grid correction, black, red, ... after it
    const int npre = 2 * T.pre, npass = npre + 2 * T.post;
#pragma unroll 1
    for (int step = 0;; ++step) {
        if (step == npre) {
#pragma unroll
            for (int j = 0; j < 2 * TAIL_PAIRS; ++j) {
                const int i = j >> 1;
                float r = 0.f;
                if ((fl >> j) & 1u) {
                    float v[6];
                    neighbours(i, j & 1, v);
                    r = b[j] - (T.from_msbg ? tail_block_resid(w[j], v, diag[j], x[j]) : ufma(diag[j], x[j], tail_uniform(w[j], v)));
                    rs[2 * (tid + i * TAIL_THREADS) + (odd[i] ^ (j & 1))] = r;
                }
                if (T.r && ((act >> j) & 1u)) T.r[at[j]] = r;
            }
            __syncthreads();
            // ---- the levels below, by the warps that cover the first of them
            const int nt = (lattice_cells(T.lv[0].d) + 31) & ~31;
            if (tid < nt) {
#pragma unroll 1
                for (int l = 0; l < T.n; ++l) {
                    const TailLow L = tail_low(T, low, l);
                    if (L.mine) {
                        const float* r = l == 0 ? rs : low + T.low[l - 1] + lattice_padded(T.lv[l - 1].d) + lattice_cells(T.lv[l - 1].d);
                        const float s = tail_restrict(r + L.child, l == 0 ? d0 : T.lv[l - 1].d);
                        const float b = L.fluid ? s : 0.f;
                        L.b[tid] = b;
                        T.lb[l][tid] = b;
                    }
                    tail_bar(nt);
                    if (l + 1 == T.n) break;
                    tail_low_smooth(L, T.sweeps, 0, T.omega, nt);
                    if (L.mine) {
                        float v[6];
                        tail_nb(L.own, L.sy, L.sz, v);
                        const float r = L.fluid ? L.b[tid] - ufma(L.diag, *L.own, tail_uniform(L.w, v)) : 0.f;
                        L.r[tid] = r;
                        if (T.r) T.lr[l][tid] = r;
                    }
                    tail_bar(nt);
                }
#pragma unroll 1
                for (int l = T.n - 1; l >= 0; --l) {
                    const TailLow L = tail_low(T, low, l);
                    if (l + 1 == T.n) {  // the coarsest
                        if (T.exact) {
                            const double* M = nex <= TAIL_INV ? inv : T.Minv;
                            const DenseView& d = T.lv[l].d;
                            for (int i = tid >> 5; i < nex; i += nt >> 5) {  // a warp per row
                                double s = 0.0;
                                for (int k = tid & 31; k < nex; k += 32) s += M[(size_t)i * nex + k] * (double)L.b[idx[k]];
                                s = warp_sum(s);
                                const int p = idx[i];
                                if ((tid & 31) == 0)
                                    L.x[pad_index(d, p % d.D[0], (p / d.D[0]) % d.D[1], p / (d.D[0] * d.D[1]))] = (float)s;
                            }
                            tail_bar(nt);
                        } else {
                            tail_low_smooth(L, T.coarsest_iters, 0, T.omega, nt);
                        }
                        if (L.mine) T.lx[l][tid] = *L.own;
                        continue;
                    }
                    if (L.fluid) *L.own += (low + T.low[l + 1])[L.parent];
                    tail_bar(nt);
                    tail_low_smooth(L, T.sweeps, 1, T.omega, nt);
                    if (L.mine) T.lx[l][tid] = *L.own;
                }
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < 2 * TAIL_PAIRS; ++j)
                if ((fl >> j) & 1u) {
                    x[j] += (low + T.low[0])[parent[j >> 1]];
                    xs[(j & 1) * np0 + cell[j >> 1]] = x[j];
                }
            __syncthreads();
        }
        if (step == npass) break;
        if (((step - npre) & 1) == (step < npre ? 0 : 1)) pass(0);
        else pass(1);
    }
    pdl_trigger();
#pragma unroll
    for (int j = 0; j < 2 * TAIL_PAIRS; ++j)
        if ((act >> j) & 1u) T.x[at[j]] = x[j];
}

// ------------------------------------------------------------------------------------------------
// Host orchestration
// ------------------------------------------------------------------------------------------------
static LevelView lview(const aw_solver* S, int m) {
    const MsbgState& G = S->g->st;
    const MGLevel& L = S->lv[m];
    LevelView v;
    v.g = G.geo;
    v.res = L.res.p;
    for (int k = 0; k < 4; ++k) v.off[k] = L.off[k].p;
    return v;
}
static DenseView dview(const MGLevel& L) {
    DenseView d;
    d.D[0] = L.D[0];
    d.D[1] = L.D[1];
    d.D[2] = L.D[2];
    return d;
}
static XStore xstore(aw_solver* S, int m) {
    MGLevel& L = S->lv[m];
    XStore x;
    if (m == 0 && S->x0) {
        x.f = S->x0;
        return x;
    }
    if (L.half) {
        x.h = L.xh.p;
        x.scale = L.xscale.p;
    } else {
        x.f = L.x.p;
    }
    return x;
}
static const float* bptr(aw_solver* S, int m) { return (m == 0 && S->b0) ? S->b0 : S->lv[m].b.p; }
static Coef3 coef(const MGLevel& L) { return Coef3{{L.W[0].p, L.W[1].p, L.W[2].p}}; }
// Slots per CTA.  One-cell blocks take 64 slots (a quarter of the threads), not 256: a level's
// slot image is sized for its largest group, and 256 one-cell slots (70 KB in FP32, 98 KB in FP64)
// held every CTA of the level to 3 (or 2) per SM.  At 64 the image stays under 18 KB (25 KB in FP64)
// and 6 CTAs fit per SM (poisson_256 to 1e-6: 8.05 to 5.90 ms; dam_drop_128 solve 2.08 to 1.86 ms).
// Blocks of 2^3 cells take 16 slots (half the threads) rather than 32: more, shorter CTAs on the
// small levels (dam_drop_128 solve 1.86 to 1.76 ms).
static int slots_per_cta(int r) {
    return r == 1 ? 64 : (r == 2 ? 16 : std::max(1, std::min(256, 256 / (r * r * r))));
}

// Build the CTA batches of one block-structured level from its per-block resolutions.
static aw_status build_batches(MGLevel& L, const Geo& geo) {
    const int nb = (int)L.h_res.size();
    std::vector<int4> desc[3];
    std::vector<int> blocks[3];
    std::vector<int> by_res[3][17];
    for (int b = 0; b < nb; ++b) {
        const int r = L.h_res[b];
        if (!r) continue;
        int c[3];
        bcoord(geo, b, c);
        by_res[(c[0] + c[1] + c[2]) & 1][r].push_back(b);
        by_res[2][r].push_back(b);
    }
    for (int k = 0; k < 3; ++k) {
        for (int r = 16; r >= 1; --r) {
            const std::vector<int>& list = by_res[k][r];
            const int G = slots_per_cta(r);
            for (size_t i = 0; i < list.size(); i += G) {
                const int cnt = (int)std::min<size_t>(G, list.size() - i);
                desc[k].push_back(make_int4((int)(blocks[k].size() + i), cnt, r, 0));
            }
            blocks[k].insert(blocks[k].end(), list.begin(), list.end());
            if (!list.empty()) {
                const int Gm = std::min<int>(G, (int)list.size());
                const size_t X3 = (size_t)(r + 2) * (r + 2) * (r + 2);
                L.smem_smooth = std::max(L.smem_smooth, slot_image_bytes(Gm, r, sizeof(float)));
                L.smem_x64 = std::max(L.smem_x64, slot_image_bytes(Gm, r, sizeof(double)));
                L.smem_meta = std::max(L.smem_meta, (size_t)Gm * NMETA * 4 + 16);
                L.smem_prolong = std::max(L.smem_prolong, (size_t)Gm * (X3 * 4 + NMETA * 4) + 16);
            }
        }
        L.ndesc[k] = (int)desc[k].size();
        L.nslots[k] = (int)blocks[k].size();
    }
    // one allocation and one copy: the descriptors, the blocks, then room for the metadata
    size_t q[3], o = 0, host;
    std::vector<int4> img;
    for (int k = 0; k < 3; ++k) img.insert(img.end(), desc[k].begin(), desc[k].end());
    for (int k = 0; k < 3; ++k) {
        q[k] = img.size();
        img.resize(img.size() + (blocks[k].size() + 3) / 4);
        if (!blocks[k].empty()) memcpy(img.data() + q[k], blocks[k].data(), blocks[k].size() * sizeof(int));
    }
    host = img.size();
    size_t tot = host;
    for (int k = 0; k < 3; ++k) tot += (NMETA * blocks[k].size() + 3) / 4;
    AW_TRY(L.batches.ensure(std::max<size_t>(tot, 1)));
    if (host) AW_CUDA(cudaMemcpy(L.batches.p, img.data(), host * sizeof(int4), cudaMemcpyHostToDevice));
    size_t m = host;
    for (int k = 0; k < 3; ++k) {
        L.desc[k] = L.batches.p + o;
        o += desc[k].size();
        L.blk[k] = reinterpret_cast<int*>(L.batches.p + q[k]);
        L.meta[k] = reinterpret_cast<int*>(L.batches.p + m);
        m += (NMETA * blocks[k].size() + 3) / 4;
    }
    return AW_OK;
}
static Batch batch(const MGLevel& L, int k) { return Batch{L.desc[k], L.meta[k], L.nslots[k]}; }

// Slot metadata of one batch of level m, laid out in batch order (field-major): block id, offsets,
// the six face neighbours (cell offset, kind, block) and the block's cells on the adjacent levels.
// One thread per slot, from the level arrays already on the device (no host copy of the offsets).
__global__ void k_build_meta(Geo geo, const int* __restrict__ blocks, int n, MetaSrc h, MetaSrc finer, MetaSrc coarser,
                             int* __restrict__ mt) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const int b = blocks[j];
    const int r = h.res[b];
    auto F = [&](int f, int v) { mt[(size_t)f * n + j] = v; };
    F(MF_BLOCK, b);
    for (int q = 0; q < 4; ++q) F(MF_OFF + q, (int)h.off[q][b]);
    int c[3];
    bcoord(geo, b, c);
    for (int a = 0; a < 3; ++a)
        for (int sd = 0; sd < 2; ++sd) {
            const int f = MF_NB + 3 * (2 * a + sd);
            int nc[3] = {c[0], c[1], c[2]};
            nc[a] += sd ? 1 : -1;
            int o = 0, kind = NB_NONE, nbk = 0;
            if (inside(geo, nc)) {
                const int q = bidx(geo, nc[0], nc[1], nc[2]);
                const int rn = h.res[q];
                if (rn) {
                    o = (int)h.off[0][q];
                    kind = rn == r ? NB_SAME : (rn < r ? NB_COARSE : NB_FINE);
                    nbk = q;
                }
            }
            F(f, o);
            F(f + 1, kind);
            F(f + 2, nbk);
        }
    F(MF_FINE_OFF, finer.res ? (int)finer.off[0][b] : 0);
    F(MF_FINE_RES, finer.res ? finer.res[b] : 0);
    F(MF_COARSE_OFF, coarser.res ? (int)coarser.off[0][b] : 0);
    F(MF_COARSE_RES, coarser.res ? coarser.res[b] : 0);
}
static MetaSrc meta_src(const MGLevel* L) {
    MetaSrc m{};
    if (!L) return m;
    m.res = L->res.p;
    for (int k = 0; k < 4; ++k) m.off[k] = L->off[k].p;
    return m;
}
// The slot metadata of level m's three batches, built on the device.
static aw_status build_meta(MGLevel& L, const Geo& geo, const MGLevel* finer, const MGLevel* coarser, cudaStream_t s) {
    for (int k = 0; k < 3; ++k) {
        const int n = L.nslots[k];
        if (!n) continue;
        k_build_meta<<<nblk(n), 256, 0, s>>>(geo, L.blk[k], n, meta_src(&L), meta_src(finer), meta_src(coarser),
                                            L.meta[k]);
        AW_LAUNCH();
    }
    return AW_OK;
}
static bool fv(const aw_solver* S) { return S->d.operator_mode == AW_OPERATOR_FV; }

static Uniform uniform_of(aw_solver* S, int m) {
    MGLevel& L = S->lv[m];
    Uniform U{};
    if (L.dense) {
        for (int a = 0; a < 3; ++a) U.D[a] = L.D[a];
        U.msbg = 0;
    } else {
        for (int a = 0; a < 3; ++a) U.D[a] = S->g->st.geo.D[a];
        U.msbg = 1;
        U.L = lview(S, m);
    }
    U.A.d = dview(L);
    for (int a = 0; a < 3; ++a) U.A.W[a] = L.W[a].p;
    U.A.fluid = L.fluid.p;
    U.fluid = L.fluid.p;
    return U;
}

// A V-cycle kernel launch, as a programmatic dependent of the kernel before it in the stream (the
// kernels call pdl_wait before reading what it wrote).  After uniform_check the first one is an ordinary
// launch: the records' weights and masks, read before the wait, are what that launch's predecessor wrote.
template <typename... KArgs, typename... Args>
static aw_status launch_dep(aw_solver* S, void (*k)(KArgs...), unsigned grid, unsigned block, size_t smem,
                            cudaStream_t s, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = S->use_pdl && !S->full_next ? 1 : 0;
    S->full_next = false;
    AW_CUDA(cudaLaunchKernelEx(&cfg, k, std::forward<Args>(args)...));
    AW_LAUNCH();
    return AW_OK;
}

static aw_status zero_x(aw_solver* S, int m, cudaStream_t s) {
    MGLevel& L = S->lv[m];
    if (L.half) {
        AW_CUDA(cudaMemsetAsync(L.xh.p, 0, L.ncell() * sizeof(__half), s));
        AW_CUDA(cudaMemsetAsync(L.xscale.p, 0, S->g->st.nb * sizeof(float), s));
    } else if (m == 0 && S->x0) {
        AW_CUDA(cudaMemsetAsync(S->x0, 0, L.ncell() * sizeof(float), s));
    } else {
        AW_CUDA(cudaMemsetAsync(L.x.p, 0, L.ncell() * sizeof(float), s));
    }
    return AW_OK;
}

// Red-black block Gauss-Seidel on level m.  The post-smoothing of an FV V-cycle (reverse) runs the
// adjoint order: block colours and cell colours black before red, so that the V-cycle is a
// symmetric preconditioner for CG.  Reference mode keeps the reference's order (VCycle.cuh:251-304).
static aw_status smooth_level(aw_solver* S, int m, int iterations, cudaStream_t s, bool post = false) {
    MGLevel& L = S->lv[m];
    const int cf = fv(S) ? 1 : 0;
    const int rev = post && fv(S) ? 1 : 0;
    if (L.dense) {
        DenseArgs A{dview(L), {L.W[0].p, L.W[1].p, L.W[2].p}, L.fluid.p};
        size_t n = L.ncell();
        for (int it = 0; it < iterations; ++it)
            for (int k = 0; k < 2; ++k) {
                AW_TRY(launch_dep(S, k_dense_smooth, nblk(n), 256, 0, s, A, L.x.p, (const float*)L.b.p, rev ? 1 - k : k,
                                  S->d.omega));
            }
        return AW_OK;
    }
    const int nb = S->g->st.nb;
    // a negative activation threshold keeps every block active: no status arrays
    const bool act = S->d.theta >= 0.f;
    if (act) AW_CUDA(cudaMemsetAsync(L.status[0].p, 1, nb, s));
    SmoothParams P{S->d.omega, S->d.target_reduction, S->d.theta, S->d.block_iterations, cf, rev};
    LevelView V = lview(S, m);
    XStore x = xstore(S, m);
    int cur = 0;
    for (int it = 0; it < iterations; ++it) {
        if (act) AW_CUDA(cudaMemsetAsync(L.status[cur ^ 1].p, 0, nb, s));
        for (int k = 0; k < 2; ++k) {
            const int rb = rev ? 1 - k : k;
            if (!L.ndesc[rb]) continue;
            AW_TRY(launch_dep(S, k_smooth, (unsigned)L.ndesc[rb], 256, L.smem_smooth, s, V, x, bptr(S, m), coef(L),
                              (const uint8_t*)L.fluid.p, batch(L, rb),
                              (const uint8_t*)(act ? L.status[cur].p : nullptr), act ? L.status[cur ^ 1].p : nullptr, P));
        }
        cur ^= 1;
    }
    return AW_OK;
}

static aw_status residual_level(aw_solver* S, int m, double* part, cudaStream_t s) {
    MGLevel& L = S->lv[m];
    const int cf = fv(S) ? 1 : 0;
    if (L.dense) {
        DenseArgs A{dview(L), {L.W[0].p, L.W[1].p, L.W[2].p}, L.fluid.p};
        return launch_dep(S, k_dense_residual, nblk(L.ncell()), 256, 0, s, A, (const float*)L.x.p, (const float*)L.b.p,
                          L.r.p);
    }
    XStore x = xstore(S, m);
    if (L.ndesc[2]) {
        AW_TRY(launch_dep(S, k_residual<SrcX>, (unsigned)L.ndesc[2], 256, L.smem_smooth, s, SrcX{x}, bptr(S, m), coef(L),
                          (const uint8_t*)L.fluid.p, batch(L, 2), cf, L.r.p, (double*)nullptr, part));
    }
    return AW_OK;
}

static aw_status restrict_level(aw_solver* S, int m, cudaStream_t s) {
    MGLevel& F = S->lv[m];
    MGLevel& K = S->lv[m + 1];
    const int cf = fv(S) ? 1 : 0;
    if (K.dense) {
        LevelView Fv = F.dense ? LevelView{} : lview(S, m);
        if (F.dense) Fv.g = S->g->st.geo;
        return launch_dep(S, k_dense_restrict, nblk(K.ncell()), 256, 0, s, dview(K), (const uint8_t*)K.fluid.p, K.b.p,
                          F.dense ? 0 : 1, Fv, dview(F), (const float*)F.r.p);
    }
    if (K.ndesc[2]) {
        AW_TRY(launch_dep(S, k_restrict, (unsigned)K.ndesc[2], 256, K.smem_meta, s, (const float*)F.r.p, K.b.p,
                          (const uint8_t*)K.fluid.p, cf, batch(K, 2)));
    }
    return AW_OK;
}

static aw_status prolong_level(aw_solver* S, int m, cudaStream_t s) {
    MGLevel& F = S->lv[m];
    MGLevel& K = S->lv[m + 1];
    const int cf = fv(S) ? 1 : 0;
    if (K.dense) {
        LevelView Fv = F.dense ? LevelView{} : lview(S, m);
        if (F.dense) Fv.g = S->g->st.geo;
        size_t n = F.dense ? F.ncell() : (size_t)S->g->st.nb;
        XStore xf = F.dense ? XStore{} : xstore(S, m);
        AW_CHECK_ARG(F.dense || xf.f, "FP16 storage on the one-cell MSBG level is not supported");
        return launch_dep(S, k_dense_prolong, nblk(n), 256, 0, s, dview(K), (const float*)K.x.p, F.dense ? 0 : 1, Fv, xf,
                          dview(F), F.x.p, (const uint8_t*)F.fluid.p);
    }
    if (F.ndesc[2]) {
        AW_TRY(launch_dep(S, k_prolong, (unsigned)F.ndesc[2], 256, F.half ? F.smem_prolong : F.smem_meta, s, xstore(S, m),
                          xstore(S, m + 1), (const uint8_t*)F.fluid.p, cf, batch(F, 2)));
    }
    return AW_OK;
}

static aw_status coarsest(aw_solver* S, int m, cudaStream_t s) {
    MGLevel& L = S->lv[m];
    if (fv(S) && S->exact) {
        Uniform U = uniform_of(S, m);
        float* x = L.dense ? L.x.p : (m == 0 && S->x0 ? S->x0 : L.x.p);
        return launch_dep(S, k_coarse_apply, EXACT_CAP / 8, 256, 0, s, U, (const int*)S->ex_idx.p, (const int*)S->ex_n.p,
                          (const double*)S->Minv.p, bptr(S, m), x);
    }
    return smooth_level(S, m, S->d.coarsest_iterations, s);
}

// Levels S->tail and below as one launch (k_dense_tail), from x = 0; b of level S->tail is in place.
static DenseTail tail_args(aw_solver* S) {
    const int m = S->tail, last = (int)S->lv.size() - 1;
    MGLevel& F = S->lv[m];
    DenseTail T{};
    for (int a = 0; a < 3; ++a) {
        T.top.d.D[a] = F.dense ? F.D[a] : S->g->st.geo.D[a];
        T.top.W[a] = F.W[a].p;
    }
    T.top.fluid = F.fluid.p;
    T.from_msbg = F.dense ? 0 : 1;
    if (!F.dense) T.F = lview(S, m);
    T.x = F.x.p;
    T.b = F.b.p;
    T.r = S->keep_r ? F.r.p : nullptr;
    T.n = last - m;
    for (int j = 0; j < T.n; ++j) {
        MGLevel& L = S->lv[m + 1 + j];
        T.lv[j] = DenseArgs{dview(L), {L.W[0].p, L.W[1].p, L.W[2].p}, L.fluid.p};
        T.lx[j] = L.x.p;
        T.lb[j] = L.b.p;
        T.lr[j] = L.r.p;
    }
    T.pre = F.dense ? S->d.dense_sweeps : S->d.pre_smooth;
    T.post = F.dense ? S->d.dense_sweeps : S->d.post_smooth;
    T.local = S->d.block_iterations;
    T.sweeps = S->d.dense_sweeps;
    T.coarsest_iters = S->d.coarsest_iterations;
    T.exact = S->exact ? 1 : 0;
    T.omega = S->d.omega;
    if (S->exact) {
        T.idx = S->ex_idx.p;
        T.ex_n = S->ex_n.p;
        T.Minv = S->Minv.p;
    }
    return T;
}
static aw_status dense_tail(aw_solver* S, cudaStream_t s) {
    DenseTail T = tail_args(S);
    const size_t smem = tail_layout(T);
    return launch_dep(S, k_dense_tail, 1, TAIL_THREADS, smem, s, T);
}

static aw_status vcycle(aw_solver* S, int m, cudaStream_t s) {
    const int last = (int)S->lv.size() - 1;
    if (m == last) return coarsest(S, m, s);
    MGLevel& L = S->lv[m];
    AW_TRY(smooth_level(S, m, L.dense ? S->d.dense_sweeps : S->d.pre_smooth, s));
    AW_TRY(residual_level(S, m, nullptr, s));
    AW_TRY(restrict_level(S, m, s));
    if (S->tail && m + 1 == S->tail) {
        AW_TRY(dense_tail(S, s));
    } else {
        AW_TRY(zero_x(S, m + 1, s));
        AW_TRY(vcycle(S, m + 1, s));
    }
    AW_TRY(prolong_level(S, m, s));
    AW_TRY(smooth_level(S, m, L.dense ? S->d.dense_sweeps : S->d.post_smooth, s, true));
    return AW_OK;
}

// ---- the register-resident kernels of aw_uniform.cuh --------------------------------------------
// Slots, warps and slot records of every block-structured level.  All levels list their blocks in one
// order (colour 0 then 1, native resolutions descending: a level's resolutions then descend too), in
// one device allocation filled by one copy.
static aw_status build_uniform(aw_solver* S, cudaStream_t s) {
    const Geo& geo = S->g->st.geo;
    const std::vector<int>& res = S->lv[0].h_res;
    const int nl = S->nmsbg;
    size_t cnt[2][UNI_MAX_RES + 1] = {}, at[2][UNI_MAX_RES + 1];
    auto each = [&](auto f) {
        int b = 0;
        for (int z = 0; z < geo.D[2]; ++z)
            for (int y = 0; y < geo.D[1]; ++y)
                for (int x = 0; x < geo.D[0]; ++x, ++b)
                    if (res[b]) f(b, (x + y + z) & 1, res[b]);
    };
    each([&](int, int k, int r) { ++cnt[k][r]; });
    size_t n = 0;
    for (int k = 0; k < 2; ++k)
        for (int r = UNI_MAX_RES; r >= 1; --r) {
            at[k][r] = n;
            n += cnt[k][r];
        }
    // host image: the blocks of the slots, then every level's warp descriptors
    std::vector<int> img(n);
    each([&](int b, int k, int r) { img[at[k][r]++] = b; });
    size_t ndesc[UNI_MAX_LEVELS] = {}, d0[UNI_MAX_LEVELS] = {};
    if (img.size() & 1) img.push_back(0);
    for (int m = 0; m < nl; ++m) {
        d0[m] = img.size();
        size_t first = 0;
        for (int k = 0; k < 2; ++k) {
            const size_t w0 = ndesc[m];
            for (int r = UNI_MAX_RES >> m; r >= 1; r >>= 1) {
                size_t c = 0;  // native resolutions that are r here (1 takes all that vanish)
                for (int q = 1; q <= UNI_MAX_RES; q <<= 1)
                    if (std::max(q >> m, 1) == r) c += cnt[k][q];
                const size_t G = (size_t)uni_blocks_per_warp(r);
                for (size_t i = 0; i < c; i += G, ++ndesc[m]) {
                    img.push_back((int)(first + i));
                    img.push_back((int)std::min(G, c - i) | (r << 8));
                }
                first += c;
            }
            S->lv[m].uwarps[k] = (int)(ndesc[m] - w0);
        }
    }
    auto q16 = [](size_t bytes) { return (bytes + 15) / 16; };
    size_t tot = q16(img.size() * sizeof(int)), o_rec[UNI_MAX_LEVELS], o_wt[UNI_MAX_LEVELS], o_mask[UNI_MAX_LEVELS], o_gen[UNI_MAX_LEVELS];
    for (int m = 0; m < nl; ++m) {
        o_rec[m] = tot;
        o_wt[m] = o_rec[m] + n * UREC;
        o_mask[m] = o_wt[m] + 2 * n;
        o_gen[m] = o_mask[m] + q16(ndesc[m] * 32 * sizeof(uint16_t));
        tot = o_gen[m] + q16(ndesc[m]);
    }
    AW_TRY(S->uslab.ensure(std::max<size_t>(tot, 1)));
    if (!n) return AW_OK;
    AW_CUDA(cudaMemcpyAsync(S->uslab.p, img.data(), img.size() * sizeof(int), cudaMemcpyHostToDevice, s));
    const int* blk = reinterpret_cast<const int*>(S->uslab.p);
    for (int m = 0; m < nl; ++m) {
        MGLevel& L = S->lv[m];
        L.udesc = reinterpret_cast<int2*>(S->uslab.p) + d0[m] / 2;
        L.urec = S->uslab.p + o_rec[m];
        L.uwt = reinterpret_cast<float4*>(S->uslab.p + o_wt[m]);
        L.umask = reinterpret_cast<uint16_t*>(S->uslab.p + o_mask[m]);
        L.ugeneral = reinterpret_cast<uint8_t*>(S->uslab.p + o_gen[m]);
        k_build_records<<<nblk(n), 256, 0, s>>>(geo, blk, (int)n, meta_src(&L), meta_src(m + 1 < nl ? &S->lv[m + 1] : nullptr),
                                                reinterpret_cast<int*>(L.urec));
        AW_LAUNCH();
    }
    // the levels that k_uni_low walks (AW_NO_UNIFORM_LOW keeps a launch per step)
    S->low = nl - 1;
    if (getenv("AW_NO_UNIFORM_LOW") == nullptr)
        while (S->low > 0 && S->lv[S->low - 1].uwarps[0] + S->lv[S->low - 1].uwarps[1] <= ULOW_WARPS) --S->low;
    return AW_OK;
}

static UniView uview(const MGLevel& L, int k) {  // k: colour 0, 1, or 2 for both
    UniView V;
    V.desc = L.udesc;
    V.rec = L.urec;
    V.wt = L.uwt;
    V.mask = L.umask;
    V.general = L.ugeneral;
    V.W = coef(L);
    V.first = k == 1 ? L.uwarps[0] : 0;
    V.nwarp = k == 2 ? L.uwarps[0] + L.uwarps[1] : L.uwarps[k];
    return V;
}
static unsigned ugrid(const UniView& V) { return (unsigned)((V.nwarp + UWARPS - 1) / UWARPS); }
template <bool HALF>
static UX<HALF> ux(const XStore& x) {
    return UX<HALF>{x.f, x.h, x.scale};
}

// Weights, fluid masks and states of every block on every level.  In the blocks without fluid, which the
// kernels leave out, it clears r, and x and b where they are the solver's to write: on every level but the
// finest, and there too with own_x0 (the preconditioner of a CG solve), with the vectors whose old
// values a later kernel would read or add there: the directions, or the FP32 form's -A d.
static aw_status uniform_check(aw_solver* S, bool own_x0, cudaStream_t s) {
    UCheckAll K{};
    unsigned grid = 1;
    for (int m = 0; m < S->nmsbg; ++m) {
        MGLevel& L = S->lv[m];
        K.v[m] = uview(L, 2);
        UCheck& c = K.k[m];
        c.fluid = L.fluid.p;
        c.r = L.r.p;
        if (m > 0 || own_x0) {
            c.b = L.b.p;
            c.x = L.half ? nullptr : L.x.p;
            c.xh = L.half ? L.xh.p : nullptr;
            c.scale = L.xscale.p;
        }
        if (m == 0 && own_x0 && S->d.precision == AW_PRECISION_MIXED) {
            c.d0 = S->cg_d.p;
            c.d1 = S->cg_d2.p;
        }
        if (m == 0 && own_x0 && S->d.precision == AW_PRECISION_FP32_PCG) c.q = S->cg32_q.p;
        c.wt = L.uwt;
        c.mask = L.umask;
        c.general = L.ugeneral;
        c.count = reinterpret_cast<int*>(S->norm.p + 1) + m;
        grid = std::max(grid, ugrid(K.v[m]));
    }
    AW_CUDA(cudaMemsetAsync(S->norm.p + 1, 0, UNI_MAX_LEVELS * sizeof(int), s));
    k_uni_check<<<dim3(grid, S->nmsbg), UNT, 0, s>>>(K);
    AW_LAUNCH();
    S->full_next = true;
    return AW_OK;
}

// One colour of one smoothing iteration on level m in the given mode.
template <bool HALF, int MODE, bool HC>
static aw_status uni_smooth_t(aw_solver* S, int m, int k, int rev, cudaStream_t s) {
    MGLevel& L = S->lv[m];
    const UniView V = uview(L, k);
    if (!V.nwarp) return AW_OK;
    const bool prol = MODE == UM_PROLONG_ALL || MODE == UM_PROLONG_OWN;
    const USmooth<HALF, HC> K{V, ux<HALF>(xstore(S, m)), prol ? ux<HC>(xstore(S, m + 1)) : UX<HC>{}, bptr(S, m),
                              S->d.omega, (int)S->d.block_iterations, rev};
    if ((S->gen >> m) & 1u) return launch_dep(S, k_uni_smooth<HALF, MODE, HC, true>, ugrid(V), UNT, 0, s, K);
    return launch_dep(S, k_uni_smooth<HALF, MODE, HC, false>, ugrid(V), UNT, 0, s, K);
}
static aw_status uni_smooth(aw_solver* S, int m, int k, int rev, int mode, cudaStream_t s) {
    const bool half = S->lv[m].half && !(m == 0 && S->x0);
    if (mode == UM_PROLONG_ALL || mode == UM_PROLONG_OWN) {
        const bool hc = S->lv[m + 1].half, all = mode == UM_PROLONG_ALL;
        if (hc) return all ? uni_smooth_t<false, UM_PROLONG_ALL, true>(S, m, k, rev, s)
                           : uni_smooth_t<false, UM_PROLONG_OWN, true>(S, m, k, rev, s);
        return all ? uni_smooth_t<false, UM_PROLONG_ALL, false>(S, m, k, rev, s)
                   : uni_smooth_t<false, UM_PROLONG_OWN, false>(S, m, k, rev, s);
    }
    switch (mode) {
        case UM_ZERO_ALL:
            return half ? uni_smooth_t<true, UM_ZERO_ALL, false>(S, m, k, rev, s)
                        : uni_smooth_t<false, UM_ZERO_ALL, false>(S, m, k, rev, s);
        case UM_ZERO_OWN:
            return half ? uni_smooth_t<true, UM_ZERO_OWN, false>(S, m, k, rev, s)
                        : uni_smooth_t<false, UM_ZERO_OWN, false>(S, m, k, rev, s);
        default:
            return half ? uni_smooth_t<true, UM_PLAIN, false>(S, m, k, rev, s)
                        : uni_smooth_t<false, UM_PLAIN, false>(S, m, k, rev, s);
    }
}

// r = b - A x of level m: into out (r, or restricted), with the sum of r^2 into *sum when given
static aw_status uni_residual(aw_solver* S, int m, const XStore& x, const float* b, const UOut& out, double* sum,
                              cudaStream_t s) {
    const UniView V = uview(S->lv[m], 2);
    if (!V.nwarp) return AW_OK;
    const bool gen = (S->gen >> m) & 1u;
    if (x.h)
        return launch_dep(S, gen ? k_uni_residual<true, true> : k_uni_residual<true, false>, ugrid(V), UNT, 0, s, V,
                          ux<true>(x), b, out, S->partials.p, S->ticket.p, sum);
    return launch_dep(S, gen ? k_uni_residual<false, true> : k_uni_residual<false, false>, ugrid(V), UNT, 0, s, V,
                      ux<false>(x), b, out, S->partials.p, S->ticket.p, sum);
}

// Levels m .. and below as one launch of k_uni_low (or two around the coarser part); S->low <= m.
static aw_status uni_vcycle(aw_solver* S, int m, bool zero, cudaStream_t s);
static aw_status uni_low(aw_solver* S, int m, bool zero, cudaStream_t s) {
    const int end = S->nmsbg - 1;  // the level below the walk
    ULow K{};
    bool gen = false;
    for (int k = m; k <= end; ++k) {
        MGLevel& L = S->lv[k];
        const XStore x = xstore(S, k);
        K.lv[k] = ULowLevel{uview(L, 2), L.uwarps[0], x.f, x.h, x.scale, bptr(S, k), UOut{}};
        if (k < end) {
            K.lv[k].out.r = S->keep_r ? L.r.p : nullptr;
            K.lv[k].out.bc = S->lv[k + 1].b.p;
            K.lv[k].out.fluid_c = S->lv[k + 1].fluid.p;
            gen = gen || ((S->gen >> k) & 1u);
        }
    }
    K.first = m;
    K.last = end - 1;
    K.pre = S->d.pre_smooth;
    K.post = S->d.post_smooth;
    K.iters = (int)S->d.block_iterations;
    K.omega = S->d.omega;
    K.zero = zero;
    K.exact = S->exact && end == (int)S->lv.size() - 1 && S->lv[end].ncell() <= (size_t)ULOW_EXACT && S->lv[end].maxres == 1;
    if (K.exact) {
        K.idx = S->ex_idx.p;
        K.ex_n = S->ex_n.p;
        K.Minv = S->Minv.p;
        K.cell = S->lv[end].off[0].p;
        K.xb = S->lv[end].b.p;
    }
    auto launch = [&](bool down, bool up) {
        K.down = down;
        K.up = up;
        return launch_dep(S, gen ? k_uni_low<true> : k_uni_low<false>, 1, ULOW_THREADS, 0, s, K);
    };
    if (K.exact) return launch(true, true);
    AW_TRY(launch(true, false));
    if (S->tail && end == S->tail) AW_TRY(dense_tail(S, s));
    else AW_TRY(uni_vcycle(S, end, true, s));
    return launch(false, true);
}

// The V-cycle by the register-resident kernels: the steps of vcycle() with the
// residual restricted as it is taken, levels starting at zero without a clearing pass (zero: this
// level does), and the correction of an FP32 level added where its first post-smoothing reads it.
// Every level's x and b, and with keep_r its r, hold afterwards what vcycle() leaves there.
static aw_status uni_vcycle(aw_solver* S, int m, bool zero, cudaStream_t s) {
    const int last = (int)S->lv.size() - 1;
    MGLevel& L = S->lv[m];
    if (m == last || L.dense) {
        if (zero) AW_TRY(zero_x(S, m, s));
        return vcycle(S, m, s);
    }
    if (m >= S->low && m < S->nmsbg - 1) return uni_low(S, m, zero, s);
    if (zero && S->d.pre_smooth == 0) AW_TRY(zero_x(S, m, s));
    for (int it = 0; it < S->d.pre_smooth; ++it)
        for (int k = 0; k < 2; ++k) {
            const int mode = zero && it == 0 ? (k == 0 ? UM_ZERO_ALL : UM_ZERO_OWN) : UM_PLAIN;
            AW_TRY(uni_smooth(S, m, k, 0, mode, s));
        }
    MGLevel& K = S->lv[m + 1];
    const XStore x = xstore(S, m);
    UOut out{};
    if (S->keep_r || K.dense) out.r = L.r.p;
    if (!K.dense) {
        out.bc = K.b.p;
        out.fluid_c = K.fluid.p;
    }
    AW_TRY(uni_residual(S, m, x, bptr(S, m), out, nullptr, s));
    int mode = UM_PLAIN;
    const bool tail = S->tail && m + 1 == S->tail;
    if (K.dense) {
        AW_TRY(restrict_level(S, m, s));
        if (tail) {
            AW_TRY(dense_tail(S, s));
        } else {
            AW_TRY(zero_x(S, m + 1, s));
            AW_TRY(vcycle(S, m + 1, s));
        }
        AW_TRY(prolong_level(S, m, s));
    } else {
        if (tail) AW_TRY(dense_tail(S, s));
        else AW_TRY(uni_vcycle(S, m + 1, true, s));
        if (x.h || S->d.post_smooth == 0) {
            const UniView V = uview(L, 2);
            if (x.h && K.half)
                AW_TRY(launch_dep(S, k_uni_prolong<true, true>, ugrid(V), UNT, 0, s, V, ux<true>(x), ux<true>(xstore(S, m + 1))));
            else if (x.h)
                AW_TRY(launch_dep(S, k_uni_prolong<true, false>, ugrid(V), UNT, 0, s, V, ux<true>(x), ux<false>(xstore(S, m + 1))));
            else if (K.half)
                AW_TRY(launch_dep(S, k_uni_prolong<false, true>, ugrid(V), UNT, 0, s, V, ux<false>(x), ux<true>(xstore(S, m + 1))));
            else
                AW_TRY(launch_dep(S, k_uni_prolong<false, false>, ugrid(V), UNT, 0, s, V, ux<false>(x), ux<false>(xstore(S, m + 1))));
        } else {
            mode = UM_PROLONG_ALL;
        }
    }
    for (int it = 0; it < S->d.post_smooth; ++it)
        for (int k = 1; k >= 0; --k) {
            const int md = it == 0 && mode == UM_PROLONG_ALL ? (k == 1 ? UM_PROLONG_ALL : UM_PROLONG_OWN) : UM_PLAIN;
            AW_TRY(uni_smooth(S, m, k, 1, md, s));
        }
    return AW_OK;
}

}  // namespace aw

using namespace aw;

// ================================================================================================
// C ABI
// ================================================================================================
extern "C" aw_status aw_solver_default_desc(int32_t mode, aw_solver_desc* d) {
    AW_CHECK_ARG(d && (mode == AW_OPERATOR_FV || mode == AW_OPERATOR_REFERENCE), "bad argument");
    memset(d, 0, sizeof *d);
    d->operator_mode = mode;
    d->precision = AW_PRECISION_FP32;
    d->mg_levels = 0;
    d->pre_smooth = 2;
    d->post_smooth = 2;
    d->coarsest_iterations = 50;
    d->dense_sweeps = 2;
    d->max_cycles = 100;
    d->tolerance = 1e-6;
    if (mode == AW_OPERATOR_REFERENCE) {
        d->block_iterations = 10;     // MAX_BLOCK_ITER
        d->omega = 0.85714f;          // OMEGA
        d->target_reduction = 0.33f;  // TARGET_RESIDUAL_REDUCTION
        d->theta = 1e-4f;             // Smoother.cuh:286
    } else {
        d->block_iterations = 2;
        // Over-relaxed block Gauss-Seidel.  With the symmetric V-cycle preconditioning CG, 1.35
        // reaches 1e-6 on the 4-level poisson_256 layout in 5 iterations (6 at 1.0) and needs 7
        // instead of 9 on the 34.7M-particle dam_drop2_256 step; at 1.5 and above the smoothing
        // degrades and the iteration counts rise again.
        d->omega = 1.35f;
        d->target_reduction = 0.33f;
        d->theta = -1.0f;  // every block stays active (no residual-threshold deactivation)
    }
    return AW_OK;
}

static int ilog2(int v) {
    int l = 0;
    while ((1 << l) < v) ++l;
    return l;
}

// Coefficients of the block-structured levels from BETA_COEFF_* (stream-ordered): level 0 takes
// them as they are, coarser levels average them (k_coarse_bbar); FV mode multiplies by the face
// geometry (k_conductance), reference mode coarsens with galerkinCoarsen (MSBG.cuh:378-498).
static aw_status build_coefficients(aw_solver* S, cudaStream_t s) {
    MsbgState& G = S->g->st;
    const bool ref = S->d.operator_mode == AW_OPERATOR_REFERENCE;
    const int nb = G.nb;
    for (int m = 0; m < S->nmsbg; ++m) {
        MGLevel& L = S->lv[m];
        LevelView V = lview(S, m);
        Face3 bb{{L.bbar[0].p, L.bbar[1].p, L.bbar[2].p}};
        if (m == 0) {
            for (int a = 0; a < 3; ++a)
                AW_CUDA(cudaMemcpyAsync(L.bbar[a].p, G.ch[AW_BETA_COEFF_X + a], L.nface(a) * sizeof(float),
                                        cudaMemcpyDeviceToDevice, s));
        } else {
            MGLevel& P = S->lv[m - 1];
            Face3 fb{{P.bbar[0].p, P.bbar[1].p, P.bbar[2].p}};
            k_coarse_bbar<<<dim3(nb, 3), 128, 0, s>>>(lview(S, m - 1), V, fb, bb);
            AW_LAUNCH();
        }
        if (!ref) {
            k_conductance<<<dim3(nb, 3), 128, 0, s>>>(V, bb, Face3{{L.W[0].p, L.W[1].p, L.W[2].p}});
            AW_LAUNCH();
            continue;
        }
        for (int a = 0; a < 3; ++a) {
            if (m == 0) {
                AW_CUDA(cudaMemcpyAsync(L.W[a].p, L.bbar[a].p, L.nface(a) * sizeof(float), cudaMemcpyDeviceToDevice,
                                        s));
            } else {
                AW_CUDA(cudaMemsetAsync(L.W[a].p, 0, L.nface(a) * sizeof(float), s));
                k_galerkin_ref<<<nb, 256, 0, s>>>(G.geo, G.level.p, a, m, S->lv[m - 1].W[a].p, L.W[a].p,
                                                  S->lv[m - 1].off[1 + a].p, L.off[1 + a].p);
                AW_LAUNCH();
            }
        }
    }
    // uniform levels below one cell per block (FV mode): 1/rho averaged down face by face, so that
    // their operator follows the density of the finer levels
    for (int m = S->nmsbg; m < (int)S->lv.size(); ++m) {
        MGLevel& L = S->lv[m];
        const MGLevel& P = S->lv[m - 1];
        const bool from_msbg = m == S->nmsbg;
        for (int a = 0; a < 3; ++a) {
            k_dense_bbar<<<nblk(L.nface(a)), 256, 0, s>>>(dview(L), a, from_msbg ? 1 : 0, lview(S, m - 1),
                                                           P.bbar[a].p, dview(P), L.bbar[a].p);
            AW_LAUNCH();
            k_dense_conductance<<<nblk(L.nface(a)), 256, 0, s>>>(dview(L), a, L.H, L.bbar[a].p, L.W[a].p);
            AW_LAUNCH();
        }
    }
    return AW_OK;
}

extern "C" aw_status aw_solver_update_coefficients(aw_solver* S, aw_stream s) {
    AW_CHECK_ARG(S, "null solver");
    S->coef_dirty = true;
    return build_coefficients(S, (cudaStream_t)s);
}

// The multigrid hierarchy of the grid's current layout, built into S.  Every device buffer grows
// only: a re-layout whose levels fit the previous ones reuses their storage, so rebuilding the
// solver after aw_flip_rebuild_levels allocates and frees nothing in the common case.
static void reset_level(MGLevel& L) {
    L.dense = false;
    L.D[0] = L.D[1] = L.D[2] = 0;
    L.H = 0.f;
    L.half = false;
    L.h_res.clear();
    for (int k = 0; k < 4; ++k) L.tot[k] = 0;
    for (int k = 0; k < 3; ++k) {
        L.ndesc[k] = L.nslots[k] = 0;
    }
    L.smem_smooth = L.smem_x64 = L.smem_prolong = L.smem_meta = 0;
    L.maxres = 0;
}

// The stencils assume 2:1 grading between face neighbours.
static aw_status check_grading(const MsbgState& G) {
    const Geo& geo = G.geo;
    for (int b = 0; b < G.nb; ++b) {
        if ((int)G.h_level[b] >= geo.L) continue;
        int c[3];
        bcoord(geo, b, c);
        for (int a = 0; a < 3; ++a) {
            int nc[3] = {c[0], c[1], c[2]};
            nc[a] += 1;
            if (!inside(geo, nc)) continue;
            uint32_t nl = G.h_level[bidx(geo, nc[0], nc[1], nc[2])];
            if ((int)nl < geo.L && std::abs((int)nl - (int)G.h_level[b]) > 1)
                return set_error(AW_ERR_INVALID_ARGUMENT,
                                 "level map is not 2:1 graded (block %d); run aw_msbg_enforce_grading first", b);
        }
    }
    return AW_OK;
}

static aw_status solver_build(aw_solver* S) {
    aw_msbg* g = S->g;
    MsbgState& G = g->st;
    S->exact = false;
    S->coef_dirty = true;
    S->smem_max = S->smem_max64 = 0;
    for (aw_solver::Cycle& c : S->solve_cycle) c.drop();
    S->call_cycle.drop();
    for (aw_solver::Loop& l : S->cgloop) l.drop();
    S->vcycle_called = false;
    S->x0 = nullptr;
    S->b0 = nullptr;
    const bool ref = S->d.operator_mode == AW_OPERATOR_REFERENCE;
    const int nb = G.nb;
    int M = S->d.mg_levels > 0 ? S->d.mg_levels : (ref ? G.geo.L : ilog2(G.geo.R0) + 1);
    if (!ref) M = std::min(M, ilog2(G.geo.R0) + 1);
    cudaStream_t s = 0;
    if (S->lv.size() < (size_t)M) S->lv.resize(M);
    DBuf<uint32_t>& off4 = G.scratch_off4;
    AW_TRY(off4.ensure(4 * (size_t)nb));
    int nlev = M;
    for (int m = 0; m < M; ++m) {
        MGLevel& L = S->lv[m];
        reset_level(L);
        AW_TRY(L.res.ensure(nb));
        AW_TRY(level_offsets(G, m, ref ? 1 : 0, off4.p, L.res.p, L.tot, s));
        for (int k = 0; k < 4; ++k) {
            AW_TRY(L.off[k].ensure(nb));
            AW_CUDA(cudaMemcpy(L.off[k].p, off4.p + (size_t)k * nb, nb * sizeof(uint32_t), cudaMemcpyDeviceToDevice));
        }
        L.h_res.resize(nb);
        AW_CUDA(cudaMemcpy(L.h_res.data(), L.res.p, nb * sizeof(int), cudaMemcpyDeviceToHost));
        for (int b = 0; b < nb; ++b) L.maxres = std::max(L.maxres, L.h_res[b]);
        if (L.maxres == 0) {
            nlev = m;
            break;
        }
        AW_TRY(build_batches(L, G.geo));
        if (S->d.theta >= 0.f) {  // the activation flags of smooth_level
            AW_TRY(L.status[0].ensure(nb));
            AW_TRY(L.status[1].ensure(nb));
        }
        L.half = (S->d.precision == AW_PRECISION_MIXED) && m >= 1 && m < M - 1 + (ref ? 0 : 1) && L.maxres > 1;
        size_t nc = L.ncell();
        AW_TRY(L.x.ensure(nc));
        AW_TRY(L.b.ensure(nc));
        AW_TRY(L.r.ensure(nc));
        AW_TRY(L.fluid.ensure(nc + 16));  // whole 32-bit words are staged
        AW_CUDA(cudaMemset(L.x.p, 0, nc * sizeof(float)));
        AW_CUDA(cudaMemset(L.b.p, 0, nc * sizeof(float)));
        AW_CUDA(cudaMemset(L.fluid.p, 1, nc + 16));
        if (L.half) {
            AW_TRY(L.xh.ensure(nc));
            AW_TRY(L.xscale.ensure(nb));
            AW_CUDA(cudaMemset(L.xh.p, 0, nc * sizeof(__half)));
            AW_CUDA(cudaMemset(L.xscale.p, 0, nb * sizeof(float)));
        }
        for (int a = 0; a < 3; ++a) {
            AW_TRY(L.W[a].ensure(L.nface(a)));
            AW_TRY(L.bbar[a].ensure(L.nface(a)));
        }
    }
    S->nmsbg = nlev;
    for (int m = 0; m < S->nmsbg; ++m) {
        MGLevel& L = S->lv[m];
        AW_TRY(build_meta(L, G.geo, m > 0 ? &S->lv[m - 1] : nullptr, m + 1 < S->nmsbg ? &S->lv[m + 1] : nullptr, s));
        S->smem_max = std::max({S->smem_max, L.smem_smooth, L.smem_prolong, L.smem_meta});
        S->smem_max64 = std::max(S->smem_max64, L.smem_x64);
    }
    // the register-resident kernels take FV levels of at most 8^3 blocks without activation flags or
    // per-block early exit (the FV defaults; k_smooth tracks block residuals otherwise)
    const bool track = S->d.target_reduction > 0.f && (S->d.block_iterations > 2 ||
                                                      (S->d.block_iterations == 2 && S->d.target_reduction >= 1.f));
    S->uni = !ref && S->d.theta < 0.f && !track && G.geo.R0 <= UNI_MAX_RES && S->nmsbg > 0 &&
             S->nmsbg <= UNI_MAX_LEVELS && getenv("AW_NO_UNIFORM") == nullptr;
    if (S->uni) AW_TRY(build_uniform(S, s));
    // uniform continuation below one cell per block (FV mode)
    size_t used = (size_t)S->nmsbg;
    if (!ref && S->nmsbg > 0 && S->lv[S->nmsbg - 1].maxres == 1) {
        int Dd[3] = {G.geo.D[0], G.geo.D[1], G.geo.D[2]};
        float H = G.geo.bs;
        while (Dd[0] % 2 == 0 && Dd[1] % 2 == 0 && Dd[2] % 2 == 0 && (long)Dd[0] * Dd[1] * Dd[2] > 64) {
            if (S->lv.size() <= used) S->lv.emplace_back();
            MGLevel& L = S->lv[used++];
            reset_level(L);
            L.dense = true;
            for (int a = 0; a < 3; ++a) L.D[a] = Dd[a] / 2;
            H *= 2.f;
            L.H = H;
            size_t nc = L.ncell();
            AW_TRY(L.x.ensure(nc));
            AW_TRY(L.b.ensure(nc));
            AW_TRY(L.r.ensure(nc));
            AW_TRY(L.fluid.ensure(nc));
            AW_CUDA(cudaMemset(L.x.p, 0, nc * sizeof(float)));
            AW_CUDA(cudaMemset(L.b.p, 0, nc * sizeof(float)));
            for (int a = 0; a < 3; ++a) {
                AW_TRY(L.W[a].ensure(L.nface(a)));
                AW_TRY(L.bbar[a].ensure(L.nface(a)));
            }
            for (int a = 0; a < 3; ++a) Dd[a] /= 2;
        }
        S->lv.resize(used);  // levels beyond the new hierarchy are released
        // the coarsest level is uniform: factorise it densely when small enough
        MGLevel& C = S->lv.back();
        size_t npos = C.dense ? C.ncell() : (size_t)nb;
        if (npos <= (size_t)EXACT_POS_CAP) {
            AW_TRY(S->M.ensure((size_t)EXACT_CAP * EXACT_CAP));
            AW_TRY(S->Minv.ensure((size_t)EXACT_CAP * EXACT_CAP));
            AW_TRY(S->ex_idx.ensure(EXACT_CAP));
            AW_TRY(S->ex_pos.ensure(npos));
            AW_TRY(S->ex_prev.ensure(npos));
            AW_CUDA(cudaMemset(S->ex_prev.p, 0xFF, npos));
            AW_TRY(S->ex_n.ensure(1));
            AW_CUDA(cudaMemset(S->ex_n.p, 0, sizeof(int)));
            S->exact = true;
        }
    }
    S->lv.resize(used);
    // coefficients of every level
    AW_TRY(build_coefficients(S, 0));
    // always opted in: static shared memory (k_smooth's per-slot state) counts against the default 48 KB too
    AW_TRY(allow_smem<k_smooth>(S->smem_max));
    AW_TRY(allow_smem<k_residual<SrcX>>(S->smem_max));
    AW_TRY(allow_smem<k_prolong>(S->smem_max));
    AW_TRY(allow_smem<k_restrict>(S->smem_max));
    AW_TRY(allow_smem<k_residual<SrcD>>(S->smem_max64));
    AW_TRY(allow_smem<k_apply_dot>(S->smem_max64));
    if (S->d.precision == AW_PRECISION_MIXED) {
        const size_t nc0 = S->lv[0].ncell();
        AW_TRY(S->cg_r.ensure(nc0));
        AW_TRY(S->cg_d.ensure(nc0));
        AW_TRY(S->cg_d2.ensure(nc0));
        AW_TRY(S->cg_q.ensure(nc0));
        AW_TRY(S->cg_sc.ensure(4));
        AW_TRY(S->cg_zero.ensure(nc0));
        AW_CUDA(cudaMemset(S->cg_zero.p, 0, nc0 * sizeof(float)));
        AW_CUDA(cudaMemset(S->cg_d.p, 0, nc0 * sizeof(double)));
        AW_CUDA(cudaMemset(S->cg_d2.p, 0, nc0 * sizeof(double)));
        AW_CUDA(cudaMemset(S->cg_r.p, 0, nc0 * sizeof(double)));
        AW_CUDA(cudaMemset(S->cg_q.p, 0, nc0 * sizeof(double)));
        AW_TRY(S->cgst.ensure(4));
        AW_TRY(S->cgprm.ensure(2));
    }
    if (S->d.precision == AW_PRECISION_FP32_PCG) {
        const size_t nc0 = S->lv[0].ncell();
        AW_TRY(S->cg32_d.ensure(std::max<size_t>(nc0, 1)));
        AW_TRY(S->cg32_q.ensure(std::max<size_t>(nc0, 1)));
        AW_TRY(S->cg32_sc.ensure(4));
        AW_TRY(S->cg_zero.ensure(std::max<size_t>(nc0, 1)));
        AW_TRY(S->partials32.ensure(4096));
        AW_CUDA(cudaMemset(S->cg_zero.p, 0, std::max<size_t>(nc0, 1) * sizeof(float)));
        AW_CUDA(cudaMemset(S->cg32_d.p, 0, std::max<size_t>(nc0, 1) * sizeof(float)));
        AW_CUDA(cudaMemset(S->cg32_q.p, 0, std::max<size_t>(nc0, 1) * sizeof(float)));
    }
    // partial sums: one per CTA of the widest launch (batches and uniform warps hold at least one block)
    size_t nparts = (size_t)nb + 2048;
    AW_TRY(S->partials.ensure(nparts));
    AW_TRY(S->norm.ensure(1 + UNI_MAX_LEVELS / 2));  // a squared norm; uniform_check's count per level
    AW_TRY(S->ticket.ensure(1));
    AW_CUDA(cudaMemset(S->ticket.p, 0, sizeof(unsigned)));
    S->use_graph = getenv("AW_NO_GRAPH") == nullptr;
    S->use_pdl = getenv("AW_NO_PDL") == nullptr;
    S->use_devloop = getenv("AW_NO_DEVLOOP") == nullptr;
    // the tail as one launch (FV mode): from the first level of at most TAIL_TOP cells that is uniform or,
    // where k_smooth neither tracks residuals nor deactivates blocks, the one-cell MSBG level below level 0;
    // the uniform levels under it have at most TAIL_MAX_CELLS cells (AW_NO_DENSE_TAIL keeps one launch per
    // step).  An 8th of 4096 cells is 512, so any level that qualifies has such levels under it.
    S->tail = 0;
    if (!ref && S->nmsbg > 0 && getenv("AW_NO_DENSE_TAIL") == nullptr) {
        const int nl = (int)S->lv.size();
        int j = S->nmsbg;
        if (j > 1 && nb <= TAIL_TOP && S->d.theta < 0.f && !track && S->lv[j - 1].maxres == 1 && !S->lv[j - 1].half) --j;
        else
            while (j < nl && S->lv[j].ncell() > (size_t)TAIL_TOP) ++j;
        bool ok = j < nl - 1 && nl - 1 - j <= TAIL_MAX;
        for (int k = j + 1; ok && k < nl; ++k) ok = S->lv[k].dense && S->lv[k].ncell() <= (size_t)TAIL_MAX_CELLS;
        if (ok) {
            S->tail = j;
            AW_TRY(allow_smem<k_dense_tail>(200 * 1024));
            DenseTail T = tail_args(S);
            if (tail_layout(T) > 200 * 1024) S->tail = 0;  // a lattice so thin that its ghost layer dominates
        }
    }

    AW_CUDA(cudaDeviceSynchronize());
    return AW_OK;
}

namespace aw {
aw_status solver_relayout(aw_solver* S) {
    AW_CHECK_ARG(S && S->g && S->g->st.allocated, "grid not allocated");
    AW_TRY(check_grading(S->g->st));
    AW_TRY(solver_build(S));
    return aw_solver_setup(S, nullptr, 0);
}
}  // namespace aw

extern "C" aw_status aw_solver_create(aw_msbg* g, const aw_solver_desc* d, aw_solver** out) {
    AW_CHECK_ARG(g && d && out, "null argument");
    AW_CHECK_ARG(g->st.allocated, "grid not allocated");
    AW_CHECK_ARG(d->operator_mode == AW_OPERATOR_FV || d->operator_mode == AW_OPERATOR_REFERENCE, "bad operator mode");
    AW_CHECK_ARG(d->precision == AW_PRECISION_FP32 || d->precision == AW_PRECISION_MIXED ||
                     d->precision == AW_PRECISION_FP32_PCG,
                 "bad precision");
    AW_CHECK_ARG(d->block_iterations >= 1 && d->pre_smooth >= 0 && d->post_smooth >= 0, "bad smoother settings");
    *out = nullptr;
    MsbgState& G = g->st;
    AW_TRY(check_grading(G));
    std::unique_ptr<aw_solver> S(new aw_solver());
    S->g = g;
    S->d = *d;
    AW_TRY(solver_build(S.get()));
    *out = S.release();
    // default setup: every cell fluid
    return aw_solver_setup(*out, nullptr, 0);
}

extern "C" aw_status aw_solver_destroy(aw_solver* sv) {
    delete sv;
    return AW_OK;
}

extern "C" aw_status aw_solver_setup(aw_solver* S, const uint8_t* d_fluid, aw_stream s_) {
    AW_CHECK_ARG(S, "null solver");
    cudaStream_t s = (cudaStream_t)s_;
    MsbgState& G = S->g->st;
    MGLevel& L0 = S->lv[0];
    if (d_fluid) AW_CUDA(cudaMemcpyAsync(L0.fluid.p, d_fluid, L0.ncell(), cudaMemcpyDeviceToDevice, s));
    else AW_CUDA(cudaMemsetAsync(L0.fluid.p, 1, L0.ncell(), s));
    for (int m = 1; m < (int)S->lv.size(); ++m) {
        MGLevel& L = S->lv[m];
        MGLevel& F = S->lv[m - 1];
        if (!L.dense) {
            k_coarse_fluid<<<G.nb, 128, 0, s>>>(lview(S, m - 1), lview(S, m), F.fluid.p, L.fluid.p);
        } else {
            LevelView Fv = F.dense ? LevelView{} : lview(S, m - 1);
            if (F.dense) Fv.g = G.geo;
            k_dense_fluid<<<nblk(L.ncell()), 256, 0, s>>>(dview(L), F.dense ? 0 : 1, Fv, F.fluid.p, dview(F), L.fluid.p);
        }
        AW_LAUNCH();
    }
    if (S->exact) {
        Uniform U = uniform_of(S, (int)S->lv.size() - 1);
        k_coarse_factor<<<1, 512, 0, s>>>(U, S->ex_pos.p, S->ex_idx.p, S->ex_n.p, S->M.p, S->Minv.p, S->ex_prev.p,
                                          S->coef_dirty ? 1 : 0);
        S->coef_dirty = false;
        AW_LAUNCH();
    }
    return AW_OK;
}

extern "C" aw_status aw_solver_precision(const aw_solver* S, int32_t* precision) {
    AW_CHECK_ARG(S && precision, "null argument");
    *precision = S->d.precision;
    return AW_OK;
}

extern "C" aw_status aw_solver_num_levels(const aw_solver* S, int32_t* n) {
    AW_CHECK_ARG(S && n, "null argument");
    *n = (int32_t)S->lv.size();
    return AW_OK;
}

extern "C" aw_status aw_solver_level_array(aw_solver* S, int32_t m, int32_t which, void** p, uint32_t* count) {
    AW_CHECK_ARG(S && p && m >= 0 && m < (int)S->lv.size(), "bad argument");
    MGLevel& L = S->lv[m];
    uint32_t c = 0;
    void* q = nullptr;
    switch (which) {
        case 0: q = L.half ? (void*)L.xh.p : (void*)L.x.p; c = (uint32_t)L.ncell(); break;
        case 1: q = L.b.p; c = (uint32_t)L.ncell(); break;
        case 2: q = L.r.p; c = (uint32_t)L.ncell(); break;
        case 3: case 4: case 5: q = L.W[which - 3].p; c = (uint32_t)L.nface(which - 3); break;
        case 6: q = L.fluid.p; c = (uint32_t)L.ncell(); break;
        case 7: case 8: case 9: case 10:
            AW_CHECK_ARG(!L.dense, "offsets exist on block-structured levels only");
            q = L.off[which - 7].p;
            c = (uint32_t)S->g->st.nb;
            break;
        case 11:
            AW_CHECK_ARG(!L.dense, "res exists on block-structured levels only");
            q = L.res.p;
            c = (uint32_t)S->g->st.nb;
            break;
        default: return set_error(AW_ERR_INVALID_ARGUMENT, "unknown level array %d", which);
    }
    *p = q;
    if (count) *count = c;
    return AW_OK;
}

extern "C" aw_status aw_smoother_solve_level(aw_solver* S, int32_t m, int32_t iterations, aw_stream s) {
    AW_CHECK_ARG(S && m >= 0 && m < (int)S->lv.size() && iterations >= 0, "bad argument");
    return smooth_level(S, m, iterations, (cudaStream_t)s);
}
extern "C" aw_status aw_mg_residual(aw_solver* S, int32_t m, aw_stream s) {
    AW_CHECK_ARG(S && m >= 0 && m < (int)S->lv.size(), "bad argument");
    return residual_level(S, m, nullptr, (cudaStream_t)s);
}
extern "C" aw_status aw_mg_restrict(aw_solver* S, int32_t m, aw_stream s) {
    AW_CHECK_ARG(S && m >= 0 && m + 1 < (int)S->lv.size(), "bad argument");
    return restrict_level(S, m, (cudaStream_t)s);
}
extern "C" aw_status aw_mg_prolongate(aw_solver* S, int32_t m, aw_stream s) {
    AW_CHECK_ARG(S && m >= 0 && m + 1 < (int)S->lv.size(), "bad argument");
    return prolong_level(S, m, (cudaStream_t)s);
}
// One V-cycle of the current solve; zero: the level-0 x starts at zero (whatever it holds).
static aw_status solve_vcycle(aw_solver* S, bool zero, cudaStream_t s) {
    if (S->uni) return uni_vcycle(S, 0, zero, s);
    if (zero) AW_TRY(zero_x(S, 0, s));
    return vcycle(S, 0, s);
}
// ... replayed from a CUDA graph (captured on first use for the current level-0 x/b and form): aw_vcycle_run's
// (call), or the one of aw_solve's two that fits, else in the place of the one used longer ago.
static aw_status run_vcycle(aw_solver* S, bool call, bool zero, cudaStream_t s) {
    if (!S->use_graph) return solve_vcycle(S, zero, s);
    const void* x0 = S->x0 ? (const void*)S->x0 : (const void*)S->lv[0].x.p;
    const void* b0 = S->b0 ? (const void*)S->b0 : (const void*)S->lv[0].b.p;
    const unsigned form = 2 * S->gen + (zero ? 1u : 0u);
    auto fits = [&](const aw_solver::Cycle& c) { return c.exec && c.x0 == x0 && c.b0 == b0 && c.form == form; };
    if (!call && !fits(S->solve_cycle[S->solve_last])) S->solve_last ^= 1;
    aw_solver::Cycle& C = call ? S->call_cycle : S->solve_cycle[S->solve_last];
    if (!fits(C)) {
        C.drop();
        if (!S->cap) AW_CUDA(cudaStreamCreateWithFlags(&S->cap, cudaStreamNonBlocking));
        const unsigned long long l0 = g_launches;
        AW_CUDA(cudaStreamBeginCapture(S->cap, cudaStreamCaptureModeThreadLocal));
        aw_status st = solve_vcycle(S, zero, S->cap);
        cudaGraph_t graph = nullptr;
        cudaError_t e = cudaStreamEndCapture(S->cap, &graph);
        C.kernels = g_launches - l0;
        g_launches = l0;
        if (st != AW_OK) {
            if (graph) cudaGraphDestroy(graph);
            return st;
        }
        if (e != cudaSuccess) return set_error(AW_ERR_CUDA, "V-cycle capture: %s", cudaGetErrorString(e));
        e = cudaGraphInstantiate(&C.exec, graph, 0);
        cudaGraphDestroy(graph);
        if (e != cudaSuccess) {
            C.exec = nullptr;
            return set_error(AW_ERR_CUDA, "V-cycle graph instantiate: %s", cudaGetErrorString(e));
        }
        C.x0 = x0;
        C.b0 = b0;
        C.form = form;
    }
    AW_CUDA(cudaGraphLaunch(C.exec, s));
    g_launches += C.kernels;
    return AW_OK;
}

extern "C" aw_status aw_solver_coarsest_solve(aw_solver* S, aw_stream s) {
    AW_CHECK_ARG(S, "null solver");
    return coarsest(S, (int)S->lv.size() - 1, (cudaStream_t)s);
}
extern "C" aw_status aw_vcycle_run(aw_solver* S, aw_stream s) {
    AW_CHECK_ARG(S, "null solver");
    S->keep_r = true;
    if (!S->uni) return vcycle(S, 0, (cudaStream_t)s);
    AW_TRY(uniform_check(S, false, (cudaStream_t)s));
    S->gen = (1u << S->nmsbg) - 1;  // no host read here: the kernels that take any block
    // replayed from a graph (a launch each costs the host more than the kernels take) from the second call
    // on (building it costs about one call), unless the caller is capturing this stream
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    AW_CUDA(cudaStreamIsCapturing((cudaStream_t)s, &cap));
    if (!S->vcycle_called || cap != cudaStreamCaptureStatusNone) {
        S->vcycle_called = true;
        return solve_vcycle(S, false, (cudaStream_t)s);
    }
    return run_vcycle(S, true, false, (cudaStream_t)s);
}

// *out = sqrt of the sum in S->norm[0], read back with uniform_check's counts (syncs)
static aw_status fetch_norm(aw_solver* S, cudaStream_t s, double* out) {
    if (!S->h_norm) AW_CUDA(cudaHostAlloc((void**)&S->h_norm, 4 * sizeof(double), cudaHostAllocDefault));
    AW_CUDA(cudaMemcpyAsync(S->h_norm, S->norm.p, (1 + UNI_MAX_LEVELS / 2) * sizeof(double), cudaMemcpyDeviceToHost, s));
    AW_CUDA(cudaStreamSynchronize(s));
    *out = std::sqrt(S->h_norm[0]);
    return AW_OK;
}
static aw_status read_norm(aw_solver* S, int nparts, cudaStream_t s, double* out) {
    k_reduce_sum<<<1, 256, 0, s>>>(S->partials.p, nparts, S->norm.p);
    AW_LAUNCH();
    return fetch_norm(S, s, out);
}

// r = b - A p into r (FP32) and r64, and ||r||: the true residual of the outer loops (FP32 or FP64 p)
static aw_status true_residual(aw_solver* S, const float* p32, const double* p64, const float* b, float* r, double* r64,
                               cudaStream_t s, double* norm) {
    MGLevel& L0 = S->lv[0];
    const int cf = fv(S) ? 1 : 0;
    XStore xp;
    xp.f = const_cast<float*>(p32);
    if (S->uni) {
        UOut out{};
        out.r = r;
        out.r64 = r64;
        const UniView V = uview(L0, 2);
        if (!V.nwarp) AW_CUDA(cudaMemsetAsync(S->norm.p, 0, sizeof(double), s));
        else if (p64) {
            (S->gen & 1u ? k_uni_residual64<true> : k_uni_residual64<false>)<<<ugrid(V), UNT, 0, s>>>(
                V, USrcD{p64}, b, out, S->partials.p, S->ticket.p, S->norm.p);
            AW_LAUNCH();
        } else {
            AW_TRY(uni_residual(S, 0, xp, b, out, S->norm.p, s));
        }
        return fetch_norm(S, s, norm);
    }
    if (L0.ndesc[2]) {
        if (p64)
            k_residual<SrcD><<<L0.ndesc[2], 256, L0.smem_x64, s>>>(SrcD{p64}, b, coef(L0), L0.fluid.p, batch(L0, 2), cf, r,
                                                                   r64, S->partials.p);
        else
            k_residual<SrcX><<<L0.ndesc[2], 256, L0.smem_smooth, s>>>(SrcX{xp}, b, coef(L0), L0.fluid.p, batch(L0, 2), cf,
                                                                      r, r64, S->partials.p);
        AW_LAUNCH();
    }
    return read_norm(S, L0.ndesc[2], s, norm);
}

// One mixed-precision CG iteration: z = V(r) (r in FP32 in the level-0 right-hand side), rho = r . z,
// d = z + (rho / rho_old) d, q = -A d with d . q, then k_cg_update.  The same kernels in the
// device-side loop (h given) and in the host-driven one.
static aw_status cg_iteration(aw_solver* S, double* p, unsigned ndot, cudaStream_t s, const cudaGraphConditionalHandle* h) {
    MGLevel& L0 = S->lv[0];
    const size_t nc = L0.ncell();
    const int cf = fv(S) ? 1 : 0;
    double* sc = S->cg_sc.p;
    if (h) AW_TRY(solve_vcycle(S, true, s));
    else AW_TRY(run_vcycle(S, false, true, s));
    AW_TRY(launch_dep(S, k_dot64, ndot, 256, 0, s, (const double*)S->cg_r.p, (const float*)L0.x.p,
                      (const uint8_t*)L0.fluid.p, nc, S->partials.p, S->ticket.p, sc + 0));
    CgVec K{};
    if (S->uni) {
        K.d0 = S->cg_d.p;
        K.d1 = S->cg_d2.p;
        UOut out{};
        out.r64 = S->cg_q.p;
        const UniView V = uview(L0, 2);
        AW_TRY(launch_dep(S, S->gen & 1u ? k_uni_apply<true> : k_uni_apply<false>, ugrid(V), UNT, 0, s, V, (const float*)L0.x.p, S->cg_d.p, S->cg_d2.p, out,
                          (const double*)sc, (const int*)S->cgst.p, S->partials.p, S->ticket.p, sc + 2));
    } else {
        K.d0 = K.d1 = S->cg_d.p;
        AW_TRY(launch_dep(S, k_cg_direction, nblk(nc), 256, 0, s, S->cg_d.p, (const float*)L0.x.p,
                          (const uint8_t*)L0.fluid.p, (const double*)sc, (const int*)(S->cgst.p + 1), nc));
        AW_TRY(launch_dep(S, k_apply_dot, (unsigned)L0.ndesc[2], 256, L0.smem_x64, s, SrcD{S->cg_d.p}, S->cg_zero.p,
                          coef(L0), L0.fluid.p, batch(L0, 2), cf, S->cg_q.p, S->partials.p));
        AW_TRY(launch_dep(S, k_reduce_sum, 1, 256, 0, s, S->partials.p, L0.ndesc[2], sc + 2));
    }
    K.p = p;
    K.r = S->cg_r.p;
    K.rf = L0.b.p;
    K.qn = S->cg_q.p;
    K.sc = sc;
    K.fluid = L0.fluid.p;
    K.air = cf ? 0 : 1;
    K.n = nc;
    K.norm2 = S->norm.p;
    K.prm = S->cgprm.p;
    K.st = S->cgst.p;
    if (h) return launch_dep(S, k_cg_update<true>, ndot, 256, 0, s, K, S->partials.p, S->ticket.p, *h);
    return launch_dep(S, k_cg_update<false>, ndot, 256, 0, s, K, S->partials.p, S->ticket.p, cudaGraphConditionalHandle{});
}

// Mixed-precision CG iterations on the device until the recursive residual falls below the
// tolerance, turns NaN or the iteration limit is reached: one graph whose while node repeats the
// iteration; the update kernel's last CTA sets the loop condition, so no host round trip separates
// iterations.  The graph is built per pressure array and form.  Returns false (state unchanged) when
// the device cannot build such a graph; the caller then keeps the host loop.
static bool cg_devloop_build(aw_solver* S, aw_solver::Loop& C, double* p, unsigned ndot) {
    C.drop();
    if (!S->cap && cudaStreamCreateWithFlags(&S->cap, cudaStreamNonBlocking) != cudaSuccess) return false;
    cudaGraph_t g = nullptr;
    if (cudaGraphCreate(&g, 0) != cudaSuccess) return false;
    bool ok = false;
    cudaGraphConditionalHandle h;
    cudaGraphNodeParams cp = {};
    cudaGraphNode_t node;
    if (cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault) == cudaSuccess) {
        cp.type = cudaGraphNodeTypeConditional;
        cp.conditional.handle = h;
        cp.conditional.type = cudaGraphCondTypeWhile;
        cp.conditional.size = 1;
        if (cudaGraphAddNode(&node, g, nullptr, 0, &cp) == cudaSuccess) {
            cudaGraph_t body = cp.conditional.phGraph_out[0];
            const unsigned long long l0 = g_launches;
            if (cudaStreamBeginCaptureToGraph(S->cap, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal) ==
                cudaSuccess) {
                const aw_status st = cg_iteration(S, p, ndot, S->cap, &h);
                cudaGraph_t out = nullptr;
                const cudaError_t e = cudaStreamEndCapture(S->cap, &out);
                C.kernels = g_launches - l0;
                g_launches = l0;
                ok = st == AW_OK && e == cudaSuccess && cudaGraphInstantiate(&C.exec, g, 0) == cudaSuccess;
            }
        }
    }
    cudaGraphDestroy(g);
    if (!ok) {
        C.exec = nullptr;
        cudaGetLastError();
        return false;
    }
    C.p = p;
    C.gen = S->gen;
    return true;
}

// aw_solve on arrays that start on 16 bytes: the kernels take two cells of a level array at a time
static aw_status solve_aligned(aw_solver* S, const float* d_b, void* d_p, int32_t* cycles, double* final_rel,
                               cudaStream_t s) {
    MGLevel& L0 = S->lv[0];
    const int cf = fv(S) ? 1 : 0;
    const size_t nc = L0.ncell();
    int nsm = 148;
    {
        int dev = 0;
        if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    }
    // reductions over the level-0 cells: at most 8 CTAs per SM, two cells per thread and step, grid-stride
    const unsigned ndot = (unsigned)std::max<size_t>(1, std::min<size_t>({(size_t)nsm * 8, nc / 512 + 1, S->partials.n}));
    // (19 MB a cycle at poisson_256's size: 2860 to 2910 us a solve when the mixed form stored it)
    S->keep_r = S->d.precision == AW_PRECISION_FP32;
    // the blocks' coefficients and masks, ||b||
    if (S->uni) AW_TRY(uniform_check(S, S->d.precision != AW_PRECISION_FP32, s));
    k_sumsq<<<ndot, 256, 0, s>>>(d_b, L0.fluid.p, nc, cf, S->partials.p, S->ticket.p, S->norm.p);
    AW_LAUNCH();
    double bn;
    AW_TRY(fetch_norm(S, s, &bn));
    if (!(bn == bn) || std::isinf(bn)) return set_error(AW_ERR_NAN, "right-hand side contains NaN/Inf");
    if (bn == 0.0) bn = 1.0;
    S->gen = 0;
    for (int m = 0; S->uni && m < S->nmsbg; ++m) {
        int c;
        memcpy(&c, reinterpret_cast<const char*>(S->h_norm + 1) + m * sizeof(int), sizeof c);
        if (c) S->gen |= 1u << m;
    }
    const int nlist = L0.ndesc[2];
    int it = 0;
    double rel = 0;
    aw_status st = AW_OK;
    if (S->d.precision == AW_PRECISION_FP32) {
        S->x0 = (float*)d_p;
        S->b0 = d_b;
        for (;; ++it) {
            double rn;
            st = true_residual(S, (const float*)d_p, nullptr, d_b, L0.r.p, nullptr, s, &rn);
            if (st != AW_OK) break;
            rel = rn / bn;
            if (!(rel == rel)) {
                st = set_error(AW_ERR_NAN, "residual became NaN after %d cycles", it);
                break;
            }
            if (rel < S->d.tolerance) break;
            if (it >= S->d.max_cycles) {
                st = set_error(AW_ERR_NOT_CONVERGED, "relative residual %.3e after %d cycles", rel, it);
                break;
            }
            st = run_vcycle(S, false, false, s);
            if (st != AW_OK) break;
        }
        S->x0 = nullptr;
        S->b0 = nullptr;
    } else if (S->d.precision == AW_PRECISION_FP32_PCG) {
        // Conjugate gradients preconditioned by the same V-cycle as the mixed form, with the pressure,
        // residual, direction and every scalar in FP32 (the like-for-like FP32 baseline of the mixed
        // precision).  r lives in the level-0 right-hand side array, the V-cycle's input.
        float* p = (float*)d_p;
        float* sc = S->cg32_sc.p;
        const unsigned ndot32 = (unsigned)std::min<size_t>((size_t)nsm * 8, S->partials32.n);
        XStore xd;
        xd.f = S->cg32_d.p;
        auto launch_err = [&](const char* what) -> aw_status {
            ++g_launches;
            cudaError_t e = cudaGetLastError();
            return e == cudaSuccess ? AW_OK : set_error(AW_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
        };
        auto read_norm32 = [&](double* out) -> aw_status {
            k_reduce_sum32<<<1, 256, 0, s>>>(S->partials32.p, (int)ndot32, sc + 3);
            AW_TRY(launch_err("k_reduce_sum32"));
            AW_CUDA(cudaMemcpyAsync(S->h_norm, sc + 3, sizeof(float), cudaMemcpyDeviceToHost, s));
            AW_CUDA(cudaStreamSynchronize(s));
            float f;
            memcpy(&f, S->h_norm, sizeof f);
            *out = std::sqrt((double)f);
            return AW_OK;
        };
        // r = b - A p into the V-cycle's input; its norm (FP64 partial sums) for the stopping test
        auto residual32 = [&](double* out) -> aw_status {
            return true_residual(S, p, nullptr, d_b, L0.b.p, nullptr, s, out);
        };
        double rn = 0;
        st = residual32(&rn);
        bool restart = true;
        while (st == AW_OK) {
            rel = rn / bn;
            if (!(rel == rel)) {
                st = set_error(AW_ERR_NAN, "residual became NaN after %d iterations", it);
                break;
            }
            if (rel < S->d.tolerance) {
                if (restart) break;
                st = residual32(&rn);
                restart = true;
                continue;
            }
            if (it >= S->d.max_cycles) {
                st = set_error(AW_ERR_NOT_CONVERGED, "relative residual %.3e after %d iterations", rel, it);
                break;
            }
            st = run_vcycle(S, false, true, s);
            if (st != AW_OK) break;
            // the kernels of one iteration as programmatic dependents of one another
            if ((st = launch_dep(S, k_dot32, ndot32, 256, 0, s, L0.b.p, L0.x.p, L0.fluid.p, nc, S->partials32.p)) != AW_OK) break;
            if ((st = launch_dep(S, k_reduce_sum32, 1, 256, 0, s, S->partials32.p, (int)ndot32, sc + 0)) != AW_OK) break;
            if ((st = launch_dep(S, k_cg_direction32, nblk(nc), 256, 0, s, S->cg32_d.p, L0.x.p, L0.fluid.p, sc,
                                 restart ? 1 : 0, nc)) != AW_OK)
                break;
            if (S->uni) {
                UOut out{};
                out.r = S->cg32_q.p;
                st = uni_residual(S, 0, xd, nullptr, out, nullptr, s);
            } else {
                st = launch_dep(S, k_residual<SrcX>, (unsigned)nlist, 256, L0.smem_smooth, s, SrcX{xd}, S->cg_zero.p,
                                coef(L0), L0.fluid.p, batch(L0, 2), cf, S->cg32_q.p, (double*)nullptr,
                                (double*)nullptr);
            }
            if (st != AW_OK) break;
            if ((st = launch_dep(S, k_dot32, ndot32, 256, 0, s, S->cg32_d.p, S->cg32_q.p, L0.fluid.p, nc,
                                 S->partials32.p)) != AW_OK)
                break;
            if ((st = launch_dep(S, k_reduce_sum32, 1, 256, 0, s, S->partials32.p, (int)ndot32, sc + 2)) != AW_OK) break;
            if ((st = launch_dep(S, k_cg_update32, ndot32, 256, 0, s, p, L0.b.p, S->cg32_d.p, S->cg32_q.p, sc, L0.fluid.p,
                                 nc, S->partials32.p)) != AW_OK)
                break;
            if ((st = launch_dep(S, k_copy_scalar32, 1, 1, 0, s, sc, 1, 0)) != AW_OK) break;
            ++it;
            restart = false;
            st = read_norm32(&rn);
        }
    } else {
        // Mixed precision: conjugate gradients preconditioned by the FP32 V-cycle (FP16-stored coarse
        // corrections), with the residual, the search direction and the pressure accumulation in
        // FP64 and the FP64 coarsest solve inside the V-cycle.  A stand-alone V-cycle iteration
        // stalls or diverges on free-surface domains with four levels; as a preconditioner the same
        // cycle converges on every configuration.  The iterations run in a device-side loop
        // (cg_devloop_build) when the device can build it, else with one host read (||r||) each.
        double* p = (double*)d_p;
        auto residual64 = [&](double* out) -> aw_status {
            return true_residual(S, nullptr, p, d_b, L0.b.p, S->cg_r.p, s, out);
        };
        double rn = 0;
        st = residual64(&rn);
        bool restart = true;
        if (!S->h_cg) AW_CUDA(cudaHostAlloc((void**)&S->h_cg, 4 * sizeof(double), cudaHostAllocDefault));
        while (st == AW_OK) {
            rel = rn / bn;
            if (!(rel == rel)) {
                st = set_error(AW_ERR_NAN, "residual became NaN after %d iterations", it);
                break;
            }
            if (rel < S->d.tolerance) {
                if (restart) break;  // rn is a true residual
                // confirm with the true FP64 residual (the recursive one can drift)
                st = residual64(&rn);
                restart = true;
                continue;
            }
            if (it >= S->d.max_cycles) {
                st = set_error(AW_ERR_NOT_CONVERGED, "relative residual %.3e after %d iterations", rel, it);
                break;
            }
            auto fits = [&](const aw_solver::Loop& l) { return l.exec && l.p == (const void*)p && l.gen == S->gen; };
            if (!fits(S->cgloop[S->cgloop_last])) S->cgloop_last ^= 1;
            aw_solver::Loop& loop = S->cgloop[S->cgloop_last];
            if (S->use_graph && S->use_devloop && !fits(loop) && !cg_devloop_build(S, loop, p, ndot))
                S->use_devloop = false;  // no such graph on this device: the host loop below
            if (restart) {
                // {iterations, restart flag, limit} and {||b||, tolerance}, kept on the device by the iterations
                const int st0[4] = {it, 1, S->d.max_cycles, 0};
                const double prm[2] = {bn, S->d.tolerance};
                memcpy(S->h_cg, st0, sizeof st0);
                memcpy(S->h_cg + 2, prm, sizeof prm);
                AW_CUDA(cudaMemcpyAsync(S->cgst.p, S->h_cg, sizeof st0, cudaMemcpyHostToDevice, s));
                AW_CUDA(cudaMemcpyAsync(S->cgprm.p, S->h_cg + 2, sizeof prm, cudaMemcpyHostToDevice, s));
                restart = false;
            }
            if (S->use_graph && S->use_devloop) {
                // iterations on the device until the recursive residual converges, turns NaN or the
                // limit is reached; then one read-back of ||r||^2 and the iteration count
                AW_CUDA(cudaGraphLaunch(loop.exec, s));
                AW_CUDA(cudaMemcpyAsync(S->h_cg, S->norm.p, sizeof(double), cudaMemcpyDeviceToHost, s));
                AW_CUDA(cudaMemcpyAsync(S->h_cg + 1, S->cgst.p, sizeof(int), cudaMemcpyDeviceToHost, s));
                AW_CUDA(cudaStreamSynchronize(s));
                int it1 = 0;
                memcpy(&it1, S->h_cg + 1, sizeof(int));
                g_launches += loop.kernels * (unsigned long long)(it1 - it);
                it = it1;
                rn = std::sqrt(S->h_cg[0]);
                continue;
            }
            st = cg_iteration(S, p, ndot, s, nullptr);
            ++it;
            if (st == AW_OK) st = fetch_norm(S, s, &rn);  // ||r|| from k_cg_update
        }
    }
    if (cycles) *cycles = it;
    if (final_rel) *final_rel = rel;
    return st;
}

// The caller's arrays may start at any element (a view): one that is not on 16 bytes is solved in an aligned
// copy, 0.2 GB of traffic at 4.7M cells beside the solve's own, and p is copied back whatever the status.
extern "C" aw_status aw_solve(aw_solver* S, const float* d_b, void* d_p, int32_t* cycles, double* final_rel,
                              aw_stream s_) {
    AW_CHECK_ARG(S && d_b && d_p, "null argument");
    cudaStream_t s = (cudaStream_t)s_;
    const size_t nc = S->lv[0].ncell();
    const size_t pbytes = nc * (S->d.precision == AW_PRECISION_MIXED ? sizeof(double) : sizeof(float));
    auto aligned = [](const void* q) { return ((uintptr_t)q & 15u) == 0; };
    const float* b = d_b;
    void* p = d_p;
    if (!aligned(d_b)) {
        AW_TRY(S->b_copy.ensure(std::max<size_t>(nc, 1)));
        AW_CUDA(cudaMemcpyAsync(S->b_copy.p, d_b, nc * sizeof(float), cudaMemcpyDeviceToDevice, s));
        b = S->b_copy.p;
    }
    if (!aligned(d_p)) {
        AW_TRY(S->p_copy.ensure(std::max<size_t>((pbytes + 7) / 8, 1)));
        AW_CUDA(cudaMemcpyAsync(S->p_copy.p, d_p, pbytes, cudaMemcpyDeviceToDevice, s));
        p = S->p_copy.p;
    }
    const aw_status st = solve_aligned(S, b, p, cycles, final_rel, s);
    if (p != d_p && st != AW_ERR_CUDA) {
        AW_CUDA(cudaMemcpyAsync(d_p, p, pbytes, cudaMemcpyDeviceToDevice, s));
        AW_CUDA(cudaStreamSynchronize(s));
    }
    return st;
}
