// sm_103a kernels for the SwiftLink MCMC hot path.
//
// Samplers (one chain's descent graph per chain, bit-packed [chain][M][W]):
//  * lsampler_kernel<T,G> -- L-sampler, one group of G = 32, 16 or 8 lanes per
//                            (chain, locus): T=double with the reference's
//                            operation order (bit-exact decisions), T=float
//                            the batched form.  The form compiled per
//                            pedigree lives in sl_lsjit.cc.
//  * lsampler_quad_kernel<T> -- the same with four lanes per task, eight tasks
//                            per warp: the form that runs unless another is
//                            asked for or the peel sequence does not suit it.
//  * si_kernel<T>, si_quad_kernel<T>, si_select_kernel -- sequential imputation
//                            passes (one-sided L-steps from a start locus), 32
//                            or 4 lanes each, and the best pass.
//  * fag_kernel           -- M-sampler likelihoods, thread per (chain, locus):
//                            founder-allele graph with one meiosis toggled
//                            (exact mode, and fast mode past the warp form's
//                            shared-memory limit).
//  * msweep_kernel<G>     -- fast mode: a chain's whole M-sweep by one cluster.
//  * fag_warp_kernel<G>   -- fast-mode likelihoods in lane groups of G (chains
//                            whose share of loci does not fit a cluster).
//  * ffbs_exact_runs_kernel, ffbs_exact_kernel -- exact mode: forward filter of
//                            one meiosis in runs that start anew, backward
//                            sampling as a composition of choices.
//  * ffbs_scan_kernel     -- the same as block-wide scans (fast mode).
//  * loglik_*_kernel      -- log P(G, graph) of (graph, map) chain pairs (MC3).
// Scorer:
//  * lod_kernel<T,R,L>    -- trait peel at every (graph, interval, position), L
//                            lanes per task; T=double is the plain FP64 form,
//                            R=true rescales every rfunction by a power of two
//                            and carries the exponent.
//  * lod_prog_kernel      -- the FP32 rescaled peel as a slot-program
//                            interpreter (specialised forms: sl_jit.cc).
//  * trait_adjoint_kernel, trait_adjoint_thr_kernel -- the hand-written
//                            adjoint of the rescaled peel, a warp or a thread
//                            per task (the form compiled per pedigree lives
//                            in sl_adjjit.cc).
//  * lod_merge_kernel, chain_merge_kernel -- FP64 log-sum accumulation.
// Run graph: run_init / chain_iter / chain_advance kernels drive each chain's
// WHILE and SWITCH nodes; choose / shuffle / set_key draw the iteration's
// choices; lfreq_kernel precomputes the allele frequencies' log2 per chain map.
//
// FP64 arithmetic on decision paths uses __dmul_rn/__dadd_rn/__ddiv_rn so no
// multiply-add is contracted and the doubles match the reference's.

#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <float.h>
#include <limits.h>
#include <stdint.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <utility>

#include "sl_flips.h"
#include "sl_internal.h"
#include "sl_philox.cuh"

namespace sl {

namespace cg = cooperative_groups;

// Raises a kernel's dynamic shared-memory limit on the current device when a
// launch needs more than it was given so far.  The attribute is per device
// and contexts on several devices or threads may launch the same kernel, so
// the record is keyed by (kernel, device) and taken under a lock.
static cudaError_t ensure_smem(const void* func, size_t bytes) {
    if (bytes <= 48 * 1024) return cudaSuccess;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    static std::mutex mu;
    static std::map<std::pair<const void*, int>, size_t> given;
    std::lock_guard<std::mutex> lock(mu);
    size_t& have = given[std::make_pair(func, dev)];
    if (bytes <= have) return cudaSuccess;
    e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) have = bytes;
    else cudaGetLastError();   // reported here; the next launch, perhaps another context's, asks for the last error
    return e;
}

#define DMUL __dmul_rn
#define DADD __dadd_rn
#define DSUB __dsub_rn
#define DDIV __ddiv_rn
#define FULLMASK 0xffffffffu

__device__ __forceinline__ int dgbit(const uint32_t* col, int b) { return (col[b >> 5] >> (b & 31)) & 1; }
__device__ __forceinline__ int digit(int ext, int pos) { return (ext >> (2 * pos)) & 3; }
__device__ __forceinline__ void set_status(int* st, int code) { atomicCAS(st, 0, code); }

// maternal / paternal allele of a phased state: U=0, A=1
__device__ __forceinline__ int mat_allele(int s) { return (s == AA || s == AU) ? 1 : 0; }
__device__ __forceinline__ int pat_allele(int s) { return (s == AA || s == UA) ? 1 : 0; }

__device__ __forceinline__ double philox_u01(uint64_t key, uint64_t c_hi, uint64_t c_lo) {
    return sl_philox_u01(key, c_hi, c_lo);
}

// Where uniform draws come from: a caller-supplied array (bit-exact replay of
// the reference) or the Philox stream (device-driven runs).  `unit` is the
// locus (L-sampler) or the meiosis step (M-sampler) within the sweep.
// `key` (device memory, may be null) overrides seed and iteration: a
// captured graph replayed every iteration reads them there.
struct Draws {
    const double* u;
    int64_t chain_stride, unit_stride;
    uint64_t seed, iter;
    int stage;
    const uint64_t* key;
    __device__ __forceinline__ double get(int chain_rel, int chain, int64_t unit, int64_t k) const {
        if (u) return u[chain_rel * chain_stride + unit * unit_stride + k];
        const uint64_t sd = key ? key[0] : seed, it = key ? key[1] : iter;
        uint64_t hi = ((uint64_t)chain << 40) ^ (it << 4) ^ (uint64_t)stage;
        return philox_u01(sd, hi, ((uint64_t)unit << 24) ^ (uint64_t)k);
    }
    // The same draw rounded down to a float: for a float x, get() < (double)x
    // exactly when get_rd() < x (no float lies between a draw and the one below
    // it), without the FP64 units, of which an SM has two.
    __device__ __forceinline__ float get_rd(int chain_rel, int chain, int64_t unit, int64_t k) const {
        if (u) return __double2float_rd(u[chain_rel * chain_stride + unit * unit_stride + k]);
        const uint64_t sd = key ? key[0] : seed, it = key ? key[1] : iter;
        const uint64_t hi = ((uint64_t)chain << 40) ^ (it << 4) ^ (uint64_t)stage;
        return __ull2float_rd(sl_philox_bits(sd, hi, ((uint64_t)unit << 24) ^ (uint64_t)k)) * 0x1p-53f;
    }
};
// the draw to compare a probability of type T with
template <typename T>
__device__ __forceinline__ T draw_for(const Draws& d, int chain_rel, int chain, int64_t unit, int64_t k) {
    if constexpr (sizeof(T) == 4) return d.get_rd(chain_rel, chain, unit, k);
    else return d.get(chain_rel, chain, unit, k);
}

__global__ void set_key_kernel(uint64_t* key, uint64_t seed, uint64_t iter) {
    key[0] = seed;
    key[1] = iter;
}

// Arithmetic of the L-sampler: FP64 without contraction (the reference's
// doubles) or plain FP32 for the fast sampler mode.
template <typename T>
struct Ls;
template <>
struct Ls<double> {
    static __device__ __forceinline__ double mul(double a, double b) { return DMUL(a, b); }
    static __device__ __forceinline__ double add(double a, double b) { return DADD(a, b); }
    static __device__ __forceinline__ double sub(double a, double b) { return DSUB(a, b); }
    static __device__ __forceinline__ double div(double a, double b) { return DDIV(a, b); }
};
template <>
struct Ls<float> {   // rounded operations, never contracted: the kernel specialised at run time matches them
    static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
    static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
    static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
    static __device__ __forceinline__ float div(float a, float b) { return __fdiv_rn(a, b); }
};

// The lanes working on one L-sampler task: a whole warp (G = 32), half of one
// or a quarter (G = 16 or 8; two or four tasks per warp, for pedigrees whose
// rfunctions have few allowed cells).  Shuffles and ballots stay within the
// group, whose tasks may diverge from the warp's other groups; lane numbers
// are the group's own.
template <int G>
struct Lanes {
    static_assert(G == 32 || G == 16 || G == 8, "a lane group is 32, 16 or 8 lanes of one warp");
    unsigned mask;
    // the group's lanes: G consecutive lanes starting at a multiple of G
    __device__ __forceinline__ Lanes() : mask(G == 32 ? FULLMASK : (((1u << G) - 1u) << (threadIdx.x & (32 - G)))) {}
    template <typename V>
    __device__ __forceinline__ V shfl(V v, int src) const { return __shfl_sync(mask, v, src, G); }
    template <typename V>
    __device__ __forceinline__ V shfl_xor(V v, int d) const { return __shfl_xor_sync(mask, v, d, G); }
    template <typename V>
    __device__ __forceinline__ V shfl_up(V v, int d) const { return __shfl_up_sync(mask, v, d, G); }
    __device__ __forceinline__ unsigned ballot(bool p) const {
        const unsigned b = __ballot_sync(mask, p);
        return G == 32 ? b : (b >> (threadIdx.x & (32 - G))) & ((1u << G) - 1u);
    }
    __device__ __forceinline__ void sync() const { __syncwarp(mask); }
};

// ---------------------------------------------------------------------------
// L-sampler
// ---------------------------------------------------------------------------

// Recombination distributions of one child's two meioses for every parental
// state (SamplerRfunction::get_recombination_distribution,
// sampler_rfunction.cc:102-157): d[side*8 + state*2 + allele].
template <typename T>
__device__ void ls_dist_one(const ProblemDev& P, int person, const uint32_t* colL, const uint32_t* colR,
                            int l, T th, T an, T th2, T an2, T* d) {
    using A = Ls<T>;
    for (int side = 0; side < 2; ++side) {
        const int b = 2 * (person - P.F) + side;
        T* s = d + side * 8;
        s[UU * 2 + 0] = T(1); s[UU * 2 + 1] = T(0);
        s[AA * 2 + 0] = T(0); s[AA * 2 + 1] = T(1);
        T tmp0 = T(0.5), tmp1 = T(0.5);
        if (colL) {   // a left neighbour (absent at locus 0 and when imputation ignores it)
            const bool cross = dgbit(colL, b) != 0;
            tmp0 = A::mul(tmp0, cross ? th2 : an2);
            tmp1 = A::mul(tmp1, cross ? an2 : th2);
        }
        if (colR) {
            const bool cross = dgbit(colR, b) != 0;
            tmp0 = A::mul(tmp0, cross ? th : an);
            tmp1 = A::mul(tmp1, cross ? an : th);
        }
        const T total = A::add(tmp0, tmp1);
        const T uau = A::div(tmp1, total);
        s[AU * 2 + 0] = uau;
        s[AU * 2 + 1] = A::sub(T(1), uau);
        const T uua = A::div(tmp0, total);
        s[UA * 2 + 0] = uua;
        s[UA * 2 + 1] = A::sub(T(1), uua);
    }
}

template <typename T, int G>
__device__ __forceinline__ void ls_dists(const ProblemDev& P, const OpDev& op, const int32_t* opd,
                                         const uint32_t* colL, const uint32_t* colR, int l, T th, T an, T th2, T an2,
                                         T* dist, int lane) {
    const int nch = op.type == CHILD ? 1 : (op.type == PARENT ? op.n_child : 0);
    for (int c = lane; c < nch; c += G) {
        const int person = op.type == CHILD ? op.peel : opd[op.child_at + 4 * c];
        ls_dist_one<T>(P, person, colL, colR, l, th, an, th2, an2, dist + 16 * c);
    }
}

// A cell of op k in the compact layout, with the peel node's state v: ext
// holds the dense digits of (cutset states, v) as in peel_matrix.h:37-45, rk
// the states' ranks and bits each position's rank bits (2 bits per position,
// the peel node at position c), bad the positions whose state is not allowed
// (only the peel node's can be, the cell itself being valid).
struct LsCell {
    int ext, rk, bits, bad;
};

// A task's compact rfunctions: the first `cap` cells in the task's shared
// memory, the rest (at the few loci whose rfunctions need more) in its slice
// of a global spill buffer.  Sizing the shared part for nearly every locus
// rather than the largest keeps more tasks resident on an SM.
template <typename T>
struct LsArena {
    T* sh;
    T* gl;
    int cap;
    __device__ __forceinline__ T ld(int o) const { return o < cap ? sh[o] : gl[o - cap]; }
    __device__ __forceinline__ void st(int o, T v) const {
        if (o < cap) sh[o] = v;
        else gl[o - cap] = v;
    }
};

// One presum entry (cell, peel state v) in the reference's product order
// (sampler_rfunction.cc:190-287, rfunction.cc:116-142); a previous rfunction
// is read at its compact index, or as zero where the dense matrix held zero.
template <typename T>
__device__ T ls_term(const OpDev& op, const int32_t* opd, const LsArena<T>& Am, const uint16_t* off, const T* dist,
                     const LsCell& x, int v, T tv) {
    using A = Ls<T>;
    const int ext = x.ext;
    T tmp = tv;
    if (op.type == CHILD) {
        const int mt = digit(ext, op.mpos), pt = digit(ext, op.fpos);
        const T tr = A::mul(dist[mt * 2 + mat_allele(v)], dist[8 + pt * 2 + pat_allele(v)]);
        tmp = A::mul(tmp, tr);
    }
    const int32_t* pd = opd + op.prev_at;
    const int32_t* po = opd + op.prev_ops_at;
    for (int j = 0; j < op.n_prev; ++j) {
        const int pc = pd[1];
        int idx = 0, sh = 0, bad = 0;
        for (int q = 0; q < pc; ++q) {
            const int pos = pd[2 + q];
            idx |= ((x.rk >> (2 * pos)) & 3) << sh;
            sh += (x.bits >> (2 * pos)) & 3;
            bad |= (x.bad >> pos) & 1;
        }
        tmp = A::mul(tmp, bad ? T(0) : Am.ld(off[po[j]] + idx));
        pd += 2 + pc;
    }
    if (op.type == PARENT) {
        T cp = T(1);
        const int32_t* cd = opd + op.child_at;
        for (int c = 0; c < op.n_child; ++c, cd += 4) {
            const int kt = digit(ext, cd[1]), other = digit(ext, cd[2]);
            const int mt = cd[3] ? v : other, pt = cd[3] ? other : v;
            const T tr = A::mul(dist[c * 16 + mt * 2 + mat_allele(kt)], dist[c * 16 + 8 + pt * 2 + pat_allele(kt)]);
            cp = A::mul(cp, tr);
        }
        tmp = A::mul(tmp, cp);
    }
    return tmp;
}

// The L-sampler's compact rfunctions.  At locus l a member whose genotype-
// elimination mask allows s states takes b = 0, 1 or 2 bits (s = 1, 2, 3-4)
// of a cell's index, holding the rank of its state among the allowed ones, in
// cutset order; op k's cells are the 2^B_k indices (B_k the sum of its
// members' bits) at offset off[k] of the task's arena, a prefix sum over the
// ops worked out at the start of each task.  Only cells whose members are all
// in allowed states are stored -- on the 400-member pedigree at most 1,350
// values against 11,485 for dense 4^c matrices -- and exactly those are the
// cells the dense layout could hold non-zero: a gather that would reach a
// dense cell with a disallowed state reads zero instead, and a rank past the
// allowed count (s = 3) marks an invalid cell.
__device__ __forceinline__ int rank_bits(int mask) {
    const int s = __popc(mask);
    return s <= 1 ? 0 : (s == 2 ? 1 : 2);
}
__device__ __forceinline__ int state_rank(int mask, int v) { return __popc(mask & ((1 << v) - 1)); }
__device__ __forceinline__ int state_of_rank(int mask, int r) {   // the r-th allowed state (r < popc(mask))
    for (int i = 0; i < r; ++i) mask &= mask - 1;
    return __ffs(mask) - 1;
}

// A task's shared bytes: the rfunctions [ls_arena, compact], the children's
// transmission distributions [16 per child], the sampled states [N], the
// locus's genotype codes and masks [N], its neighbours' descent-graph words
// [2 W], its prior row [16] and the ops' compact offsets [K + 1] (16-bit); each part
// 16-byte aligned, so every task's base is aligned.  (The backward pass's
// draws are made as it goes, one per operation: storing them took K doubles,
// a third of a task on the 400-member pedigree.)
__host__ __device__ __forceinline__ size_t al16(size_t x) { return (x + 15) & ~(size_t)15; }
template <typename T>
__host__ __device__ __forceinline__ size_t ls_draws_at(const ProblemDev& P) {
    return al16((size_t)P.ls_cap * sizeof(T) + (size_t)P.max_child * 16 * sizeof(T) + (size_t)P.N);
}
template <typename T>
__host__ __device__ __forceinline__ size_t ls_gcol_at(const ProblemDev& P) {
    return ls_draws_at<T>(P);
}
template <typename T>
__host__ __device__ __forceinline__ size_t ls_cols_at(const ProblemDev& P) {
    return al16(ls_gcol_at<T>(P) + (size_t)P.N);
}
template <typename T>
__host__ __device__ __forceinline__ size_t ls_pri_at(const ProblemDev& P) {
    return al16(ls_cols_at<T>(P) + 8 * (size_t)P.W);
}
template <typename T>
__host__ __device__ __forceinline__ size_t ls_off_at(const ProblemDev& P) {
    return al16(ls_pri_at<T>(P) + 16 * sizeof(T));
}
template <typename T>
__host__ __device__ __forceinline__ size_t ls_warp_bytes(const ProblemDev& P) {
    return al16(ls_off_at<T>(P) + 2 * ((size_t)P.K + 1));   // 16-bit offsets: the arena holds < 65,536 cells
}

// Task slot s's part of the spill buffer of chain `chain` (null when no
// locus spills, or past the buffer's slots).  Every chain has its own slots:
// the run graph launches the chains' sweeps concurrently; a launch over
// several chains runs its tasks slot by slot in the first chain's slots.
template <typename T>
__device__ __forceinline__ T* ls_spill_slice(const ProblemDev& P, int chain, int64_t s) {
    if (P.ls_spill_cells <= 0 || s >= P.ls_spill_slots || chain < 0 || chain >= P.ls_spill_chains) return nullptr;
    return (T*)P.ls_spill + ((size_t)chain * P.ls_spill_slots + s) * P.ls_spill_cells;
}

// Block-shared copies of the peel's operations and their lists: every lane
// reads them at every operation, and L1 holds little beside the arenas.
__host__ __device__ __forceinline__ size_t ls_tables_bytes(const ProblemDev& P) {
    return P.ls_stage_ops ? al16((size_t)P.K * sizeof(OpDev)) + al16((size_t)P.opdata_n * 4) : 0;
}

__device__ __forceinline__ void ls_stage_tables(const ProblemDev& P, unsigned char* smem, const OpDev*& ops,
                                                const int32_t*& opd) {
    if (!P.ls_stage_ops) {   // tables too large to share a block's shared memory with the arenas
        ops = P.ops;
        opd = P.opdata;
        return;
    }
    int32_t* so = (int32_t*)smem;
    int32_t* sd = (int32_t*)(smem + al16((size_t)P.K * sizeof(OpDev)));
    const int32_t* src = (const int32_t*)P.ops;
    const int nw = P.K * (int)(sizeof(OpDev) / 4);
    for (int i = threadIdx.x; i < nw; i += blockDim.x) so[i] = src[i];
    for (int i = threadIdx.x; i < P.opdata_n; i += blockDim.x) sd[i] = P.opdata[i];
    ops = (const OpDev*)so;
    opd = sd;
}

// One warp per (chain, locus) task; the listed loci must be pairwise
// non-adjacent so each task owns its descent-graph column.
// One L-sampler step at locus l of one chain, by one warp
// (LocusSampler::step, locus_sampler2.cc:128-159): hasL / hasR say whether the
// neighbouring columns take part (set_locus(l, ignore_left, ignore_right),
// sampler_rfunction.h:84-101).  Draws are taken at indices base, base + 1, ...
// of the unit's stream.  Returns the number of draws used, or -1 when the
// locus has likelihood 0; *logroot (lane 0) receives log of the peel's result.
template <typename T, int G>
__device__ int ls_locus(const ProblemDev& P, const OpDev* ops, const int32_t* opd, uint32_t* dg, int cr, int chain,
                        int l, bool hasL, bool hasR, const Draws& draws, int64_t unit, int64_t base,
                        unsigned char* wsmem, T* spill, int lane, int* status, double* logroot) {
    using Ar = Ls<T>;
    const Lanes<G> L;
    constexpr bool kRescale = sizeof(T) == 4;   // FP32: each rfunction scaled to a maximum of about 1
    const LsArena<T> A{(T*)wsmem, spill, P.ls_cap};
    T* dist = A.sh + P.ls_cap;
    int8_t* assign = (int8_t*)(dist + 16 * P.max_child);
    uint16_t* off = (uint16_t*)(wsmem + ls_off_at<T>(P));
    uint32_t* colC = dg + ((size_t)chain * P.M + l) * P.W;
    // the locus's inputs copied to the task's shared memory first
    uint8_t* sg = (uint8_t*)(wsmem + ls_gcol_at<T>(P));
    uint32_t* sL = (uint32_t*)(wsmem + ls_cols_at<T>(P));
    uint32_t* sR = sL + P.W;
    T* spri = (T*)(wsmem + ls_pri_at<T>(P));
    {
        const uint8_t* gsrc = P.geno + (size_t)l * P.N;
        for (int i = lane; i < P.N; i += G) sg[i] = gsrc[i];
        for (int w = lane; w < P.W; w += G) {
            if (hasL) sL[w] = colC[w - P.W];
            if (hasR) sR[w] = colC[w + P.W];
        }
        for (int i = lane; i < 16; i += G) {
            if constexpr (sizeof(T) == 4) spri[i] = (T)P.prior_f[(size_t)l * 16 + i];
            else spri[i] = (T)P.prior[(size_t)l * 16 + i];
        }
        L.sync();
    }
    const uint32_t* colL = hasL ? sL : nullptr;
    const uint32_t* colR = hasR ? sR : nullptr;
    T th = T(1), an = T(1), th2 = T(1), an2 = T(1);
    if constexpr (sizeof(T) == 4) {
        const float* tf = P.c_theta_f + (size_t)chain * (P.M - 1);
        if (hasL) { th2 = tf[l - 1]; an2 = 1.f - th2; }
        if (hasR) { th = tf[l]; an = 1.f - th; }
    } else {
        const double* td = P.c_theta + (size_t)chain * (P.M - 1);
        if (hasL) { th2 = td[l - 1]; an2 = DSUB(1.0, td[l - 1]); }
        if (hasR) { th = td[l]; an = DSUB(1.0, td[l]); }
    }
    const uint8_t* gcol = sg;
    const T* pri = spri;
    int scale = 0;
    // the ops' compact offsets at this locus: each lane sums the cells of a
    // run of ops, a scan over the group turns the sums into offsets
    {
        const int per = (P.K + G - 1) / G, k0 = min(P.K, lane * per), k1 = min(P.K, k0 + per);
        int sum = 0;
        for (int k = k0; k < k1; ++k) {
            const OpDev& op = ops[k];
            int b = 0;
            for (int q = 0; q < op.c; ++q) b += rank_bits((gcol[opd[op.cut_at + q]] >> 4) & 15);
            sum += 1 << b;
        }
        int incl = sum;
        for (int dd = 1; dd < G; dd <<= 1) {
            const int o = L.shfl_up(incl, dd);
            if (lane >= dd) incl += o;
        }
        int run = incl - sum;
        for (int k = k0; k < k1; ++k) {
            const OpDev& op = ops[k];
            int b = 0;
            for (int q = 0; q < op.c; ++q) b += rank_bits((gcol[opd[op.cut_at + q]] >> 4) & 15);
            off[k] = (uint16_t)run;
            run += 1 << b;
        }
        if (lane == G - 1) off[P.K] = (uint16_t)incl;
        L.sync();
        if (L.shfl(incl, G - 1) > P.ls_arena || (spill == nullptr && L.shfl(incl, G - 1) > P.ls_cap)) {
            // cannot happen: the arena (shared part and spill) holds the most any locus needs
            if (lane == 0) set_status(status, ST_ILLEGAL_DG);
            return -1;
        }
    }
    // forward peel over the valid cells of every rfunction
    for (int k = 0; k < P.K; ++k) {
        const OpDev op = ops[k];
        ls_dists<T, G>(P, op, opd, colL, colR, l, th, an, th2, an2, dist, lane);
        L.sync();
        const int32_t* cut = opd + op.cut_at;
        // the op's members: allowed states (4 bits each) and rank bits, the peel node last
        unsigned long long mk = 0;
        int bits = 0, B = 0;
        for (int q = 0; q < op.c; ++q) {
            const int m = (gcol[cut[q]] >> 4) & 15, b = rank_bits(m);
            mk |= (unsigned long long)m << (4 * q);
            bits |= b << (2 * q);
            B += b;
        }
        const int mp = (gcol[op.peel] >> 4) & 15;
        bits |= rank_bits(mp) << (2 * op.c);
        const int ncell = 1 << B;
        const T* trait = pri + 4 * (gcol[op.peel] & 3);
        const int ob = off[k];
        T mx = T(0);
        // one (cell, state) term per lane, four lanes per cell; the cell's
        // total adds its terms in state order from zero, as the reference's
        // loop does (a skipped term is an exact zero)
        const int nitem = 4 * ncell, grp = lane & ~3, v = lane & 3;
        const T tv = trait[v];
        LsCell x;
        x.bits = bits;
        x.bad = ((mp >> v) & 1) ? 0 : 1 << op.c;
        const int vrank = state_rank(mp, v);
        for (int it0 = 0; it0 < nitem; it0 += G) {
            const int cell = (it0 + lane) >> 2;
            T term = T(0);
            if (it0 + lane < nitem && tv != T(0)) {
                // decode the compact index into states and ranks
                int rem = cell, ext = 0, rk = 0;
                bool ok = true;
                for (int q = 0; q < op.c; ++q) {
                    const int m = (int)(mk >> (4 * q)) & 15, b = (bits >> (2 * q)) & 3;
                    const int r = rem & ((1 << b) - 1);
                    rem >>= b;
                    ok &= r < __popc(m);
                    ext |= state_of_rank(m, r & 3) << (2 * q);
                    rk |= r << (2 * q);
                }
                if (ok) {
                    x.ext = ext | (v << (2 * op.c));
                    x.rk = rk | (vrank << (2 * op.c));
                    term = ls_term<T>(op, opd, A, off, dist, x, v, tv);
                }
            }
            const T t0 = L.shfl(term, grp), t1 = L.shfl(term, grp + 1);
            const T t2 = L.shfl(term, grp + 2), t3 = L.shfl(term, grp + 3);
            if (v == 0 && it0 + lane < nitem) {
                const T total = Ar::add(Ar::add(Ar::add(Ar::add(T(0), t0), t1), t2), t3);
                A.st(ob + cell, total);
                mx = total > mx ? total : mx;
            }
        }
        if (kRescale) {
            // the sampling draws from ratios within one rfunction, so a
            // power-of-two factor per rfunction changes no decision
            for (int dd = G / 2; dd >= 1; dd >>= 1) {
                const T o = L.shfl_xor(mx, dd);
                mx = o > mx ? o : mx;
            }
            if (mx > T(0)) {
                // every rfunction enters the root exactly once, so the root's
                // logarithm is the scaled root's plus the removed exponents
                const int ex = ilogbf((float)mx);
                scale += ex;
                const float f = scalbnf(1.0f, -ex);
                L.sync();   // the cells other lanes of the group wrote (some maybe in the global spill)
                for (int cell = lane; cell < ncell; cell += G) A.st(ob + cell, (T)((float)A.ld(ob + cell) * f));
            }
        }
        L.sync();
    }
    const T root = A.ld(off[P.K - 1]);
    if (root == T(0)) {
        if (lane == 0) set_status(status, ST_ZERO_LIK);
        L.sync();
        return -1;
    }
    if (lane == 0 && logroot) *logroot = log((double)root) + (double)scale * 0.69314718055994530942;
    for (int i = lane; i < P.N; i += G) assign[i] = -1;
    L.sync();
    // backward sampling of ordered genotypes (SamplerRfunction::sample); the
    // group's last lane draws the operation's uniform (one per operation, in
    // the backward order) while the others work out its terms
    for (int k = P.K - 1; k >= 0; --k) {
        const OpDev op = ops[k];
        const double rdraw = lane == G - 1 ? draws.get(cr, chain, unit, base + (P.K - 1 - k)) : 0.0;
        ls_dists<T, G>(P, op, opd, colL, colR, l, th, an, th2, an2, dist, lane);
        L.sync();
        const int32_t* cut = opd + op.cut_at;
        const T* trait = pri + 4 * (gcol[op.peel] & 3);
        // the sampled cutset states as a compact cell (invalid where a state
        // is not allowed: the dense matrix held zero there)
        int ext = 0, rk = 0, bits = 0;
        bool known = true, ok = true;
        for (int q = 0; q < op.c; ++q) {
            const int a = assign[cut[q]];
            const int m = (gcol[cut[q]] >> 4) & 15;
            known &= a >= 0;
            ok &= ((m >> (a & 3)) & 1) != 0;
            ext |= (a & 3) << (2 * q);
            rk |= state_rank(m, a & 3) << (2 * q);
            bits |= rank_bits(m) << (2 * q);
        }
        const int mp = (gcol[op.peel] >> 4) & 15;
        T pv = T(0);
        if (lane < 4 && known && ok) {
            const T tv = trait[lane];
            if (tv != T(0)) {
                LsCell x;
                x.ext = ext | (lane << (2 * op.c));
                x.rk = rk | (state_rank(mp, lane) << (2 * op.c));
                x.bits = bits | (rank_bits(mp) << (2 * op.c));
                x.bad = ((mp >> lane) & 1) ? 0 : 1 << op.c;
                pv = ls_term<T>(op, opd, A, off, dist, x, lane, tv);
            }
        }
        const double rk_draw = L.shfl(rdraw, G - 1);
        const T p0 = L.shfl(pv, 0), p1 = L.shfl(pv, 1);
        const T p2 = L.shfl(pv, 2), p3 = L.shfl(pv, 3);
        if (lane == 0) {
            if (!known) set_status(status, ST_ILLEGAL_DG);
            T pd[4] = {p0, p1, p2, p3};
            const T tot = Ar::add(Ar::add(Ar::add(p0, p1), p2), p3);
            if (tot != T(0))
                for (int v = 0; v < 4; ++v) pd[v] = Ar::div(pd[v], tot);
            const double r = rk_draw;
            T acc = T(0);
            int lastv = 0, pick = -1;
            for (int v = 0; v < 4; ++v) {
                acc = Ar::add(acc, pd[v]);
                if (r < (double)acc) { pick = v; break; }
                if (pd[v] != T(0)) lastv = v;
            }
            assign[op.peel] = (int8_t)(pick >= 0 ? pick : lastv);
        }
        L.sync();
    }
    // meiosis indicators (locus_sampler2.cc:32-125) in person order, maternal
    // first: bit b = 2 (person - F) + parent, so 32 consecutive meioses are one
    // descent-graph word.  A lane takes one meiosis; a draw is consumed only
    // below a homozygous parent, and a ballot prefix gives each draw its index.
    {
        int64_t cursor = base + P.K;
        const int nb = 2 * P.Nnf;
        for (int w = 0; w < P.W; ++w) {
            uint32_t word = 0;
            for (int h = 0; h < 32; h += G) {
                const int b = 32 * w + h + lane;
                int mi = 0, need = 0;
                T p0 = T(1), p1 = T(1);
                if (b < nb) {
                    const int i = P.F + (b >> 1), par = b & 1;
                    const int tr = assign[i];
                    const int ptr = assign[par == 0 ? P.mother[i] : P.father[i]];
                    const int allele = par == 0 ? ((tr == UU || tr == UA) ? 0 : 1) : ((tr == UU || tr == AU) ? 0 : 1);
                    if (ptr == UA || ptr == AU) {
                        mi = allele == 0 ? (ptr == UA ? 0 : 1) : (ptr == UA ? 1 : 0);
                    } else {
                        need = 1;
                        if (hasL) {
                            const int d = dgbit(colL, b);
                            p0 = Ar::mul(p0, d == 0 ? an2 : th2);
                            p1 = Ar::mul(p1, d == 1 ? an2 : th2);
                        }
                        if (hasR) {
                            const int d = dgbit(colR, b);
                            p0 = Ar::mul(p0, d == 0 ? an : th);
                            p1 = Ar::mul(p1, d == 1 ? an : th);
                        }
                    }
                }
                const unsigned nmask = L.ballot(need);
                if (need) {
                    const double r = draws.get(cr, chain, unit, cursor + __popc(nmask & ((1u << lane) - 1u)));
                    mi = (r < (double)Ar::div(p0, Ar::add(p0, p1))) ? 0 : 1;
                }
                cursor += __popc(nmask);
                word |= L.ballot(mi != 0) << h;
            }
            if (lane == 0) colC[w] = word;   // bits past 2 Nnf stay zero
        }
        L.sync();
        return (int)(cursor - base);
    }
}

// One task per (chain, locus), G lanes each (a warp, or half of one); the
// listed loci must be pairwise non-adjacent so each task owns its
// descent-graph column.
template <typename T, int G>
__global__ void __launch_bounds__(128) lsampler_kernel(ProblemDev P, uint32_t* dg, int first, int nchain,
                                                       const int32_t* loci, int nloci, Draws draws,
                                                       const uint8_t* sel, int want, int* status) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int kPer = 32 / G;   // tasks per warp
    const int tpb = (blockDim.x >> 5) * kPer, slot = (threadIdx.x >> 5) * kPer + ((threadIdx.x & 31) / G);
    const int lane = threadIdx.x & (G - 1);
    const OpDev* ops;
    const int32_t* opd;
    ls_stage_tables(P, smem, ops, opd);
    __syncthreads();
    unsigned char* wsmem = smem + ls_tables_bytes(P) + (size_t)slot * ls_warp_bytes<T>(P);
    T* spill = ls_spill_slice<T>(P, first, (int64_t)blockIdx.x * tpb + slot);
    if (P.ls_spill_cells > 0 && !spill) {   // the launch has more task slots than the spill buffer: never run past it
        if (lane == 0) set_status(status, ST_ILLEGAL_DG);
        return;
    }
    const int64_t ntask = (int64_t)nchain * nloci;
    for (int64_t t = (int64_t)blockIdx.x * tpb + slot; t < ntask; t += (int64_t)gridDim.x * tpb) {
        const int cr = (int)(t / nloci);
        if (sel && sel[cr] != want) continue;
        const int l = loci[t % nloci];
        ls_locus<T, G>(P, ops, opd, dg, cr, first + cr, l, l > 0, l < P.M - 1, draws, l, 0, wsmem, spill, lane,
                       status, nullptr);
    }
}

// ---------------------------------------------------------------------------
// L-sampler with four lanes per (chain, locus) task, eight tasks per warp.
//
// The steps, products and draws of ls_locus, bit for bit; what differs is how
// the work lies on the warp.  Lane v of a task's four works out the terms of
// the peel node's state v, four cells of an rfunction at a time; with most
// members typed an op has one to four cells, so the eight tasks go through an
// op together and its description is read once for them, from a packed form of
// the operations in the block's shared memory (P.quad_prog).  The transmission
// distributions, which ls_locus works out again for every child, op and pass
// (four divisions each), take only four values per locus -- a child's indicator
// at the left and the right neighbour -- and are tabled once per task; likewise
// the indicator probabilities of the last phase.  A task's shared memory holds
// a byte per member and the neighbours' columns; the rfunctions, compact as
// there, lie in shared memory when eight tasks' fit (kQuadSharedArena), else
// in a global arena that stays in L1 and L2.
//
// Bound by issue: 400,000 warp instructions per eight tasks of the 400-member
// pedigree, 58% of the issue slots with 15 warps on an SM.  The loops stay
// rolled: unrolled by the compiler, warps at different operations waited for
// instructions (8 chains of that pedigree 12.7 ms a sweep, rolled 6.4).
// Measured, a sweep (the fastest of 32, 16 and 8 lanes before): 400 members,
// 10,000 SNPs, one chain 4.2 -> 2.2 ms, 8 chains 30.1 -> 5.7, 32 chains 123 ->
// 22.3; 120 members, 2,000 SNPs, one chain 0.86 -> 0.59, 10 chains 2.1 -> 0.71;
// 30 members, 200 SNPs, one chain 0.23 -> 0.17.
// ---------------------------------------------------------------------------
constexpr int kQuadTasks = 8;                       // tasks per warp
constexpr int kQuadWarps = 8;                       // most warps per block
constexpr size_t kQuadSharedArena = 20 * 1024;      // most shared bytes per warp with the rfunctions in them

__host__ __device__ __forceinline__ size_t quad_cols_at(const ProblemDev& P) { return al16((size_t)P.N * kQuadTasks); }
__host__ __device__ __forceinline__ size_t quad_off_at(const ProblemDev& P) {
    return quad_cols_at(P) + al16((size_t)2 * P.W * 4 * kQuadTasks);
}
template <typename T>
__host__ __device__ __forceinline__ size_t quad_tab_at(const ProblemDev& P) {
    return quad_off_at(P) + al16((size_t)2 * P.K * kQuadTasks);
}
// [32] transmission values and [16] priors per task, then the rfunctions
template <typename T>
__host__ __device__ __forceinline__ size_t quad_arena_at(const ProblemDev& P) {
    return quad_tab_at<T>(P) + 48 * sizeof(T) * kQuadTasks;
}
template <typename T>
__host__ __device__ __forceinline__ size_t quad_arena_bytes(const ProblemDev& P) {
    return al16((size_t)(P.ls_arena | 1) * sizeof(T) * kQuadTasks);
}
template <typename T>
__host__ __device__ __forceinline__ bool quad_arena_shared(const ProblemDev& P) {
    return quad_arena_at<T>(P) + quad_arena_bytes<T>(P) <= kQuadSharedArena;
}
template <typename T>
__host__ __device__ __forceinline__ size_t quad_warp_bytes(const ProblemDev& P) {
    return quad_arena_at<T>(P) + (quad_arena_shared<T>(P) ? quad_arena_bytes<T>(P) : 0);
}
// shared bytes of a block's copy of the operations (0: they stay in global memory)
__host__ __device__ __forceinline__ size_t quad_prog_bytes(const ProblemDev& P) {
    return P.quad_prog_words <= 8 * 1024 ? al16((size_t)P.quad_prog_words * 4) : 0;
}
// bits 2 r and 2 r + 1 of entry m: the r-th state that mask m allows
__device__ __forceinline__ unsigned quad_states(int m) {
    unsigned s = 0;
    int r = 0;
    for (int v = 0; v < 4; ++v)
        if ((m >> v) & 1) {
            s |= (unsigned)v << (2 * r);
            ++r;
        }
    return s;
}

// One operation of P.quad_prog: word 0 its sizes (below), word 1 the peel node,
// then the cutset members, two to a word; per previous rfunction its op and
// cutset size, then its keys' positions (four bits each; the peel node's is c);
// per child (for a child peel, the peel node itself) its first meiosis, and for
// a parent peel its position, the other parent's and whether the peel node is
// its mother.
struct QuadOp {
    const uint32_t *cuts, *prevs, *kids;
    int type, c, n_prev, n_kid, mpos, fpos, peel;
    __device__ __forceinline__ explicit QuadOp(const uint32_t* w) {
        const uint32_t h = w[0];
        peel = (int)w[1];
        c = h & 15;
        type = (h >> 4) & 7;
        n_prev = (h >> 7) & 31;
        n_kid = (h >> 12) & 31;
        mpos = (h >> 17) & 15;
        fpos = (h >> 21) & 15;
        cuts = w + 2;
        prevs = cuts + ((c + 1) >> 1);
        kids = prevs + 2 * n_prev;
    }
    __device__ __forceinline__ int cut(int q) const { return (int)(cuts[q >> 1] >> (16 * (q & 1))) & 0xffff; }
};

// What a task's lanes share: byte arrays [members][8], words [2 W][8], and so on.
template <typename T>
struct Quad {
    const ProblemDev& P;
    const uint32_t* prog;   // the operations (QuadOp)
    const uint16_t* at;     // [K] each one's first word
    const uint16_t* parent; // [2 Nnf] the parent of each meiosis
    uint8_t* geno;     // bits 0-1 genotype code, bits 2-3 the sampled state, bits 4-7 allowed states
    uint32_t* cols;    // the left neighbour's words, then the right one's
    uint16_t* off;     // each op's first cell
    T* tab;            // [indicators of the two neighbours][parent's state][allele]
    T* pri;            // [genotype code][state]
    T* A;              // this task's rfunctions
    int task, v;
    __device__ __forceinline__ int mem(int i) const { return geno[i * kQuadTasks + task]; }
    __device__ __forceinline__ int bits2(int b) const {   // meiosis b's indicators: left, right << 1
        const int w = b >> 5;
        return (int)((cols[w * kQuadTasks + task] >> (b & 31)) & 1u) |
               (int)((cols[(P.W + w) * kQuadTasks + task] >> (b & 31)) & 1u) << 1;
    }
    // the probability that a parent in state st passes on `allele` (ls_dist_one's d[2 st + allele])
    __device__ __forceinline__ T dist(int ind, int st, int allele) const {
        return tab[(8 * ind + 2 * st + allele) * kQuadTasks + task];
    }
    // the op's children's indicators, four bits each in order
    __device__ __forceinline__ unsigned long long children(const QuadOp& op) const {
        unsigned long long x = 0;
#pragma unroll 1
        for (int c = 0; c < op.n_kid; ++c) {
            const int b = (int)op.kids[c] & 0xffff;
            x |= (unsigned long long)(bits2(b) | bits2(b + 1) << 2) << (4 * c);
        }
        return x;
    }
    // ls_term of NC cells for this lane's state (tv its prior, vbit whether it is
    // allowed): ext and rk hold each cell's states and ranks, two bits a position.
    // Every index read is inside its rfunction, whatever the cell.
    template <int NC>
    __device__ __forceinline__ void term(const QuadOp& op, unsigned long long ch, const int (&ext)[NC],
                                         const int (&rk)[NC], int bits, bool vbit, T tv, T (&t)[NC]) const {
        using Ar = Ls<T>;
#pragma unroll
        for (int n = 0; n < NC; ++n) t[n] = tv;
        if (op.type == CHILD) {
            const int m = 8 * ((int)ch & 3) + mat_allele(v), p = 8 * ((int)(ch >> 2) & 3) + pat_allele(v);
#pragma unroll
            for (int n = 0; n < NC; ++n)
                t[n] = Ar::mul(t[n], Ar::mul(tab[(m + 2 * digit(ext[n], op.mpos)) * kQuadTasks + task],
                                             tab[(p + 2 * digit(ext[n], op.fpos)) * kQuadTasks + task]));
        }
#pragma unroll 1
        for (int j = 0; j < op.n_prev; ++j) {
            const uint32_t w = op.prevs[2 * j];
            uint32_t keys = op.prevs[2 * j + 1];
            int idx[NC], sh = 0;
#pragma unroll
            for (int n = 0; n < NC; ++n) idx[n] = 0;
            bool good = true;
#pragma unroll 1
            for (int q = (int)w >> 16; q > 0; --q, keys >>= 4) {
                const int pos = keys & 15, p2 = 2 * pos;
#pragma unroll
                for (int n = 0; n < NC; ++n) idx[n] |= ((rk[n] >> p2) & 3) << sh;
                sh += (bits >> p2) & 3;
                good &= vbit || pos != op.c;
            }
            const T* a = A + off[(w & 0xffff) * kQuadTasks + task];
#pragma unroll
            for (int n = 0; n < NC; ++n) t[n] = Ar::mul(t[n], good ? a[idx[n]] : T(0));
        }
        if (op.type == PARENT) {
            T cp[NC];
#pragma unroll
            for (int n = 0; n < NC; ++n) cp[n] = T(1);
#pragma unroll 1
            for (int c = 0; c < op.n_kid; ++c) {
                const uint32_t w = op.kids[c];
                const int ind = (int)(ch >> (4 * c)), kp = 2 * ((w >> 16) & 15), op2 = 2 * ((w >> 20) & 15);
                const bool mum = (w >> 24) & 1;
#pragma unroll
                for (int n = 0; n < NC; ++n) {
                    const int kt = (ext[n] >> kp) & 3, other = (ext[n] >> op2) & 3;
                    cp[n] = Ar::mul(cp[n], Ar::mul(dist(ind & 3, mum ? v : other, mat_allele(kt)),
                                                   dist((ind >> 2) & 3, mum ? other : v, pat_allele(kt))));
                }
            }
#pragma unroll
            for (int n = 0; n < NC; ++n) t[n] = Ar::mul(t[n], cp[n]);
        }
    }
};

// What the forward pass knows of an op at a task.
struct QuadCells {
    unsigned long long perm;   // each member's allowed states by rank (8 bits a member)
    int bits, three;           // rank bits (2 bits a position, the peel node's last); members with three states
    int vext, vrank;           // this lane's state and rank in the peel node's position
    bool vbit;                 // the state is allowed
};

// The totals of cells first .. first + NC - 1 of an op, on all four lanes of each task.
template <typename T, int NC>
__device__ __forceinline__ void quad_cells(const Quad<T>& Q, const QuadOp& op, const QuadCells& x,
                                           unsigned long long ch, int first, int ncell, T tv, int q0, T (&total)[NC]) {
    using Ar = Ls<T>;
    int ext[NC], rk[NC], rem[NC];
    bool ok[NC];
#pragma unroll
    for (int n = 0; n < NC; ++n) {
        ext[n] = x.vext;
        rk[n] = x.vrank;
        rem[n] = first + n;
        ok[n] = first + n < ncell;
    }
#pragma unroll 1
    for (int q = 0; q < op.c; ++q) {
        const int b = (x.bits >> (2 * q)) & 3, mask = (1 << b) - 1;
        const unsigned pq = (unsigned)(x.perm >> (8 * q)) & 255u;
        const bool three = (x.three >> q) & 1;
#pragma unroll
        for (int n = 0; n < NC; ++n) {
            const int r = rem[n] & mask;
            rem[n] >>= b;
            ok[n] &= !(three && r == 3);
            ext[n] |= (int)((pq >> (2 * r)) & 3u) << (2 * q);
            rk[n] |= r << (2 * q);
        }
    }
    T t[NC];
    Q.term(op, ch, ext, rk, x.bits, x.vbit, tv, t);
#pragma unroll
    for (int n = 0; n < NC; ++n) {
        const T tn = ok[n] ? t[n] : T(0);
        const T t0 = __shfl_sync(FULLMASK, tn, q0), t1 = __shfl_sync(FULLMASK, tn, q0 + 1);
        const T t2 = __shfl_sync(FULLMASK, tn, q0 + 2), t3 = __shfl_sync(FULLMASK, tn, q0 + 3);
        total[n] = Ar::add(Ar::add(Ar::add(Ar::add(T(0), t0), t1), t2), t3);
    }
}

// ls_locus by four lanes; `live` false: a lane group without a task, which
// goes along with the warp on a task of another's inputs and writes nothing.
template <typename T>
__device__ int quad_locus(Quad<T>& Q, const unsigned* states, uint32_t* colC, int cr, int chain, int l, bool hasL,
                          bool hasR, bool live, const Draws& draws, int64_t unit, int64_t base, int* status,
                          double* logroot) {
    using Ar = Ls<T>;
    constexpr bool kRescale = sizeof(T) == 4;
    const ProblemDev& P = Q.P;
    const int lane = threadIdx.x & 31, q0 = lane & ~3, v = Q.v, task = Q.task;
    // the locus's inputs: genotypes, neighbours' columns, transmission values, priors
    {
        const uint8_t* gsrc = P.geno + (size_t)l * P.N;
#pragma unroll 8
        for (int i = v; i < P.N; i += 4) Q.geno[i * kQuadTasks + task] = gsrc[i] & 0xf3;
        for (int w = v; w < P.W; w += 4) {
            Q.cols[w * kQuadTasks + task] = hasL ? colC[w - P.W] : 0u;
            Q.cols[(P.W + w) * kQuadTasks + task] = hasR ? colC[w + P.W] : 0u;
        }
    }
    T th = T(1), an = T(1), th2 = T(1), an2 = T(1);
    if constexpr (sizeof(T) == 4) {
        const float* tf = P.c_theta_f + (size_t)chain * (P.M - 1);
        if (hasL) { th2 = tf[l - 1]; an2 = 1.f - th2; }
        if (hasR) { th = tf[l]; an = 1.f - th; }
    } else {
        const double* td = P.c_theta + (size_t)chain * (P.M - 1);
        if (hasL) { th2 = td[l - 1]; an2 = DSUB(1.0, td[l - 1]); }
        if (hasR) { th = td[l]; an = DSUB(1.0, td[l]); }
    }
    T pick0;   // lane v: the probability of indicator 0 below a homozygous parent, neighbours' indicators v
    {
        T t0 = T(0.5), t1 = T(0.5), p0 = T(1), p1 = T(1);
        if (hasL) {
            const bool cross = v & 1;
            t0 = Ar::mul(t0, cross ? th2 : an2);
            t1 = Ar::mul(t1, cross ? an2 : th2);
            p0 = Ar::mul(p0, cross ? th2 : an2);
            p1 = Ar::mul(p1, cross ? an2 : th2);
        }
        if (hasR) {
            const bool cross = v >> 1;
            t0 = Ar::mul(t0, cross ? th : an);
            t1 = Ar::mul(t1, cross ? an : th);
            p0 = Ar::mul(p0, cross ? th : an);
            p1 = Ar::mul(p1, cross ? an : th);
        }
        const T total = Ar::add(t0, t1), uau = Ar::div(t1, total), uua = Ar::div(t0, total);
        const T d[8] = {T(1), T(0), T(0), T(1), uau, Ar::sub(T(1), uau), uua, Ar::sub(T(1), uua)};   // UU, AA, AU, UA
        for (int i = 0; i < 8; ++i) Q.tab[(8 * v + i) * kQuadTasks + task] = d[i];
        pick0 = Ar::div(p0, Ar::add(p0, p1));
        for (int i = v; i < 16; i += 4) {
            if constexpr (sizeof(T) == 4) Q.pri[i * kQuadTasks + task] = (T)P.prior_f[(size_t)l * 16 + i];
            else Q.pri[i * kQuadTasks + task] = (T)P.prior[(size_t)l * 16 + i];
        }
    }
    __syncwarp();
    int scale = 0, run = 0;
    T root = T(0);
    // forward peel over the valid cells of every rfunction
#pragma unroll 1
    for (int k = 0; k < P.K; ++k) {
        const QuadOp op(Q.prog + Q.at[k]);
        QuadCells x;
        x.perm = 0;
        x.bits = x.three = 0;
        int B = 0;
#pragma unroll 1
        for (int q = 0; q < op.c; ++q) {
            const int m = Q.mem(op.cut(q)) >> 4, b = rank_bits(m);
            x.perm |= (unsigned long long)states[m] << (8 * q);
            x.bits |= b << (2 * q);
            B += b;
            x.three |= (__popc(m) == 3) << q;
        }
        const int gp = Q.mem(op.peel), mp = gp >> 4;
        const int ncell = 1 << B;
        const T tv = Q.pri[(4 * (gp & 3) + v) * kQuadTasks + task];
        x.vbit = (mp >> v) & 1;
        x.bits |= rank_bits(mp) << (2 * op.c);
        x.vrank = x.vbit ? state_rank(mp, v) << (2 * op.c) : 0;
        x.vext = v << (2 * op.c);
        const unsigned long long ch = Q.children(op);
        const int most = __reduce_max_sync(FULLMASK, B);   // the warp's widest task
        const int ob = run;
        // all four lanes have each total; up to four cells wait in registers (cell v in lane v) for the scaling
        T mx = T(0), mine = T(0);
        if (most < 2) {
            T t[2];
            quad_cells<T, 2>(Q, op, x, ch, 0, ncell, tv, q0, t);
            mx = t[0] > mx ? t[0] : mx;
            mx = t[1] > mx ? t[1] : mx;
            mine = v == 0 ? t[0] : t[1];
        } else {
#pragma unroll 1
            for (int cell = 0; cell < 1 << most; cell += 4) {
                T t[4];
                quad_cells<T, 4>(Q, op, x, ch, cell, ncell, tv, q0, t);
#pragma unroll
                for (int n = 0; n < 4; ++n) mx = t[n] > mx ? t[n] : mx;
                const T m = v == 0 ? t[0] : v == 1 ? t[1] : v == 2 ? t[2] : t[3];
                if (cell == 0) mine = m;
                if (ncell > 4 && cell < ncell) Q.A[ob + cell + v] = m;
            }
        }
        if (k == P.K - 1) root = __shfl_sync(FULLMASK, mine, q0);
        if (kRescale) {
            float f = 1.f;
            if (mx > T(0)) {
                const int ex = ilogbf((float)mx);
                scale += ex;
                f = scalbnf(1.0f, -ex);
                if (k == P.K - 1) root = (T)((float)root * f);
            }
            if (ncell > 4) {
                if (mx > T(0))
#pragma unroll 1
                    for (int cell = v; cell < ncell; cell += 4) Q.A[ob + cell] = (T)((float)Q.A[ob + cell] * f);
            } else if (v < ncell) {
                Q.A[ob + v] = mx > T(0) ? (T)((float)mine * f) : mine;
            }
        } else if (ncell <= 4 && v < ncell) {
            Q.A[ob + v] = mine;
        }
        if (v == 0) Q.off[k * kQuadTasks + task] = (uint16_t)ob;
        run += ncell;
        __syncwarp();
    }
    bool fail = false;
    if (root == T(0)) {
        if (live && v == 0) set_status(status, ST_ZERO_LIK);
        fail = true;
    }
    if (v == 0 && logroot && !fail) *logroot = log((double)root) + (double)scale * 0.69314718055994530942;
    // backward sampling of ordered genotypes: lane v draws the uniforms of every fourth operation
    T draw = T(0);
#pragma unroll 1
    for (int j = 0; j < P.K; ++j) {
        const int k = P.K - 1 - j;
        const QuadOp op(Q.prog + Q.at[k]);
        if ((j & 3) == 0 && j + v < P.K && live && !fail) draw = draw_for<T>(draws, cr, chain, unit, base + j + v);
        int ext[1] = {v << (2 * op.c)}, rk[1] = {0}, bits = 0;
        bool ok = true;
#pragma unroll 1
        for (int q = 0; q < op.c; ++q) {
            const int g = Q.mem(op.cut(q)), a = (g >> 2) & 3, m = g >> 4;
            const bool in = (m >> a) & 1;
            ok &= in;
            ext[0] |= a << (2 * q);
            rk[0] |= in ? state_rank(m, a) << (2 * q) : 0;
            bits |= rank_bits(m) << (2 * q);
        }
        const int gp = Q.mem(op.peel), mp = gp >> 4;
        const T tv = Q.pri[(4 * (gp & 3) + v) * kQuadTasks + task];
        const bool vbit = (mp >> v) & 1;
        rk[0] |= vbit ? state_rank(mp, v) << (2 * op.c) : 0;
        bits |= rank_bits(mp) << (2 * op.c);
        T pt[1];
        Q.term(op, Q.children(op), ext, rk, bits, vbit, tv, pt);
        const T pv = ok ? pt[0] : T(0);
        const T r = __shfl_sync(FULLMASK, draw, q0 + (j & 3));
        const T p0 = __shfl_sync(FULLMASK, pv, q0), p1 = __shfl_sync(FULLMASK, pv, q0 + 1);
        const T p2 = __shfl_sync(FULLMASK, pv, q0 + 2), p3 = __shfl_sync(FULLMASK, pv, q0 + 3);
        const T tot = Ar::add(Ar::add(Ar::add(p0, p1), p2), p3);
        // lane v divides its own term; the four quotients are added up in order
        const T d = tot != T(0) ? Ar::div(pv, tot) : pv;
        const T d0 = __shfl_sync(FULLMASK, d, q0), d1 = __shfl_sync(FULLMASK, d, q0 + 1);
        const T d2 = __shfl_sync(FULLMASK, d, q0 + 2), d3 = __shfl_sync(FULLMASK, d, q0 + 3);
        const T a0 = Ar::add(T(0), d0), a1 = Ar::add(a0, d1), a2 = Ar::add(a1, d2), a3 = Ar::add(a2, d3);
        int pick;
        if (r < a0) pick = 0;
        else if (r < a1) pick = 1;
        else if (r < a2) pick = 2;
        else if (r < a3) pick = 3;
        else pick = d3 != T(0) ? 3 : d2 != T(0) ? 2 : d1 != T(0) ? 1 : 0;
        if (v == 0) Q.geno[op.peel * kQuadTasks + task] = (uint8_t)((gp & 0xf3) | pick << 2);
        __syncwarp();
    }
    // meiosis indicators in person order, maternal first, four at a time; a
    // draw is consumed only below a homozygous parent
    int64_t cursor = base + P.K;
    const int nb = 2 * P.Nnf;
#pragma unroll 1
    for (int w = 0; w < P.W; ++w) {
        uint32_t word = 0;
#pragma unroll 1
        for (int h = 0; h < 32; h += 4) {
            const int b = 32 * w + h + v;
            if (32 * w + h >= nb) break;   // the same for the whole warp
            int mi = 0, need = 0, ind = 0;
            if (b < nb) {
                const int i = P.F + (b >> 1), par = b & 1;
                const int tr = (Q.mem(i) >> 2) & 3;
                const int ptr = (Q.mem(Q.parent[b]) >> 2) & 3;
                const int allele = par == 0 ? ((tr == UU || tr == UA) ? 0 : 1) : ((tr == UU || tr == AU) ? 0 : 1);
                if (ptr == UA || ptr == AU) mi = (allele == 0) == (ptr == UA) ? 0 : 1;
                else {
                    need = 1;
                    ind = Q.bits2(b);
                }
            }
            const unsigned nmask = (__ballot_sync(FULLMASK, need) >> q0) & 15u;
            const T p = __shfl_sync(FULLMASK, pick0, q0 + ind);
            if (need && live && !fail) {
                const T r = draw_for<T>(draws, cr, chain, unit, cursor + __popc(nmask & ((1u << v) - 1u)));
                mi = r < p ? 0 : 1;
            }
            cursor += __popc(nmask);
            word |= ((__ballot_sync(FULLMASK, mi != 0) >> q0) & 15u) << h;
        }
        if (v == 0 && live && !fail) colC[w] = word;   // bits past 2 Nnf stay zero
    }
    __syncwarp();
    return fail ? -1 : (int)(cursor - base);
}

// A warp's Quad over its shared memory; arena: its part of the global one.
template <typename T>
__device__ __forceinline__ Quad<T> quad_bind(const ProblemDev& P, const uint32_t* prog, unsigned char* wsm, T* arena) {
    const int lane = threadIdx.x & 31, task = lane >> 2;
    T* rf = quad_arena_shared<T>(P) ? (T*)(wsm + quad_arena_at<T>(P)) : arena;
    T* tab = (T*)(wsm + quad_tab_at<T>(P));
    const uint16_t* at = (const uint16_t*)(prog + P.quad_prog_words - P.quad_tail_words);
    return Quad<T>{P, prog, at, at + P.K, wsm, (uint32_t*)(wsm + quad_cols_at(P)), (uint16_t*)(wsm + quad_off_at(P)), tab,
                   tab + 32 * kQuadTasks, rf + (size_t)task * (P.ls_arena | 1), task, lane & 3};
}

// The block's copies of the operations and of quad_states.
__device__ __forceinline__ const uint32_t* quad_stage(const ProblemDev& P, unsigned char* smem, unsigned* states) {
    const uint32_t* prog = P.quad_prog;
    if (quad_prog_bytes(P)) {
        uint32_t* sp = (uint32_t*)smem;
        for (int i = threadIdx.x; i < P.quad_prog_words; i += blockDim.x) sp[i] = prog[i];
        prog = sp;
    }
    if (threadIdx.x < 16) states[threadIdx.x] = quad_states(threadIdx.x);
    __syncthreads();
    return prog;
}

// This launch's warp w of chains from `first` on: its part of the global arena
// (null: the rfunctions are in shared memory).
template <typename T>
__device__ __forceinline__ T* quad_arena_slice(const ProblemDev& P, int first, int64_t w) {
    if (quad_arena_shared<T>(P)) return nullptr;
    return (T*)P.quad_arena + ((size_t)first * P.quad_warps + w) * (quad_arena_bytes<T>(P) / sizeof(T));
}

template <typename T>
__global__ void __launch_bounds__(32 * kQuadWarps) lsampler_quad_kernel(ProblemDev P, uint32_t* dg, int first,
                                                                        int nchain, const int32_t* loci, int nloci,
                                                                        Draws draws, const uint8_t* sel, int want,
                                                                        int* status) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ unsigned states[16];
    const uint32_t* prog = quad_stage(P, smem, states);
    const int warp = threadIdx.x >> 5;
    const int wpb = blockDim.x >> 5;
    const int64_t gw = (int64_t)blockIdx.x * wpb + warp, nw = (int64_t)gridDim.x * wpb;
    Quad<T> Q = quad_bind<T>(P, prog, smem + quad_prog_bytes(P) + warp * quad_warp_bytes<T>(P),
                             quad_arena_slice<T>(P, first, gw));
    const int64_t ntask = (int64_t)nchain * nloci;
    for (int64_t g = gw; g * kQuadTasks < ntask; g += nw) {
        const int64_t t = min(g * kQuadTasks + Q.task, ntask - 1);
        const int cr = (int)(t / nloci), l = loci[t % nloci];
        const bool live = g * kQuadTasks + Q.task < ntask && !(sel && sel[cr] != want);
        if (!__any_sync(FULLMASK, live)) continue;
        uint32_t* colC = dg + ((size_t)(first + cr) * P.M + l) * P.W;
        quad_locus<T>(Q, states, colC, cr, first + cr, l, l > 0, l < P.M - 1, live, draws, l, 0, status, nullptr);
    }
}

// Sequential imputation (LocusSampler::start_from, locus_sampler2.cc:214-241),
// one warp per chain: the start locus with neither neighbour, then leftwards
// with the right neighbour only, then rightwards with the left neighbour only;
// draws are consumed in one sequence (unit `unit`), the weight is the sum of
// log(root) over the steps (-DBL_MAX when a locus has likelihood 0).
// npass independent passes of every chain run as separate warps: pass q of
// chain cr writes the graph set at dg + q * pass_stride, draws from the
// Philox stream of pass draws.iter + q, starts at starts[q * nchain + cr] and
// leaves its weight at weights[q * nchain + cr].
template <typename T>
__global__ void __launch_bounds__(128) si_kernel(ProblemDev P, uint32_t* dg, int first, int nchain,
                                                 const int32_t* starts, Draws draws, int64_t unit, double* weights,
                                                 int* status, int npass, int64_t pass_stride) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int wpb = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const OpDev* ops;
    const int32_t* opd;
    ls_stage_tables(P, smem, ops, opd);
    __syncthreads();
    unsigned char* wsmem = smem + ls_tables_bytes(P) + (size_t)warp * ls_warp_bytes<T>(P);
    T* spill = ls_spill_slice<T>(P, first, (int64_t)blockIdx.x * wpb + warp);
    if (P.ls_spill_cells > 0 && !spill) {
        if (lane == 0) set_status(status, ST_ILLEGAL_DG);
        return;
    }
    for (int t = blockIdx.x * wpb + warp; t < nchain * npass; t += gridDim.x * wpb) {
        const int cr = t % nchain, q = t / nchain;
        const int chain = first + cr, M = P.M, start = starts[t];
        uint32_t* dgq = dg + (size_t)q * pass_stride;
        Draws dq = draws;
        dq.iter = draws.iter + (uint64_t)q;
        int64_t base = 0;
        double w = 0.0;
        bool ok = true;
        for (int v = 0; v < M && ok; ++v) {
            const int l = v == 0 ? start : (v <= start ? start - v : v);
            const bool hasL = v > start && l > 0;
            const bool hasR = v > 0 && v <= start && l < M - 1;
            double lr = 0.0;
            const int used = ls_locus<T, 32>(P, ops, opd, dgq, cr, chain, l, hasL, hasR, dq, unit, base, wsmem,
                                             spill, lane, status, &lr);
            if (used < 0) {
                ok = false;
                break;
            }
            base += used;
            w += __shfl_sync(FULLMASK, lr, 0);
        }
        if (lane == 0) weights[t] = ok ? w : -DBL_MAX;
        __syncwarp();
    }
}

// The same by four lanes per pass (quad_locus), eight passes a warp; a pass
// that met a locus of likelihood 0 goes along with its warp and writes nothing
// more.  1,000 passes of 301 loci of the 120-member pedigree: 133 -> 74 ms, bound
// by one pass's chain of loci (125 warps on the whole GPU).
template <typename T>
__global__ void __launch_bounds__(32 * kQuadWarps) si_quad_kernel(ProblemDev P, uint32_t* dg, int first, int nchain,
                                                                  const int32_t* starts, Draws draws, int64_t unit,
                                                                  double* weights, int* status, int npass,
                                                                  int64_t pass_stride) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ unsigned states[16];
    const uint32_t* prog = quad_stage(P, smem, states);
    const int warp = threadIdx.x >> 5, wpb = blockDim.x >> 5, M = P.M;
    const int64_t gw = (int64_t)blockIdx.x * wpb + warp, nw = (int64_t)gridDim.x * wpb;
    Quad<T> Q = quad_bind<T>(P, prog, smem + quad_prog_bytes(P) + warp * quad_warp_bytes<T>(P),
                             quad_arena_slice<T>(P, 0, gw));
    const int64_t ntask = (int64_t)nchain * npass;
    for (int64_t g = gw; g * kQuadTasks < ntask; g += nw) {
        const int64_t t = min(g * kQuadTasks + Q.task, ntask - 1);
        const int cr = (int)(t % nchain), q = (int)(t / nchain), chain = first + cr, start = starts[t];
        const bool mine = g * kQuadTasks + Q.task < ntask;
        uint32_t* graph = dg + (size_t)q * pass_stride + (size_t)chain * M * P.W;
        Draws dq = draws;
        dq.iter = draws.iter + (uint64_t)q;
        int64_t base = 0;
        double w = 0.0;
        bool ok = mine;
        for (int k = 0; k < M && __any_sync(FULLMASK, ok); ++k) {
            const int l = k == 0 ? start : (k <= start ? start - k : k);
            const bool hasL = k > start && l > 0;
            const bool hasR = k > 0 && k <= start && l < M - 1;
            double lr = 0.0;
            const int used = quad_locus<T>(Q, states, graph + (size_t)l * P.W, cr, chain, l, hasL, hasR, ok, dq, unit,
                                           base, status, &lr);
            if (used < 0) ok = false;
            base += used;
            w += lr;
        }
        if (mine && Q.v == 0) weights[t] = ok ? w : -DBL_MAX;
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// Founder allele graph likelihood (FounderAlleleGraph4::likelihood,
// founder_allele_graph4.cc:34-442), one thread per (chain, locus).  The
// per-thread state lives in shared memory as structure-of-arrays over the
// block's threads (element i of thread t at [i * S + t]) so a warp's accesses
// to the same field hit 32 consecutive banks.
// ---------------------------------------------------------------------------
// Probability arithmetic of the founder-allele graph.  ProbExact is the
// reference's FP64 (bit-exact); ProbLog2 works on log2 values in FP32 for the
// fast sampler mode, where only the normalised pair of likelihoods is used:
// products become sums and a zero likelihood is -inf.
struct ProbExact {
    using T = double;
    static __device__ __forceinline__ T zero() { return 0.0; }
    static __device__ __forceinline__ T one() { return 1.0; }
    static __device__ __forceinline__ T mul(T a, T b) { return DMUL(a, b); }
    static __device__ __forceinline__ T add(T a, T b) { return DADD(a, b); }
    static __device__ __forceinline__ T from(double x) { return x; }
    static __device__ __forceinline__ bool is_zero(T a) { return a == 0.0; }
};
struct ProbLog2 {
    using T = float;
    static __device__ __forceinline__ T zero() { return -INFINITY; }
    static __device__ __forceinline__ T one() { return 0.f; }
    static __device__ __forceinline__ T mul(T a, T b) { return a + b; }
    static __device__ __forceinline__ T add(T a, T b) {
        if (a == -INFINITY) return b;
        if (b == -INFINITY) return a;
        const T m = fmaxf(a, b), d = fminf(a, b) - m;
        return m + log2f(1.f + exp2f(d));
    }
    static __device__ __forceinline__ T from(double x) { return x > 0.0 ? log2f((float)x) : -INFINITY; }
    static __device__ __forceinline__ bool is_zero(T a) { return a == -INFINITY; }
};

// Founder-allele groups are kept in a union-find whose links carry a swap
// parity: the reference relabels every member of the absorbed component and
// swaps its two allele assignments when merging (combine_components,
// founder_allele_graph4.cc:491-541); here the absorbed component's root is
// linked under the survivor's root with parity = swap, and a member's
// assignment in its group's frame is its stored pair read through the
// accumulated parity.  Group ids, the fixed/active flags and every FP64
// product follow the reference's order exactly, so the likelihood is the
// same double.  IX is uint8_t when 2F <= 255 (founder-allele and group ids
// fit a byte), else uint16_t.
template <typename IX, typename PT>
struct Fag {
    PT* pr0;          // [2F][S] prob[0][group]
    PT* pr1;          // [2F][S]
    IX* edge;         // [2N][S] founder allele of each person's maternal/paternal allele
    IX* up;           // [2F][S] union-find parent of a founder allele
    uint8_t* fl;      // [2F][S] bit0 parity to parent, bit1 in a group, bits 2-3 a0, bits 4-5 a1
    int8_t* fx;       // [2F][S] group fixed: -1 unfixed, 0/1 fixed, 2 inactive
    IX* root;         // [2F][S] root founder allele of a group id
    IX* gid;          // [2F][S] group id of a root founder allele
    int S, t;
    __device__ __forceinline__ PT& p0(int g) { return pr0[g * S + t]; }
    __device__ __forceinline__ PT& p1(int g) { return pr1[g * S + t]; }
    __device__ __forceinline__ PT& pw(int w, int g) { return w == 0 ? p0(g) : p1(g); }
    __device__ __forceinline__ IX& e(int i) { return edge[i * S + t]; }
};

__host__ __device__ inline size_t fag_per_thread(int N, int F, int fast) {
    const size_t ix = (2 * F <= 255) ? 1 : 2;
    const size_t pb = fast ? 4 : 8;
    return (size_t)2 * F * 2 * pb + (size_t)2 * N * ix + (size_t)2 * F * (3 * ix + 2);
}

// Shared bytes of a block of S threads: the FAG arrays plus the staged
// person tables (order, mother, father as int16 and typed as uint8).
__host__ __device__ inline size_t fag_block_bytes(int N, int F, int S, int fast) {
    size_t tables = ((size_t)N * 7 + 15) & ~(size_t)15;
    return ((fag_per_thread(N, F, fast) * S + 15) & ~(size_t)15) + tables;
}

template <typename IX, typename PT>
__device__ __forceinline__ Fag<IX, PT> fag_bind(unsigned char* p, int N, int F, int S, int t) {
    Fag<IX, PT> s;
    s.S = S;
    s.t = t;
    s.pr0 = (PT*)p;
    s.pr1 = s.pr0 + (size_t)2 * F * S;
    s.edge = (IX*)(s.pr1 + (size_t)2 * F * S);
    s.up = s.edge + (size_t)2 * N * S;
    s.root = s.up + (size_t)2 * F * S;
    s.gid = s.root + (size_t)2 * F * S;
    s.fl = (uint8_t*)(s.gid + (size_t)2 * F * S);
    s.fx = (int8_t*)(s.fl + (size_t)2 * F * S);
    return s;
}

__device__ __forceinline__ int fag_legal(int obs, int x, int y) {
    if (obs == G_HETERO) return x != y;
    if (obs == G_HOMOZ_A) return x == G_HOMOZ_A && y == G_HOMOZ_A;
    return x == G_HOMOZ_B && y == G_HOMOZ_B;
}

__device__ __forceinline__ int fag_other(int obs, int x) {
    if (obs == G_HETERO) return x == G_HOMOZ_A ? G_HOMOZ_B : G_HOMOZ_A;
    if (obs == G_HOMOZ_A) return x == G_HOMOZ_A ? G_HOMOZ_A : G_UNTYPED;
    return x == G_HOMOZ_B ? G_HOMOZ_B : G_UNTYPED;
}

// Root of a founder allele's component and the parity from the allele to it,
// compressing the path.
template <typename FS>
__device__ __forceinline__ int fag_find(FS& s, int fa, int& parity) {
    int r = fa, p = 0;
    while (true) {
        const int u = s.up[r * s.S + s.t];
        if (u == r) break;
        p ^= s.fl[r * s.S + s.t] & 1;
        r = u;
    }
    int x = fa, px = p;
    while (x != r) {
        const int u = s.up[x * s.S + s.t];
        const uint8_t f = s.fl[x * s.S + s.t];
        s.up[x * s.S + s.t] = r;
        s.fl[x * s.S + s.t] = (uint8_t)((f & ~1) | px);
        px ^= f & 1;
        x = u;
    }
    parity = p;
    return r;
}

// A founder allele as the reference sees it: its group id (-1 = none) and its
// two allele assignments in its group's frame.
struct FaView {
    int group, a0, a1;
    __device__ __forceinline__ int a(int w) const { return w ? a1 : a0; }
};

template <typename FS>
__device__ __forceinline__ FaView fag_view(FS& s, int fa) {
    FaView v;
    const uint8_t f = s.fl[fa * s.S + s.t];
    if (!(f & 2)) { v.group = -1; v.a0 = v.a1 = 0; return v; }
    int par;
    const int r = fag_find(s, fa, par);
    const uint8_t g = s.fl[fa * s.S + s.t];
    const int s0 = (g >> 2) & 3, s1 = (g >> 4) & 3;
    v.group = s.gid[r * s.S + s.t];
    v.a0 = par ? s1 : s0;
    v.a1 = par ? s0 : s1;
    return v;
}

// Put founder allele fa in group g with assignment value `val` in slot w (the
// other slot unset, as in the reference), linked straight to the group's root.
template <typename FS>
__device__ __forceinline__ void fag_join(FS& s, int fa, int g, int w, int val) {
    const int r = s.root[g * s.S + s.t];
    s.up[fa * s.S + s.t] = r;
    s.fl[fa * s.S + s.t] = (uint8_t)(2 | (val << (w == 0 ? 2 : 4)));
}

template <typename FS>
__device__ __forceinline__ void fag_join2(FS& s, int fa, int g, int v0, int v1) {
    const int r = s.root[g * s.S + s.t];
    s.up[fa * s.S + s.t] = r;
    s.fl[fa * s.S + s.t] = (uint8_t)(2 | (v0 << 2) | (v1 << 4));
}

template <typename FS>
__device__ __forceinline__ void fag_new_root(FS& s, int fa, int g, int v0, int v1) {
    s.up[fa * s.S + s.t] = fa;
    s.fl[fa * s.S + s.t] = (uint8_t)(2 | (v0 << 2) | (v1 << 4));
    s.root[g * s.S + s.t] = fa;
    s.gid[fa * s.S + s.t] = g;
}

// combine_components(c1, c2, flip) (founder_allele_graph4.cc:491-541)
template <typename PP, typename FS>
__device__ __forceinline__ void fag_combine(FS& s, int c1, int c2, bool flip) {
    const int r1 = s.root[c1 * s.S + s.t], r2 = s.root[c2 * s.S + s.t];
    s.up[r2 * s.S + s.t] = r1;
    s.fl[r2 * s.S + s.t] = (uint8_t)((s.fl[r2 * s.S + s.t] & ~1) | (flip ? 1 : 0));
    if (flip) {
        s.p0(c1) = PP::mul(s.p0(c1), s.p1(c2));
        s.p1(c1) = PP::mul(s.p1(c1), s.p0(c2));
    } else {
        s.p0(c1) = PP::mul(s.p0(c1), s.p0(c2));
        s.p1(c1) = PP::mul(s.p1(c1), s.p1(c2));
    }
    s.fx[c2 * s.S + s.t] = 2;
}

// Edges of the column (FounderAlleleGraph4::reset, founder_allele_graph4.cc:
// 543-569) with one meiosis optionally toggled, which equals flip() and its
// propagation (founder_allele_graph4.cc:571-597).
template <typename FS>
__device__ void fag_edges(int N, int F, const int16_t* order, const int16_t* mo, const int16_t* fa,
                          const uint32_t* col, FS& s, int flip_b) {
    for (int n = 0; n < N; ++n) {
        const int pid = order[n];
        if (pid < F) {
            s.e(2 * pid) = 2 * pid;
            s.e(2 * pid + 1) = 2 * pid + 1;
        } else {
            const int b = 2 * (pid - F);
            const int vm = dgbit(col, b) ^ (flip_b == b);
            const int vp = dgbit(col, b + 1) ^ (flip_b == b + 1);
            s.e(2 * pid) = s.e(2 * mo[pid] + vm);
            s.e(2 * pid + 1) = s.e(2 * fa[pid] + vp);
        }
    }
}

template <typename PP, typename FS>
__device__ typename PP::T fag_like(int N, int F, const uint8_t* typed, const uint8_t* gcol, double minor_d, FS& s) {
    using T = typename PP::T;
    const int nfa = 2 * F;
    const T major = PP::from(DSUB(1.0, minor_d)), minor = PP::from(minor_d);
    for (int i = 0; i < nfa; ++i) s.fl[i * s.S + s.t] = 0;
    int gi = 0;
#define FREQ(g) ((g) == G_HOMOZ_A ? major : minor)
#define FX(g) s.fx[(g) * s.S + s.t]
#define ZERO PP::zero()
    for (int i = 0; i < N; ++i) {
        if (!typed[i]) continue;
        const int g = gcol[i] & 3;
        if (g == G_UNTYPED) continue;
        const int mfa = s.e(2 * i), pfa = s.e(2 * i + 1);
        if (mfa == pfa) {
            if (g == G_HETERO) return ZERO;
            const FaView m = fag_view(s, mfa);
            if (m.group != -1) {
                const int g1 = m.group;
                const int f1 = FX(g1);
                if (f1 != -1) {
                    if (g != m.a(f1)) return ZERO;
                } else {
                    if (m.a(0) == g) { FX(g1) = 0; s.p1(g1) = ZERO; }
                    else if (m.a(1) == g) { FX(g1) = 1; s.p0(g1) = ZERO; }
                    else return ZERO;
                }
            } else {
                fag_new_root(s, mfa, gi, g, 0);
                FX(gi) = 0;
                s.p0(gi) = FREQ(g);
                s.p1(gi) = ZERO;
                ++gi;
            }
            continue;
        }
        const FaView m = fag_view(s, mfa);
        const FaView p = fag_view(s, pfa);
        const int g1 = m.group, g2 = p.group;
        if (g1 != -1) {
            int f1 = FX(g1);
            if (g2 != -1) {
                if (g1 == g2) {
                    if (f1 != -1) {
                        if (!fag_legal(g, m.a(f1), p.a(f1))) return ZERO;
                    } else {
                        const int l0 = fag_legal(g, m.a(0), p.a(0));
                        const int l1 = fag_legal(g, m.a(1), p.a(1));
                        if (l0) {
                            if (!l1) { FX(g1) = 0; s.p1(g1) = ZERO; }
                        } else {
                            if (l1) { FX(g1) = 1; s.p0(g1) = ZERO; }
                            else return ZERO;
                        }
                    }
                } else {
                    int f2 = FX(g2);
                    if (f1 != -1) {
                        if (f2 != -1) {
                            if (!fag_legal(g, m.a(f1), p.a(f2))) return ZERO;
                        } else {
                            const int l0 = fag_legal(g, m.a(f1), p.a(0));
                            const int l1 = fag_legal(g, m.a(f1), p.a(1));
                            if (l0) f2 = 0; else if (l1) f2 = 1; else return ZERO;
                        }
                    } else if (f2 != -1) {
                        const int l0 = fag_legal(g, m.a(0), p.a(f2));
                        const int l1 = fag_legal(g, m.a(1), p.a(f2));
                        if (l0) f1 = 0; else if (l1) f1 = 1; else return ZERO;
                    } else {
                        const int l0 = fag_legal(g, m.a(0), p.a(0));
                        const int l1 = fag_legal(g, m.a(1), p.a(0));
                        const int l2 = fag_legal(g, m.a(0), p.a(1));
                        const int l3 = fag_legal(g, m.a(1), p.a(1));
                        if (!(l0 || l1 || l2 || l3)) return ZERO;
                        if (l0 && !(l1 || l2 || l3)) { f1 = 0; f2 = 0; }
                        else if (l1 && !(l0 || l2 || l3)) { f1 = 1; f2 = 0; }
                        else if (l2 && !(l0 || l1 || l3)) { f1 = 0; f2 = 1; }
                        else if (l3 && !(l0 || l1 || l2)) { f1 = 1; f2 = 1; }
                        else if (l0 && l3 && !(l1 || l2)) { f1 = -1; f2 = -1; }
                        else if (l1 && l2 && !(l0 || l3)) { f1 = -2; f2 = -2; }
                        else { f1 = -1; f2 = -1; }
                    }
                    if (f1 != f2) {
                        FX(g1) = (int8_t)f1;
                        s.pw(1 - f1, g1) = ZERO;
                        s.pw(1 - f2, g2) = ZERO;
                        fag_combine<PP>(s, g1, g2, true);
                    } else if (f1 == -2) {
                        FX(g1) = -1;
                        fag_combine<PP>(s, g1, g2, true);
                    } else {
                        FX(g1) = (int8_t)f1;
                        if (f1 != -1) {
                            s.pw(1 - f1, g1) = ZERO;
                            s.pw(1 - f2, g2) = ZERO;
                        }
                        fag_combine<PP>(s, g1, g2, false);
                    }
                }
            } else {
                if (f1 != -1) {
                    const int t0 = fag_other(g, m.a(f1));
                    if (t0 == G_UNTYPED) return ZERO;
                    fag_join(s, pfa, g1, f1, t0);
                    s.pw(f1, g1) = PP::mul(s.pw(f1, g1), FREQ(t0));
                } else {
                    const int t0 = fag_other(g, m.a(0));
                    const int t1 = fag_other(g, m.a(1));
                    if (t0 != G_UNTYPED) {
                        if (t1 != G_UNTYPED) {
                            fag_join2(s, pfa, g1, t0, t1);
                            s.p0(g1) = PP::mul(s.p0(g1), FREQ(t0));
                            s.p1(g1) = PP::mul(s.p1(g1), FREQ(t1));
                        } else {
                            fag_join(s, pfa, g1, 0, t0);
                            s.p0(g1) = PP::mul(s.p0(g1), FREQ(t0));
                            s.p1(g1) = ZERO;
                            FX(g1) = 0;
                        }
                    } else {
                        if (t1 != G_UNTYPED) {
                            fag_join(s, pfa, g1, 1, t1);
                            s.p1(g1) = PP::mul(s.p1(g1), FREQ(t1));
                            s.p0(g1) = ZERO;
                            FX(g1) = 1;
                        } else return ZERO;
                    }
                }
            }
        } else if (g2 != -1) {
            const int f2 = FX(g2);
            if (f2 != -1) {
                const int t0 = fag_other(g, p.a(f2));
                if (t0 == G_UNTYPED) return ZERO;
                fag_join(s, mfa, g2, f2, t0);
                s.pw(f2, g2) = PP::mul(s.pw(f2, g2), FREQ(t0));
            } else {
                const int t0 = fag_other(g, p.a(0));
                const int t1 = fag_other(g, p.a(1));
                if (t0 != G_UNTYPED) {
                    if (t1 != G_UNTYPED) {
                        fag_join2(s, mfa, g2, t0, t1);
                        s.p0(g2) = PP::mul(s.p0(g2), FREQ(t0));
                        s.p1(g2) = PP::mul(s.p1(g2), FREQ(t1));
                    } else {
                        fag_join(s, mfa, g2, 0, t0);
                        s.p0(g2) = PP::mul(s.p0(g2), FREQ(t0));
                        s.p1(g2) = ZERO;
                        FX(g2) = 0;
                    }
                } else {
                    if (t1 != G_UNTYPED) {
                        fag_join(s, mfa, g2, 1, t1);
                        s.p1(g2) = PP::mul(s.p1(g2), FREQ(t1));
                        s.p0(g2) = ZERO;
                        FX(g2) = 1;
                    } else return ZERO;
                }
            }
        } else {
            if (g == G_HETERO) {
                fag_new_root(s, mfa, gi, G_HOMOZ_A, G_HOMOZ_B);
                fag_join2(s, pfa, gi, G_HOMOZ_B, G_HOMOZ_A);
                s.p0(gi) = PP::mul(major, minor);
                s.p1(gi) = PP::mul(major, minor);
                FX(gi) = -1;
            } else {
                fag_new_root(s, mfa, gi, g, 0);
                fag_join(s, pfa, gi, 0, g);
                s.p0(gi) = PP::mul(FREQ(g), FREQ(g));
                s.p1(gi) = ZERO;
                FX(gi) = 0;
            }
            ++gi;
        }
    }
#undef FREQ
    T ret = PP::one();
    for (int i = 0; i < gi; ++i) {
        const int f = FX(i);
        if (f == 2) continue;
        if (f != -1) ret = PP::mul(ret, s.pw(f, i));
        else ret = PP::mul(ret, PP::add(s.p0(i), s.p1(i)));
    }
#undef FX
#undef ZERO
    return ret;
}

// ---------------------------------------------------------------------------
// M-sampler, split per meiosis step into a grid-wide likelihood kernel and a
// per-chain forward-filter / backward-sample kernel (meiosis_sampler.cc:
// 17-203).  raw64[cr][locus][2] holds the exact likelihoods; raw32 holds the
// same pair divided by its larger member, for the FP32 filter.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void put_raw32(float* r32, int l, double v0, double v1) {
    const double mx = v0 > v1 ? v0 : v1;
    float a = 0.f, b = 0.f;
    if (mx > 0.0) {
        a = (float)(v0 / mx);
        b = (float)(v1 / mx);
    }
    r32[2 * l] = a;
    r32[2 * l + 1] = b;
}

__device__ __forceinline__ void put_raw32_log2(float* r32, int l, float l0, float l1) {
    const float mx = fmaxf(l0, l1);
    float a = 0.f, b = 0.f;
    if (mx != -INFINITY) {
        a = l0 == -INFINITY ? 0.f : exp2f(l0 - mx);
        b = l1 == -INFINITY ? 0.f : exp2f(l1 - mx);
    }
    r32[2 * l] = a;
    r32[2 * l + 1] = b;
}

// step < 0: reset at order[0] (raw[l][cur] = likelihood of the column);
// step >= 0: likelihoods of meiosis order[step] at both values.  With
// ProbExact, raw holds the reference's doubles; with ProbLog2 it holds log2
// likelihoods and raw32 receives each pair divided by its larger member.
template <typename IX, typename PP>
__global__ void __launch_bounds__(128) fag_kernel(ProblemDev P, uint32_t* dg, int first, int nchain,
                                                  const int32_t* order, int64_t ostride, int step,
                                                  const uint8_t* sel, int want, typename PP::T* rawbuf,
                                                  float* raw32, uint8_t* badc, int* status, int fast) {
    using T = typename PP::T;
    extern __shared__ __align__(16) unsigned char smem[];
    const int S = blockDim.x;
    const size_t per = fag_block_bytes(P.N, P.F, S, fast) - (((size_t)P.N * 7 + 15) & ~(size_t)15);
    int16_t* s_order = (int16_t*)(smem + per);
    int16_t* s_mo = s_order + P.N;
    int16_t* s_fa = s_mo + P.N;
    uint8_t* s_typed = (uint8_t*)(s_fa + P.N);
    for (int i = threadIdx.x; i < P.N; i += S) {
        s_order[i] = P.fag_order[i];
        s_mo[i] = P.mother[i];
        s_fa[i] = P.father[i];
        s_typed[i] = P.typed[i];
    }
    __syncthreads();
    Fag<IX, T> fs = fag_bind<IX, T>(smem, P.N, P.F, S, threadIdx.x);
    const int64_t ntask = (int64_t)nchain * P.M;
    const int64_t t = (int64_t)blockIdx.x * S + threadIdx.x;
    if (t >= ntask) return;
    const int cr = (int)(t / P.M);
    const int l = (int)(t % P.M);
    if (sel && sel[cr] != want) return;
    const int chain = first + cr;
    const uint32_t* col = dg + ((size_t)chain * P.M + l) * P.W;
    const int32_t* ord = order + cr * ostride;
    T* raw = rawbuf + (size_t)cr * 2 * P.M;
    const uint8_t* gcol = P.geno + (size_t)l * P.N;
    if (step < 0) {
        fag_edges(P.N, P.F, s_order, s_mo, s_fa, col, fs, -1);
        const T lk = fag_like<PP>(P.N, P.F, s_typed, gcol, P.c_minor[(size_t)chain * P.M + l], fs);
        raw[2 * l + dgbit(col, ord[0])] = lk;
        if (PP::is_zero(lk)) {
            badc[cr] = 1;
            set_status(status, ST_ILLEGAL_DG);
        }
        return;
    }
    const int m = ord[step];
    const int last = ord[step > 0 ? step - 1 : 0];
    const int tb = dgbit(col, m), t2 = dgbit(col, last);
    const T keep = raw[2 * l + t2];
    fag_edges(P.N, P.F, s_order, s_mo, s_fa, col, fs, m);
    const T lk = fag_like<PP>(P.N, P.F, s_typed, gcol, P.c_minor[(size_t)chain * P.M + l], fs);
    raw[2 * l + tb] = keep;
    raw[2 * l + 1 - tb] = lk;
    if (raw32) {
        float* r32 = raw32 + (size_t)cr * 2 * P.M;
        if (sizeof(T) == 8) {
            if (tb == 0) put_raw32(r32, l, (double)keep, (double)lk); else put_raw32(r32, l, (double)lk, (double)keep);
        } else {
            if (tb == 0) put_raw32_log2(r32, l, (float)keep, (float)lk);
            else put_raw32_log2(r32, l, (float)lk, (float)keep);
        }
    }
    if (PP::is_zero(keep) && PP::is_zero(lk)) {
        badc[cr] = 1;
        set_status(status, ST_ILLEGAL_DG);
    }
}

// ---------------------------------------------------------------------------
// Fast-mode founder-allele-graph likelihood, one group of G lanes (a warp, or
// half a warp) per (chain, locus).  The likelihood of the genotypes given the
// column's founder-allele graph (FounderAlleleGraph4::likelihood,
// founder_allele_graph4.cc:34-442) is the product over the connected
// components of the heterozygote edges of the sum, over the component's two
// colourings (allele A = major, B = minor) that satisfy every homozygote's
// fixed alleles, of the product of the founder alleles' frequencies.  Here:
//   1. the founder allele of every person's two alleles is propagated one
//      generation level at a time, the lanes splitting a level's persons;
//   2. the locus's typed persons (a list built at context creation,
//      heterozygotes first) mark their founder alleles used / fixed A /
//      fixed B (shared-memory atomicOr); a heterozygote on one founder allele
//      is a zero likelihood;
//   3. the heterozygote edges join components in a lock-free union-find with
//      parities (pf_find; a compare-and-swap hooks the larger root under the
//      smaller, so every root is its component's smallest allele whatever the
//      interleaving); an edge whose ends already share a root with equal
//      parity closes an odd cycle: zero;
//   4. a component's two colourings weigh (even members) x log2 f(A) + (odd
//      members) x log2 f(B) and the reverse, so each component needs only
//      integer counts, taken at its root; a butterfly sum over the group
//      gives log2 of the likelihood.
// ---------------------------------------------------------------------------
constexpr int kFagWarpsPerBlock = 8;
constexpr int kMswThreads = 1024;
constexpr int kFagRounds = 4;   // rounds of colour propagation along heterozygote edges

__host__ __device__ inline size_t fagw_tables(int N) {
    return (((size_t)N * 8 + 15) & ~(size_t)15) + (((size_t)4 * (N + 1) + 15) & ~(size_t)15);
}
// per lane group: e [2N] founder-allele labels of eb bytes each (1 when the
// 2F labels fit a byte: less shared memory per block, more blocks per SM),
// then Lb / fl / cnt [2F] int each, then the typed-member list [N] u16 on a
// 16-byte boundary in whole 16-byte chunks
__host__ __device__ inline size_t fagw_typ_offset(int N, int F, int eb) {
    return (((((size_t)2 * eb * N + 15) & ~(size_t)15) + (size_t)2 * F * 12) + 15) & ~(size_t)15;
}
__host__ __device__ inline size_t fagw_warp_bytes(int N, int F, int eb) {
    return fagw_typ_offset(N, F, eb) + (size_t)16 * ((N + 7) / 8);
}
// per block: the shared tables and one locus's arrays per lane group (G lanes)
size_t fagw_block_bytes(int N, int F, int G, int eb) {
    return fagw_tables(N) + (size_t)kFagWarpsPerBlock * (32 / G) * fagw_warp_bytes(N, F, eb);
}
// bytes of a founder-allele label: one while the 2F labels fit
__host__ __device__ inline int fagw_label_bytes(int F) { return 2 * F <= 256 ? 1 : 2; }

// 16-byte global -> shared copies that complete asynchronously (cp.async,
// sm_80 and later): both addresses 16-byte aligned.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Root of founder allele x in a forest of 2 * parent + parity entries, and
// x's parity to it.  Parents have smaller indices than their children, so the
// walk ends within x steps.  On the way every other entry is pointed at its
// grandparent with the composed parity (path halving): only entries that are
// not roots are rewritten, always to an ancestor, so the forest stays valid
// whatever other lanes do meanwhile.
__device__ __forceinline__ int pf_find(volatile int* L, int x, int& parity) {
    int p = 0, y = x;
#pragma unroll 1
    for (int it = 0; it < 8192; ++it) {
        const int v = L[y];
        const int up = v >> 1;
        if (up == y) break;
        const int w = L[up];
        const int gp = w >> 1;
        if (gp == up) {   // up is the root
            p ^= v & 1;
            y = up;
            break;
        }
        const int pg = (v ^ w) & 1;   // parity of y to its grandparent
        L[y] = (gp << 1) | pg;
        p ^= pg;
        y = gp;
    }
    parity = p;
    return y;
}

// The tables every warp of a block shares, loaded into the block's shared memory.
struct FagwTables {
    uint2* lvl;         // [N] members by generation level: x = member, y = 2 mother | 2 father << 16
    int32_t* lvl_off;   // [n_lvl + 1]
};

__device__ FagwTables fagw_load_tables(const ProblemDev& P, unsigned char* smem) {
    const int N = P.N;
    FagwTables t;
    t.lvl = (uint2*)smem;
    t.lvl_off = (int32_t*)(smem + (((size_t)N * 8 + 15) & ~(size_t)15));
    for (int q = threadIdx.x; q < N; q += blockDim.x) {
        const int pid = P.lvl_order[q];
        const int mo = P.mother[pid], fa = P.father[pid];
        t.lvl[q] = make_uint2((unsigned)pid, mo < 0 ? 0u : (unsigned)(2 * mo) | ((unsigned)(2 * fa) << 16));
    }
    for (int i = threadIdx.x; i <= P.n_lvl; i += blockDim.x) t.lvl_off[i] = P.lvl_off[i];
    return t;
}

// A group of G lanes (32 or 16) of a warp, aligned, working on one locus;
// every primitive runs on the full warp and is read per group.
template <int G>
struct LaneGroup {
    int gl, base;
    __device__ LaneGroup() {
        const int lane = threadIdx.x & 31;
        gl = lane & (G - 1);
        base = lane & ~(G - 1);
    }
    __device__ __forceinline__ unsigned ballot(bool p) const {
        const unsigned b = __ballot_sync(FULLMASK, p);
        return G == 32 ? b : (b >> base) & ((1u << G) - 1u);
    }
    __device__ __forceinline__ bool any(bool p) const { return ballot(p) != 0u; }
    __device__ __forceinline__ uint32_t shfl(uint32_t v, int src) const { return __shfl_sync(FULLMASK, v, src, G); }
};

// log2 of the genotypes' likelihood at locus lc given the column `col` with
// meiosis `flip` toggled (-1: as it is), by one group of G lanes (32 / G loci
// per warp, in lockstep: every loop below has the same trip count in all
// groups except the union loop, which holds no warp primitive); all lanes of
// the group return it.
template <int G, typename E>
__device__ __forceinline__ float fagw_like(const ProblemDev& P, const FagwTables& tab, unsigned char* wbase,
                                           const uint32_t* col, int chain, int lc, int flip, int* status) {
    const LaneGroup<G> grp;
    const int N = P.N, F = P.F, nfa = 2 * F, M = P.M, gl = grp.gl;
    const uint2* s_lvl = tab.lvl;
    const int32_t* s_off = tab.lvl_off;
    E* e = (E*)wbase;                                                 // [2N] founder allele of each allele
    volatile int* Lb = (volatile int*)(wbase + (((size_t)2 * sizeof(E) * N + 15) & ~(size_t)15));   // [2F] 2 * parent + parity
    int* fl = (int*)(Lb + nfa);                                       // [2F] bit0 used, bit1 fixed A, bit2 fixed B
    int* cnt = fl + nfa;                                              // [2F] per component: counts, forbidden colourings
    uint16_t* typ = (uint16_t*)(wbase + fagw_typ_offset(N, F, (int)sizeof(E)));   // [N] the locus's typed members
    // the task's global reads issued together: the column's words (lane w of
    // the group holds word w, read by shuffles), the allele frequencies'
    // log2, and the locus's typed members (member << 2 | genotype code,
    // heterozygotes first: fixed by the genotypes, listed once at context
    // creation), copied to shared memory in 16-byte asynchronous copies that
    // complete while the founder alleles are propagated
    const bool wreg = P.W <= G;
    const uint32_t toggled = 1u << (flip & 31);   // of word flip >> 5; none where flip is -1
    const uint32_t cw = wreg && gl < P.W ? col[gl] ^ (gl == flip >> 5 ? toggled : 0u) : 0u;
    const int t0 = P.typ_off[lc], ntyp = P.typ_cnt[lc], nhet = P.typ_nhet[lc];
    const float2 lfreq = P.c_lfreq[(size_t)chain * M + lc];
#pragma unroll 1
    for (int q = gl; q < (ntyp + 7) >> 3; q += G) cp_async16(typ + 8 * q, P.typ_ent + t0 + 8 * q);
    cp_async_commit();
    // 1. founder alleles, one generation level at a time
#pragma unroll 1
    for (int q = gl; q < s_off[1]; q += G) {
        const int pid = (int)s_lvl[q].x;
        e[2 * pid] = (E)(2 * pid);
        e[2 * pid + 1] = (E)(2 * pid + 1);
    }
    __syncwarp();
#pragma unroll 1
    for (int k = 1; k < P.n_lvl; ++k) {
        // every lane takes part in the shuffles, members or not
#pragma unroll 1
        for (int q0 = s_off[k]; q0 < s_off[k + 1]; q0 += G) {
            const int q = q0 + gl;
            const bool act = q < s_off[k + 1];
            const uint2 ent = act ? s_lvl[q] : make_uint2((unsigned)F, 0u);
            const int pid = (int)ent.x;
            const int b = 2 * (pid - F);
            const uint32_t w = wreg ? grp.shfl(cw, b >> 5) : col[b >> 5] ^ (b >> 5 == flip >> 5 ? toggled : 0u);
            if (!act) continue;
            const int vm = (int)((w >> (b & 31)) & 1u), vp = (int)((w >> ((b + 1) & 31)) & 1u);
            e[2 * pid] = e[(ent.y & 0xffffu) + vm];
            e[2 * pid + 1] = e[(ent.y >> 16) + vp];
        }
        __syncwarp();
    }
    // 2. fixed founder alleles: the homozygous typed members (after the
    // heterozygotes in the list) mark theirs with the colour their genotype
    // forces (no warp primitive inside: the groups' loci have lists of their
    // own lengths)
#pragma unroll 1
    for (int x = gl; x < nfa; x += G) {
        Lb[x] = x << 1;
        fl[x] = 0;
        cnt[x] = 0;
    }
    cp_async_wait_all();   // this lane's copies of the list; the barrier makes the group's visible
    __syncwarp();
    int clash = 0;
#pragma unroll 1
    for (int x = nhet + gl; x < ntyp; x += G) {
        const int ent = typ[x], i = ent >> 2, g = ent & 3;
        const int bits = g == G_HOMOZ_A ? 3 : 5;   // used, fixed A / fixed B
        const int b0 = atomicOr(&fl[e[2 * i]], bits) | bits, b1 = atomicOr(&fl[e[2 * i + 1]], bits) | bits;
        clash |= (b0 & 6) == 6 || (b1 & 6) == 6;
    }
    __syncwarp();
    // a founder allele fixed to both colours: the likelihood is zero, and the
    // components need not be worked out (most evaluated toggles end here)
    clash = grp.any(clash);
    if (__all_sync(FULLMASK, clash)) return -INFINITY;
    // 3. components of the heterozygote edges with parities: a lock-free
    // union-find forest in Lb (2 * parent + parity to the parent), each lane
    // joining its edges by hooking the larger root under the smaller with a
    // compare-and-swap (so a root is its component's smallest allele); an edge
    // whose ends already share a root must have ends of opposite parity.  A
    // failed hook means another lane's hook succeeded, so a lane retries fewer
    // than 2F times.  An edge whose two ends are both fixed only needs their
    // colours to differ: the two sides' colourings are then determined apart,
    // and the likelihood is the product of the two sides' terms, so the edge
    // joins nothing.  The ends of the other edges are marked used and joined
    // (bit 3: in the forest).  First, a heterozygote with exactly one fixed
    // end fixes the other to the opposite colour, in rounds until nothing
    // changes (at most kFagRounds): most edges then have both ends fixed, and
    // a fixed allele's colour is its component's, so its term is the same.
#pragma unroll 1
    for (int round = 0; round < kFagRounds; ++round) {
        int changed = 0;
#pragma unroll 1
        for (int q = gl; q < nhet; q += G) {
            const int i = typ[q] >> 2;
            const int u = e[2 * i], v = e[2 * i + 1];
            const int fu = fl[u] & 6, fv = fl[v] & 6;
            if ((fu != 0) == (fv != 0)) continue;   // both ends fixed, or neither
            const int cf = fu ? fu : fv;
            const int opp = cf == 2 ? 4 : (cf == 4 ? 2 : 6);
            atomicOr(&fl[fu ? v : u], opp | 1);
            changed = 1;
        }
        __syncwarp();
        if (!__any_sync(FULLMASK, changed)) break;   // the whole warp, as its groups share the loop
    }
    int bad = clash;
#pragma unroll 1
    for (int q = gl; q < nhet; q += G) {
        const int i = typ[q] >> 2;   // the heterozygotes lead the list
        const int u = e[2 * i], v = e[2 * i + 1];
        if (u == v) {   // one founder allele cannot give both alleles of a heterozygote
            bad = 1;
            continue;
        }
        const int fu = fl[u], fv = fl[v];
        if ((fu & 6) && (fv & 6)) {
            if (fu & fv & 6) bad = 1;   // both ends forced to the same colour
            continue;
        }
        atomicOr(&fl[u], 9);
        atomicOr(&fl[v], 9);
        for (int tries = 0;; ++tries) {
            if (tries > nfa) {
                bad = 1;
                set_status(status, ST_ILLEGAL_DG);
                break;
            }
            int pu, pv;
            const int ru = pf_find(Lb, u, pu), rv = pf_find(Lb, v, pv);
            if (ru == rv) {
                if ((pu ^ pv) != 1) bad = 1;   // an odd cycle of heterozygote edges
                break;
            }
            const int lo = min(ru, rv), hi = max(ru, rv);
            if (atomicCAS((int*)&Lb[hi], hi << 1, (lo << 1) | (pu ^ pv ^ 1)) == (hi << 1)) break;
        }
    }
    bad = grp.any(bad);
    __syncwarp();
    // 4. sum over each component's colourings, log2: every member allele
    // contributes log2 of the major or the minor frequency, so a component
    // needs only its member count, how many members have even parity and
    // which colourings its fixed members forbid (integer shared-memory
    // atomics, the same result in any order).  A fixed allele outside the
    // forest is a component of its own: its term is added directly.
    float sum = 0.f;
    int zero = 0, forest = 0;
    const float lmaj = lfreq.x, lmin = lfreq.y;
    if (!bad)
#pragma unroll 1
        for (int x = gl; x < nfa; x += G) {
            const int f = fl[x];
            if (!(f & 1)) continue;
            if (!(f & 8)) {
                if ((f & 6) == 6) zero = 1;
                else sum += (f & 2) ? lmaj : lmin;
                continue;
            }
            forest = 1;
            int p = 0;
            const int r = pf_find(Lb, x, p);   // the forest is final: the unions are done
            // bit 16 + n: member count; bits 0-15: even-parity members; bits 29/30: colouring 0/1 forbidden
            const int add = (1 << 16) + (p ? 0 : 1);
            int forbid = 0;
            if (f & 2) forbid |= p ? (1 << 29) : (1 << 30);   // fixed A
            if (f & 4) forbid |= p ? (1 << 30) : (1 << 29);   // fixed B
            atomicAdd(&cnt[r], add);
            if (forbid) atomicOr(&cnt[r], forbid);
        }
    forest = grp.any(forest);   // no union: every term is in already
    __syncwarp();
    if (!bad && forest) {
#pragma unroll 1
        for (int x = gl; x < nfa; x += G) {
            const int c = cnt[x];
            const int n = (c >> 16) & 0x1fff, even = c & 0xffff;
            if (n == 0) continue;
            const float w0 = (float)even * lmaj + (float)(n - even) * lmin;   // root coloured A
            const float w1 = (float)even * lmin + (float)(n - even) * lmaj;   // root coloured B
            const int ok0 = !(c & (1 << 29)), ok1 = !(c & (1 << 30));
            if (ok0 && ok1) {
                const float mx = fmaxf(w0, w1);
                sum += mx + log2f(1.f + exp2f(fminf(w0, w1) - mx));
            } else if (ok0) sum += w0;
            else if (ok1) sum += w1;
            else zero = 1;
        }
    }
    zero = grp.any(zero);
    for (int dd = G / 2; dd >= 1; dd >>= 1) sum += __shfl_xor_sync(FULLMASK, sum, dd);
    __syncwarp();
    return (bad || zero) ? -INFINITY : sum;
}

// One (chain, locus) task by one group of G lanes: step < 0 stores the
// likelihood of the column at meiosis order[0]; step >= 0 the likelihoods at
// both values of meiosis order[step] (the kept one from the previous step).
// A group past the last locus (valid false) works on locus 0 and stores
// nothing.
template <int G, typename E>
__device__ __forceinline__ void fagw_task(const ProblemDev& P, const FagwTables& tab, unsigned char* wbase,
                                          const uint32_t* dg, int chain, int cr, int l, bool valid,
                                          const int32_t* ord, int step, float* rawbuf, float* raw32, uint8_t* badc,
                                          int* status) {
    const int M = P.M, lc = valid ? l : 0;
    const uint32_t* col = dg + ((size_t)chain * M + lc) * P.W;
    float* raw = rawbuf + (size_t)cr * 2 * M;
    int flip = -1, tb = 0;
    float keep = 0.f;
    if (step >= 0) {
        flip = ord[step];
        tb = dgbit(col, flip);
        keep = raw[2 * lc + dgbit(col, ord[step > 0 ? step - 1 : 0])];
    }
    const float lk = fagw_like<G, E>(P, tab, wbase, col, chain, lc, flip, status);
    if ((threadIdx.x & (G - 1)) == 0 && valid) {
        if (step < 0) {
            raw[2 * l + dgbit(col, ord[0])] = lk;
            if (lk == -INFINITY) {
                badc[cr] = 1;
                set_status(status, ST_ILLEGAL_DG);
            }
        } else {
            raw[2 * l + tb] = keep;
            raw[2 * l + 1 - tb] = lk;
            float* r32 = raw32 + (size_t)cr * 2 * M;
            if (tb == 0) put_raw32_log2(r32, l, keep, lk);
            else put_raw32_log2(r32, l, lk, keep);
            if (keep == -INFINITY && lk == -INFINITY) {
                badc[cr] = 1;
                set_status(status, ST_ILLEGAL_DG);
            }
        }
    }
    __syncwarp();
}

template <typename T>
struct Flt;
template <>
struct Flt<double> {
    static __device__ __forceinline__ double mul(double a, double b) { return DMUL(a, b); }
    static __device__ __forceinline__ double add(double a, double b) { return DADD(a, b); }
    static __device__ __forceinline__ double sub(double a, double b) { return DSUB(a, b); }
    static __device__ __forceinline__ double div(double a, double b) { return DDIV(a, b); }
};

// one locus of the exact filter (meiosis_sampler.cc:136-155): the pair (f0, f1)
// entering it becomes its own; th the recombination fraction below it
__device__ __forceinline__ void exact_filter(double a0, double a1, double th, bool bottom, double& f0, double& f1) {
    using Fl = Flt<double>;
    double g0 = a0, g1 = a1;
    if (!bottom) {
        const double ax = Fl::sub(1.0, th);
        g0 = Fl::mul(a0, Fl::add(Fl::mul(f1, th), Fl::mul(f0, ax)));
        g1 = Fl::mul(a1, Fl::add(Fl::mul(f0, th), Fl::mul(f1, ax)));
    }
    const double tot = Fl::add(g0, g1);
    f0 = Fl::div(g0, tot);
    f1 = Fl::div(g1, tot);
}

// (x o y)(v) = x(y(v)) for 2-bit maps
__device__ __forceinline__ int map_compose(int x, int y) {
    const int y0 = y & 1, y1 = (y >> 1) & 1;
    return ((x >> y0) & 1) | (((x >> y1) & 1) << 1);
}

// The exact filter and sampling of one meiosis by one warp, in the reference's
// order (meiosis_sampler.cc:136-203): all 32 lanes run the same serial recursion
// on values broadcast by shuffles from coalesced 32-locus chunks (the FP64 pipe
// costs the same per warp instruction whatever the active mask).  For the
// chains that ffbs_exact_kernel cannot split.
__device__ void ffbs_serial_chain(const ProblemDev& P, uint32_t* G, int chain, int cr, int m, int step, const Draws& draws,
                                  const double* r64, double* fb) {
    using Fl = Flt<double>;
    const int lane = threadIdx.x & 31;
    double prev0 = 0.0, prev1 = 0.0;
    for (int base = 0; base < P.M; base += 32) {
        const int i = base + lane;
        double q0 = 0.0, q1 = 0.0, th = 0.0;
        if (i < P.M) {
            q0 = r64[2 * i];
            q1 = r64[2 * i + 1];
            if (i >= 1) th = P.c_theta[(size_t)chain * (P.M - 1) + i - 1];
        }
        const int n = min(32, P.M - base);
        double k0 = 0.0, k1 = 0.0;
        for (int x = 0; x < n; ++x) {
            const double a0 = __shfl_sync(FULLMASK, q0, x), a1 = __shfl_sync(FULLMASK, q1, x);
            exact_filter(a0, a1, __shfl_sync(FULLMASK, th, x), base + x == 0, prev0, prev1);
            if (lane == x) { k0 = prev0; k1 = prev1; }
        }
        if (i < P.M) { fb[2 * i] = k0; fb[2 * i + 1] = k1; }
    }
    __syncwarp();
    // backward sampling (meiosis_sampler.cc:157-203)
    int64_t cursor = 0;
    int nxt = 0;
    for (int top = P.M - 1; top >= 0; top -= 32) {
        const int lo = max(0, top - 31);
        const int n = top - lo + 1;
        const int i = top - lane;
        const bool in = i >= lo;
        const double f0 = in ? fb[2 * i] : 0.0, f1 = in ? fb[2 * i + 1] : 0.0;
        const double th = (in && i < P.M - 1) ? P.c_theta[(size_t)chain * (P.M - 1) + i] : 0.0;
        uint32_t* wp = in ? (G + (size_t)i * P.W + (m >> 5)) : nullptr;
        const int cur = in ? (int)((*wp >> (m & 31)) & 1u) : 0;
        const int64_t c0 = cursor;
        const double dr = (c0 + lane < P.M) ? draws.get(cr, chain, step, c0 + lane) : 0.0;
        int mine = cur;
        for (int x = 0; x < n; ++x) {
            const int ii = top - x;
            double a0 = __shfl_sync(FULLMASK, f0, x), a1 = __shfl_sync(FULLMASK, f1, x);
            const double tx = __shfl_sync(FULLMASK, th, x);
            if (ii < P.M - 1) {
                const double ax = Fl::sub(1.0, tx);
                a0 = Fl::mul(a0, nxt != 0 ? tx : ax);
                a1 = Fl::mul(a1, nxt != 1 ? tx : ax);
            }
            int samp;
            if (a0 == 0.0) samp = 1;
            else if (a1 == 0.0) samp = 0;
            else {
                const double r = __shfl_sync(FULLMASK, dr, (int)(cursor - c0));
                ++cursor;
                samp = (r < Fl::div(a0, Fl::add(a0, a1))) ? 0 : 1;
            }
            nxt = samp;
            if (lane == x) mine = samp;
        }
        if (in && mine != cur) *wp ^= (1u << (m & 31));
    }
}

// The exact filter, split where it starts anew.  A locus where one of the two
// likelihoods is zero leaves the pair (0, 1) or (1, 0), exactly, whatever came
// before: 0 x / (0 x + a y) is 0 and a y / (0 + a y) is 1 for finite x and any
// a y > 0.  So a run of loci from one such locus to the next is filtered by
// itself, the same operations on the same values, and the runs side by side: a
// warp's lanes each take the run that starts at their locus.  That holds while
// no product underflows, in the filter or in the sampling (which draws where
// both of a locus's values are non-zero, one of them times theta): loci whose
// larger likelihood, or whose smaller non-zero filtered value, lies below
// kExactTiny, and any theta below kExactTheta, set the chain's flag, and
// ffbs_exact_kernel then does it all in one run.  The serial recursion is
// bound by the latency of FP64 (about 900 cycles a locus, two divisions and
// five dependent operations): an M-sweep of two chains of 30 members took 13.7
// ms at 200 SNPs and 121 ms at 2,000, in runs 2.6 and 3.6 ms; one of 120
// members and 2,000 SNPs 549 and 36 ms.
constexpr double kExactTiny = 1e-280, kExactTheta = 1e-20;

__global__ void __launch_bounds__(32) ffbs_exact_runs_kernel(ProblemDev P, int first, int nchain, const uint8_t* sel,
                                                             int want, const uint8_t* badc, const double* raw64,
                                                             double* fbbuf, int* flag, int64_t fstride) {
    const int cr = blockIdx.y, M = P.M;
    if (sel && sel[cr] != want) return;
    if (badc[cr]) return;
    const int chain = first + cr, i = blockIdx.x * 32 + threadIdx.x;
    if (i >= M) return;
    const double* r = raw64 + (size_t)cr * 2 * M;
    double* fb = fbbuf + (size_t)cr * 2 * M;
    const double* th = P.c_theta + (size_t)chain * (M - 1);
    auto anew = [&](double a0, double a1) { return (a0 == 0.0) != (a1 == 0.0); };
    double a0 = r[2 * i], a1 = r[2 * i + 1];
    if (i > 0 && !anew(a0, a1)) return;   // in another lane's run
    double f0 = 0.0, f1 = 0.0;
    bool tiny = false;
    for (int k = i;; ) {
        tiny |= !(fmax(a0, a1) >= kExactTiny);
        if (k > 0 && k == i) {
            f0 = a0 == 0.0 ? 0.0 : 1.0;
            f1 = a0 == 0.0 ? 1.0 : 0.0;
        } else {
            exact_filter(a0, a1, k > 0 ? th[k - 1] : 0.0, k == 0, f0, f1);
        }
        tiny |= k > 0 && !(th[k - 1] >= kExactTheta);
        tiny |= (f0 != 0.0 && !(f0 >= kExactTiny)) || (f1 != 0.0 && !(f1 >= kExactTiny));
        fb[2 * k] = f0;
        fb[2 * k + 1] = f1;
        if (++k >= M) break;
        a0 = r[2 * k];
        a1 = r[2 * k + 1];
        if (anew(a0, a1)) break;
    }
    if (tiny) atomicOr(flag + cr * fstride, 1);
}

// Backward sampling of one meiosis over the filtered pairs, one block per
// chain: a locus's choice given the one above, for both of that one's values,
// is worked out at all loci at once (a locus draws when both its filtered
// values are non-zero, so a suffix count gives each its draw), and the choices
// are composed from the top.  The chain's flag (see above) sends it through
// ffbs_serial_chain instead, and is cleared for the next meiosis.
__global__ void __launch_bounds__(512) ffbs_exact_kernel(ProblemDev P, uint32_t* dg, int first, int nchain,
                                                         const int32_t* order, int64_t ostride, int step, Draws draws,
                                                         const uint8_t* sel, int want, const uint8_t* badc,
                                                         const double* raw64, double* fbbuf, uint8_t* mapbuf, int* flag,
                                                         int64_t fstride) {
    __shared__ int wcnt[16], wmap[17];
    using Fl = Flt<double>;
    const int cr = blockIdx.x, M = P.M;
    if (sel && sel[cr] != want) return;
    if (badc[cr]) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    const int chain = first + cr, m = order[cr * ostride + step];
    uint32_t* G = dg + (size_t)chain * M * P.W;
    double* fb = fbbuf + (size_t)cr * 2 * M;
    uint8_t* maps = mapbuf + (size_t)cr * M;
    const double* th = P.c_theta + (size_t)chain * (M - 1);
    if (flag[cr * fstride]) {
        if (warp == 0) ffbs_serial_chain(P, G, chain, cr, m, step, draws, raw64 + (size_t)cr * 2 * M, fb);
        __syncthreads();
        if (tid == 0) flag[cr * fstride] = 0;
        return;
    }
    const int L = (M + blockDim.x - 1) / blockDim.x, s0 = min(M, tid * L), s1 = min(M, s0 + L);
    int cnt = 0;
    for (int i = s0; i < s1; ++i) cnt += fb[2 * i] != 0.0 && fb[2 * i + 1] != 0.0;
    int x = cnt;   // draws of this run and those above it in the warp
    for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_down_sync(FULLMASK, x, d);
        if (lane + d < 32) x += y;
    }
    if (lane == 0) wcnt[warp] = x;
    __syncthreads();
    int idx = x - cnt;
    for (int w = warp + 1; w < nw; ++w) idx += wcnt[w];
    int g = 2;   // identity: bit 0 = 0, bit 1 = 1
    for (int i = s1 - 1; i >= s0; --i) {
        const double f0 = fb[2 * i], f1 = fb[2 * i + 1];
        int map;
        if (f0 == 0.0) map = 3;
        else if (f1 == 0.0) map = 0;
        else {
            const double u = draws.get(cr, chain, step, idx++);
            if (i == M - 1) {
                map = (u < Fl::div(f0, Fl::add(f0, f1))) ? 0 : 3;
            } else {
                const double t = th[i], a = Fl::sub(1.0, t);
                const double x0 = Fl::mul(f0, a), y0 = Fl::mul(f1, t);   // next = 0
                const double x1 = Fl::mul(f0, t), y1 = Fl::mul(f1, a);   // next = 1
                map = (u < Fl::div(x0, Fl::add(x0, y0)) ? 0 : 1) | (u < Fl::div(x1, Fl::add(x1, y1)) ? 0 : 2);
            }
        }
        maps[i] = (uint8_t)map;
        g = map_compose(map, g);
    }
    // suffix composition: within the warp, then across warps
    for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_down_sync(FULLMASK, g, d);
        if (lane + d < 32) g = map_compose(g, y);
    }
    if (lane == 0) wmap[warp] = g;
    __syncthreads();
    if (tid == 0) {
        int acc = 2;
        wmap[nw] = 2;
        for (int w = nw - 1; w >= 0; --w) {
            acc = map_compose(wmap[w], acc);
            wmap[w] = acc;
        }
    }
    __syncthreads();
    const int tail = wmap[warp + 1];
    int above = __shfl_down_sync(FULLMASK, map_compose(g, tail), 1);
    if (lane == 31) above = tail;
    int sv = above & 1;
    for (int i = s1 - 1; i >= s0; --i) {
        sv = (maps[i] >> sv) & 1;
        uint32_t* wp = G + (size_t)i * P.W + (m >> 5);
        const uint32_t w = *wp;
        if (sv != (int)((w >> (m & 31)) & 1u)) *wp = w ^ (1u << (m & 31));
    }
}

// Fast M-sampler filter and sampling in O(M/32 + log 32) depth per chain.
// The forward filter f_i = normalise(diag(r_i) T_i f_{i-1}) is a product of
// 2x2 matrices: each lane multiplies its chunk's matrices, a warp scan
// combines the chunk products, and each lane then replays its chunk from the
// vector entering it.  Backward sampling s_i = d_i(s_{i+1}) is a composition
// of maps {0,1} -> {0,1} (2 bits each: the decision when s_{i+1} = 0 and when
// it is 1), scanned the same way from the top locus down.  A locus consumes a
// draw only when neither filtered probability is zero (meiosis_sampler.cc:
// 193-203), so draw indices come from a suffix count of such loci.
__device__ __forceinline__ void mat_norm(float& a, float& b, float& c, float& d) {
    const float mx = fmaxf(fmaxf(fabsf(a), fabsf(b)), fmaxf(fabsf(c), fabsf(d)));
    if (mx > 0.f) {
        const float inv = 1.f / mx;
        a *= inv; b *= inv; c *= inv; d *= inv;
    }
}

// Block-wide scan scratch of ffbs_scan_kernel (blockDim.x = T, a multiple of 32, <= 1024).
struct ScanScratch {
    float4* incl;   // [T] each thread's inclusive filter product
    float4* wmat;   // [32] warp products, then their inclusive scan
    int* wcnt;      // [32] draws per warp
    int* wmap;      // [33] warp decision maps, then their suffix compositions
};

__device__ __forceinline__ void mat_mul_left(float& p00, float& p01, float& p10, float& p11, float o00, float o01,
                                             float o10, float o11) {
    // p <- p * o (o is the earlier product, applied first)
    const float n00 = p00 * o00 + p01 * o10, n01 = p00 * o01 + p01 * o11;
    const float n10 = p10 * o00 + p11 * o10, n11 = p10 * o01 + p11 * o11;
    p00 = n00; p01 = n01; p10 = n10; p11 = n11;
}

// p <- diag(q) R(t) p, one locus's factor of the filter product
__device__ __forceinline__ void filter_product(float q0, float q1, float t, float& p00, float& p01, float& p10,
                                               float& p11) {
    const float a = 1.f - t;
    const float n00 = q0 * (a * p00 + t * p10), n01 = q0 * (a * p01 + t * p11);
    const float n10 = q1 * (t * p00 + a * p10), n11 = q1 * (t * p01 + a * p11);
    p00 = n00; p01 = n01; p10 = n10; p11 = n11;
}

// one locus of the filter from the vector (v0, v1) entering it
__device__ __forceinline__ void filter_locus(float q0, float q1, float t, float v0, float v1, float& f0, float& f1) {
    const float a = 1.f - t;
    f0 = q0 * (a * v0 + t * v1);
    f1 = q1 * (t * v0 + a * v1);
    const float tot = f0 + f1;
    if (tot > 0.f) { const float inv = 1.f / tot; f0 *= inv; f1 *= inv; }
    // keep the reference's exact zeros: a zero likelihood stays zero
    if (q0 == 0.f) f0 = 0.f;
    if (q1 == 0.f) f1 = 0.f;
}

// a locus's decision map from its filtered pair (both non-zero) and its draw;
// t: the recombination fraction to the locus above (last: none above).  U is
// double, or float with the draw rounded down (Draws::get_rd): the same choices.
template <typename U>
__device__ __forceinline__ int locus_map(float f0, float f1, U u, bool last, float t) {
    if (last) {
        const int v = (u < (U)(f0 / (f0 + f1))) ? 0 : 1;
        return v | (v << 1);
    }
    const float a = 1.f - t;
    const float x0 = f0 * a, y0 = f1 * t;   // next = 0
    const float x1 = f0 * t, y1 = f1 * a;   // next = 1
    const int d0 = (u < (U)(x0 / (x0 + y0))) ? 0 : 1;
    const int d1 = (u < (U)(x1 / (x1 + y1))) ? 0 : 1;
    return d0 | (d1 << 1);
}

// Fast-mode forward filter and backward sampling of one meiosis over all loci,
// one block per chain (meiosis_sampler.cc:123-203 restated as scans): each
// thread owns a run of L = ceil(M / T) loci.
//   forward:  the filter is a product of 2x2 matrices A_i = diag(r_i) R(theta_i);
//             chunk products are scanned across the block (later chunks on the
//             left, normalised to a maximum of 1), and each chunk then filters
//             its loci from the vector entering it;
//   backward: loci draw from M-1 down, a locus drawing when both filtered
//             entries are non-zero; a suffix sum of the chunks' draw counts
//             gives each chunk its first draw, so all draws are generated in
//             parallel; each locus's choice given the locus above is a 2-bit
//             map, and a suffix composition of the chunks' maps gives each
//             chunk the state entering it from above.
// The body for chain `chain` (relative index cr), meiosis m, run by a whole
// block.  upre (may be null) holds the step's draws by index, precomputed;
// with cg, the pairs and draws written by other blocks of the same launch are
// read past L1.
__device__ __forceinline__ void ffbs_scan_chain(const ProblemDev& P, uint32_t* dg, int chain, int cr, int m, int step,
                                const Draws& draws, const double* upre, const float* r, float* fb, uint8_t* maps,
                                int staged, bool cg, unsigned char* fsm) {
    const int T = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = T >> 5;
    const int M = P.M;
    uint32_t* G = dg + (size_t)chain * M * P.W;
    float* th = nullptr;        // theta as floats, [M]
    uint32_t* words = nullptr;  // the meiosis's descent-graph word at each locus, [M]
    ScanScratch sc;
    sc.incl = (float4*)fsm;
    sc.wmat = sc.incl + T;
    sc.wcnt = (int*)(sc.wmat + 32);
    sc.wmap = sc.wcnt + 32;
    unsigned char* stage = (unsigned char*)(sc.wmap + 36);
    if (staged) {
        // [r: 2M][fb: 2M][theta: M] floats, [words: M], [maps: M bytes]
        float* sr = (float*)stage;
        float* sfb = sr + 2 * M;
        th = sfb + 2 * M;
        words = (uint32_t*)(th + M);
        uint8_t* smaps = (uint8_t*)(words + M);
        for (int i = tid; i < M; i += T) words[i] = G[(size_t)i * P.W + (m >> 5)];
        for (int i = tid; i < 2 * M; i += T) sr[i] = cg ? __ldcg(r + i) : r[i];
        for (int i = tid; i < M; i += T) th[i] = i > 0 ? P.c_theta_f[(size_t)chain * (M - 1) + i - 1] : 0.f;
        r = sr;
        fb = sfb;
        maps = smaps;
    }
    __syncthreads();
    auto tof = [&](int i) { return th ? th[i] : (i > 0 ? P.c_theta_f[(size_t)chain * (M - 1) + i - 1] : 0.f); };
    const bool rcg = cg && !staged;   // the pairs still in global memory, written by other blocks
    auto rq = [&](int i) { return rcg ? __ldcg(r + i) : r[i]; };
    const int L = (M + T - 1) / T;
    const int s0 = min(M, tid * L), s1 = min(M, s0 + L);
    // chunk product P = A_{s1-1} ... A_{s0} (A_0 = diag(r_0)); an empty chunk is the identity
    float p00 = 1.f, p01 = 0.f, p10 = 0.f, p11 = 1.f;
    for (int i = s0; i < s1; ++i) {
        filter_product(rq(2 * i), rq(2 * i + 1), tof(i), p00, p01, p10, p11);
        // each pair is scaled to a maximum of 1, so 8 steps cannot underflow
        if (((i - s0) & 7) == 7) mat_norm(p00, p01, p10, p11);
    }
    mat_norm(p00, p01, p10, p11);
    // inclusive scan within the warp: S_k = P_k ... P_first
    for (int d = 1; d < 32; d <<= 1) {
        const float o00 = __shfl_up_sync(FULLMASK, p00, d), o01 = __shfl_up_sync(FULLMASK, p01, d);
        const float o10 = __shfl_up_sync(FULLMASK, p10, d), o11 = __shfl_up_sync(FULLMASK, p11, d);
        if (lane >= d) {
            mat_mul_left(p00, p01, p10, p11, o00, o01, o10, o11);
            mat_norm(p00, p01, p10, p11);
        }
    }
    if (lane == 31) sc.wmat[warp] = make_float4(p00, p01, p10, p11);
    __syncthreads();
    if (warp == 0) {
        // inclusive scan of the warp products (nw <= 32)
        float4 w = lane < nw ? sc.wmat[lane] : make_float4(1.f, 0.f, 0.f, 1.f);
        for (int d = 1; d < 32; d <<= 1) {
            const float o00 = __shfl_up_sync(FULLMASK, w.x, d), o01 = __shfl_up_sync(FULLMASK, w.y, d);
            const float o10 = __shfl_up_sync(FULLMASK, w.z, d), o11 = __shfl_up_sync(FULLMASK, w.w, d);
            if (lane >= d) {
                mat_mul_left(w.x, w.y, w.z, w.w, o00, o01, o10, o11);
                mat_norm(w.x, w.y, w.z, w.w);
            }
        }
        __syncwarp();
        if (lane < nw) sc.wmat[lane] = w;
    }
    __syncthreads();
    if (warp > 0) {
        const float4 o = sc.wmat[warp - 1];
        mat_mul_left(p00, p01, p10, p11, o.x, o.y, o.z, o.w);
        mat_norm(p00, p01, p10, p11);
    }
    sc.incl[tid] = make_float4(p00, p01, p10, p11);
    __syncthreads();
    // vector entering the chunk: S_{k-1} (1, 1)
    float v0 = 1.f, v1 = 1.f;
    if (tid > 0) {
        const float4 e = sc.incl[tid - 1];
        v0 = e.x + e.y;
        v1 = e.z + e.w;
    }
    int cnt = 0;
    for (int i = s0; i < s1; ++i) {
        float f0, f1;
        filter_locus(rq(2 * i), rq(2 * i + 1), tof(i), v0, v1, f0, f1);
        fb[2 * i] = f0;
        fb[2 * i + 1] = f1;
        cnt += (f0 != 0.f && f1 != 0.f);
        v0 = f0;
        v1 = f1;
    }
    // draws consumed by loci in higher chunks: a suffix sum over the block
    int x = cnt;
    for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_down_sync(FULLMASK, x, d);
        if (lane + d < 32) x += y;
    }
    if (lane == 0) sc.wcnt[warp] = x;
    __syncthreads();
    int above = x - cnt;
    for (int w = warp + 1; w < nw; ++w) above += sc.wcnt[w];
    // per-locus decision maps and the chunk's composed map; the chunk's draws are
    // independent of one another, so they are generated four at a time
    int gmap = 2;  // identity: bit0 = 0, bit1 = 1
    int idx = above;
    double ubuf[4];
    int ub = 4;
    for (int i = s1 - 1; i >= s0; --i) {
        const float f0 = fb[2 * i], f1 = fb[2 * i + 1];
        int dmap;
        if (f0 == 0.f) dmap = 3;
        else if (f1 == 0.f) dmap = 0;
        else {
            if (ub == 4) {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    ubuf[q] = idx + q >= M ? 0.0
                              : upre ? (cg ? __ldcg(upre + idx + q) : upre[idx + q])
                                     : draws.get(cr, chain, step, idx + q);
                ub = 0;
            }
            const double u = ubuf[ub++];
            ++idx;
            dmap = locus_map(f0, f1, u, i == M - 1, i == M - 1 ? 0.f : tof(i + 1));
        }
        maps[i] = (uint8_t)dmap;
        gmap = map_compose(dmap, gmap);
    }
    // suffix composition x_k = G_k o G_{k+1} o ... o G_{T-1}: within the warp,
    // then across warps
    int xm = gmap;
    for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_down_sync(FULLMASK, xm, d);
        if (lane + d < 32) xm = map_compose(xm, y);
    }
    if (lane == 0) sc.wmap[warp] = xm;
    __syncthreads();
    if (tid == 0) {
        int acc = 2;
        sc.wmap[nw] = 2;
        for (int w = nw - 1; w >= 0; --w) {
            acc = map_compose(sc.wmap[w], acc);
            sc.wmap[w] = acc;     // warp w's maps composed with every warp above it
        }
    }
    __syncthreads();
    // the state entering this chunk from above: x_{k+1} applied to anything
    // (the chunk holding locus M-1 ends in a constant map)
    const int tail = sc.wmap[warp + 1];
    const int full = map_compose(xm, tail);
    int above_map = __shfl_down_sync(FULLMASK, full, 1);
    if (lane == 31) above_map = tail;
    int sv = above_map & 1;
    for (int i = s1 - 1; i >= s0; --i) {
        sv = (maps[i] >> sv) & 1;
        uint32_t* wp = G + (size_t)i * P.W + (m >> 5);
        const uint32_t w = words ? words[i] : *wp;
        const int cur = (int)((w >> (m & 31)) & 1u);
        if (sv != cur) *wp = w ^ (1u << (m & 31));
    }
}

__global__ void __launch_bounds__(1024, 1) ffbs_scan_kernel(ProblemDev P, uint32_t* dg, int first, int nchain,
                                                         const int32_t* order, int64_t ostride, int step,
                                                         Draws draws, const uint8_t* sel, int want,
                                                         const uint8_t* badc, const float* raw32, float* fbbuf,
                                                         uint8_t* mapbuf, int staged, const double* ubuf) {
    extern __shared__ __align__(16) unsigned char fsm[];
    const int cr = blockIdx.x;
    if (cr >= nchain) return;
    if (sel && sel[cr] != want) return;
    if (badc[cr]) return;
    const int M = P.M;
    ffbs_scan_chain(P, dg, first + cr, cr, order[cr * ostride + step], step, draws,
                    ubuf ? ubuf + (size_t)cr * M : nullptr,
                    raw32 + (size_t)cr * 2 * M, fbbuf + (size_t)cr * 2 * M, mapbuf + (size_t)cr * M, staged, false,
                    fsm);
}

// ---------------------------------------------------------------------------
// Fast M-sampler likelihoods of one meiosis step: grid (blocks per chain,
// chains), one warp per locus (fagw_task).  With ubuf, the first 32-locus
// slice of warps also draws the step's uniforms by index, one per lane, so
// ffbs_scan_kernel only reads them.
// ---------------------------------------------------------------------------
template <int G, typename E>
__global__ void __launch_bounds__(kFagWarpsPerBlock * 32) fag_warp_kernel(ProblemDev P, uint32_t* dg, int first,
                                                                         const int32_t* order, int64_t ostride,
                                                                         int step, Draws draws, const uint8_t* sel,
                                                                         int want, float* rawbuf, float* raw32,
                                                                         uint8_t* badc, int* status, double* ubuf) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int cr = blockIdx.y;
    if (sel && sel[cr] != want) return;
    const int M = P.M;
    const FagwTables tab = fagw_load_tables(P, smem);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kLoci = 32 / G;   // loci per warp
    const int chain = first + cr;
    const int32_t* ord = order + cr * ostride;
    const int gw = blockIdx.x * kFagWarpsPerBlock + warp;
    if (ubuf && step >= 0 && gw * 32 + lane < M)
        ubuf[(size_t)cr * M + gw * 32 + lane] = draws.get(cr, chain, step, gw * 32 + lane);
    const int gi = lane / G, l = gw * kLoci + gi;
    if (gw * kLoci < M)
        fagw_task<G, E>(P, tab,
                        smem + fagw_tables(P.N) + ((size_t)warp * kLoci + gi) * fagw_warp_bytes(P.N, P.F, (int)sizeof(E)),
                        dg, chain,
                     cr, l, l < M, ord, step, rawbuf, raw32, badc, status);
}

// Threads per chain of ffbs_scan_kernel: runs of about 2 loci (the scan is
// on every meiosis step's critical path; shorter runs shorten its serial parts).
int ffbs_scan_threads(int M) {
    int t = ((M + 1) / 2 + 31) / 32 * 32;
    return t < 32 ? 32 : (t > 1024 ? 1024 : t);
}

// Shared bytes: the scan scratch, then (when staged) the chain's arrays.
size_t ffbs_scan_scratch(int T) { return (size_t)16 * T + 16 * 32 + 4 * 32 + 4 * 36; }
size_t ffbs_scan_smem(int M) { return ffbs_scan_scratch(ffbs_scan_threads(M)) + (size_t)6 * 4 * M + (size_t)M + 16; }

// ---------------------------------------------------------------------------
// Fast-mode M-sweep of one chain by one thread-block cluster.
//
// Every meiosis step needs the likelihood of each locus with the meiosis
// toggled, then a filter and a backward draw along all loci.  As two launches
// per meiosis (fag_warp_kernel, ffbs_scan_kernel) the step of a 120-member,
// 2,000-SNP chain took 27 us: two dependent launches and a scan on one SM.
// Here a cluster of CS blocks keeps the chain for the whole sweep: a block
// owns the loci of its share of ffbs_scan_kernel's warps, holds their columns
// (when they fit), current likelihoods and filter state in shared memory, and
// meets the others three times per meiosis in cluster barriers, to pass on the
// scans' warp totals through distributed shared memory.  The scans keep that
// kernel's threads, runs and order of operations (a "virtual" warp v of the
// chain is warp v - rank * vpb of block rank), so graphs are the same bit for
// bit, whatever CS.
//
// Most toggled likelihoods follow from the genotypes and the current one
// (P.mflip, built with the context, meiosis_flips in sl_host.cc): where the
// two founder alleles that the meiosis chooses between are both fixed to one
// colour by homozygous members above it, or nobody below it is typed, the
// toggled graph has the same terms in the same places, and its likelihood is
// the current one; where they are fixed to opposite colours and the
// transmitted one is known, the toggled graph is impossible.  More follows
// from the graph as it is (P.mrel, relatives_rule).  The rest (one in 25 to 30
// with 5% of the genotypes missing) are listed and evaluated by the block's
// warps (fagw_like).
//
// A step changes one column in 600, so the likelihoods of kMswAhead steps are
// evaluated together at the first of them, from the columns as they are then:
// one wait for the evaluations (5 us each, however few there are) instead of
// four, and a fuller block waits for 4 steps' sum instead of each step's most.
// Where a column has changed since, a step decides the locus anew and, if need
// be, evaluates it itself (one step in two to four of the whole cluster).
//
// Measured, a sweep of every chain, as launches per meiosis, by a cluster, with
// the steps evaluated together: 400 members, 10,000 SNPs, one chain 39 | 16.6 |
// 13.3 ms, 8 chains 128 | 20.8 | 17.8, 32 chains 397 | 37.4 | 35.5; 120 members,
// 2,000 SNPs, one chain 3.3 | 2.22 | 1.86, 10 chains 5.1 | 2.77 | 2.20 (11 us a
// meiosis), 160 chains 53 | 8.9 | 8.6; 30 members, 200 SNPs 0.41 | 0.33 (by a
// cluster).  Bound by the evaluated likelihoods
// (issue with 32 warps on an SM: 23,000 of a 400-member step's 60,000 cycles;
// 4,800 of 25,000 for 120 members), by waiting for the block with the most of
// them (13,000; 5,600) and by the scans' serial runs and barriers.
// ---------------------------------------------------------------------------
struct MswShape {
    int cs;        // blocks per cluster
    int nw, run;   // virtual warps of the chain, loci per virtual thread
    int vpb;       // virtual warps per block
    int nl;        // loci per block
    int threads;   // per block
    int staged;    // the columns are kept in shared memory
    size_t task, xch, loci, cols, bytes;   // shared offsets: tasks' scratch, exchange, per-locus arrays, columns; all bytes
};

// Steps whose likelihoods are evaluated together, a locus's index and step
// among them in 16 bits, and how many likelihoods a block keeps (what does not
// fit is evaluated at its step; one locus in 25 is evaluated at a step, so 4
// steps fill 16% of nl).  3 or 5 steps measured within 2% of 4, 8 steps 5% slower.
constexpr int kMswAhead = 4, kMswStepShift = 13;
__host__ __device__ constexpr int msw_kept(int nl) { return nl / 4; }

// per-locus arrays of a block: filter pairs (8), current and toggled
// likelihood, theta (one more) and draw index (4 each), what was evaluated
// ahead (6 for each that is kept), masks (five for each step ahead, and the
// columns changed), the list of loci to evaluate (2) and the decision maps (1)
static size_t msw_locus_bytes(int nl) {
    return al16((size_t)nl * (8 + 4 * 4 + 2 + 1) + 4 + (size_t)msw_kept(nl) * 6 +
                4 * (size_t)(5 * kMswAhead + 1) * (nl / 32));
}

// Shared memory a block of msweep_kernel may take.
constexpr size_t kMswSmem = 200 * 1024;

// The shape with up to `cs` blocks per cluster; false when a block's share
// does not fit its shared memory.  A block has a warp for every four of its
// loci, up to 32: of 8, 16 and 32 warps the most are the fastest or as fast.  A
// sweep with 8 | 16 | 32: 30 members, 200 SNPs 0.354 | 0.328 | 0.329 ms; 120 members,
// 2,000 SNPs, one chain 2.27 | 1.92 | 1.86, 160 chains 8.6 with any; 400 members, 10,000
// SNPs, one chain 26.0 | 17.2 | 13.3, 32 chains 59.9 | 36.2 | 35.5.
static bool msw_shape(const ProblemDev& P, int G, int eb, int cs, MswShape* out) {
    MswShape s;
    s.nw = ffbs_scan_threads(P.M) / 32;
    s.run = (P.M + s.nw * 32 - 1) / (s.nw * 32);
    if (cs > s.nw) cs = s.nw;
    s.vpb = (s.nw + cs - 1) / cs;
    s.cs = (s.nw + s.vpb - 1) / s.vpb;
    s.nl = s.vpb * 32 * s.run;
    s.task = fagw_tables(P.N);
    for (int warps = std::min(kMswThreads / 32, std::max(4, s.nl / 4)); warps >= std::max(4, s.vpb); warps /= 2) {
        s.threads = 32 * warps;
        s.xch = s.task + (size_t)warps * (32 / G) * fagw_warp_bytes(P.N, P.F, eb);
        s.loci = s.xch + 16 * 32 + 4 * 32 + 4 * 32 + 16;
        s.cols = s.loci + msw_locus_bytes(s.nl);
        s.bytes = s.cols + al16((size_t)4 * P.W * s.nl);
        s.staged = s.bytes <= kMswSmem;   // else the columns stay in global memory
        if (!s.staged) s.bytes = s.cols;
        *out = s;
        if (s.bytes <= kMswSmem && s.nl <= 1 << kMswStepShift) return true;
    }
    return false;
}

// One of a meiosis's relatives (P.mrel) at 32 loci: its entry and the two bits
// of its genotype codes.  Lane r of a warp holds relative r.
struct Relative {
    uint32_t entry, c0, c1;
};
__device__ __forceinline__ Relative load_relative(const ProblemDev& P, int m, int word, int lane) {
    Relative r;
    r.entry = P.mrel[(size_t)m * kRelatives + lane];
    r.c0 = r.c1 = 0u;
    if (r.entry != kNoRelative && word < P.mflip_words) {
        const uint32_t* g = P.gplane + (size_t)(r.entry & 0xffffu) * 2 * P.mflip_words + word;
        r.c0 = g[0];
        r.c1 = g[P.mflip_words];
    }
    return r;
}

// relatives_rule at a warp's 32 loci: lane r holds relative r, lane l locus
// l's column and the meiosis's own indicator tb there.
__device__ __forceinline__ void flips_by_relatives(const ProblemDev& P, int m, const Relative& own,
                                                   const uint32_t* col, int tb, uint32_t* same, uint32_t* never) {
    relatives_rule(
        m, P.F, __ballot_sync(FULLMASK, tb), [&](int r) { return __shfl_sync(FULLMASK, own.entry, r); },
        [&](int r) { return __shfl_sync(FULLMASK, own.c0, r); }, [&](int r) { return __shfl_sync(FULLMASK, own.c1, r); },
        [&](int b) { return __ballot_sync(FULLMASK, (col[b >> 5] >> (b & 31)) & 1u); }, same, never);
}

template <int G, typename E>
__global__ void __launch_bounds__(kMswThreads, 1) msweep_kernel(ProblemDev P, MswShape sh, uint32_t* dg, int first,
                                                             const int32_t* order, int64_t ostride, int nm,
                                                             Draws draws, const uint8_t* sel, int want, int* status) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int cr = blockIdx.y;
    if (sel && sel[cr] != want) return;   // the whole cluster
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, NT = blockDim.x;
    const int M = P.M, W = P.W, chain = first + cr;
    const int nw = sh.nw, L = sh.run;
    const int lo = rank * sh.nl, nl = max(0, min(M, lo + sh.nl) - lo);
    const FagwTables tab = fagw_load_tables(P, smem);
    constexpr int kLoci = 32 / G;   // loci per warp
    unsigned char* scratch = smem + sh.task + (size_t)(warp * kLoci + lane / G) * fagw_warp_bytes(P.N, P.F, (int)sizeof(E));
    float4* wmat = (float4*)(smem + sh.xch);   // every virtual warp's filter product
    int* wcnt = (int*)(wmat + 32);             // its draws (bit 30: an impossible pair somewhere in its block)
    int* wmap = wcnt + 32;                     // its decision map
    int* ctl = wmap + 32;                      // [0, 1] loci to evaluate at even and odd steps, [2] impossible pair,
                                               // [3] likelihoods to evaluate ahead
    float2* pr = (float2*)(smem + sh.loci);    // [nl] the step's pair, then the filtered pair
    float* cur = (float*)(pr + sh.nl);         // [nl] log2 likelihood of the column
    float* tog = cur + sh.nl;                  // [nl] with the meiosis toggled
    float* th = tog + sh.nl;                   // [nl + 1] theta to the locus below
    int* didx = (int*)(th + sh.nl + 1);        // [nl] draws above the locus in its block's run
    const int nmw = sh.nl / 32, MW = P.mflip_words, kept = msw_kept(sh.nl);
    float* eval = (float*)(didx + sh.nl);            // [kept] likelihoods evaluated ahead
    uint32_t* msk = (uint32_t*)(eval + kept);        // [step ahead][nl / 32][5]: what the genotypes say (same, never),
                                                     // same, to evaluate, evaluated
    uint32_t* changed = msk + kMswAhead * 5 * nmw;   // [nl / 32] columns changed since the evaluation ahead
    uint16_t* ahead = (uint16_t*)(changed + nmw);    // [kept] locus | step << kMswStepShift
    uint16_t* list = ahead + kept;
    uint8_t* maps = (uint8_t*)(list + sh.nl);
    uint32_t* gcol = dg + ((size_t)chain * M + lo) * W;
    uint32_t* col = sh.staged ? (uint32_t*)(smem + sh.cols) : gcol;
    const int32_t* ord = order + cr * ostride;
    if (sh.staged)
#pragma unroll 1
        for (int i = tid; i < nl * W; i += NT) col[i] = gcol[i];
#pragma unroll 1
    for (int i = tid; i <= nl; i += NT) th[i] = lo + i > 0 && lo + i < M ? P.c_theta_f[(size_t)chain * (M - 1) + lo + i - 1] : 0.f;
    if (tid < 4) ctl[tid] = 0;
    __syncthreads();
    // the likelihood of every column as it is
#pragma unroll 1
    for (int h = warp * kLoci; h < nl; h += (NT >> 5) * kLoci) {
        const int i = h + lane / G;
        const bool valid = i < nl;
        const int q = valid ? i : h;
        const float lk = fagw_like<G, E>(P, tab, scratch, col + (size_t)q * W, chain, lo + q, -1, status);
        if ((lane & (G - 1)) == 0 && valid) {
            cur[i] = lk;
            if (lk == -INFINITY) {
                ctl[2] = 1;
                set_status(status, ST_ILLEGAL_DG);
            }
        }
    }
    cluster.sync();   // every block runs before the first write to another's shared memory
    const int vw = rank * sh.vpb + warp;                  // this warp's virtual warp
    const bool scans = warp < sh.vpb && vw < nw;
    const int s0 = min(M, (vw * 32 + lane) * L) - lo, s1 = min(M, (vw * 32 + lane + 1) * L) - lo;   // its run of loci
    int na = 0;   // likelihoods evaluated ahead
    // a meiosis at 32 loci: the loci where its toggling is known to change nothing, and those to evaluate
    auto classify = [&](int m, int w, uint32_t of, uint32_t same, uint32_t never, auto relative, uint32_t* out_same) {
        const int i = 32 * w + lane;
        const bool in = i < nl;
        const uint32_t* mine = col + (size_t)(in ? i : 32 * w) * W;
        if (__any_sync(FULLMASK, in && ((of & ~(same | never)) >> lane) & 1))
            flips_by_relatives(P, m, relative(), mine, (mine[m >> 5] >> (m & 31)) & 1, &same, &never);
        *out_same = same;
        return __ballot_sync(FULLMASK, in && (cur[in ? i : 0] == -INFINITY || !(((same | never) >> lane) & 1)));
    };
#pragma unroll 1
    for (int j = 0; j < nm; ++j) {
        const int m = ord[j], mw = m >> 5, mb = m & 31, s = j % kMswAhead;
        if (s == 0) {
            // this step and the next ones as the columns are now; a task's genotypes are read while the one before goes on
            const int tasks = min(kMswAhead, nm - j) * nmw;
            uint32_t gs = 0u, gn = 0u;
            Relative rel = {kNoRelative, 0u, 0u};
            auto read = [&](int t) {
                const int q = t / nmw, gw = (lo >> 5) + t - q * nmw;
                if (t >= tasks || gw >= MW) return;
                const int m2 = ord[j + q];
                gs = P.mflip[(size_t)m2 * 2 * MW + gw];
                gn = P.mflip[((size_t)m2 * 2 + 1) * MW + gw];
                rel = load_relative(P, m2, gw, lane);
            };
            read(warp);
#pragma unroll 1
            for (int t = warp; t < tasks; t += NT >> 5) {
                const int q = t / nmw, w = t - q * nmw;
                if (q == 0 && lane == 0) changed[w] = 0u;
                const uint32_t ts = gs, tn = gn;
                const Relative tr = rel;
                read(t + (NT >> 5));
                if (32 * w >= nl) continue;
                uint32_t same;
                const uint32_t hard = classify(ord[j + q], w, FULLMASK, ts, tn, [&] { return tr; }, &same);
                int at = 0;
                if (lane == 0 && hard) at = atomicAdd(&ctl[3], __popc(hard));
                at = __shfl_sync(FULLMASK, at, 0) + __popc(hard & ((1u << lane) - 1u));
                const bool mine = (hard >> lane) & 1 && at < kept;
                if (mine) ahead[at] = (uint16_t)((32 * w + lane) | q << kMswStepShift);
                const uint32_t has = __ballot_sync(FULLMASK, mine);
                if (lane < 5) msk[t * 5 + lane] = lane == 0 ? ts : lane == 1 ? tn : lane == 2 ? same : lane == 3 ? hard : has;
            }
            __syncthreads();
            na = min(ctl[3], kept);
        }
        // the step's pairs: from the genotypes where they decide, evaluated ahead, else listed
#pragma unroll 1
        for (int i0 = warp * 32; i0 < nl; i0 += NT) {
            const int i = i0 + lane, w = i0 >> 5;
            const bool in = i < nl;
            const uint32_t* k = msk + (s * nmw + w) * 5;
            const uint32_t ch = changed[w];
            uint32_t same = k[2], hard = k[3];
            const uint32_t has = k[4] & ~ch;
            if (ch) {
                uint32_t sn;
                const uint32_t hn = classify(m, w, ch, k[0], k[1], [&] { return load_relative(P, m, (lo >> 5) + w, lane); }, &sn);
                same = (same & ~ch) | (sn & ch);
                hard = (hard & ~ch) | (hn & ch);
            }
            if (in) {
                const bool sm = (same >> lane) & 1;
                const int tb = (col[(size_t)i * W + mw] >> mb) & 1;
                if (!((has >> lane) & 1)) {
                    tog[i] = sm ? cur[i] : -INFINITY;
                    pr[i] = sm ? make_float2(1.f, 1.f) : make_float2(tb ? 0.f : 1.f, tb ? 1.f : 0.f);
                }
            }
            hard &= ~has;
            int at = 0;
            if (lane == 0 && hard) at = atomicAdd(&ctl[j & 1], __popc(hard));
            at = __shfl_sync(FULLMASK, at, 0);
            if ((hard >> lane) & 1) list[at + __popc(hard & ((1u << lane) - 1u))] = (uint16_t)i;
        }
        // the pair of column i whose toggled likelihood is lk
        auto take = [&](int i, float lk) {
            const float keep = cur[i];
            const int tb = (col[(size_t)i * W + mw] >> mb) & 1;
            tog[i] = lk;
            float r2[2];
            put_raw32_log2(r2, 0, tb ? lk : keep, tb ? keep : lk);
            pr[i] = make_float2(r2[0], r2[1]);
            if (keep == -INFINITY && lk == -INFINITY) {
                ctl[2] = 1;
                set_status(status, ST_ILLEGAL_DG);
            }
        };
        __syncthreads();
        const int nh = ctl[j & 1];
        if (tid == 0) ctl[(j + 1) & 1] = ctl[3] = 0;
        if (s > 0)
#pragma unroll 1
            for (int e = tid; e < na; e += NT) {
                const int a = ahead[e], i = a & ((1 << kMswStepShift) - 1);
                if (a >> kMswStepShift == s && !((changed[i >> 5] >> (i & 31)) & 1)) take(i, eval[e]);
            }
        // what is to be evaluated: ahead when the step is the first of its group, then the step's own list
        const int n0 = s == 0 ? na : 0;
#pragma unroll 1
        for (int h = warp * kLoci; h < n0 + nh; h += (NT >> 5) * kLoci) {
            const bool valid = h + lane / G < n0 + nh;
            const int k = valid ? h + lane / G : h;
            const int e = k < n0 ? ahead[k] : list[k - n0];
            const int i = k < n0 ? e & ((1 << kMswStepShift) - 1) : e, q = k < n0 ? e >> kMswStepShift : 0;
            const float lk = fagw_like<G, E>(P, tab, scratch, col + (size_t)i * W, chain, lo + i, ord[j + q], status);
            if ((lane & (G - 1)) == 0 && valid) {
                if (q == 0) take(i, lk);
                else eval[k] = lk;
            }
        }
        __syncthreads();
        // forward filter: run products, scanned within the warp, the warp totals passed to every block
        float p00 = 1.f, p01 = 0.f, p10 = 0.f, p11 = 1.f;
        if (scans) {
#pragma unroll 1
            for (int i = s0; i < s1; ++i) {
                const float2 q = pr[i];
                filter_product(q.x, q.y, th[i], p00, p01, p10, p11);
                // each pair is scaled to a maximum of 1, so 8 steps cannot underflow
                if (((i - s0) & 7) == 7) mat_norm(p00, p01, p10, p11);
            }
            mat_norm(p00, p01, p10, p11);
            for (int d = 1; d < 32; d <<= 1) {
                const float o00 = __shfl_up_sync(FULLMASK, p00, d), o01 = __shfl_up_sync(FULLMASK, p01, d);
                const float o10 = __shfl_up_sync(FULLMASK, p10, d), o11 = __shfl_up_sync(FULLMASK, p11, d);
                if (lane >= d) {
                    mat_mul_left(p00, p01, p10, p11, o00, o01, o10, o11);
                    mat_norm(p00, p01, p10, p11);
                }
            }
            const float4 tot = make_float4(__shfl_sync(FULLMASK, p00, 31), __shfl_sync(FULLMASK, p01, 31),
                                           __shfl_sync(FULLMASK, p10, 31), __shfl_sync(FULLMASK, p11, 31));
            if (lane < sh.cs) *cluster.map_shared_rank(&wmat[vw], lane) = tot;
        }
        cluster.sync();
        int cnt = 0, x = 0;
        if (scans) {
            float4 w = lane < nw ? wmat[lane] : make_float4(1.f, 0.f, 0.f, 1.f);
            float4 below = vw > 0 ? wmat[vw - 1] : w;   // the product of the thread below lane 0's
            for (int d = 1; d < 32; d <<= 1) {
                const float o00 = __shfl_up_sync(FULLMASK, w.x, d), o01 = __shfl_up_sync(FULLMASK, w.y, d);
                const float o10 = __shfl_up_sync(FULLMASK, w.z, d), o11 = __shfl_up_sync(FULLMASK, w.w, d);
                if (lane >= d) {
                    mat_mul_left(w.x, w.y, w.z, w.w, o00, o01, o10, o11);
                    mat_norm(w.x, w.y, w.z, w.w);
                }
            }
            if (vw > 0) {
                const int o = vw - 1;
                mat_mul_left(p00, p01, p10, p11, __shfl_sync(FULLMASK, w.x, o), __shfl_sync(FULLMASK, w.y, o),
                             __shfl_sync(FULLMASK, w.z, o), __shfl_sync(FULLMASK, w.w, o));
                mat_norm(p00, p01, p10, p11);
            }
            if (vw > 1) {
                const int o = vw - 2;
                mat_mul_left(below.x, below.y, below.z, below.w, __shfl_sync(FULLMASK, w.x, o),
                             __shfl_sync(FULLMASK, w.y, o), __shfl_sync(FULLMASK, w.z, o),
                             __shfl_sync(FULLMASK, w.w, o));
                mat_norm(below.x, below.y, below.z, below.w);
            }
            // the vector entering the run: S_{k-1} (1, 1)
            float v0 = __shfl_up_sync(FULLMASK, __fadd_rn(p00, p01), 1);
            float v1 = __shfl_up_sync(FULLMASK, __fadd_rn(p10, p11), 1);
            if (lane == 0) {
                v0 = vw > 0 ? __fadd_rn(below.x, below.y) : 1.f;
                v1 = vw > 0 ? __fadd_rn(below.z, below.w) : 1.f;
            }
#pragma unroll 1
            for (int i = s0; i < s1; ++i) {
                const float2 q = pr[i];
                float f0, f1;
                filter_locus(q.x, q.y, th[i], v0, v1, f0, f1);
                pr[i] = make_float2(f0, f1);
                cnt += (f0 != 0.f && f1 != 0.f);
                v0 = f0;
                v1 = f1;
            }
            // draws consumed by loci in higher runs: a suffix sum
            x = cnt;
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_down_sync(FULLMASK, x, d);
                if (lane + d < 32) x += y;
            }
            const int tot = __shfl_sync(FULLMASK, x, 0) | (ctl[2] ? 1 << 30 : 0);
            if (lane < sh.cs) *cluster.map_shared_rank(&wcnt[vw], lane) = tot;
        }
        cluster.sync();
        // draws above this block's loci, and whether any block met an impossible pair (the chain then stays as it is)
        int above = 0, bad = 0;
        {
            const int c = lane < nw ? wcnt[lane] : 0;
            bad = __any_sync(FULLMASK, c >> 30);
            // draws of the virtual warps above the block's, then of those above this one within it
            const int hi = (rank + 1) * sh.vpb;
            int s = lane >= hi ? c & 0x3fffffff : 0;
            s = __reduce_add_sync(FULLMASK, s);
            above = s;
        }
        if (bad) break;   // every block of the cluster leaves here together
        if (scans) {
            int rel = x - cnt;   // draws above this run in the block
#pragma unroll 1
            for (int v = vw + 1; v < min(nw, (rank + 1) * sh.vpb); ++v) rel += wcnt[v] & 0x3fffffff;
#pragma unroll 1
            for (int i = s1 - 1; i >= s0; --i) {
                const float2 f = pr[i];
                didx[i] = rel;
                rel += f.x != 0.f && f.y != 0.f;
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int i = tid; i < nl; i += NT) {
            const float2 f = pr[i];
            int dmap;
            if (f.x == 0.f) dmap = 3;
            else if (f.y == 0.f) dmap = 0;
            else dmap = locus_map(f.x, f.y, draws.get_rd(cr, chain, j, above + didx[i]), lo + i == M - 1, th[i + 1]);
            maps[i] = (uint8_t)dmap;
        }
        __syncthreads();
        int xm = 2;   // identity: bit0 = 0, bit1 = 1
        if (scans) {
#pragma unroll 1
            for (int i = s1 - 1; i >= s0; --i) xm = map_compose(maps[i], xm);
            // suffix composition within the warp
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_down_sync(FULLMASK, xm, d);
                if (lane + d < 32) xm = map_compose(xm, y);
            }
            const int tot = __shfl_sync(FULLMASK, xm, 0);
            if (lane < sh.cs) *cluster.map_shared_rank(&wmap[vw], lane) = tot;
        }
        cluster.sync();
        if (scans) {
            // every virtual warp above this one, composed
            int tail = lane > vw && lane < nw ? wmap[lane] : 2;
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_down_sync(FULLMASK, tail, d);
                if (lane + d < 32) tail = map_compose(tail, y);
            }
            tail = __shfl_sync(FULLMASK, tail, 0);
            // the state entering this run from above (the run holding locus M - 1 ends in a constant map)
            int in = __shfl_down_sync(FULLMASK, map_compose(xm, tail), 1);
            if (lane == 31) in = tail;
            int sv = in & 1;
#pragma unroll 1
            for (int i = s1 - 1; i >= s0; --i) {
                sv = (maps[i] >> sv) & 1;
                const uint32_t w = col[(size_t)i * W + mw];
                if (sv != (int)((w >> mb) & 1u)) {
                    col[(size_t)i * W + mw] = w ^ (1u << mb);
                    cur[i] = tog[i];
                    atomicOr(&changed[i >> 5], 1u << (i & 31));
                }
            }
        }
        __syncthreads();
    }
    __syncthreads();
    if (sh.staged)
#pragma unroll 1
        for (int i = tid; i < nl * W; i += NT) gcol[i] = col[i];
}

// ---------------------------------------------------------------------------
// Trait peel LOD scorer: one warp per (graph, interval, position).
// ---------------------------------------------------------------------------
__device__ __forceinline__ int phased_trait(int m, int p, int i, int j) {
    // rfunction.cc:98-114 with affected_trait (rfunction.h:82-107)
    const int ma = (m == AA) || (m == AU && i == 0) || (m == UA && i == 1);
    const int pa = (p == AA) || (p == AU && j == 0) || (p == UA && j == 1);
    if (ma) return pa ? AA : AU;
    return pa ? UA : UU;
}

template <typename T>
struct Arith;
template <>
struct Arith<double> {
    static __device__ __forceinline__ double mul(double a, double b) { return DMUL(a, b); }
    static __device__ __forceinline__ double add(double a, double b) { return DADD(a, b); }
};
template <>
struct Arith<float> {
    static __device__ __forceinline__ float mul(float a, float b) { return a * b; }
    static __device__ __forceinline__ float add(float a, float b) { return a + b; }
};

// TraitRfunction::get_recombination_probability (trait_rfunction.cc:9-24)
template <typename T>
__device__ __forceinline__ T trait_rec(int bits, int i, int j, T th, T an, T th2, T an2) {
    using Ar = Arith<T>;
    T tmp = ((bits & 1) == i) ? an : th;                      // maternal, locus
    tmp = Ar::mul(tmp, (((bits >> 2) & 1) == i) ? an2 : th2); // maternal, locus + 1
    tmp = Ar::mul(tmp, (((bits >> 1) & 1) == j) ? an : th);   // paternal, locus
    tmp = Ar::mul(tmp, (((bits >> 3) & 1) == j) ? an2 : th2); // paternal, locus + 1
    return tmp;
}

__device__ __forceinline__ int person_bits(const ProblemDev& P, const uint32_t* colL, const uint32_t* colR,
                                           int person) {
    const int b = 2 * (person - P.F);
    return dgbit(colL, b) | (dgbit(colL, b + 1) << 1) | (dgbit(colR, b) << 2) | (dgbit(colR, b + 1) << 3);
}

// L lanes a position, which share the cells of its rfunctions.  The FP64 pipe
// bounds it (16 cycles for a warp's instruction, however many lanes it has), so:
// several positions to a warp, since a two-member cutset has 16 cells and many
// have 4; the recombination terms of a child from 16 products made once a
// position (four multiplications for each of a cell's four terms before); the
// recombination sum from the count of crossovers (one lane's 2 (N - F) additions
// before); and matrices that lie where a dead one lay (reuse_arena), for 28
// warps to an SM instead of 8.  Four graphs of 45 members and 401 SNPs (8,000
// positions): 0.92 ms with a warp a position; 0.58 with 16 lanes, 0.36 with the
// products, 0.25 with the smaller arena, the pipe at 74%.
template <typename T, bool RESCALE, int L>
__global__ void __launch_bounds__(128) lod_kernel(ProblemDev P, const uint32_t* graphs, int64_t graph_words,
                                                  int G, double* vals, int* status) {
    using Ar = Arith<T>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int per = blockDim.x / L, at = threadIdx.x / L, lane = threadIdx.x & (L - 1);
    T* A = (T*)(smem + (size_t)at * (P.arena + 16) * sizeof(T));
    T* quarter_rec = A + P.arena;   // [bits ^ (5 i | 10 j)]: a quarter of trait_rec(bits, i, j)
    const int n = P.n_lod;
    const int64_t npos = (int64_t)(P.M - 1) * n;
    const int64_t ntask = (int64_t)G * npos;
    // at - at % (32 / L): a warp's positions go round together, those past the end on the last one's data
    for (int64_t t0 = (int64_t)blockIdx.x * per + at; t0 - at % (32 / L) < ntask; t0 += (int64_t)gridDim.x * per) {
        const int64_t t = min(t0, ntask - 1);
        const int b = (int)(t / npos);
        const int64_t pidx = t % npos;
        const int l = (int)(pidx / n), o = (int)(pidx % n);
        const uint32_t* colL = graphs + (size_t)b * graph_words + (size_t)l * P.W;
        const uint32_t* colR = colL + P.W;
        // TraitRfunction::set_thetas (trait_rfunction.h:50-56)
        const double thd = DMUL(P.partial[l], (double)(o + 1));
        const double th2d = DMUL(P.partial[l], (double)(n + 1 - (o + 1)));
        const T th = (T)thd, an = (T)DSUB(1.0, thd), th2 = (T)th2d, an2 = (T)DSUB(1.0, th2d);
        for (int e = lane; e < 16; e += L)
            quarter_rec[e] = Ar::mul((T)0.25, trait_rec<T>(e, 0, 0, th, an, th2, an2));
        __syncwarp();
        int scale = 0;
        for (int k = 0; k < P.K; ++k) {
            const OpDev op = P.ops[k];
            const int ncell = 1 << (2 * op.c);
            const int32_t* cut = P.opdata + op.cut_at;
            const double* trait = P.dprob + 4 * op.peel;
            T* out = A + op.mat_off;
            T mx = (T)0;
            for (int cell = lane; cell < ncell; cell += L) {
                bool valid = true;
                for (int q = 0; q < op.c; ++q) valid &= ((P.dmask[cut[q]] >> digit(cell, q)) & 1) != 0;
                T total = (T)0;
                if (valid) {
                    if (op.type == CHILD) {
                        const int mt = digit(cell, op.mpos), pt = digit(cell, op.fpos);
                        const int bits = person_bits(P, colL, colR, op.peel);
                        for (int i = 0; i < 2; ++i)
                            for (int j = 0; j < 2; ++j) {
                                const int kt = phased_trait(mt, pt, i, j);
                                const double tvd = trait[kt];
                                if (tvd == 0.0) continue;
                                const int ext = cell | (kt << (2 * op.c));
                                T tmp = (T)tvd;
                                const int32_t* pd = P.opdata + op.prev_at;
                                for (int jj = 0; jj < op.n_prev; ++jj) {
                                    int idx = 0;
                                    for (int q = 0; q < pd[1]; ++q) idx |= digit(ext, pd[2 + q]) << (2 * q);
                                    tmp = Ar::mul(tmp, A[pd[0] + idx]);
                                    pd += 2 + pd[1];
                                }
                                tmp = Ar::mul(tmp, quarter_rec[bits ^ (5 * i | 10 * j)]);
                                total = Ar::add(total, tmp);
                            }
                    } else if (op.type == PARENT) {
                        for (int a = 0; a < 4; ++a) {
                            const double tvd = trait[a];
                            if (tvd == 0.0) continue;
                            const int ext = cell | (a << (2 * op.c));
                            T tmp = (T)tvd;
                            const int32_t* pd = P.opdata + op.prev_at;
                            for (int jj = 0; jj < op.n_prev; ++jj) {
                                int idx = 0;
                                for (int q = 0; q < pd[1]; ++q) idx |= digit(ext, pd[2 + q]) << (2 * q);
                                tmp = Ar::mul(tmp, A[pd[0] + idx]);
                                pd += 2 + pd[1];
                            }
                            T cp = (T)1;
                            int mt = a, pt = a;
                            const int32_t* cd = P.opdata + op.child_at;
                            for (int c = 0; c < op.n_child; ++c, cd += 4) {
                                const int kt = digit(ext, cd[1]), other = digit(ext, cd[2]);
                                if (cd[3]) pt = other; else mt = other;
                                const int bits = person_bits(P, colL, colR, cd[0]);
                                T ct = (T)0;
                                for (int i = 0; i < 2; ++i)
                                    for (int j = 0; j < 2; ++j) {
                                        if (phased_trait(mt, pt, i, j) != kt) continue;
                                        ct = Ar::add(ct, quarter_rec[bits ^ (5 * i | 10 * j)]);
                                    }
                                cp = Ar::mul(cp, ct);
                            }
                            tmp = Ar::mul(tmp, cp);
                            total = Ar::add(total, tmp);
                        }
                    } else {
                        for (int a = 0; a < 4; ++a) {
                            const double tvd = trait[a];
                            if (tvd == 0.0) continue;
                            const int ext = cell | (a << (2 * op.c));
                            T tmp = (T)tvd;
                            const int32_t* pd = P.opdata + op.prev_at;
                            for (int jj = 0; jj < op.n_prev; ++jj) {
                                int idx = 0;
                                for (int q = 0; q < pd[1]; ++q) idx |= digit(ext, pd[2 + q]) << (2 * q);
                                tmp = Ar::mul(tmp, A[pd[0] + idx]);
                                pd += 2 + pd[1];
                            }
                            total = Ar::add(total, tmp);
                        }
                    }
                }
                out[cell] = total;
                mx = total > mx ? total : mx;
            }
            __syncwarp();
            if (RESCALE) {
                for (int s = L / 2; s > 0; s >>= 1) {
                    const T o2 = __shfl_xor_sync(FULLMASK, mx, s);
                    mx = o2 > mx ? o2 : mx;
                }
                if (mx > (T)0) {
                    if constexpr (sizeof(T) == 8) {
                        const int e = ilogb(mx);
                        const T f = scalbn(1.0, -e);
                        for (int cell = lane; cell < ncell; cell += L) out[cell] *= f;
                        scale += e;
                    } else {
                        // FP32: the largest cell to 2^scale_to (LI_SCALE, sl_internal.h)
                        const int e = ilogbf(mx) - op.scale_to;
                        for (int cell = lane; cell < ncell; cell += L) out[cell] = ldexpf(out[cell], -e);
                        scale += e;
                    }
                }
                __syncwarp();
            }
        }
        // DescentGraph::get_recombination_prob (descent_graph.cc:212-242) by the count of crossovers
        const double r = (double)A[P.ops[P.K - 1].mat_off];
        int cross = 0;
        for (int w = lane; w < P.W; w += L) cross += __popc(colL[w] ^ colR[w]);
        for (int s = L / 2; s > 0; s >>= 1) cross += __shfl_xor_sync(FULLMASK, cross, s);
        if (lane == 0 && t0 < ntask) {
            const double rec = DADD(DMUL((double)cross, P.log_theta[l]), DMUL((double)(2 * P.Nnf - cross), P.log_itheta[l]));
            double v;
            if (r <= 0.0) {
                if (!P.lod_zero_ok) set_status(status, ST_LOD_NONPOS);
                v = -DBL_MAX;
            } else {
                v = log(r) + (double)scale * 0.69314718055994530942 - rec - P.marker_trans;
            }
            vals[t] = v;
        }
        __syncwarp();
    }
}

// Batched trait peel: one thread per (graph, interval, position) runs the
// compiled LI_* program; every lane of a warp executes the same instruction
// stream (uniform loads of the program) on its own recombination terms, with
// its FP32 slots in shared memory at [slot][thread].  Each rfunction's cells
// are rescaled by a power of two after they are computed; the exponents are
// summed and restored in FP64 at the end.
__global__ void __launch_bounds__(128) lod_prog_kernel(ProblemDev P, const uint32_t* graphs, int64_t graph_words,
                                                       int G, double* vals, int* status) {
    extern __shared__ float sh[];
    const int S = blockDim.x;
    float* A = sh + threadIdx.x;
    const int n = P.n_lod;
    const int64_t npos = (int64_t)(P.M - 1) * n;
    const int64_t ntask = (int64_t)G * npos;
    for (int64_t t = (int64_t)blockIdx.x * S + threadIdx.x; t < ntask; t += (int64_t)gridDim.x * S) {
        const int b = (int)(t / npos);
        const int64_t pidx = t % npos;
        const int l = (int)(pidx / n), o = (int)(pidx % n);
        const uint32_t* colL = graphs + (size_t)b * graph_words + (size_t)l * P.W;
        const uint32_t* colR = colL + P.W;
        const float th = P.partial_f[l] * (float)(o + 1), an = 1.f - th;
        const float th2 = P.partial_f[l] * (float)(n - o), an2 = 1.f - th2;
        int scale = 0;
        float result = 0.f;
        const int32_t* pc = P.prog;
        while (true) {
            const int op = __ldg(pc);
            if (op == LI_CELL) {
                const int dst = __ldg(pc + 1), nt = __ldg(pc + 2);
                pc += 3;
                float total = 0.f;
                for (int q = 0; q < nt; ++q) {
                    const int nf = __ldg(pc);
                    float v = __ldg(P.pconst + __ldg(pc + 1));
                    pc += 2;
                    for (int f = 0; f < nf; ++f) v *= A[__ldg(pc + f) * S];
                    pc += nf;
                    total += v;
                }
                A[dst * S] = total;
            } else if (op == LI_REC) {
                const int child = __ldg(pc + 1), dst = __ldg(pc + 2);
                pc += 3;
                const int bits = person_bits(P, colL, colR, child);
                A[(dst + 0) * S] = 0.25f * trait_rec<float>(bits, 0, 0, th, an, th2, an2);
                A[(dst + 1) * S] = 0.25f * trait_rec<float>(bits, 0, 1, th, an, th2, an2);
                A[(dst + 2) * S] = 0.25f * trait_rec<float>(bits, 1, 0, th, an, th2, an2);
                A[(dst + 3) * S] = 0.25f * trait_rec<float>(bits, 1, 1, th, an, th2, an2);
            } else if (op == LI_SUM) {
                const int dst = __ldg(pc + 1), ns = __ldg(pc + 2);
                float v = 0.f;
                for (int q = 0; q < ns; ++q) v += A[__ldg(pc + 3 + q) * S];
                A[dst * S] = v;
                pc += 3 + ns;
            } else if (op == LI_SCALE) {
                const int first = __ldg(pc + 1), cnt = __ldg(pc + 2), target = __ldg(pc + 3);
                pc += 4;
                float mx = 0.f;
                for (int q = 0; q < cnt; ++q) mx = fmaxf(mx, A[(first + q) * S]);
                if (mx > 0.f) {
                    // ldexpf: exact for any exponent, a subnormal maximum included
                    const int e = ilogbf(mx) - target;
                    for (int q = 0; q < cnt; ++q) A[(first + q) * S] = ldexpf(A[(first + q) * S], -e);
                    scale += e;
                }
            } else {
                const int rs = __ldg(pc + 1);
                result = rs >= 0 ? A[rs * S] : 0.f;
                break;
            }
        }
        // DescentGraph::get_recombination_prob (descent_graph.cc:212-242) by crossover count
        int cross = 0;
        for (int w = 0; w < P.W; ++w) cross += __popc(colL[w] ^ colR[w]);
        const double rec = cross * P.log_theta[l] + (2 * P.Nnf - cross) * P.log_itheta[l];
        double v;
        if (!(result > 0.f)) {
            if (!P.lod_zero_ok) set_status(status, ST_LOD_NONPOS);
            v = -DBL_MAX;
        } else {
            // log of an FP32 value in FP32 (error ~1e-7, far inside the LOD tolerance)
            v = (double)logf(result) + (double)scale * 0.69314718055994530942 - rec - P.marker_trans;
        }
        vals[t] = v;
    }
}

// Adjoint of the trait peel (the reverse sum-product of TraitRfunction's
// peel, trait_rfunction.cc:28-137), one warp per (graph, interval, position)
// task with the rfunctions in the warp's shared memory, dense [4^c] per op
// (every cell and term kept: a zero disease probability still has a
// derivative with respect to the model).
//
// Forward: as the FP32 scorer, one (cell, term) item per lane -- a child
// peel's terms are its four transmissions (i, j), the others' the peel node's
// four states -- each rfunction scaled so its largest cell is 2^scale_to, the
// exponent kept.  Reverse: B[root] = 1 / root; op k's cell adjoint times
// 2^-e_k (its scaling) is spread over the item's factors: to each previous
// rfunction's cell (shared-memory atomics: cells of op k that differ only in
// members outside that cutset meet there), to the peel node's disease
// probability (its derivatives by the three penetrances and the frequency)
// and, through the children's recombination terms, to theta_L and theta_R.
// The exponents are constants of the pass, so working on scaled values gives
// d log L exactly.
//
// Memory (AdjDev): with one segment every matrix is kept from the forward
// pass (store).  When that does not fit the per-warp budget the ops are split
// into segments: the first forward pass keeps only matrices a later segment
// reads, and before each earlier segment's reverse pass its other matrices
// are recomputed from the kept ones (recompute instead of store; one extra
// forward pass).  graphs == nullptr peels without a graph (every
// recombination term 1/4, Peeler::calc_trait_prob): one task, no theta
// derivatives.  grad[task - task0][6] = d log L / d (theta_L, theta_R,
// pen x3, frequency), FP64.
constexpr int kAdjMaxPrev = 8;

struct AdjTask {
    const uint32_t* colL;
    const uint32_t* colR;
    float th, an, th2, an2;
    bool graph;
};

// 0.25 x the recombination term of (i, j) and its derivatives by theta_L and
// theta_R (TraitRfunction::get_recombination_probability, trait_rfunction.cc:9-24)
__device__ __forceinline__ void adj_rec(const AdjTask& T, int bits, int i, int j, float& r, float& dl, float& dr) {
    if (!T.graph) {
        r = 0.25f;
        dl = dr = 0.f;
        return;
    }
    const bool ml = (bits & 1) == i, mr = ((bits >> 2) & 1) == i;
    const bool pl = ((bits >> 1) & 1) == j, pr = ((bits >> 3) & 1) == j;
    const float x0 = ml ? T.an : T.th, x1 = mr ? T.an2 : T.th2, x2 = pl ? T.an : T.th, x3 = pr ? T.an2 : T.th2;
    const float s0 = ml ? -1.f : 1.f, s1 = mr ? -1.f : 1.f, s2 = pl ? -1.f : 1.f, s3 = pr ? -1.f : 1.f;
    r = 0.25f * (x0 * x1 * x2 * x3);
    dl = 0.25f * (s0 * x1 * x2 * x3 + x0 * x1 * s2 * x3);
    dr = 0.25f * (x0 * s1 * x2 * x3 + x0 * x1 * x2 * s3);
}

// Op k's recombination terms at this task, for a child peel its child's and
// for a parent peel each child's: for (i, j) = 2i + j, 0.25 x the term and its
// derivatives by theta_L and theta_R at rt[12 c + b], rt[12 c + 4 + b],
// rt[12 c + 8 + b] (the warp's scratch; its items read them).
__device__ __forceinline__ void adj_rtab(const ProblemDev& P, const AdjTask& T, const OpDev& op, float* rt, int lane) {
    const int nch = op.type == CHILD ? 1 : (op.type == PARENT ? op.n_child : 0);
    for (int q = lane; q < 4 * nch; q += 32) {
        const int c = q >> 2, b = q & 3;
        const int child = op.type == CHILD ? op.peel : P.opdata[op.child_at + 4 * c];
        const int bits = T.graph ? person_bits(P, T.colL, T.colR, child) : 0;
        float r, dl, dr;
        adj_rec(T, bits, b >> 1, b & 1, r, dl, dr);
        rt[12 * c + b] = r;
        rt[12 * c + 4 + b] = dl;
        rt[12 * c + 8 + b] = dr;
    }
    __syncwarp();
}

// Child c's transmission mask of an item of a parent peel (AdjDev::items).
__device__ __forceinline__ uint32_t adj_mask(const uint32_t* w, int pw, int c) {
    return c < 7 ? (w[0] >> (2 + 4 * c)) & 15u : (w[1 + pw + (c - 7) / 8] >> (4 * ((c - 7) % 8))) & 15u;
}

// The item's product of recombination factors (and, with D, its derivatives
// by theta_L and theta_R by the product rule as it is built): a child peel's
// one term, a parent peel's per-child sums of the transmissions its mask
// lets through, in transmission order.
template <bool D>
__device__ __forceinline__ void adj_R(const OpDev& op, const uint32_t* w, int pw, int t, const float* rt, float& R,
                                      float& dRl, float& dRr) {
    R = 1.f;
    dRl = dRr = 0.f;
    if (op.type == CHILD) {
        R = rt[t];
        if (D) {
            dRl = rt[4 + t];
            dRr = rt[8 + t];
        }
    } else if (op.type == PARENT) {
        for (int c = 0; c < op.n_child; ++c) {
            const uint32_t mask = adj_mask(w, pw, c);
            float sc = 0.f, sl = 0.f, sr = 0.f;
#pragma unroll
            for (int b = 0; b < 4; ++b)
                if (mask & (1u << b)) {
                    sc += rt[12 * c + b];
                    if (D) {
                        sl += rt[12 * c + 4 + b];
                        sr += rt[12 * c + 8 + b];
                    }
                }
            if (D) {
                dRl = dRl * sc + R * sl;
                dRr = dRr * sc + R * sr;
            }
            R *= sc;
        }
    }
}

// 2^-e as a float multiplier when it is a normal number (the op's scaling,
// exact), else 0 (the caller then scales with ldexpf).
__device__ __forceinline__ float adj_pow2(int e) {
    return (e >= -127 && e <= 126) ? __int_as_float((127 - e) << 23) : 0.f;
}

// Forward of op k: its scaled matrix in A, its exponent in E[k].  One item
// per lane: the peel node's disease probability times the previous
// rfunctions' cells times the recombination factors; the four items of a
// cell added by shuffles.
__device__ void adj_forward(const ProblemDev& P, const AdjDev& D, const AdjTask& T, int k, float* A, int* E, float* rt,
                            int lane) {
    const OpDev op = P.ops[k];
    adj_rtab(P, T, op, rt, lane);
    const int ncell = 1 << (2 * op.c), nitem = 4 * ncell;
    const int nw = adj_item_words(op.n_prev, op.n_child), pw = (op.n_prev + 1) / 2;
    const uint32_t* tab = D.items + D.item_at[k];
    float* out = A + D.aoff[k];
    const float* dp = D.dprob + 4 * op.peel;
    float mx = 0.f;
    for (int it0 = 0; it0 < nitem; it0 += 32) {
        const int item = it0 + lane, cell = item >> 2, t = item & 3;
        float term = 0.f;
        if (item < nitem) {
            const uint32_t* w = tab + (size_t)item * nw;
            term = dp[w[0] & 3u];
            for (int j = 0; j < op.n_prev; ++j) term *= A[(w[1 + (j >> 1)] >> (16 * (j & 1))) & 0xffffu];
            float R, dl, dr;
            adj_R<false>(op, w, pw, t, rt, R, dl, dr);
            term *= R;
        }
        const int grp = lane & ~3;
        const float t0 = __shfl_sync(FULLMASK, term, grp), t1 = __shfl_sync(FULLMASK, term, grp + 1);
        const float t2 = __shfl_sync(FULLMASK, term, grp + 2), t3 = __shfl_sync(FULLMASK, term, grp + 3);
        if (t == 0 && item < nitem) {
            const float total = ((t0 + t1) + t2) + t3;
            out[cell] = total;
            mx = fmaxf(mx, total);
        }
    }
    for (int dd = 16; dd >= 1; dd >>= 1) mx = fmaxf(mx, __shfl_xor_sync(FULLMASK, mx, dd));
    const int e = mx > 0.f ? ilogbf(mx) - op.scale_to : 0;
    const float sc = adj_pow2(e);
    __syncwarp();
    for (int cell = lane; cell < ncell; cell += 32) out[cell] = sc != 0.f ? out[cell] * sc : ldexpf(out[cell], -e);
    if (lane == 0) E[k] = e;
    __syncwarp();
}

// The items of op k in the reverse pass, NP previous rfunctions (unrolled).
template <int NP>
__device__ __forceinline__ void adj_reverse_items(const OpDev& op, const uint32_t* tab, int nw, int pw, int nitem,
                                                  const float* bk, int e, const float* A, float* B, const float* dp,
                                                  const float4* dg, const float* rt, int lane, float* acc) {
    const float sc = adj_pow2(e);
    float gl = 0.f, gr = 0.f, g0 = 0.f, g1 = 0.f, g2 = 0.f, g3 = 0.f;
    for (int it0 = 0; it0 < nitem; it0 += 32) {
        const int item = it0 + lane, cell = item >> 2, t = item & 3;
        if (item >= nitem) break;
        const float gd = sc != 0.f ? bk[cell] * sc : ldexpf(bk[cell], -e);   // the cell's adjoint before its scaling
        if (gd == 0.f) continue;
        const uint32_t* w = tab + (size_t)item * nw;
        const int s = (int)(w[0] & 3u);
        float a[NP > 0 ? NP : 1];
        int off[NP > 0 ? NP : 1];
        float pp = 1.f;
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            off[j] = (int)((w[1 + (j >> 1)] >> (16 * (j & 1))) & 0xffffu);
            a[j] = A[off[j]];
            pp *= a[j];
        }
        float R, dRl, dRr;
        adj_R<true>(op, w, pw, t, rt, R, dRl, dRr);
        const float c = dp[s];
        const float wgt = gd * pp;
        const float4 dc = dg[s];
        g0 += wgt * R * dc.x;
        g1 += wgt * R * dc.y;
        g2 += wgt * R * dc.z;
        g3 += wgt * R * dc.w;
        gl += wgt * c * dRl;
        gr += wgt * c * dRr;
        // each factor's adjoint: the product of the others, by prefix and suffix products
        float pre[NP > 0 ? NP : 1];
        float run = gd * c * R;
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            pre[j] = run;
            run *= a[j];
        }
        float suf = 1.f;
#pragma unroll
        for (int j = NP - 1; j >= 0; --j) {
            const float v = pre[j] * suf;
            if (v != 0.f) atomicAdd(B + off[j], v);
            suf *= a[j];
        }
    }
    acc[0] += gl;
    acc[1] += gr;
    acc[2] += g0;
    acc[3] += g1;
    acc[4] += g2;
    acc[5] += g3;
}

// Reverse of op k: adjoints into the previous rfunctions' cells (B), the
// model derivatives into g.
__device__ void adj_reverse(const ProblemDev& P, const AdjDev& D, const AdjTask& T, int k, const float* A, float* B,
                            const int* E, float* rt, int lane, double* g) {
    const OpDev op = P.ops[k];
    adj_rtab(P, T, op, rt, lane);
    const int ncell = 1 << (2 * op.c), nitem = 4 * ncell;
    const int nw = adj_item_words(op.n_prev, op.n_child), pw = (op.n_prev + 1) / 2;
    const uint32_t* tab = D.items + D.item_at[k];
    const float* bk = B + D.aoff[k];
    const float* dp = D.dprob + 4 * op.peel;
    const float4* dg = D.dgrad + 4 * op.peel;
    const int e = E[k];
    float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    switch (op.n_prev) {
#define SL_ADJ_NP(n) \
        case n: adj_reverse_items<n>(op, tab, nw, pw, nitem, bk, e, A, B, dp, dg, rt, lane, acc); break;
        SL_ADJ_NP(0) SL_ADJ_NP(1) SL_ADJ_NP(2) SL_ADJ_NP(3) SL_ADJ_NP(4)
        SL_ADJ_NP(5) SL_ADJ_NP(6) SL_ADJ_NP(7) SL_ADJ_NP(8)
#undef SL_ADJ_NP
        default: break;
    }
    for (int q = 0; q < 6; ++q) g[q] += (double)acc[q];
    __syncwarp();
}

__global__ void __launch_bounds__(128) trait_adjoint_kernel(ProblemDev P, AdjDev D, const uint32_t* graphs,
                                                            int64_t graph_words, int64_t task0, int64_t ntask,
                                                            double* grad, int* status) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int wpb = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* A = (float*)(smem + (size_t)warp * D.warp_bytes);
    float* B = A + D.half;
    int* E = (int*)(B + D.half);
    float* rt = (float*)(E + P.K);   // [12 max_child] the op's recombination terms
    const int n = P.n_lod;
    const int64_t npos = (int64_t)(P.M - 1) * n;
    for (int64_t u = (int64_t)blockIdx.x * wpb + warp; u < ntask; u += (int64_t)gridDim.x * wpb) {
        const int64_t t = task0 + u;
        AdjTask T;
        T.graph = graphs != nullptr;
        T.colL = T.colR = nullptr;
        T.th = T.an = T.th2 = T.an2 = 0.f;
        if (T.graph) {
            const int b = (int)(t / npos);
            const int64_t pidx = t % npos;
            const int l = (int)(pidx / n), o = (int)(pidx % n);
            T.colL = graphs + (size_t)b * graph_words + (size_t)l * P.W;
            T.colR = T.colL + P.W;
            T.th = P.partial_f[l] * (float)(o + 1);
            T.an = 1.f - T.th;
            T.th2 = P.partial_f[l] * (float)(n - o);
            T.an2 = 1.f - T.th2;
        }
        // first forward pass: every op; matrices not kept are overwritten by later segments
        for (int k = 0; k < P.K; ++k) adj_forward(P, D, T, k, A, E, rt, lane);
        const float root = A[D.aoff[P.K - 1]];
        double g[6] = {0, 0, 0, 0, 0, 0};
        if (!(root > 0.f)) {
            if (lane == 0) {
                if (!P.lod_zero_ok) set_status(status, ST_LOD_NONPOS);
                for (int q = 0; q < 6; ++q) grad[u * 6 + q] = __longlong_as_double(0x7ff8000000000000LL);   // NaN
            }
            __syncwarp();
            continue;
        }
        for (int i = lane; i < D.half; i += 32) B[i] = 0.f;
        __syncwarp();
        for (int sg = D.nseg - 1; sg >= 0; --sg) {
            const int k0 = D.seg[sg], k1 = D.seg[sg + 1];
            if (sg < D.nseg - 1) {
                // recompute the segment's matrices that were not kept, zero their adjoints
                for (int k = k0; k < k1; ++k)
                    if (!D.keep[k]) adj_forward(P, D, T, k, A, E, rt, lane);
                for (int k = k0; k < k1; ++k)
                    if (!D.keep[k])
                        for (int i = lane; i < (1 << (2 * P.ops[k].c)); i += 32) B[D.aoff[k] + i] = 0.f;
                __syncwarp();
            } else if (lane == 0) {
                B[D.aoff[P.K - 1]] = 1.0f / root;
            }
            __syncwarp();
            for (int k = k1 - 1; k >= k0; --k) adj_reverse(P, D, T, k, A, B, E, rt, lane, g);
        }
        for (int q = 0; q < 6; ++q) {
            double v = g[q];
            for (int dd = 16; dd >= 1; dd >>= 1) v += __shfl_xor_sync(FULLMASK, v, dd);
            if (lane == 0) grad[u * 6 + q] = v;
        }
        __syncwarp();
    }
}

// The same adjoint with one thread per task: each thread's matrices and
// adjoints live in global memory, a column of the arena per resident thread
// (float offset o of thread r at o * nthr + r, so the threads of a warp, all
// at the same item, touch one 128-byte line), and every item of an op is the
// thread's own serial loop, so small rfunctions leave no lane idle and the
// adjoints need no atomics.  Matrices are stored unscaled with their
// exponents; a factor is scaled as it is read, which gives the scaled form's
// values exactly.  Same plan (offsets, segments, kept matrices) and item
// tables as the warp form.
struct AdjThr {
    float* A;       // arena base of this thread: A[o * nthr]
    float* B;       // adjoints: B[o * nthr]
    int* E;         // exponents: E[k * nthr]
    int64_t nthr;
};

// The thread's recombination terms of op k, rt[12 c + b] as in adj_rtab.
__device__ __forceinline__ void adj_rtab_thr(const ProblemDev& P, const AdjTask& T, const OpDev& op, float* rt) {
    const int nch = op.type == CHILD ? 1 : (op.type == PARENT ? op.n_child : 0);
    for (int c = 0; c < nch; ++c) {
        const int child = op.type == CHILD ? op.peel : P.opdata[op.child_at + 4 * c];
        const int bits = T.graph ? person_bits(P, T.colL, T.colR, child) : 0;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            float r, dl, dr;
            adj_rec(T, bits, b >> 1, b & 1, r, dl, dr);
            rt[12 * c + b] = r;
            rt[12 * c + 4 + b] = dl;
            rt[12 * c + 8 + b] = dr;
        }
    }
}

// Factor j's scale and exponent for op k's previous rfunctions.
__device__ __forceinline__ void adj_prev_scales(const ProblemDev& P, const AdjThr& R, const OpDev& op, float* sj,
                                                int* ej) {
    const int32_t* po = P.opdata + op.prev_ops_at;
    for (int j = 0; j < op.n_prev; ++j) {
        ej[j] = R.E[(int64_t)po[j] * R.nthr];
        sj[j] = adj_pow2(ej[j]);
    }
}

__device__ __forceinline__ float adj_scaled(float v, float sc, int e) { return sc != 0.f ? v * sc : ldexpf(v, -e); }

__device__ void adj_forward_thr(const ProblemDev& P, const AdjDev& D, const AdjTask& T, const AdjThr& R, int k,
                                float* rt) {
    const OpDev op = P.ops[k];
    adj_rtab_thr(P, T, op, rt);
    float sj[kAdjMaxPrev];
    int ej[kAdjMaxPrev];
    adj_prev_scales(P, R, op, sj, ej);
    const int ncell = 1 << (2 * op.c);
    const int nw = adj_item_words(op.n_prev, op.n_child), pw = (op.n_prev + 1) / 2;
    const uint32_t* tab = D.items + D.item_at[k];
    float* out = R.A + (int64_t)D.aoff[k] * R.nthr;
    const float* dp = D.dprob + 4 * op.peel;
    float mx = 0.f;
    for (int cell = 0; cell < ncell; ++cell) {
        float tv[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const uint32_t* w = tab + (size_t)(4 * cell + t) * nw;
            float term = dp[w[0] & 3u];
            for (int j = 0; j < op.n_prev; ++j) {
                const int off = (int)((w[1 + (j >> 1)] >> (16 * (j & 1))) & 0xffffu);
                term *= adj_scaled(R.A[(int64_t)off * R.nthr], sj[j], ej[j]);
            }
            float Rr, dl, dr;
            adj_R<false>(op, w, pw, t, rt, Rr, dl, dr);
            tv[t] = term * Rr;
        }
        const float total = ((tv[0] + tv[1]) + tv[2]) + tv[3];
        out[(int64_t)cell * R.nthr] = total;
        mx = fmaxf(mx, total);
    }
    R.E[(int64_t)k * R.nthr] = mx > 0.f ? ilogbf(mx) - op.scale_to : 0;
}

template <int NP>
__device__ __forceinline__ void adj_reverse_thr_items(const OpDev& op, const uint32_t* tab, int nw, int pw, int ncell,
                                                      const AdjThr& R, const float* bk, float sk, int ek,
                                                      const float* sj, const int* ej, const float* dp,
                                                      const float4* dg, const float* rt, float* acc) {
    float gl = 0.f, gr = 0.f, g0 = 0.f, g1 = 0.f, g2 = 0.f, g3 = 0.f;
    for (int cell = 0; cell < ncell; ++cell) {
        const float gd = adj_scaled(bk[(int64_t)cell * R.nthr], sk, ek);   // the cell's adjoint before its scaling
        if (gd == 0.f) continue;
#pragma unroll 1
        for (int t = 0; t < 4; ++t) {
            const uint32_t* w = tab + (size_t)(4 * cell + t) * nw;
            const int s = (int)(w[0] & 3u);
            float a[NP > 0 ? NP : 1];
            int off[NP > 0 ? NP : 1];
            float pp = 1.f;
#pragma unroll
            for (int j = 0; j < NP; ++j) {
                off[j] = (int)((w[1 + (j >> 1)] >> (16 * (j & 1))) & 0xffffu);
                a[j] = adj_scaled(R.A[(int64_t)off[j] * R.nthr], sj[j], ej[j]);
                pp *= a[j];
            }
            float Rr, dRl, dRr;
            adj_R<true>(op, w, pw, t, rt, Rr, dRl, dRr);
            const float c = dp[s];
            const float wgt = gd * pp;
            const float4 dc = dg[s];
            g0 += wgt * Rr * dc.x;
            g1 += wgt * Rr * dc.y;
            g2 += wgt * Rr * dc.z;
            g3 += wgt * Rr * dc.w;
            gl += wgt * c * dRl;
            gr += wgt * c * dRr;
            float pre[NP > 0 ? NP : 1];
            float run = gd * c * Rr;
#pragma unroll
            for (int j = 0; j < NP; ++j) {
                pre[j] = run;
                run *= a[j];
            }
            float suf = 1.f;
#pragma unroll
            for (int j = NP - 1; j >= 0; --j) {
                const float v = pre[j] * suf;
                if (v != 0.f) R.B[(int64_t)off[j] * R.nthr] += v;
                suf *= a[j];
            }
        }
    }
    acc[0] += gl;
    acc[1] += gr;
    acc[2] += g0;
    acc[3] += g1;
    acc[4] += g2;
    acc[5] += g3;
}

__device__ void adj_reverse_thr(const ProblemDev& P, const AdjDev& D, const AdjTask& T, const AdjThr& R, int k,
                                float* rt, double* g) {
    const OpDev op = P.ops[k];
    adj_rtab_thr(P, T, op, rt);
    float sj[kAdjMaxPrev];
    int ej[kAdjMaxPrev];
    adj_prev_scales(P, R, op, sj, ej);
    const int ncell = 1 << (2 * op.c);
    const int nw = adj_item_words(op.n_prev, op.n_child), pw = (op.n_prev + 1) / 2;
    const uint32_t* tab = D.items + D.item_at[k];
    const float* bk = R.B + (int64_t)D.aoff[k] * R.nthr;
    const int ek = R.E[(int64_t)k * R.nthr];
    const float sk = adj_pow2(ek);
    const float* dp = D.dprob + 4 * op.peel;
    const float4* dg = D.dgrad + 4 * op.peel;
    float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    switch (op.n_prev) {
#define SL_ADJ_NP(n) \
        case n: adj_reverse_thr_items<n>(op, tab, nw, pw, ncell, R, bk, sk, ek, sj, ej, dp, dg, rt, acc); break;
        SL_ADJ_NP(0) SL_ADJ_NP(1) SL_ADJ_NP(2) SL_ADJ_NP(3) SL_ADJ_NP(4)
        SL_ADJ_NP(5) SL_ADJ_NP(6) SL_ADJ_NP(7) SL_ADJ_NP(8)
#undef SL_ADJ_NP
        default: break;
    }
    for (int q = 0; q < 6; ++q) g[q] += (double)acc[q];
}

__global__ void __launch_bounds__(128, 6) trait_adjoint_thr_kernel(ProblemDev P, AdjDev D, const uint32_t* graphs,
                                                                int64_t graph_words, int64_t task0, int64_t ntask,
                                                                double* grad, int* status, float* arena, int* expo) {
    const int64_t nthr = (int64_t)gridDim.x * blockDim.x;
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    AdjThr R;
    R.nthr = nthr;
    R.A = arena + r;
    R.B = arena + (int64_t)D.half * nthr + r;
    R.E = expo + r;
    float rt[12 * 32];   // the op's recombination terms (local memory)
    const int n = P.n_lod;
    const int64_t npos = (int64_t)(P.M - 1) * n;
    for (int64_t u = r; u < ntask; u += nthr) {
        const int64_t t = task0 + u;
        AdjTask T;
        T.graph = graphs != nullptr;
        T.colL = T.colR = nullptr;
        T.th = T.an = T.th2 = T.an2 = 0.f;
        if (T.graph) {
            const int b = (int)(t / npos);
            const int64_t pidx = t % npos;
            const int l = (int)(pidx / n), o = (int)(pidx % n);
            T.colL = graphs + (size_t)b * graph_words + (size_t)l * P.W;
            T.colR = T.colL + P.W;
            T.th = P.partial_f[l] * (float)(o + 1);
            T.an = 1.f - T.th;
            T.th2 = P.partial_f[l] * (float)(n - o);
            T.an2 = 1.f - T.th2;
        }
        for (int k = 0; k < P.K; ++k) adj_forward_thr(P, D, T, R, k, rt);
        const int kr = P.K - 1;
        const int er = R.E[(int64_t)kr * nthr];
        const float root = adj_scaled(R.A[(int64_t)D.aoff[kr] * nthr], adj_pow2(er), er);
        double g[6] = {0, 0, 0, 0, 0, 0};
        if (!(root > 0.f)) {
            if (!P.lod_zero_ok) set_status(status, ST_LOD_NONPOS);
            for (int q = 0; q < 6; ++q) grad[u * 6 + q] = __longlong_as_double(0x7ff8000000000000LL);   // NaN
            continue;
        }
        for (int i = 0; i < D.half; ++i) R.B[(int64_t)i * nthr] = 0.f;
        for (int sg = D.nseg - 1; sg >= 0; --sg) {
            const int k0 = D.seg[sg], k1 = D.seg[sg + 1];
            if (sg < D.nseg - 1) {
                // recompute the segment's matrices that were not kept, zero their adjoints
                for (int k = k0; k < k1; ++k)
                    if (!D.keep[k]) adj_forward_thr(P, D, T, R, k, rt);
                for (int k = k0; k < k1; ++k)
                    if (!D.keep[k])
                        for (int i = 0; i < (1 << (2 * P.ops[k].c)); ++i) R.B[(int64_t)(D.aoff[k] + i) * nthr] = 0.f;
            } else {
                R.B[(int64_t)D.aoff[kr] * nthr] = 1.0f / root;
            }
            for (int k = k1 - 1; k >= k0; --k) adj_reverse_thr(P, D, T, R, k, rt, g);
        }
        for (int q = 0; q < 6; ++q) grad[u * 6 + q] = g[q];
    }
}

// log_sum (logarithms.cc:14-25)
__device__ __forceinline__ double log_sum(double a, double b) {
    if (a == -DBL_MAX) return b;
    if (b == -DBL_MAX) return a;
    return log(exp(b - a) + 1.0) + a;
}

// LODscores::add in graph order (lod_score.h:74-80)
__global__ void lod_merge_kernel(const double* vals, int G, int64_t npos, double* acc, uint8_t* init) {
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < npos; p += (int64_t)gridDim.x * blockDim.x) {
        double a = acc[p];
        uint8_t ini = init ? init[p] : 1;   // without flags, acc starts at -DBL_MAX
        for (int b = 0; b < G; ++b) {
            const double v = vals[(size_t)b * npos + p];
            a = ini ? log_sum(v, a) : v;
            ini = 1;
        }
        acc[p] = a;
        if (init) init[p] = ini;
    }
}

// Per-chain shuffled meiosis order for device-driven M-sweeps (the reference
// shuffles m_ordering each sweep, markov_chain.cc:346): Fisher-Yates with
// Philox draws.
__global__ void shuffle_kernel(const int32_t* base, int nm, int32_t* out, int first, int nchain, uint64_t seed,
                               uint64_t iter) {
    const int cr = blockIdx.x * blockDim.x + threadIdx.x;
    if (cr >= nchain) return;
    const int chain = first + cr;
    int32_t* o = out + (size_t)cr * nm;
    for (int i = 0; i < nm; ++i) o[i] = base[i];
    const uint64_t hi = ((uint64_t)chain << 40) ^ (iter << 4) ^ 3u;
    for (int i = nm - 1; i > 0; --i) {
        const double u = philox_u01(seed, hi, (uint64_t)i);
        int j = (int)(u * (double)(i + 1));
        if (j > i) j = i;
        const int32_t t = o[i];
        o[i] = o[j];
        o[j] = t;
    }
}

// One uniform per chain decides L- or M-sweep (markov_chain.cc:336-352).
__global__ void choose_kernel(int first, int nchain, uint64_t seed, uint64_t iter, double lprob, uint8_t* is_l) {
    const int cr = blockIdx.x * blockDim.x + threadIdx.x;
    if (cr >= nchain) return;
    const uint64_t hi = ((uint64_t)(first + cr) << 40) ^ (iter << 4) ^ 7u;
    is_l[cr] = philox_u01(seed, hi, 0) < lprob ? 1 : 0;
}

// ---------------------------------------------------------------------------
// Parts of log P(G, graph) under a chain's map (DescentGraph::get_likelihood,
// descent_graph.cc:184-269), for up to four (graph chain, map chain) pairs:
// the founder-allele-graph likelihood of every locus (exact FP64, as the
// M-sampler's) and the recombination log-probability of every interval, each
// a sum in the reference's order; the host adds them up in order.
// ---------------------------------------------------------------------------
template <typename IX>
__global__ void __launch_bounds__(128) loglik_fag_kernel(ProblemDev P, const uint32_t* dg, int4 gch, int4 tch,
                                                         int npair, double* out, const Mc3Dev* m) {
    if (m) {   // the pairs of the device-side exchange, if one is due
        if (!m->active) return;
        gch = make_int4(m->gch[0], m->gch[1], m->gch[2], m->gch[3]);
        tch = make_int4(m->tch[0], m->tch[1], m->tch[2], m->tch[3]);
    }
    extern __shared__ __align__(16) unsigned char smem[];
    const int S = blockDim.x;
    const size_t per = fag_block_bytes(P.N, P.F, S, 0) - (((size_t)P.N * 7 + 15) & ~(size_t)15);
    int16_t* s_order = (int16_t*)(smem + per);
    int16_t* s_mo = s_order + P.N;
    int16_t* s_fa = s_mo + P.N;
    uint8_t* s_typed = (uint8_t*)(s_fa + P.N);
    for (int i = threadIdx.x; i < P.N; i += S) {
        s_order[i] = P.fag_order[i];
        s_mo[i] = P.mother[i];
        s_fa[i] = P.father[i];
        s_typed[i] = P.typed[i];
    }
    __syncthreads();
    Fag<IX, double> fs = fag_bind<IX, double>(smem, P.N, P.F, S, threadIdx.x);
    const int64_t t = (int64_t)blockIdx.x * S + threadIdx.x;
    if (t >= (int64_t)npair * P.M) return;
    const int k = (int)(t / P.M), l = (int)(t % P.M);
    const int g = k == 0 ? gch.x : k == 1 ? gch.y : k == 2 ? gch.z : gch.w;
    const int tc = k == 0 ? tch.x : k == 1 ? tch.y : k == 2 ? tch.z : tch.w;
    const uint32_t* col = dg + ((size_t)g * P.M + l) * P.W;
    fag_edges(P.N, P.F, s_order, s_mo, s_fa, col, fs, -1);
    out[t] = fag_like<ProbExact>(P.N, P.F, s_typed, P.geno + (size_t)l * P.N, P.c_minor[(size_t)tc * P.M + l], fs);
}

__global__ void loglik_rec_kernel(ProblemDev P, const uint32_t* dg, int4 gch, int4 tch, int npair, double* out,
                                  const Mc3Dev* m) {
    if (m) {
        if (!m->active) return;
        gch = make_int4(m->gch[0], m->gch[1], m->gch[2], m->gch[3]);
        tch = make_int4(m->tch[0], m->tch[1], m->tch[2], m->tch[3]);
    }
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int I = P.M - 1;
    if (t >= (int64_t)npair * I) return;
    const int k = (int)(t / I), l = (int)(t % I);
    const int g = k == 0 ? gch.x : k == 1 ? gch.y : k == 2 ? gch.z : gch.w;
    const int tc = k == 0 ? tch.x : k == 1 ? tch.y : k == 2 ? tch.z : tch.w;
    const uint32_t* colL = dg + ((size_t)g * P.M + l) * P.W;
    const uint32_t* colR = colL + P.W;
    const double lt = P.c_log_theta[(size_t)tc * I + l], la = P.c_log_itheta[(size_t)tc * I + l];
    double r = 0.0;
    for (int b = 0; b < 2 * P.Nnf; ++b) r = DADD(r, dgbit(colL, b) != dgbit(colR, b) ? lt : la);
    out[t] = r;
}

// Exchange two chains' descent graphs.
__global__ void swap_graphs_kernel(uint32_t* dg, size_t words, int a, int b) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t x = dg[(size_t)a * words + i];
        dg[(size_t)a * words + i] = dg[(size_t)b * words + i];
        dg[(size_t)b * words + i] = x;
    }
}

cudaError_t launch_loglik_parts(const ProblemDev& P, const uint32_t* dg, const int* gch, const int* tch, int npair,
                                double* fag_out, double* rec_out, cudaStream_t s, const Mc3Dev* m) {
    const int S = 64;
    const size_t smem = fag_block_bytes(P.N, P.F, S, 0);
    const int wide = 2 * P.F > 255 ? 1 : 0;
    {
        cudaError_t e = ensure_smem(wide ? (const void*)loglik_fag_kernel<uint16_t> : (const void*)loglik_fag_kernel<uint8_t>,
                                    smem);
        if (e != cudaSuccess) return e;
    }
    const int4 g4 = gch ? make_int4(gch[0], gch[1], gch[2], gch[3]) : make_int4(0, 0, 0, 0);
    const int4 t4 = tch ? make_int4(tch[0], tch[1], tch[2], tch[3]) : make_int4(0, 0, 0, 0);
    const int64_t nf = (int64_t)npair * P.M;
    if (wide)
        loglik_fag_kernel<uint16_t><<<(int)((nf + S - 1) / S), S, smem, s>>>(P, dg, g4, t4, npair, fag_out, m);
    else
        loglik_fag_kernel<uint8_t><<<(int)((nf + S - 1) / S), S, smem, s>>>(P, dg, g4, t4, npair, fag_out, m);
    const int64_t nr = (int64_t)npair * (P.M - 1);
    loglik_rec_kernel<<<(int)((nr + 127) / 128), 128, 0, s>>>(P, dg, g4, t4, npair, rec_out, m);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// MC3 exchanges on the device (Mc3::run, mc3.cc:117-158).  After a spurt that
// ends on a multiple of the exchange period, a uniformly chosen adjacent pair
// (r, r + 1) swaps graphs with probability min(1, exp((xy + yx) - (xx + yy))),
// the four log-likelihoods of DescentGraph::get_likelihood2 (descent_graph.cc:
// 184-269).  Both uniforms come from the Philox stream: stage 9, counter high
// word (0x3ff << 40) ^ (spurt end << 4), draws 0 and 1.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t mc3_hi(int64_t it_end) {
    return (0x3ffull << 40) ^ ((uint64_t)it_end << 4) ^ 9u;
}

// The proposal after the spurt ending at it_end (rp->end when rp is given;
// one thread).
__global__ void mc3_pick_kernel(Mc3Dev* m, const RunParams* rp, int64_t it_end, int C) {
    if (rp) it_end = rp->end;
    m->it_end = it_end;
    m->active = (C >= 2 && m->period > 0 && it_end % m->period == 0) ? 1 : 0;
    if (!m->active) return;
    int r = (int)((C - 1) * philox_u01(m->seed, mc3_hi(it_end), 0));
    if (r > C - 2) r = C - 2;
    m->r = r;
    const int g[4] = {r, r + 1, r + 1, r}, t[4] = {r, r + 1, r, r + 1};   // xx, yy, xy, yx
    for (int k = 0; k < 4; ++k) {
        m->gch[k] = g[k];
        m->tch[k] = t[k];
    }
}

// The decision (one block of 256): each pair's log-likelihood from its parts
// in the reference's order -- the interval log-probabilities added from 0.0,
// marker transmission first, then the log of every locus's founder-allele-graph
// likelihood (LOG_ZERO = -DBL_MAX for an illegal graph), joined by log_product
// (descent_graph.cc:184-269, logarithms.cc:27-29) -- the acceptance, the swap
// and the counts.  The logs are taken in parallel (in place); one thread per
// pair then sums in order.
__global__ void __launch_bounds__(256) mc3_decide_kernel(Mc3Dev* m, int M, double marker_trans, double* fag,
                                                         const double* rec, uint32_t* dg, size_t words,
                                                         int64_t* accept, int64_t* propose) {
    __shared__ int s_zero[4];
    __shared__ double s_ll[4];
    __shared__ int s_acc;
    if (!m->active) return;
    const int tid = threadIdx.x;
    if (tid < 4) s_zero[tid] = 0;
    __syncthreads();
    for (int i = tid; i < 4 * M; i += 256) {
        const double f = fag[i];
        if (f == 0.0) atomicOr(&s_zero[i / M], 1);
        else fag[i] = log(f);
    }
    __syncthreads();
    if (tid < 4) {
        const double LOG_ZERO = -DBL_MAX;
        double r = 0.0;
        const double* rk = rec + (size_t)tid * (M - 1);
        for (int l = 0; l < M - 1; ++l) r += rk[l];
        const double trans = marker_trans + r;
        double prior = 0.0;
        if (s_zero[tid]) {
            prior = LOG_ZERO;
        } else {
            const double* fk = fag + (size_t)tid * M;
            for (int l = 0; l < M; ++l) prior += fk[l];
        }
        s_ll[tid] = (trans == LOG_ZERO || prior == LOG_ZERO) ? LOG_ZERO : trans + prior;
    }
    __syncthreads();
    if (tid == 0) {
        const double ratio = (s_ll[2] + s_ll[3]) - (s_ll[0] + s_ll[1]);
        const double u = philox_u01(m->seed, mc3_hi(m->it_end), 1);
        const int r = m->r;
        propose[r] += 1;
        s_acc = (u == 0.0 || log(u) < fmin(0.0, ratio)) ? 1 : 0;
        if (s_acc) accept[r] += 1;
    }
    __syncthreads();
    if (s_acc) {
        uint32_t* a = dg + (size_t)m->r * words;
        uint32_t* b = a + words;
        for (size_t i = tid; i < words; i += 256) {
            const uint32_t x = a[i];
            a[i] = b[i];
            b[i] = x;
        }
    }
}

// The persistent MC3 run's spurt bounds: the next spurt [next, end) into the
// run parameters (one thread, first node of the outer loop's body).
__global__ void mc3_begin_kernel(Mc3Dev* m, RunParams* rp) {
    const int64_t it0 = m->next;
    int64_t it1 = m->period > 0 ? (it0 / m->period + 1) * m->period : m->total;
    if (it1 > m->total) it1 = m->total;
    rp->first = it0;
    rp->end = it1;
}

// After the spurt and its exchange: the next spurt, and (set) whether the
// outer loop runs again.
__global__ void mc3_end_kernel(Mc3Dev* m, const RunParams* rp, cudaGraphConditionalHandle h, int set) {
    m->next = rp->end;
    if (set) cudaGraphSetConditional(h, m->next < m->total ? 1u : 0u);
}

cudaError_t launch_mc3_exchange(const ProblemDev& P, Mc3Dev* m, const RunParams* rp, int64_t it_end, int C,
                                uint32_t* dg, double* fag, double* rec, int64_t* accept, int64_t* propose,
                                cudaStream_t s) {
    mc3_pick_kernel<<<1, 1, 0, s>>>(m, rp, it_end, C);
    cudaError_t e = launch_loglik_parts(P, dg, nullptr, nullptr, 4, fag, rec, s, m);
    if (e != cudaSuccess) return e;
    mc3_decide_kernel<<<1, 256, 0, s>>>(m, P.M, P.marker_trans, fag, rec, dg, (size_t)P.M * P.W, accept, propose);
    return cudaGetLastError();
}

// Set conditional handles of the graph this kernel is a node of (up to 64 per launch).
struct CondSet {
    cudaGraphConditionalHandle h[64];
    int n;
    unsigned v;
};

__global__ void cond_set_kernel(CondSet cs) {
    if ((int)threadIdx.x < cs.n) cudaGraphSetConditional(cs.h[threadIdx.x], cs.v);
}

cudaError_t launch_cond_set(const cudaGraphConditionalHandle* h, int n, unsigned v, cudaStream_t s) {
    for (int i = 0; i < n; i += 64) {
        CondSet cs;
        cs.n = n - i < 64 ? n - i : 64;
        cs.v = v;
        for (int k = 0; k < cs.n; ++k) cs.h[k] = h[i + k];
        cond_set_kernel<<<1, 64, 0, s>>>(cs);
    }
    return cudaGetLastError();
}

cudaError_t launch_mc3_begin(Mc3Dev* m, RunParams* rp, cudaStream_t s) {
    mc3_begin_kernel<<<1, 1, 0, s>>>(m, rp);
    return cudaGetLastError();
}

cudaError_t launch_mc3_end(Mc3Dev* m, const RunParams* rp, cudaGraphConditionalHandle h, int set, cudaStream_t s) {
    mc3_end_kernel<<<1, 1, 0, s>>>(m, rp, h, set);
    return cudaGetLastError();
}

cudaError_t launch_swap_graphs(uint32_t* dg, size_t words, int a, int b, cudaStream_t s) {
    int64_t grid = (int64_t)((words + 255) / 256);
    if (grid > 1024) grid = 1024;
    swap_graphs_kernel<<<(int)grid, 256, 0, s>>>(dg, words, a, b);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Kernels of the run graph: every chain iterates on its own inside a WHILE
// node (MarkovChain::run, markov_chain.cc:335-392, per replicate chain).
// ---------------------------------------------------------------------------
__global__ void run_init_kernel(const RunParams* rp, int64_t* it, int C) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < C) it[c] = rp->first;
}

// Start of an iteration of chain c: the L/M choice (the same draw as
// choose_kernel), the meiosis order of an M-sweep (the same draws and swaps as
// shuffle_kernel, the uniforms generated by the warp), the chain's Philox key
// and whether the iteration scores.  One warp.
__global__ void chain_iter_kernel(const RunParams* rp, const int64_t* it_arr, int c, uint64_t* key,
                                  const int32_t* base, int nm, int32_t* order, const double* temp,
                                  cudaGraphConditionalHandle hsw, cudaGraphConditionalHandle hscore) {
    extern __shared__ double su[];
    const int lane = threadIdx.x;
    const int64_t it = it_arr[c];
    if (it >= rp->end) {
        if (lane == 0) {
            cudaGraphSetConditional(hsw, 2);   // neither sweep
            cudaGraphSetConditional(hscore, 0);
        }
        return;
    }
    const uint64_t seed = rp->seed, iter = (uint64_t)it;
    const uint64_t hic = ((uint64_t)c << 40) ^ (iter << 4) ^ 7u;
    const bool is_l = philox_u01(seed, hic, 0) < rp->lprob;
    if (!is_l) {
        const uint64_t hi = ((uint64_t)c << 40) ^ (iter << 4) ^ 3u;
        for (int i = 1 + lane; i < nm; i += 32) su[i] = philox_u01(seed, hi, (uint64_t)i);
        for (int i = lane; i < nm; i += 32) order[i] = base[i];
        __syncwarp();
        if (lane == 0)
            for (int i = nm - 1; i > 0; --i) {
                int j = (int)(su[i] * (double)(i + 1));
                if (j > i) j = i;
                const int32_t t = order[i];
                order[i] = order[j];
                order[j] = t;
            }
    }
    if (lane == 0) {
        key[0] = seed;
        key[1] = iter;
        cudaGraphSetConditional(hsw, is_l ? 0 : 1);
        // only the chains at temperature 1 are scored (markov_chain.cc:173-174)
        cudaGraphSetConditional(hscore, (it >= rp->burnin && it % rp->period == 0 && temp[c] == 1.0) ? 1 : 0);
    }
}

__global__ void chain_advance_kernel(const RunParams* rp, int64_t* it_arr, int c, cudaGraphConditionalHandle hwhile) {
    const int64_t next = it_arr[c] + 1;
    it_arr[c] = next;
    cudaGraphSetConditional(hwhile, next < rp->end ? 1 : 0);
}

// Fold the chains' LOD tables into the context's, chain by chain
// (LODscores::merge_results, lod_score.h:98-105), and clear them.
__global__ void chain_merge_kernel(double* acc_c, uint8_t* init_c, int C, int64_t npos, double* acc, uint8_t* init) {
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < npos; p += (int64_t)gridDim.x * blockDim.x) {
        double a = acc[p];
        uint8_t ini = init[p];
        for (int c = 0; c < C; ++c) {
            const size_t q = (size_t)c * npos + p;
            if (!init_c[q]) continue;
            a = ini ? log_sum(a, acc_c[q]) : acc_c[q];
            ini = 1;
            init_c[q] = 0;
        }
        acc[p] = a;
        init[p] = ini;
    }
}

cudaError_t launch_run_init(const RunParams* rp, int64_t* it, int C, cudaStream_t s) {
    run_init_kernel<<<(C + 127) / 128, 128, 0, s>>>(rp, it, C);
    return cudaGetLastError();
}

cudaError_t launch_chain_iter(const RunParams* rp, const int64_t* it, int c, uint64_t* key, const int32_t* base,
                              int nm, int32_t* order, const double* temp, cudaGraphConditionalHandle hsw,
                              cudaGraphConditionalHandle hscore, cudaStream_t s) {
    chain_iter_kernel<<<1, 32, sizeof(double) * (nm > 0 ? nm : 1), s>>>(rp, it, c, key, base, nm, order, temp, hsw,
                                                                        hscore);
    return cudaGetLastError();
}

cudaError_t launch_chain_advance(const RunParams* rp, int64_t* it, int c, cudaGraphConditionalHandle hwhile,
                                 cudaStream_t s) {
    chain_advance_kernel<<<1, 1, 0, s>>>(rp, it, c, hwhile);
    return cudaGetLastError();
}

cudaError_t launch_chain_merge(double* acc_c, uint8_t* init_c, int C, int64_t npos, double* acc, uint8_t* init,
                               cudaStream_t s) {
    int64_t grid = (npos + 255) / 256;
    if (grid > 4096) grid = 4096;
    chain_merge_kernel<<<(int)grid, 256, 0, s>>>(acc_c, init_c, C, npos, acc, init);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Host-side launchers
// ---------------------------------------------------------------------------
size_t lsampler_smem_per_warp(const ProblemDev& P) {
    return P.ls_fast ? ls_warp_bytes<float>(P) : ls_warp_bytes<double>(P);
}

size_t lsampler_smem_shared(const ProblemDev& P) { return ls_tables_bytes(P); }


template <typename T, int G>
static cudaError_t launch_lsampler_g(const ProblemDev& P, uint32_t* dg, int first, int nchain, const int32_t* loci,
                                     int nloci, const Draws& d, const uint8_t* sel, int want, int* status,
                                     cudaStream_t s, int grid_cap, int wpb) {
    const int tpb = wpb * (32 / G);
    const size_t smem = ls_tables_bytes(P) + (size_t)tpb * ls_warp_bytes<T>(P);
    {
        cudaError_t e = ensure_smem((const void*)lsampler_kernel<T, G>, smem);
        if (e != cudaSuccess) return e;
    }
    const int64_t ntask = (int64_t)nchain * nloci;
    int64_t grid = (ntask + tpb - 1) / tpb;
    if (grid > grid_cap) grid = grid_cap;
    if (grid < 1) grid = 1;
    lsampler_kernel<T, G><<<(int)grid, wpb * 32, smem, s>>>(P, dg, first, nchain, loci, nloci, d, sel, want, status);
    return cudaGetLastError();
}

// The most L-sampler tasks an SM keeps resident, over the three lane groups,
// for blocks of wpb warps' worth of tasks (launch_lsampler's shapes): the
// occupancy of each kernel with its shared memory and registers.
template <typename T, int G>
static int ls_resident_g(const ProblemDev& P, int wpb) {
    const int tpb = wpb * (32 / G);
    const size_t smem = ls_tables_bytes(P) + (size_t)tpb * ls_warp_bytes<T>(P);
    if (ensure_smem((const void*)lsampler_kernel<T, G>, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    int blocks = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, (const void*)lsampler_kernel<T, G>, wpb * 32, smem) !=
        cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return blocks * tpb;
}

template <typename T>
static int ls_resident_t(const ProblemDev& P, int wpb) {
    const int a = ls_resident_g<T, 32>(P, wpb);
    const int b = ls_resident_g<T, 16>(P, wpb > 1 ? wpb / 2 : 1);
    const int c = ls_resident_g<T, 8>(P, wpb > 3 ? wpb / 4 : 1);
    return std::max(a, std::max(b, c));
}

int lsampler_resident_tasks(const ProblemDev& P, int wpb) {
    return P.ls_fast ? ls_resident_t<float>(P, wpb) : ls_resident_t<double>(P, wpb);
}

// Bytes of global arena a warp of the four-lane kernel needs (0: none, its
// rfunctions are in shared memory), and its shared bytes per block.
size_t quad_arena_per_warp(const ProblemDev& P) {
    if (P.ls_fast) return quad_arena_shared<float>(P) ? 0 : quad_arena_bytes<float>(P);
    return quad_arena_shared<double>(P) ? 0 : quad_arena_bytes<double>(P);
}
size_t quad_block_bytes(const ProblemDev& P, int warps) {
    return quad_prog_bytes(P) + warps * (P.ls_fast ? quad_warp_bytes<float>(P) : quad_warp_bytes<double>(P));
}

// Warps per block of the four-lane kernel: one block of as many as the SM's
// share of the warps that `load` chains' half-sweeps are, up to 8 and to what
// fits -- few warps are spread over the SMs, many share their block's copy of
// the operations (400 members, a sweep of 8 chains: 6.4 ms with 4 warps a block,
// 5.7 with 8).
static int quad_warps_per_block(const ProblemDev& P, int64_t load, int nloci, int sms) {
    const int64_t warps = load * ((nloci + kQuadTasks - 1) / kQuadTasks);
    int w = (int)std::max<int64_t>(1, std::min<int64_t>(kQuadWarps, (warps + sms - 1) / sms));
    while (w > 1 && quad_block_bytes(P, w) > 110 * 1024) --w;   // two blocks to an SM
    if (quad_arena_per_warp(P)) w = (int)std::min<int64_t>(w, P.quad_warps);   // the arena's slices
    return w;
}

template <typename T>
static cudaError_t launch_quad(const ProblemDev& P, uint32_t* dg, int first, int nchain, const int32_t* loci, int nloci,
                               const Draws& d, const uint8_t* sel, int want, int* status, cudaStream_t s, int wpb) {
    const size_t smem = quad_block_bytes(P, wpb);
    cudaError_t e = ensure_smem((const void*)lsampler_quad_kernel<T>, smem);
    if (e != cudaSuccess) return e;
    const int per = kQuadTasks * wpb;
    int64_t grid = ((int64_t)nchain * nloci + per - 1) / per;
    if (quad_arena_per_warp(P)) grid = std::min(grid, nchain * (P.quad_warps / wpb));   // slots of the arena
    lsampler_quad_kernel<T><<<(int)grid, 32 * wpb, smem, s>>>(P, dg, first, nchain, loci, nloci, d, sel, want, status);
    return cudaGetLastError();
}

// Whether launch_lsampler's block for `lanes` (32, 16 or 8) fits the most shared
// memory that a block may have: two and four tasks to a warp are the least that
// those lane groups take.
bool lsampler_fits(const ProblemDev& P, int wpb, int lanes) {
    const int tasks = lanes == 32 ? wpb : lanes == 16 ? 2 * std::max(1, wpb / 2) : 4 * std::max(1, wpb / 4);
    return ls_tables_bytes(P) + tasks * lsampler_smem_per_warp(P) <= 227 * 1024;
}

// lanes = 32, 16, 8 or 4 lanes per (chain, locus) task; all draw the same graphs.
cudaError_t launch_lsampler(const ProblemDev& P, uint32_t* dg, int first, int nchain, const int32_t* loci, int nloci,
                            const double* u, int64_t ucs, int64_t uls, uint64_t seed, uint64_t iter,
                            const uint8_t* sel, int want, int* status, cudaStream_t s, int grid_cap, int wpb,
                            const uint64_t* key, int lanes, int load, int sms) {
    Draws d{u, ucs, uls, seed, iter, 1, key};
    if (lanes == 4) {
        const int w4 = quad_warps_per_block(P, std::max(load, nchain), nloci, sms);
        if (P.ls_fast) return launch_quad<float>(P, dg, first, nchain, loci, nloci, d, sel, want, status, s, w4);
        return launch_quad<double>(P, dg, first, nchain, loci, nloci, d, sel, want, status, s, w4);
    }
    if (lanes == 8) {
        // four tasks per warp: a quarter of the warps per block keeps the block's shared memory
        const int w8 = std::max(1, wpb / 4);
        if (P.ls_fast) return launch_lsampler_g<float, 8>(P, dg, first, nchain, loci, nloci, d, sel, want, status, s,
                                                          grid_cap, w8);
        return launch_lsampler_g<double, 8>(P, dg, first, nchain, loci, nloci, d, sel, want, status, s, grid_cap, w8);
    }
    if (lanes == 16) {
        // two tasks per warp: half as many warps per block keeps the block's shared memory
        const int w16 = std::max(1, wpb / 2);
        if (P.ls_fast) return launch_lsampler_g<float, 16>(P, dg, first, nchain, loci, nloci, d, sel, want, status, s,
                                                           grid_cap, w16);
        return launch_lsampler_g<double, 16>(P, dg, first, nchain, loci, nloci, d, sel, want, status, s, grid_cap, w16);
    }
    if (P.ls_fast)
        return launch_lsampler_g<float, 32>(P, dg, first, nchain, loci, nloci, d, sel, want, status, s, grid_cap, wpb);
    return launch_lsampler_g<double, 32>(P, dg, first, nchain, loci, nloci, d, sel, want, status, s, grid_cap, wpb);
}

// Keep each chain's best imputation: over the batch's passes in pass order,
// the first whose weight beats the best so far (SequentialImputation::run,
// sequential_imputation.cc:14-43: `tmp_prob > best_prob`, starting from
// LOG_ZERO); its graph is copied in.  One block per chain.
__global__ void si_select_kernel(const uint32_t* scratch, uint32_t* dg, int first, int nchain, size_t words,
                                 const double* w, double* best, int npass) {
    for (int cr = blockIdx.x; cr < nchain; cr += gridDim.x) {
        double bw = best[cr];
        int bq = -1;
        for (int q = 0; q < npass; ++q)
            if (w[(size_t)q * nchain + cr] > bw) {
                bw = w[(size_t)q * nchain + cr];
                bq = q;
            }
        __syncthreads();
        if (bq < 0) continue;
        const uint32_t* src = scratch + ((size_t)bq * nchain + cr) * words;
        for (size_t i = threadIdx.x; i < words; i += blockDim.x) dg[(size_t)(first + cr) * words + i] = src[i];
        __syncthreads();
        if (threadIdx.x == 0) best[cr] = bw;
    }
}

template <typename T>
static cudaError_t launch_si_quad(const ProblemDev& P, uint32_t* dg, int first, int nchain, const int32_t* starts,
                                  const Draws& d, double* weights, int* status, cudaStream_t s, int npass,
                                  int64_t pass_stride, int sms) {
    const int64_t ntask = (int64_t)nchain * npass;
    const int wpb = quad_warps_per_block(P, 1, (int)ntask, sms), per = kQuadTasks * wpb;
    const size_t smem = quad_block_bytes(P, wpb);
    cudaError_t e = ensure_smem((const void*)si_quad_kernel<T>, smem);
    if (e != cudaSuccess) return e;
    int64_t grid = (ntask + per - 1) / per;
    if (quad_arena_per_warp(P)) grid = std::min(grid, P.quad_warps / wpb);   // slices of the call's arena
    si_quad_kernel<T><<<(int)grid, 32 * wpb, smem, s>>>(P, dg, first, nchain, starts, d, 0, weights, status, npass,
                                                        pass_stride);
    return cudaGetLastError();
}

// quad: by four lanes per pass (P.quad_prog set, its arena there)
cudaError_t launch_si(const ProblemDev& P, uint32_t* dg, int first, int nchain, const int32_t* starts,
                      const double* u, int64_t ucs, uint64_t seed, uint64_t pass, double* weights, int* status,
                      cudaStream_t s, int wpb, int npass, int64_t pass_stride, int grid_cap, bool quad, int sms) {
    if (quad) {
        const Draws dr{u, ucs, 0, seed, pass, 5, nullptr};
        if (P.ls_fast)
            return launch_si_quad<float>(P, dg, first, nchain, starts, dr, weights, status, s, npass, pass_stride, sms);
        return launch_si_quad<double>(P, dg, first, nchain, starts, dr, weights, status, s, npass, pass_stride, sms);
    }
    const size_t smem = ls_tables_bytes(P) + wpb * lsampler_smem_per_warp(P);
    {
        cudaError_t e = ensure_smem(P.ls_fast ? (const void*)si_kernel<float> : (const void*)si_kernel<double>, smem);
        if (e != cudaSuccess) return e;
    }
    Draws d{u, ucs, 0, seed, pass, 5, nullptr};
    int grid = (nchain * npass + wpb - 1) / wpb;
    if (grid > grid_cap) grid = grid_cap;
    if (P.ls_fast)
        si_kernel<float><<<grid, wpb * 32, smem, s>>>(P, dg, first, nchain, starts, d, 0, weights, status, npass,
                                                      pass_stride);
    else
        si_kernel<double><<<grid, wpb * 32, smem, s>>>(P, dg, first, nchain, starts, d, 0, weights, status, npass,
                                                       pass_stride);
    return cudaGetLastError();
}

cudaError_t launch_si_select(const uint32_t* scratch, uint32_t* dg, int first, int nchain, size_t words,
                             const double* w, double* best, int npass, cudaStream_t s) {
    si_select_kernel<<<nchain < 1024 ? nchain : 1024, 256, 0, s>>>(scratch, dg, first, nchain, words, w, best, npass);
    return cudaGetLastError();
}

// Lanes per founder-allele graph: two loci per warp (16 lanes each: 17% fewer
// instructions per locus) when the context holds enough chains to be
// throughput-bound and a column fits in 16 words (with longer columns the
// 400-member pedigree's M-sweeps were 16% slower than with 32 lanes).
static int fagw_lanes(const ProblemDev& P, int chains) { return chains >= 8 && P.W <= 16 ? 16 : 32; }

static const void* msw_kernel(int G, int eb) {
    return G == 16 ? (eb == 1 ? (const void*)msweep_kernel<16, uint8_t> : (const void*)msweep_kernel<16, uint16_t>)
                   : (eb == 1 ? (const void*)msweep_kernel<32, uint8_t> : (const void*)msweep_kernel<32, uint16_t>);
}

static void msw_config(const MswShape& sh, int nchain, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at) {
    *cfg = cudaLaunchConfig_t{};
    cfg->gridDim = dim3((unsigned)sh.cs, (unsigned)nchain);
    cfg->blockDim = dim3((unsigned)sh.threads);
    cfg->dynamicSmemBytes = sh.bytes;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = (unsigned)sh.cs;
    at->val.clusterDim.y = 1;
    at->val.clusterDim.z = 1;
    cfg->attrs = at;
    cfg->numAttrs = 1;
}

// Whether fast M-sweeps run as clusters: the genotypes' masks are there and
// some shape fits (the component counts are 13-bit fields).
static bool msw_fits(const ProblemDev& P, int G, int eb) {
    MswShape sh;
    return P.mflip && !P.ms_launches && 2 * P.F < 8192 && msw_shape(P, G, eb, 16, &sh);
}

// The most blocks per cluster, of the sizes that give every block as many scan
// warps (16, 11, 8, 7, 6, 5, 4, 3, 2, 1 for 32 scan warps), at which `load`
// chains' clusters are all resident, by the occupancy calculator; the fewest
// that fit when none is.  A sweep of the 400-member, 10,000-SNP pedigree took
// 20.4, 30.8 and 48.4 ms with 16, 8 and 4 blocks for one chain, 101, 77 and 49 ms
// for 32 chains; of the 120-member one 2.2, 2.4 and 3.2 ms for one, 31, 15 and
// 7.8 ms (6.7 with 2 blocks) for 80 chains (before likelihoods were evaluated
// ahead).  With the sizes between the powers of two: 400 members, 8 chains (11
// blocks instead of 8) 23.0 -> 19.8 ms, 16 chains 37.4 -> 29.5, 24 chains 37.4 ->
// 32.7; 120 members, 40 chains 3.64 -> 3.05, 16 chains 2.65 -> 2.53.
static cudaError_t msw_choose(const ProblemDev& P, int G, int eb, int load, MswShape* out) {
    const void* mk = msw_kernel(G, eb);
    cudaError_t e = cudaFuncSetAttribute(mk, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    int last = 0;
    for (int cs = 16; cs >= 1 && e == cudaSuccess; --cs) {
        MswShape sh;
        if (!msw_shape(P, G, eb, cs, &sh)) break;
        if (sh.cs == last) continue;   // as many scan warps a block as the size before
        last = sh.cs;
        *out = sh;
        if ((e = ensure_smem(mk, sh.bytes)) != cudaSuccess) break;
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at;
        msw_config(sh, load, &cfg, &at);
        int active = 0;
        if ((e = cudaOccupancyMaxActiveClusters(&active, mk, &cfg)) == cudaSuccess && active >= load) break;
    }
    return e;
}

// Kernels of one fast M-sweep of nm meioses in a context of `chains` chains.
int64_t msweep_launches(const ProblemDev& P, int chains, int nm) {
    return msw_fits(P, fagw_lanes(P, chains), fagw_label_bytes(P.F)) ? 1 : 1 + 2 * (int64_t)nm;
}

template <typename IX, typename PP>
static cudaError_t launch_msampler_t(const ProblemDev& P, uint32_t* dg, int first, int nchain, const int32_t* meioses,
                                     int64_t mstride, int nm, const double* u, int64_t ucs, uint64_t seed,
                                     uint64_t iter, const uint8_t* sel, int want, typename PP::T* raw, float* raw32,
                                     void* fb, uint8_t* badc, uint8_t* maps, int* status, int fag_threads, int exact,
                                     cudaStream_t s, const uint64_t* key, double* ubuf, int chains, int load) {
    const int fast = exact ? 0 : 1;
    Draws d{u, ucs, P.M, seed, iter, 2, key};
    const int G = fagw_lanes(P, chains), eb = fagw_label_bytes(P.F);
    if (!exact && msw_fits(P, G, eb)) {
        MswShape sh;
        cudaError_t e = msw_choose(P, G, eb, std::max(load, nchain), &sh);
        if (e != cudaSuccess) return e;
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at;
        msw_config(sh, nchain, &cfg, &at);
        cfg.stream = s;
        void* args[] = {(void*)&P, (void*)&sh, (void*)&dg, (void*)&first, (void*)&meioses, (void*)&mstride,
                        (void*)&nm, (void*)&d, (void*)&sel, (void*)&want, (void*)&status};
        return cudaLaunchKernelExC(&cfg, msw_kernel(G, eb), args);
    }
    cudaError_t e0 = cudaMemsetAsync(badc, 0, (size_t)nchain, s);
    if (e0 != cudaSuccess) return e0;
    if (exact) {   // the chains' flags (ffbs_exact_kernel), the first word of each one's part of ubuf
        e0 = cudaMemset2DAsync(ubuf, sizeof(double) * P.M, 0, sizeof(int), (size_t)nchain, s);
        if (e0 != cudaSuccess) return e0;
    }
    const size_t smem = fag_block_bytes(P.N, P.F, fag_threads, fast);
    {
        cudaError_t e = ensure_smem((const void*)fag_kernel<IX, PP>, smem);
        if (e != cudaSuccess) return e;
    }
    const int scan_threads = ffbs_scan_threads(P.M);
    size_t scan_smem = ffbs_scan_smem(P.M);
    int staged = 1;
    if (scan_smem > 200 * 1024) {   // long maps: read the chain's arrays from global memory
        scan_smem = ffbs_scan_scratch(scan_threads);
        staged = 0;
    }
    if (!exact) {
        cudaError_t e = ensure_smem((const void*)ffbs_scan_kernel, scan_smem);
        if (e != cudaSuccess) return e;
    }
    const int64_t ntask = (int64_t)nchain * P.M;
    const int grid = (int)((ntask + fag_threads - 1) / fag_threads);
    // fast mode: one warp per (chain, locus), else the thread-per-locus kernel
    // in log2 (component counts are 13-bit fields)
    const size_t wsm = fagw_block_bytes(P.N, P.F, G, eb);
    const bool warp_like = !exact && wsm <= 200 * 1024 && 2 * P.F < 8192;
    const void* fk = G == 16 ? (eb == 1 ? (const void*)fag_warp_kernel<16, uint8_t> : (const void*)fag_warp_kernel<16, uint16_t>)
                             : (eb == 1 ? (const void*)fag_warp_kernel<32, uint8_t> : (const void*)fag_warp_kernel<32, uint16_t>);
    if (warp_like) {
        cudaError_t e = ensure_smem(fk, wsm);
        if (e != cudaSuccess) return e;
    }
    const int lpb = kFagWarpsPerBlock * (32 / G);   // loci per block
    const dim3 wgrid((unsigned)((P.M + lpb - 1) / lpb), (unsigned)nchain);
    double* upre = warp_like ? ubuf : nullptr;
    for (int j = -1; j < nm; ++j) {
        if (!warp_like)
            fag_kernel<IX, PP><<<grid, fag_threads, smem, s>>>(P, dg, first, nchain, meioses, mstride, j, sel, want,
                                                               raw, exact ? nullptr : raw32, badc, status, fast);
        else {
            float* rawf = (float*)raw;
            void* args[] = {(void*)&P, (void*)&dg, (void*)&first, (void*)&meioses, (void*)&mstride, (void*)&j,
                            (void*)&d, (void*)&sel, (void*)&want, (void*)&rawf, (void*)&raw32, (void*)&badc,
                            (void*)&status, (void*)&upre};
            cudaError_t e = cudaLaunchKernel(fk, wgrid, dim3(kFagWarpsPerBlock * 32), args, wsm, s);
            if (e != cudaSuccess) return e;
        }
        if (j < 0) continue;
        if (exact) {
            ffbs_exact_runs_kernel<<<dim3((unsigned)((P.M + 31) / 32), (unsigned)nchain), 32, 0, s>>>(
                P, first, nchain, sel, want, badc, (const double*)raw, (double*)fb, (int*)ubuf, 2 * (int64_t)P.M);
            const int bt = std::min(512, (P.M + 31) / 32 * 32);
            ffbs_exact_kernel<<<nchain, bt, 0, s>>>(P, dg, first, nchain, meioses, mstride, j, d, sel, want, badc,
                                                    (const double*)raw, (double*)fb, maps, (int*)ubuf,
                                                    2 * (int64_t)P.M);
        } else
            ffbs_scan_kernel<<<nchain, scan_threads, scan_smem, s>>>(P, dg, first, nchain, meioses, mstride, j, d, sel,
                                                                     want, badc, raw32, (float*)fb, maps, staged,
                                                                     upre);
    }
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Descent graphs from the caller's int32 [locus][person][2] arrays into packed
// columns.  Where the device reads the host's pages itself
// (cudaDevAttrPageableMemoryAccessUsesHostPageTables: Grace over NVLink-C2C)
// this kernel takes the caller's memory as it lies: 8 graphs of the 400-member,
// 10,000-SNP pedigree (256 MB) packed in 1.0 ms, where the host's 16 cores took
// 3.2 ms with the copy.  Bound by the link (200 GB/s for a plain read of host
// pages); founders' entries are not read.
// ---------------------------------------------------------------------------
constexpr int kPackWords = 4;   // words a warp has in flight

// A warp per four words of the packed graphs: bit b of a column is int32 2F + b of its 2N.
__global__ void __launch_bounds__(256) pack_kernel(const int32_t* __restrict__ src, int N, int F, int W, int64_t words,
                                                   uint32_t* dst) {
    const int lane = threadIdx.x & 31, nb = 2 * (N - F);
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5), gw = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    for (int64_t i0 = gw * kPackWords; i0 < words; i0 += nw * kPackWords) {
        int v[kPackWords];
#pragma unroll
        for (int k = 0; k < kPackWords; ++k) {
            const int64_t i = i0 + k, c = i / W;
            const int b = 32 * (int)(i - c * W) + lane;
            v[k] = i < words && b < nb ? __ldcs(src + c * 2 * N + 2 * F + b) : 0;
        }
#pragma unroll
        for (int k = 0; k < kPackWords; ++k) {
            const unsigned x = __ballot_sync(FULLMASK, v[k] & 1);
            if (lane == 0 && i0 + k < words) dst[i0 + k] = x;
        }
    }
}

cudaError_t launch_pack(const int32_t* src, int n, int N, int F, int M, int W, uint32_t* dst, int sms, cudaStream_t s) {
    const int64_t words = (int64_t)n * M * W, need = (words + 8 * kPackWords - 1) / (8 * kPackWords);
    pack_kernel<<<(int)std::min<int64_t>(need, 8 * (int64_t)sms), 256, 0, s>>>(src, N, F, W, words, dst);
    return cudaGetLastError();
}
// log2 of each chain's major and minor allele frequency at each locus, in
// the founder-allele kernel's arithmetic (FP32 logs of the rounded frequencies)
__global__ void lfreq_kernel(const double* minor, float2* out, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double m = minor[i];
        out[i] = make_float2(log2f((float)(1.0 - m)), log2f((float)m));
    }
}

cudaError_t launch_lfreq(const double* minor, float2* out, int64_t n, cudaStream_t s) {
    int64_t grid = (n + 255) / 256;
    if (grid > 4096) grid = 4096;
    if (grid < 1) grid = 1;
    lfreq_kernel<<<(int)grid, 256, 0, s>>>(minor, out, n);
    return cudaGetLastError();
}

cudaError_t launch_set_key(uint64_t* key, uint64_t seed, uint64_t iter, cudaStream_t s) {
    set_key_kernel<<<1, 1, 0, s>>>(key, seed, iter);
    return cudaGetLastError();
}

cudaError_t launch_msampler(const ProblemDev& P, uint32_t* dg, int first, int nchain, const int32_t* meioses,
                            int64_t mstride, int nm, const double* u, int64_t ucs, uint64_t seed, uint64_t iter,
                            const uint8_t* sel, int want, double* raw64, float* raw32, void* fb, uint8_t* badc,
                            uint8_t* maps, int* status, int fag_threads, int exact, cudaStream_t s,
                            const uint64_t* key, double* ubuf, int chains, int load) {
    // the fast mode keeps log2 likelihoods as floats in the first half of the raw buffer
    float* rawl = (float*)raw64;
    if (2 * P.F <= 255) {
        if (exact)
            return launch_msampler_t<uint8_t, ProbExact>(P, dg, first, nchain, meioses, mstride, nm, u, ucs, seed,
                                                         iter, sel, want, raw64, raw32, fb, badc, maps, status,
                                                         fag_threads, exact, s, key, ubuf, chains, load);
        return launch_msampler_t<uint8_t, ProbLog2>(P, dg, first, nchain, meioses, mstride, nm, u, ucs, seed, iter,
                                                    sel, want, rawl, raw32, fb, badc, maps, status, fag_threads,
                                                    exact, s, key, ubuf, chains, load);
    }
    if (exact)
        return launch_msampler_t<uint16_t, ProbExact>(P, dg, first, nchain, meioses, mstride, nm, u, ucs, seed, iter,
                                                      sel, want, raw64, raw32, fb, badc, maps, status, fag_threads,
                                                      exact, s, key, ubuf, chains, load);
    return launch_msampler_t<uint16_t, ProbLog2>(P, dg, first, nchain, meioses, mstride, nm, u, ucs, seed, iter, sel,
                                                 want, rawl, raw32, fb, badc, maps, status, fag_threads, exact, s,
                                                 key, ubuf, chains, load);
}

size_t fag_smem(int N, int F, int threads, int fast) { return fag_block_bytes(N, F, threads, fast); }

// Warps a block of the FP64 scorer takes, of 1 to 4: as many as leave the most
// warps resident with `warp` shared bytes each (28: what their registers allow).
// A grid that was sized for one lane count and blocks cut to 100 KB left one
// warp on an SM where three fit: 4,336 cells, 32 lanes 4.06 -> 1.87 ms, 10,220
// cells 30 -> 15.
constexpr size_t kLodBlock = 227 * 1024, kLodSM = 228 * 1024;
static int lod64_warps(size_t warp) {
    int best = 1;
    size_t most = 0;
    for (int w = 4; w >= 1; --w) {
        if (w * warp > kLodBlock) continue;
        const size_t resident = std::min<size_t>(28, w * (kLodSM / (w * warp + 1024)));
        if (resident > most) {
            most = resident;
            best = w;
        }
    }
    return best;
}

template <bool RESCALE, int L>
static cudaError_t launch_lod_lanes(const ProblemDev& P, const uint32_t* graphs, int64_t graph_words, int G,
                                    double* vals, int* status, cudaStream_t s) {
    const int64_t ntask = (int64_t)G * (P.M - 1) * P.n_lod;
    const size_t warp = (size_t)(32 / L) * (P.arena + 16) * sizeof(double);
    const int wpb = lod64_warps(warp), per = wpb * (32 / L);
    const int64_t grid = std::max<int64_t>(1, std::min<int64_t>(INT_MAX, (ntask + per - 1) / per));
    const void* k = (const void*)lod_kernel<double, RESCALE, L>;
    const cudaError_t e = ensure_smem(k, wpb * warp);
    if (e != cudaSuccess) return e;
    lod_kernel<double, RESCALE, L><<<(int)grid, wpb * 32, wpb * warp, s>>>(P, graphs, graph_words, G, vals, status);
    return cudaGetLastError();
}

// Lanes to a position: by the arena (P.arena cells), which bounds the positions on
// an SM, and which grows with the widest cutset, whose cells more lanes share.
//  * up to 600 cells, 16 lanes, and 8 from 20,000 positions (128 to an SM, more
//    than the warps of 4 that are resident there): at 8 the FP64 pipe gives its
//    whole rate to fewer idle lanes, but a position takes half as long again.
//    32 | 16 | 8 lanes, plain form, 45 members, 156 cells: 2,000 positions 0.162 |
//    0.129 | 0.177 ms, 8,000 0.465 | 0.252 | 0.272, 40,000 2.14 | 1.13 | 1.05; 528
//    cells (120 members, rescaled) 0.69 | 0.53 | 0.73, 2.28 | 1.58 | 1.77, 10.5 |
//    5.96 | 5.69;
//  * up to 1,000, 16: 672 cells (45 members, 4 loops) 0.353 | 0.374 | 0.594, 1.14 |
//    1.26 | 1.31, 5.24 | 4.59 | 5.06; 788 cells (120 members, 4 loops, rescaled)
//    0.73 | 0.59 | 0.83, 2.41 | 1.69 | 1.83, 11.1 | 7.5 | 8.0;
//  * above, 32, which every arena that a context accepts leaves room for (8 need
//    four arenas in a warp, 16 two): 1,088 cells 0.44 | 0.55 | 0.99, 1.48 | 1.76 |
//    2.94, 6.6 | 6.7 | 10.8 (1,256 cells of 120 members 0.93 | 0.99 | 1.54, 16.1 |
//    13.8 | 21.0 at 40,000); 2,216 cells 12.6 | 18.9 | 34.5; 4,336 cells 27.5 | 49.1
//    | 147; 8,784 cells 139 | 413, 8 do not fit; 15,728 cells 490, 16 do not fit.
template <bool RESCALE>
static cudaError_t launch_lod64(const ProblemDev& P, const uint32_t* graphs, int64_t graph_words, int G, double* vals,
                                int* status, cudaStream_t s) {
    if (P.arena > 1000) return launch_lod_lanes<RESCALE, 32>(P, graphs, graph_words, G, vals, status, s);
    if (P.arena <= 600 && (int64_t)G * (P.M - 1) * P.n_lod >= 20000)
        return launch_lod_lanes<RESCALE, 8>(P, graphs, graph_words, G, vals, status, s);
    return launch_lod_lanes<RESCALE, 16>(P, graphs, graph_words, G, vals, status, s);
}

cudaError_t launch_lod(const ProblemDev& P, int precision, const uint32_t* graphs, int64_t graph_words, int G,
                       double* vals, int* status, cudaStream_t s, int grid_cap, int wpb) {
    const int64_t ntask = (int64_t)G * (P.M - 1) * P.n_lod;
    if (precision == 0) return launch_lod64<false>(P, graphs, graph_words, G, vals, status, s);
    if (precision == 2) return launch_lod64<true>(P, graphs, graph_words, G, vals, status, s);
    if (P.prog) {
        const int S = P.prog_threads;
        const size_t smem = (size_t)S * P.prog_slots * sizeof(float);
        {
            cudaError_t e = ensure_smem((const void*)lod_prog_kernel, smem);
            if (e != cudaSuccess) return e;
        }
        int64_t pgrid = (ntask + S - 1) / S;
        if (pgrid > grid_cap * 4) pgrid = grid_cap * 4;
        lod_prog_kernel<<<(int)pgrid, S, smem, s>>>(P, graphs, graph_words, G, vals, status);
    } else {
        const size_t smem = (size_t)wpb * (P.arena + 16) * sizeof(float);
        {
            cudaError_t e = ensure_smem((const void*)lod_kernel<float, true, 32>, smem);
            if (e != cudaSuccess) return e;
        }
        int64_t grid = (ntask + wpb - 1) / wpb;
        if (grid > grid_cap) grid = grid_cap;
        if (grid < 1) grid = 1;
        lod_kernel<float, true, 32><<<(int)grid, wpb * 32, smem, s>>>(P, graphs, graph_words, G, vals, status);
    }
    return cudaGetLastError();
}

cudaError_t launch_trait_adjoint(const ProblemDev& P, const AdjDev& D, const uint32_t* graphs, int64_t graph_words,
                                 int64_t task0, int64_t ntask, double* grad, int* status, cudaStream_t s, int sms) {
    const int wpb = (int)std::max<int64_t>(1, std::min<int64_t>(4, (200 * 1024) / std::max(1, D.warp_bytes)));
    const size_t smem = (size_t)wpb * D.warp_bytes;
    {
        cudaError_t e = ensure_smem((const void*)trait_adjoint_kernel, smem);
        if (e != cudaSuccess) return e;
    }
    int blocks = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, (const void*)trait_adjoint_kernel, wpb * 32, smem) !=
            cudaSuccess || blocks < 1)
        blocks = 1;
    int64_t grid = (ntask + wpb - 1) / wpb;
    grid = std::min<int64_t>(grid, (int64_t)sms * blocks);
    trait_adjoint_kernel<<<(int)std::max<int64_t>(1, grid), wpb * 32, smem, s>>>(P, D, graphs, graph_words, task0,
                                                                                 ntask, grad, status);
    return cudaGetLastError();
}

// Resident blocks of 128 threads per SM of the one-thread-per-task form.
int trait_adjoint_thr_blocks() {
    int blocks = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, (const void*)trait_adjoint_thr_kernel, 128, 0) !=
            cudaSuccess || blocks < 1) {
        cudaGetLastError();
        blocks = 1;
    }
    return blocks;
}

// One block of 128 threads per 128 threads of the arena (arena_threads, the
// resident threads of every SM); the threads stride over the tasks.
cudaError_t launch_trait_adjoint_thr(const ProblemDev& P, const AdjDev& D, const uint32_t* graphs, int64_t graph_words,
                                     int64_t task0, int64_t ntask, double* grad, int* status, float* arena, int* expo,
                                     int64_t arena_threads, cudaStream_t s) {
    const int64_t blocks = arena_threads / 128;
    if (blocks < 1) return cudaErrorInvalidValue;
    trait_adjoint_thr_kernel<<<(int)blocks, 128, 0, s>>>(P, D, graphs, graph_words, task0, ntask, grad, status, arena,
                                                         expo);
    return cudaGetLastError();
}

cudaError_t launch_lod_merge(const double* vals, int G, int64_t npos, double* acc, uint8_t* init, cudaStream_t s) {
    const int threads = 256;
    int64_t grid = (npos + threads - 1) / threads;
    if (grid > 65535) grid = 65535;
    lod_merge_kernel<<<(int)grid, threads, 0, s>>>(vals, G, npos, acc, init);
    return cudaGetLastError();
}

cudaError_t launch_shuffle(const int32_t* base, int nm, int32_t* out, int first, int nchain, uint64_t seed,
                           uint64_t iter, cudaStream_t s) {
    shuffle_kernel<<<(nchain + 63) / 64, 64, 0, s>>>(base, nm, out, first, nchain, seed, iter);
    return cudaGetLastError();
}

cudaError_t launch_choose(int first, int nchain, uint64_t seed, uint64_t iter, double lprob, uint8_t* is_l,
                          cudaStream_t s) {
    choose_kernel<<<(nchain + 63) / 64, 64, 0, s>>>(first, nchain, seed, iter, lprob, is_l);
    return cudaGetLastError();
}

}  // namespace sl
