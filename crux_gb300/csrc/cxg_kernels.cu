// Device kernels of the pruning likelihood on sm_103a.
//
// Layout in HBM: a CL buffer of K active components over ppad patterns is
// [K][U][ppad] 16-byte units (FP32: U = 1, a float4 of the four states;
// FP64: U = 2, two double2), so that the threads of a warp, one pattern
// each, move 512 contiguous bytes per instruction.  Leaves are one uint8
// state mask per pattern.  Scalers are one FP64 log scale (plain form) or
// one int32 power-of-two exponent (FP32 form) per pattern.
//
// Kernels:
//   pmat_kernel     P(t) = V diag(exp(lambda r t)) V^-1 per (child edge,
//                   component), FP64, clipped at 0 (CxLik.c:258-292), plus
//                   the 16-entry message table of every leaf child.
//   walk_kernel<T>  one CTA per tile of patterns, one thread per pattern,
//                   walks the whole node-update list (patterns are
//                   independent through the entire post-order,
//                   CxLik.c:314-596, so no grid-wide sync is needed).  CLs
//                   produced and consumed within the walk stay in a
//                   shared-memory stack (slots assigned by the host), so HBM
//                   sees the write-through of every parent, the staged leaf
//                   masks and CLs cached by earlier runs.  Then it
//                   aggregates the root (CxLik.c:598-632) and reduces the
//                   weighted site lnLs with a compensated sum.
//   qdecomp_kernel  FP64 eigensystem of a reversible 4x4 Q by Jacobi
//                   rotations of the symmetrised matrix (CxLik.c:59-250).
#include <math.h>

#include <mutex>

#include "cxg_internal.h"
#include "cxg_device.cuh"

namespace cxg {

// ---------------------------------------------------------------------------
// P matrices, written into the op records.
// ---------------------------------------------------------------------------
// Four lanes per (child edge, component), see pmat_one.
// Programmatic dependent launch: a walker launched as a dependent of the
// P kernel may start (be scheduled, set up its shared memory and barriers)
// once every P block has started; it waits here, before it copies its
// first records, for the P kernel's matrices and their memory.  Without
// such a dependency both instructions do nothing.
__device__ __forceinline__ void pdl_launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

__global__ void pmat_kernel(PmatArgs a) {
    pdl_launch_dependents();
    // The walker's result words (ticket, counts, sum): it reads them only
    // after this grid has completed (stream order, or griddepcontrol.wait).
    if (a.zero != nullptr && blockIdx.x == 0 && threadIdx.x < 4) a.zero[threadIdx.x] = 0;
    const unsigned idx = (blockIdx.x * blockDim.x + threadIdx.x) >> 2;
    if (idx >= a.nchild * a.kact) return;  // the same for all four lanes
    pmat_one(a, idx, threadIdx.x & 3u);
}

// P matrices of many jobs in one launch: (edge, component) t belongs to
// the job whose prefix range [prefix[j], prefix[j+1]) holds it.
__global__ void pmat_batch_kernel(const PmatArgs *jobs, const uint32_t *prefix,
                                  uint32_t njobs, uint32_t total) {
    const unsigned t = (blockIdx.x * blockDim.x + threadIdx.x) >> 2;
    if (t >= total) return;
    unsigned lo = 0, hi = njobs;  // find j with prefix[j] <= t < prefix[j+1]
    while (hi - lo > 1) {
        const unsigned mid = (lo + hi) / 2;
        if (prefix[mid] <= t) lo = mid; else hi = mid;
    }
    pmat_one(jobs[lo], t - prefix[lo], threadIdx.x & 3u);
}

cudaError_t launch_pmat_batch(const PmatArgs *jobs, const uint32_t *prefix,
                              uint32_t njobs, uint32_t total, cudaStream_t s) {
    if (total == 0) return cudaSuccess;
    pmat_batch_kernel<<<(total + 31) / 32, 128, 0, s>>>(jobs, prefix, njobs, total);
    return cudaGetLastError();
}

cudaError_t launch_pmat(const PmatArgs &a, cudaStream_t s) {
    const unsigned n = a.nchild * a.kact;
    if (n == 0) return cudaSuccess;
    pmat_kernel<<<(n + 31) / 32, 128, 0, s>>>(a);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Compensated (Neumaier two-sum) reduction helpers.
// ---------------------------------------------------------------------------
struct Comp {
    double s, c;
};

__device__ __forceinline__ Comp comp_add(Comp a, Comp b) {
    const double s = a.s + b.s;
    const double bb = s - a.s;
    const double err = (a.s - (s - bb)) + (b.s - bb);
    return Comp{s, a.c + b.c + err};
}

__device__ __forceinline__ Comp warp_comp(Comp v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        Comp o;
        o.s = __shfl_down_sync(0xffffffffu, v.s, off);
        o.c = __shfl_down_sync(0xffffffffu, v.c, off);
        v = comp_add(v, o);
    }
    return v;
}

// Tile sum of site values (finite values; -inf sites are counted
// separately) into a.partial[tile]; the last tile of the job to finish
// folds all of the job's partials into a.total.  Thread t holds the values
// of patterns t + h * blockDim (h < NV): every group of 32 consecutive
// patterns reduces by the same shuffle tree and the groups add in pattern
// order, and warp 0 alone folds the partials, so the sums do not depend
// on the launch shape.
template <int NV>
__device__ void reduce_sites_n(const PlanArgs &a, unsigned tile_idx, const double *v,
                               const bool *neg_inf) {
    __shared__ Comp warp_part[kMaxThreads / 32];
    __shared__ unsigned ninf_block;
    __shared__ bool last;
    const unsigned nwarp = blockDim.x / 32;
    if (threadIdx.x == 0) ninf_block = 0;
    __syncthreads();
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int h = 0; h < NV; ++h) {
        if (neg_inf[h]) atomicAdd(&ninf_block, 1u);
        const Comp c = warp_comp(Comp{v[h], 0.0});
        if (lane == 0) warp_part[h * nwarp + warp] = c;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        Comp b = warp_part[0];
        for (unsigned w = 1; w < NV * nwarp; ++w) b = comp_add(b, warp_part[w]);
        a.partial[2 * tile_idx] = b.s;
        a.partial[2 * tile_idx + 1] = b.c;
        if (ninf_block) atomicAdd(a.ninf, ninf_block);
        __threadfence();
        const unsigned t = atomicAdd(a.ticket, 1u);
        last = (t == a.ntiles - 1);
    }
    __syncthreads();
    if (last && warp == 0) {
        __threadfence();
        Comp acc{0.0, 0.0};
        for (unsigned b = lane; b < a.ntiles; b += 32) {
            const volatile double *pp = a.partial;
            acc = comp_add(acc, Comp{pp[2 * b], pp[2 * b + 1]});
        }
        acc = warp_comp(acc);
        if (lane == 0) {
            a.total[0] = acc.s;
            a.total[1] = acc.c;
            *a.ticket = 0;  // ready for the next launch
        }
    }
    __syncthreads();  // warp_part / last are reused by the next item
}

__device__ __forceinline__ void reduce_sites(const PlanArgs &a, unsigned tile_idx, double v,
                                             bool neg_inf) {
    reduce_sites_n<1>(a, tile_idx, &v, &neg_inf);
}

// ---------------------------------------------------------------------------
// Plan walker.  T = double: plain form, the reference's scaler (max over
// child messages, CxLik.c:390-403 and 577-588).  T = float: FP32 form, scale
// by the power of two that puts the largest parent entry in [0.5, 1); the
// exponent is an exact integer.
// ---------------------------------------------------------------------------
template <typename T>
struct Prec;

template <>
struct Prec<double> {
    typedef double S;   // scaler type
    typedef double2 V;  // 16-byte unit
    static constexpr int U = 2;
};

template <>
struct Prec<float> {
    typedef int S;
    typedef float4 V;
    static constexpr int U = 1;
};

__device__ __forceinline__ void unpack(const float4 v, float *x) {
    x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
}
__device__ __forceinline__ float4 pack4(const float *x) {
    return make_float4(x[0], x[1], x[2], x[3]);
}

__device__ __forceinline__ float pow2f(int n) {  // n in [-126, 127]
    return __int_as_float((n + 127) << 23);
}

// Shared memory of one CTA: mbarriers [ring]; the stage ring [ring] of
// `stage` bytes, each an op record (rstride) followed, for a job that
// streams its leaves, by this tile's mask rows of the op's leaf children
// (lmax rows of tile bytes); stack slots [nslot][K][U][tile] units; slot
// scalers [nslot][tile]; and, for a job that stages its leaves, every
// leaf's mask row [nleaf][tile], loaded once per tile.  A batched launch
// lays it out for its largest job; every job uses a prefix of each region.
struct SmemLayout {
    size_t bars, ring, stage, slots, slot_sc, masks, total;
};

static __host__ __device__ SmemLayout smem_layout(int precision, unsigned kact,
                                                  unsigned tile, unsigned nslot,
                                                  unsigned ring, unsigned rstride,
                                                  unsigned lmax, unsigned nleaf) {
    const size_t U = precision == CXG_FP32 ? 1 : 2;
    const size_t sc = precision == CXG_FP32 ? 4 : 8;
    SmemLayout L;
    L.bars = 0;
    L.ring = ((size_t)ring * 8 + 127) & ~(size_t)127;
    L.stage = ((size_t)rstride + (size_t)lmax * tile + 15) & ~(size_t)15;
    L.slots = L.ring + (size_t)ring * L.stage;
    L.slot_sc = L.slots + (size_t)nslot * kact * U * tile * 16;
    L.masks = L.slot_sc + (((size_t)nslot * tile * sc + 15) & ~(size_t)15);
    L.total = L.masks + (size_t)nleaf * tile;
    return L;
}

size_t plan_smem_bytes(int precision, unsigned kact, unsigned tile, unsigned nslot,
                       unsigned ring, unsigned rstride, unsigned lmax, unsigned nleaf) {
    return smem_layout(precision, kact, tile, nslot, ring, rstride, lmax, nleaf).total;
}

// --- mbarrier and bulk-copy primitives (PTX) --------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(count)
                 : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                     smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src,
                                         uint32_t bytes, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Leaf-row pointers of op q that thread 0 reads ahead (the first
// kLeafPre; rows past them are read when the stage is issued).  Indexed
// with constants only, so they stay in registers.
constexpr int kLeafPre = 4;
__device__ __forceinline__ void read_rows(const PlanArgs &a, unsigned q,
                                          const uint8_t *(&pre)[kLeafPre]) {
    const uint8_t *const *rows = a.lrows + (size_t)q * a.lmax;
#pragma unroll
    for (int j = 0; j < kLeafPre; ++j) pre[j] = (unsigned)j < a.lmax ? rows[j] : nullptr;
}

// Start op q's stage: its record and this tile's mask rows of its leaf
// children (a.lrows[q][0..lmax), null-terminated, in the record's child
// order), all completing on the stage's mbarrier.
__device__ __forceinline__ void issue_stage(const PlanArgs &a, unsigned q,
                                            unsigned char *st, uint64_t *bar,
                                            unsigned tile_idx, unsigned tile,
                                            const uint8_t *const (&pre)[kLeafPre]) {
    const uint8_t *const *rows = a.lrows + (size_t)q * a.lmax;
    unsigned n = 0;
#pragma unroll
    for (int j = 0; j < kLeafPre; ++j)
        if (n == (unsigned)j && pre[j] != nullptr) n = j + 1;
    if (n == kLeafPre)
        while (n < a.lmax && rows[n] != nullptr) ++n;
    fence_proxy_async();
    mbar_expect_tx(bar, a.rstride + n * tile);
    bulk_g2s(st, a.rec + (size_t)q * a.rstride, a.rstride, bar);
    const size_t off = (size_t)tile_idx * tile;
#pragma unroll
    for (int j = 0; j < kLeafPre; ++j)
        if ((unsigned)j < n) bulk_g2s(st + a.rstride + (size_t)j * tile, pre[j] + off, tile, bar);
    for (unsigned j = kLeafPre; j < n; ++j)
        bulk_g2s(st + a.rstride + (size_t)j * tile, rows[j] + off, tile, bar);
}

// Attempts of mbarrier.try_wait per record wait (set_spin_limit; the
// default is kSpinLimit, 0 gives up without waiting).  Read once per tile
// by the thread that waits.
__device__ uint32_t g_spin_limit = kSpinLimit;

cudaError_t set_spin_limit(uint32_t limit) {
    return cudaMemcpyToSymbol(g_spin_limit, &limit, sizeof(limit));
}

// Spin on a phase with an iteration bound; false if it gave up.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity,
                                                  uint32_t limit = kSpinLimit) {
    for (uint32_t it = 0; it < limit; ++it)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

// After a wait gave up at op (or step) o of n: wait, with the default
// bound, for the copies still in flight into the ring -- the stages of
// ops o .. o + R - 1 -- so that none lands after the CTA has left.
// `phase` is the parity state before op o's stage was flipped.
__device__ __noinline__ void drain_ring(uint64_t *bars, uint32_t phase, unsigned o,
                                        unsigned n, unsigned R) {
    for (unsigned q = o; q < n && q < o + R; ++q) {
        const unsigned st = q % R;
        mbar_wait_bounded(&bars[st], (phase >> st) & 1u);
    }
}

// The per-op hand-off barrier of the walkers: true when every thread's
// record wait succeeded.  `ok` is uniform within each warp.
__device__ __forceinline__ bool cta_hand_off(bool ok, unsigned nthr) {
    if (nthr == 32) {
        __syncwarp();
        return ok;
    }
    return __syncthreads_and(ok) != 0;
}

// Max of n values as a balanced tree (the same value as a left-to-right
// chain: fmax is exact and ignores NaN operands either way), so the
// dependent chain is log2(n) long instead of n.
template <int N, typename X>
__device__ __forceinline__ X tree_max(const X *v) {
    if constexpr (N == 1) {
        return v[0];
    } else {
        constexpr int H = N / 2;
        return fmax(tree_max<H>(v), tree_max<N - H>(v + H));
    }
}

// --- FP32 two-child ops by kind (one thread per pattern) --------------------
// One component's message m = P x: P comes as its four columns c (column j
// holds P[0..3][j]), every entry as a product, then three fused adds, in
// column order.
__device__ __forceinline__ void pcol(const float4 (&c)[4], const float *x, float *m) {
    m[0] = c[0].x * x[0];
    m[1] = c[0].y * x[0];
    m[2] = c[0].z * x[0];
    m[3] = c[0].w * x[0];
#pragma unroll
    for (int j = 1; j < 4; ++j) {
        m[0] = fmaf(c[j].x, x[j], m[0]);
        m[1] = fmaf(c[j].y, x[j], m[1]);
        m[2] = fmaf(c[j].z, x[j], m[2]);
        m[3] = fmaf(c[j].w, x[j], m[3]);
    }
}

// An internal child's rows and exponent: from its stack slot, or from HBM
// through L2 (the rows were written by this same thread earlier in the
// walk, or by an earlier launch).
template <int KT>
__device__ __forceinline__ int load_internal(const RecChild &c, const float4 *slots,
                                             const int *slot_sc, unsigned tile,
                                             unsigned pl, unsigned p, size_t ppad,
                                             float *x) {
    if (c.src == SRC_SLOT) {
        const float4 *s = slots + (size_t)c.idx * KT * tile + pl;
#pragma unroll
        for (int k = 0; k < KT; ++k) unpack(s[(size_t)k * tile], x + 4 * k);
        return slot_sc[(size_t)c.idx * tile + pl];
    }
    const float4 *g = static_cast<const float4 *>(c.data) + p;
#pragma unroll
    for (int k = 0; k < KT; ++k) unpack(__ldcg(g + (size_t)k * ppad), x + 4 * k);
    return __ldcg(static_cast<const int *>(c.scaler) + p);
}

// One two-child op of kind `kind` (OPK_*) for the NP patterns pl[h] (in
// the tile) / p[h] (in the CL buffers) a thread owns: acc[h] becomes the
// product of the two children's messages and lns[h] the sum of their
// exponents.  acc holds the previous op's result on entry (child A of the
// F kinds), with its exponents in lns.  `ia` is child A's record index; a
// streamed leaf's row is its rank among the op's leaf children.  Each P
// row is read from shared memory once for all NP patterns.
template <int KT, bool STAGED, int NP>
__device__ __forceinline__ void op2_kind(uint32_t kind, const unsigned char *rec,
                                         const RecChild *kids, unsigned ia,
                                         float (&acc)[NP][KT * 4], int (&lns)[NP],
                                         const uint8_t *masks, const uint8_t *lrow,
                                         const float4 *slots, const int *slot_sc,
                                         unsigned tile, const unsigned (&pl)[NP],
                                         const unsigned (&p)[NP], size_t ppad) {
    const RecChild &cA = kids[ia];
    const RecChild &cB = kids[ia ^ 1u];
    const float4 *PA = reinterpret_cast<const float4 *>(rec + cA.off);
    const float4 *PB = reinterpret_cast<const float4 *>(rec + cB.off);
    auto mask = [&](const RecChild &c, unsigned rank, unsigned q) -> unsigned {
        return STAGED ? masks[(size_t)c.idx * tile + q] : lrow[(size_t)rank * tile + q];
    };
    // y = a * b, one component (states 0..3) at a time.
    auto mul4 = [](float *y, const float *a, const float4 b) {
        y[0] = a[0] * b.x;
        y[1] = a[1] * b.y;
        y[2] = a[2] * b.z;
        y[3] = a[3] * b.w;
    };
    switch (kind) {
    case OPK_LL: {
        unsigned mA[NP], mB[NP];
#pragma unroll
        for (int h = 0; h < NP; ++h) {
            mA[h] = mask(cA, ia, pl[h]);
            mB[h] = mask(cB, ia ^ 1u, pl[h]);
        }
#pragma unroll
        for (int k = 0; k < KT; ++k)
#pragma unroll
            for (int h = 0; h < NP; ++h) {
                const float4 a = PA[k * 16 + mA[h]];
                const float ax[4] = {a.x, a.y, a.z, a.w};
                mul4(acc[h] + 4 * k, ax, PB[k * 16 + mB[h]]);
            }
#pragma unroll
        for (int h = 0; h < NP; ++h) lns[h] = 0;
        return;
    }
    case OPK_FL:
    case OPK_IL: {
        // A's rows: the previous result (FL) or loaded (IL); B a leaf.
        float xA[NP][KT * 4];
        int lA[NP];
#pragma unroll
        for (int h = 0; h < NP; ++h) {
            if (kind == OPK_IL) {
                lA[h] = load_internal<KT>(cA, slots, slot_sc, tile, pl[h], p[h], ppad, xA[h]);
            } else {
#pragma unroll
                for (int q = 0; q < KT * 4; ++q) xA[h][q] = acc[h][q];
                lA[h] = lns[h];
            }
        }
        unsigned mB[NP];
#pragma unroll
        for (int h = 0; h < NP; ++h) mB[h] = mask(cB, 0, pl[h]);
#pragma unroll
        for (int k = 0; k < KT; ++k) {
            const float4 ca[4] = {PA[k * 4], PA[k * 4 + 1], PA[k * 4 + 2], PA[k * 4 + 3]};
#pragma unroll
            for (int h = 0; h < NP; ++h) {
                float m[4];
                pcol(ca, xA[h] + 4 * k, m);
                mul4(acc[h] + 4 * k, m, PB[k * 16 + mB[h]]);
            }
        }
#pragma unroll
        for (int h = 0; h < NP; ++h) lns[h] = lA[h];
        return;
    }
    case OPK_FI: {
        float xB[NP][KT * 4];
        int lB[NP];
#pragma unroll
        for (int h = 0; h < NP; ++h)
            lB[h] = load_internal<KT>(cB, slots, slot_sc, tile, pl[h], p[h], ppad, xB[h]);
#pragma unroll
        for (int k = 0; k < KT; ++k) {
            const float4 ca[4] = {PA[k * 4], PA[k * 4 + 1], PA[k * 4 + 2], PA[k * 4 + 3]};
            const float4 cb[4] = {PB[k * 4], PB[k * 4 + 1], PB[k * 4 + 2], PB[k * 4 + 3]};
#pragma unroll
            for (int h = 0; h < NP; ++h) {
                float ma[4], mb[4];
                pcol(ca, acc[h] + 4 * k, ma);
                pcol(cb, xB[h] + 4 * k, mb);
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[h][4 * k + i] = ma[i] * mb[i];
            }
        }
#pragma unroll
        for (int h = 0; h < NP; ++h) lns[h] = lns[h] + lB[h];
        return;
    }
    default: {  // OPK_II
        float xA[NP][KT * 4], xB[NP][KT * 4];
        int lA[NP], lB[NP];
#pragma unroll
        for (int h = 0; h < NP; ++h) {
            lA[h] = load_internal<KT>(cA, slots, slot_sc, tile, pl[h], p[h], ppad, xA[h]);
            lB[h] = load_internal<KT>(cB, slots, slot_sc, tile, pl[h], p[h], ppad, xB[h]);
        }
#pragma unroll
        for (int k = 0; k < KT; ++k) {
            const float4 ca[4] = {PA[k * 4], PA[k * 4 + 1], PA[k * 4 + 2], PA[k * 4 + 3]};
            const float4 cb[4] = {PB[k * 4], PB[k * 4 + 1], PB[k * 4 + 2], PB[k * 4 + 3]};
#pragma unroll
            for (int h = 0; h < NP; ++h) {
                float ma[4], mb[4];
                pcol(ca, xA[h] + 4 * k, ma);
                pcol(cb, xB[h] + 4 * k, mb);
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[h][4 * k + i] = ma[i] * mb[i];
            }
        }
#pragma unroll
        for (int h = 0; h < NP; ++h) lns[h] = lA[h] + lB[h];
        return;
    }
    }
}

// ---------------------------------------------------------------------------
// The plan walker (one pattern per thread, or G threads per pattern).
//
// A CTA owns `tile` patterns and walks the whole plan.  Its op records come
// through a ring of kStages stages of `grp` consecutive ops each: one bulk
// copy for the group's records and one per leaf child for this tile's state
// masks, all completing on the stage's mbarrier.  Warps wait once per group,
// not per op, and run apart by up to the ring: the last warp to finish a
// group refills its stage (an atomic count per stage), so no block barrier
// and no waiting warp stands between ops.
//
// What bounds it: the FP32 form moves 4 K + 1 words per pattern and op to
// HBM (the parent CL), the FP64 form is bound by the narrow FP64 pipe, and a
// small plan by the latency of one warp's op after op.  So an op is
// straight-line code per kind with no loop over children, the FP32 products
// run two rows at a time (fma.rn.f32x2: P is stored by columns and x is
// broadcast; every entry keeps its order of operations), and the record's
// header and leaf masks are read one op ahead.
// ---------------------------------------------------------------------------
__host__ __device__ inline LeanLayout lean_layout(int precision, unsigned kact, unsigned tile,
                                                  unsigned nslot, unsigned grp,
                                                  unsigned rstride, unsigned lmax) {
    const size_t U = precision == CXG_FP32 ? 1 : 2;
    const size_t sc = precision == CXG_FP32 ? 4 : 8;
    LeanLayout L;
    L.stage0 = 128;  // mbarriers, counts and flags before it
    L.stage = (size_t)grp * (rstride + (size_t)lmax * tile);
    L.slots = L.stage0 + kStages * L.stage;
    L.slot_sc = L.slots + (size_t)nslot * kact * U * tile * 16;
    L.total = L.slot_sc + (((size_t)nslot * tile * sc + 15) & ~(size_t)15);
    return L;
}

size_t lean_smem_bytes(int precision, unsigned kact, unsigned tile, unsigned nslot,
                       unsigned grp, unsigned rstride, unsigned lmax) {
    return lean_layout(precision, kact, tile, nslot, grp, rstride, lmax).total;
}

// Shared words before the stages.
struct LeanHead {
    uint64_t full[kStages];  // a group's copies have arrived
    uint32_t done[kStages];  // warps that have finished the group
    uint32_t issued;         // groups of this item copied or in flight
    uint32_t abort;          // a wait gave up
};
static_assert(sizeof(LeanHead) <= 128, "the stages start at byte 128");

// Ring position of a CTA, kept across the items it walks: the stage of the
// next group and, per stage, the parity of its next completion.
struct RingPos {
    uint32_t stage, phase;
};

// This lane's leaf row of group g: the mask array of its child (lane =
// op in the group x lmax + rank), or null.
__device__ __forceinline__ const uint8_t *group_row(const PlanArgs &a, unsigned grp, unsigned g,
                                                    unsigned lane) {
    const unsigned o0 = g * grp;
    const unsigned n = min(grp, a.nops - o0);
    return lane < n * a.lmax ? a.lrows[(size_t)o0 * a.lmax + lane] : nullptr;
}

// Copy group g (its ops' records, and `rowb` mask bytes at pattern p0 of
// every leaf child) into stage memory `st`; called by all lanes of a warp.
__device__ __forceinline__ void issue_group(const PlanArgs &a, unsigned grp, unsigned g,
                                            unsigned char *st, uint64_t *bar, unsigned tile,
                                            unsigned p0, unsigned rowb, unsigned lane,
                                            const uint8_t *row) {
    const unsigned o0 = g * grp;
    const uint32_t rec = min(grp, a.nops - o0) * a.rstride;
    const unsigned nrow = __popc(__ballot_sync(0xffffffffu, row != nullptr));
    if (lane == 0) {
        fence_proxy_async();  // the stage's readers came before (the count's acquire)
        mbar_expect_tx(bar, rec + nrow * rowb);
        bulk_g2s(st, a.rec + (size_t)o0 * a.rstride, rec, bar);
    }
    __syncwarp();
    if (row != nullptr)
        bulk_g2s(st + (size_t)grp * a.rstride + (size_t)lane * tile, row + p0, rowb, bar);
}

// Wait for a group with an iteration bound; false if it gave up or another
// warp of the CTA has.
__device__ __forceinline__ bool wait_group(uint64_t *bar, uint32_t parity, uint32_t limit,
                                           volatile uint32_t *abort) {
    for (uint32_t it = 0; it < limit; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort) return false;
    }
    return false;
}

__device__ __forceinline__ uint32_t count_done(uint32_t *p) {
    uint32_t old;
    asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;"
                 : "=r"(old)
                 : "r"(smem_u32(p))
                 : "memory");
    return old;
}

// Two packed FP32 values (a register pair).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2f(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2f(f32x2 v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float max3f(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// The four states of one component: FP32 two pairs, FP64 four doubles; and
// this thread's KT components of one pattern.
template <typename T>
struct Quad;
template <>
struct Quad<float> {
    f32x2 v[2];
};
template <>
struct Quad<double> {
    double v[4];
};
template <typename T, int KT>
struct Rows {
    Quad<T> q[KT];
};

__device__ __forceinline__ Quad<float> quad(const float4 x) {
    return Quad<float>{{pack2f(x.x, x.y), pack2f(x.z, x.w)}};
}
__device__ __forceinline__ Quad<double> quad(const double2 x, const double2 y) {
    return Quad<double>{{x.x, x.y, y.x, y.y}};
}
__device__ __forceinline__ void unquad(const Quad<float> &q, float *x) {
    unpack2f(q.v[0], x[0], x[1]);
    unpack2f(q.v[1], x[2], x[3]);
}
__device__ __forceinline__ void unquad(const Quad<double> &q, double *x) {
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = q.v[i];
}
__device__ __forceinline__ Quad<float> operator*(const Quad<float> &a, const Quad<float> &b) {
    return Quad<float>{{mul2(a.v[0], b.v[0]), mul2(a.v[1], b.v[1])}};
}
__device__ __forceinline__ Quad<double> operator*(const Quad<double> &a, const Quad<double> &b) {
    return Quad<double>{
        {a.v[0] * b.v[0], a.v[1] * b.v[1], a.v[2] * b.v[2], a.v[3] * b.v[3]}};
}

// Rows from HBM (through L2: they may have been written by this walk) and
// from the stack in shared memory; unit stride `stride`.
template <int KT>
__device__ __forceinline__ void load_l2(const float4 *p, size_t stride, Rows<float, KT> &r) {
#pragma unroll
    for (int k = 0; k < KT; ++k) r.q[k] = quad(__ldcg(p + (size_t)k * stride));
}
template <int KT>
__device__ __forceinline__ void load_l2(const double2 *p, size_t stride, Rows<double, KT> &r) {
#pragma unroll
    for (int k = 0; k < KT; ++k)
        r.q[k] = quad(__ldcg(p + (size_t)(2 * k) * stride),
                      __ldcg(p + (size_t)(2 * k + 1) * stride));
}
template <int KT>
__device__ __forceinline__ void load_smem(const float4 *p, unsigned stride, Rows<float, KT> &r) {
#pragma unroll
    for (int k = 0; k < KT; ++k) r.q[k] = quad(p[k * stride]);
}
template <int KT>
__device__ __forceinline__ void load_smem(const double2 *p, unsigned stride,
                                          Rows<double, KT> &r) {
#pragma unroll
    for (int k = 0; k < KT; ++k) r.q[k] = quad(p[2 * k * stride], p[(2 * k + 1) * stride]);
}
template <int KT>
__device__ __forceinline__ void store_rows(float4 *p, size_t stride, const Rows<float, KT> &r) {
#pragma unroll
    for (int k = 0; k < KT; ++k) {
        float x[4];
        unquad(r.q[k], x);
        p[(size_t)k * stride] = pack4(x);
    }
}
template <int KT>
__device__ __forceinline__ void store_rows(double2 *p, size_t stride,
                                           const Rows<double, KT> &r) {
#pragma unroll
    for (int k = 0; k < KT; ++k) {
        p[(size_t)(2 * k) * stride] = make_double2(r.q[k].v[0], r.q[k].v[1]);
        p[(size_t)(2 * k + 1) * stride] = make_double2(r.q[k].v[2], r.q[k].v[3]);
    }
}

// One component's message of an internal child, P x (P in shared memory:
// FP32 by columns, FP64 by rows), every entry a product and three fused adds
// in column order.
__device__ __forceinline__ Quad<float> matvec(const float4 *P, const Quad<float> &x) {
    float s[4];
    unquad(x, s);
    Quad<float> m;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const Quad<float> c = quad(P[j]);
        const f32x2 d = pack2f(s[j], s[j]);
        m.v[0] = j == 0 ? mul2(c.v[0], d) : fma2(c.v[0], d, m.v[0]);
        m.v[1] = j == 0 ? mul2(c.v[1], d) : fma2(c.v[1], d, m.v[1]);
    }
    return m;
}
__device__ __forceinline__ Quad<double> matvec(const double2 *P, const Quad<double> &x) {
    Quad<double> m;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double2 a = P[2 * i], b = P[2 * i + 1];
        double v = a.x * x.v[0];
        v = fma(a.y, x.v[1], v);
        v = fma(b.x, x.v[2], v);
        m.v[i] = fma(b.y, x.v[3], v);
    }
    return m;
}

// Largest entry of a pattern's rows.  FP32: the value (operands that are
// NaN are passed over, as fmax does).  FP64: the exponent word of the
// largest of entries that are >= 0 (the sign bit is clear, so the high words
// order as the values; a NaN orders above infinity), on the integer pipe.
template <int KT>
__device__ __forceinline__ float rows_max(const Rows<float, KT> &r) {
    float m = 0.0f;
#pragma unroll
    for (int k = 0; k < KT; ++k) {
        float x[4];
        unquad(r.q[k], x);
        m = max3f(max3f(x[0], x[1], x[2]), x[3], m);
    }
    return m;
}
template <int KT>
__device__ __forceinline__ int rows_max(const Rows<double, KT> &r) {
    int m = 0;
#pragma unroll
    for (int k = 0; k < KT; ++k) {
        const double *x = r.q[k].v;
        const int a = max(__double2hiint(x[0]), __double2hiint(x[1]));
        const int b = max(__double2hiint(x[2]), __double2hiint(x[3]));
        m = max(m, max(a, b));
    }
    return m;
}
__device__ __forceinline__ float vmax(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ int vmax(int a, int b) { return max(a, b); }

// Max over the G consecutive lanes that share a pattern.
template <int G, typename X>
__device__ __forceinline__ X group_max(X x) {
#pragma unroll
    for (int o = 1; o < G; o <<= 1) x = vmax(x, __shfl_xor_sync(0xffffffffu, x, o));
    return x;
}

// Rescale a pattern's rows by an exact power of two when their largest
// entry has fallen low.
//
// FP32: below 2^-16 (or after a product of more than two messages): to
// [0.5, 1), the exponent added to the integer scaler.  Every entry is at
// most 1, a binary op's result then keeps its largest entry far above the
// FP32 normal range's floor, and the scaling is exact, so a rescale that is
// skipped changes no mantissa.
template <int KT, int G>
__device__ __forceinline__ void rescale(Rows<float, KT> &r, int &lns, bool always) {
    const float mx = group_max<G>(rows_max(r));
    if (!(mx > 0.0f && mx <= 3.0e38f && (always || mx < 1.52587890625e-05f))) return;
    const int e0 = __float_as_int(mx) >> 23;  // biased exponent (0: subnormal)
    if (e0 >= 1 && e0 <= 252) {
        // 2^n with n = 126 - e0: the exponent frexp gives is e0 - 126.
        const float s = __int_as_float((253 - e0) << 23);
        const f32x2 ss = pack2f(s, s);
#pragma unroll
        for (int k = 0; k < KT; ++k) {
            r.q[k].v[0] = mul2(r.q[k].v[0], ss);
            r.q[k].v[1] = mul2(r.q[k].v[1], ss);
        }
        lns += e0 - 126;
        return;
    }
    int e;
    frexpf(mx, &e);
    const int n = -e, n1 = n / 2, n2 = n - n1;
    const f32x2 s1 = pack2f(pow2f(n1), pow2f(n1)), s2 = pack2f(pow2f(n2), pow2f(n2));
#pragma unroll
    for (int k = 0; k < KT; ++k) {
        r.q[k].v[0] = mul2(mul2(r.q[k].v[0], s1), s2);
        r.q[k].v[1] = mul2(mul2(r.q[k].v[1], s1), s2);
    }
    lns += e;
}
// FP64: below 2^-256 (or at 2^256), to [1, 2), and its exponent times ln 2 joins the log
// scaler.  The reference divides by the largest child message and adds its
// log on every op (CxLik.c:390-403, 577-588); the product of rows and scale
// is the same, the power of two is exact, and the FP64 pipe, which bounds
// this form, is spared a reciprocal, 4 K products and a log per op (134 to
// about 80 FP64 instructions per update).  Two children at or above 2^-256
// give products far above the normal range's floor.  Rows of zeros stay, and
// a pattern with an infinite entry ends with NaN rows, as dividing by an
// infinite scaler leaves it: its site lnL is -inf either way.
template <int KT, int G>
__device__ __forceinline__ void rescale(Rows<double, KT> &r, double &lns, bool) {
    const int hi = group_max<G>(rows_max(r));
    constexpr int kLow = (1023 - 256) << 20, kHigh = (1023 + 256) << 20;
    if (hi >= kLow && hi < kHigh) return;
    double s;
    if (hi >= 0x7ff00000) {
        s = 0.0;  // infinity times 0: NaN
        lns = INFINITY;
    } else {
        // (Below the normal range -- zeros among it -- the scale is 2^1000,
        // which brings any entry that is not 0 above 2^-256.)
        int e = hi < (1 << 20) ? -1000 : (hi >> 20) - 1023;
        e = min(max(e, -1000), 1000);
        s = __hiloint2double((1023 - e) << 20, 0);
        lns = fma((double)e, 0.69314718055994530942, lns);
    }
#pragma unroll
    for (int k = 0; k < KT; ++k)
#pragma unroll
        for (int i = 0; i < 4; ++i) r.q[k].v[i] *= s;
}

// A warp's view of the tile it walks.
template <typename T>
struct TileView {
    typedef typename Prec<T>::V V;
    typedef typename Prec<T>::S S;
    V *slots;
    S *slot_sc;
    const double *ltab;  // FP64: leaf-message tables
    size_t ppad;
    unsigned tile, pl, p, k0;
};

// An internal child's rows and scaler: from its stack slot, or from HBM
// through L2 (rows this same thread wrote earlier in the walk, or an
// earlier launch did).  `cr` is the child's descriptor in the record.
template <typename T, int KT, int G>
__device__ __forceinline__ typename Prec<T>::S child_rows(const unsigned char *cr,
                                                          const TileView<T> &w,
                                                          Rows<T, KT> &x) {
    typedef typename Prec<T>::V V;
    typedef typename Prec<T>::S S;
    constexpr int U = Prec<T>::U;
    const RecChild *c = reinterpret_cast<const RecChild *>(cr);
    const ulonglong2 ptr = *reinterpret_cast<const ulonglong2 *>(cr);
    const uint2 si = *reinterpret_cast<const uint2 *>(&c->src);
    if (si.x == SRC_SLOT) {
        load_smem<KT>(w.slots + (si.y * (KT * G) + w.k0) * U * w.tile + w.pl, w.tile, x);
        return w.slot_sc[si.y * w.tile + w.pl];
    }
    load_l2<KT>(reinterpret_cast<const V *>(ptr.x) + (size_t)w.k0 * U * w.ppad + w.p, w.ppad, x);
    return __ldcg(reinterpret_cast<const S *>(ptr.y) + w.p);
}

// Component k (of this thread's) of the message of a leaf child with state
// mask m.  FP32: from the table in the record at `area`; FP64: from table
// `tab` in HBM.
template <int KA>
__device__ __forceinline__ Quad<float> leaf_message(const unsigned char *area, unsigned,
                                                    unsigned m, const TileView<float> &w,
                                                    int k) {
    return quad(reinterpret_cast<const float4 *>(area)[(w.k0 + k) * 16 + m]);
}
template <int KA>
__device__ __forceinline__ Quad<double> leaf_message(const unsigned char *, unsigned tab,
                                                     unsigned m, const TileView<double> &w,
                                                     int k) {
    const double2 *t = reinterpret_cast<const double2 *>(
        w.ltab + (((size_t)tab * 16 + m) * KA + w.k0 + k) * 4);
    return quad(__ldg(t), __ldg(t + 1));
}

// One op.  `acc` and `lns` hold the previous op's result on entry and this
// op's on return; m0 and m1 are the state masks of its first two leaf
// children, `rows` this pattern's mask of the op's leaf children (one per
// `tile` bytes).  Two-child ops run the code of their kind (an op's kind and
// the child that plays A are in its flags), others a loop over children.
// The product of two messages and the sum of two scalers are the same in
// either order, so every path gives the same bits.
template <typename T, int KT, int G>
__device__ __forceinline__ void walk_op(const unsigned char *rec, unsigned nchild, uint32_t flags,
                                        bool first, unsigned m0, unsigned m1,
                                        const uint8_t *rows, const TileView<T> &w,
                                        Rows<T, KT> &acc, typename Prec<T>::S &lns) {
    typedef typename Prec<T>::V V;
    typedef typename Prec<T>::S S;
    constexpr int KA = KT * G;
    constexpr unsigned PB = KA * 16 * sizeof(T);                       // bytes of a P area
    constexpr unsigned LB = sizeof(T) == 4 ? KA * 16 * 4 * 4 : PB;     // of a leaf's area
    constexpr unsigned PU = 16 * sizeof(T) / 16;                       // P units per component
    constexpr unsigned A0 = sizeof(RecHead) + 2 * sizeof(RecChild);
    const unsigned ia = (flags & kOpKindA) ? 1u : 0u;
    const unsigned char *kid0 = rec + sizeof(RecHead);
    uint32_t kind = (flags >> kOpKindShift) & 7u;
    // A walk that starts inside a plan (one launch per node) holds no
    // previous result.
    if (first && (kind == OPK_FL || kind == OPK_FI)) kind = OPK_GENERIC;
    auto tab_of = [&](unsigned c) -> unsigned {
        return sizeof(T) == 8 ? reinterpret_cast<const RecChild *>(kid0)[c].tab : 0u;
    };
    auto pmat = [&](const unsigned char *area) {
        return reinterpret_cast<const V *>(area) + (size_t)w.k0 * PU;
    };
    if (kind == OPK_FL || kind == OPK_IL) {
        const unsigned char *aA = rec + A0 + (ia ? LB : 0u), *aB = rec + A0 + (ia ? 0u : PB);
        if (kind == OPK_IL) lns = child_rows<T, KT, G>(kid0 + ia * sizeof(RecChild), w, acc);
        const V *P = pmat(aA);
        const unsigned tab = tab_of(ia ^ 1u);
#pragma unroll
        for (int k = 0; k < KT; ++k)
            acc.q[k] = matvec(P + k * PU, acc.q[k]) * leaf_message<KA>(aB, tab, m0, w, k);
    } else if (kind == OPK_LL) {
        lns = S(0);
        const unsigned t0 = tab_of(0), t1 = tab_of(1);
#pragma unroll
        for (int k = 0; k < KT; ++k)
            acc.q[k] = leaf_message<KA>(rec + A0, t0, m0, w, k) *
                       leaf_message<KA>(rec + A0 + LB, t1, m1, w, k);
    } else if (kind == OPK_FI || kind == OPK_II) {
        const unsigned char *aA = rec + A0 + (ia ? PB : 0u), *aB = rec + A0 + (ia ? 0u : PB);
        Rows<T, KT> xb;
        const S lb = child_rows<T, KT, G>(kid0 + (ia ^ 1u) * sizeof(RecChild), w, xb);
        if (kind == OPK_II) lns = child_rows<T, KT, G>(kid0 + ia * sizeof(RecChild), w, acc);
        const V *PA = pmat(aA), *PX = pmat(aB);
        // (The previous result's products come first: the sibling's rows
        // are on their way from L2.)
#pragma unroll
        for (int k = 0; k < KT; ++k) acc.q[k] = matvec(PA + k * PU, acc.q[k]);
#pragma unroll
        for (int k = 0; k < KT; ++k) acc.q[k] = acc.q[k] * matvec(PX + k * PU, xb.q[k]);
        lns = lns + lb;
    } else {
        // Any number of children, each read from where its record says.
        lns = S(0);
        unsigned nl = 0;
#pragma unroll 1
        for (unsigned ci = 0; ci < nchild; ++ci) {
            const unsigned char *cr = kid0 + ci * sizeof(RecChild);
            const uint4 d = *reinterpret_cast<const uint4 *>(cr + 16);  // src idx tab off
            Rows<T, KT> x;
            if (d.x == SRC_LEAF) {
                const unsigned m = rows[(nl++) * w.tile];
#pragma unroll
                for (int k = 0; k < KT; ++k) x.q[k] = leaf_message<KA>(rec + d.w, d.z, m, w, k);
            } else {
                lns = lns + child_rows<T, KT, G>(cr, w, x);
                const V *P = pmat(rec + d.w);
#pragma unroll
                for (int k = 0; k < KT; ++k) x.q[k] = matvec(P + k * PU, x.q[k]);
            }
            if (ci == 0) {
                acc = x;
            } else {
#pragma unroll
                for (int k = 0; k < KT; ++k) acc.q[k] = acc.q[k] * x.q[k];
            }
            // (The FP64 form keeps a long product inside the range.)
            if (sizeof(T) == 8 && ci >= 1 && ci + 1 < nchild) rescale<KT, G>(acc, lns, false);
        }
    }
}

// Walk every op of job `a` for tile `tile_idx`, aggregate the root and
// reduce.  G consecutive threads share a pattern, each holding KT of its
// KT*G components; with G = 1 one thread owns a pattern.  Every G and every
// tile gives the same bits: scalers are maxima over the group, and the root
// sum and the tile reduction run in the G = 1 order.  Returns false if a
// bounded wait gave up.
template <typename T, int KT, int G>
__device__ bool walk_tile(const PlanArgs &a, unsigned tile_idx, const LeanLayout &Lay,
                          unsigned grp, RingPos &ring) {
    typedef typename Prec<T>::S S;
    typedef typename Prec<T>::V V;
    constexpr int U = Prec<T>::U;
    extern __shared__ __align__(128) unsigned char smem[];
    LeanHead &hd = *reinterpret_cast<LeanHead *>(smem);
    const unsigned nthr = blockDim.x, nwarp = nthr / 32;
    const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const unsigned tile = nthr / G;
    const unsigned p0 = tile_idx * tile;
    const unsigned g = tid % G;
    TileView<T> w;
    w.slots = reinterpret_cast<V *>(smem + Lay.slots);
    w.slot_sc = reinterpret_cast<S *>(smem + Lay.slot_sc);
    w.ltab = a.ltab;
    w.ppad = a.ppad;
    w.tile = tile;
    w.pl = tid / G;
    w.p = p0 + w.pl;
    w.k0 = g * KT;
    const unsigned p = w.p;
    // The last tile of a job may pass its padded patterns by whole warps
    // (32 / G patterns each, and the padding is to 128).
    const bool on = p < a.ppad;
    const unsigned rowb = min(tile, a.ppad - p0);
    const unsigned ngrp = (a.nops + grp - 1) / grp;
    const unsigned lmax = a.lmax;
    const uint32_t spin = g_spin_limit;
    const RingPos start = ring;

    pdl_wait();  // the records hold the P kernel's matrices
    if (warp == 0) {
        unsigned st = ring.stage;
        const unsigned n = min(ngrp, kStages);
        for (unsigned q = 0; q < n; ++q) {
            issue_group(a, grp, q, smem + Lay.stage0 + st * Lay.stage, &hd.full[st], tile, p0,
                        rowb, lane, group_row(a, grp, q, lane));
            st = st + 1 == kStages ? 0u : st + 1;
        }
        if (lane == 0) hd.issued = n;
    }

    Rows<T, KT> acc;
    S lns = S(0);
    bool ok = true;
    for (unsigned q = 0; q < ngrp; ++q) {
        unsigned char *st = smem + Lay.stage0 + ring.stage * Lay.stage;
        uint64_t *bar = &hd.full[ring.stage];
        // The group that refills this stage: its leaf rows' addresses are
        // read now, long before they are needed.
        const bool refill = q + kStages < ngrp;
        const uint8_t *row = refill ? group_row(a, grp, q + kStages, lane) : nullptr;
        ok = __all_sync(0xffffffffu, wait_group(bar, (ring.phase >> ring.stage) & 1u, spin,
                                                &hd.abort));
        ring.phase ^= 1u << ring.stage;
        if (!ok) {
            if (lane == 0) {
                atomicOr(a.err, 1u);
                *(volatile uint32_t *)&hd.abort = 1u;
            }
            break;
        }
        if (on) {
            const unsigned n = min(grp, a.nops - q * grp);
            const unsigned char *rec = st;
            const uint8_t *rows = st + (size_t)grp * a.rstride + w.pl;
            // The first record's header and masks; then each op reads the
            // next one's ahead.
            ulonglong2 h0 = *reinterpret_cast<const ulonglong2 *>(rec);
            uint4 h1 = *reinterpret_cast<const uint4 *>(rec + 16);
            unsigned m0 = lmax > 0 ? rows[0] : 0u, m1 = lmax > 1 ? rows[tile] : 0u;
            for (unsigned b = 0; b < n; ++b) {
                const unsigned char *nrec = rec + a.rstride;
                const uint8_t *nrows = rows + (size_t)lmax * tile;
                ulonglong2 n0 = h0;
                uint4 n1 = h1;
                unsigned nm0 = 0u, nm1 = 0u;
                if (b + 1 < n) {
                    n0 = *reinterpret_cast<const ulonglong2 *>(nrec);
                    n1 = *reinterpret_cast<const uint4 *>(nrec + 16);
                    if (lmax > 0) nm0 = nrows[0];
                    if (lmax > 1) nm1 = nrows[tile];
                }
                walk_op<T, KT, G>(rec, h1.x, h1.z, (q | b) == 0u, m0, m1, rows, w, acc, lns);
                rescale<KT, G>(acc, lns, h1.x > 2u);
                if (!(h1.z & REC_NO_HBM)) {
                    store_rows<KT>(reinterpret_cast<V *>(h0.x) + (size_t)w.k0 * U * w.ppad + p,
                                   w.ppad, acc);
                    if (g == 0) reinterpret_cast<S *>(h0.y)[p] = lns;
                }
                if ((int)h1.y >= 0) {
                    store_rows<KT>(w.slots + (h1.y * (KT * G) + w.k0) * U * tile + w.pl, tile,
                                   acc);
                    if (g == 0) w.slot_sc[h1.y * tile + w.pl] = lns;
                }
                if (G > 1) __syncwarp();  // lane g = 0's scaler is read by the group
                rec = nrec;
                rows = nrows;
                h0 = n0;
                h1 = n1;
                m0 = nm0;
                m1 = nm1;
            }
        }
        if (refill) {
            // The last warp to finish the group hands its stage on.
            __syncwarp();
            unsigned last = 1;
            if (nwarp > 1) {
                if (lane == 0) {
                    last = count_done(&hd.done[ring.stage]) == nwarp - 1;
                    if (last) hd.done[ring.stage] = 0;
                }
                last = __shfl_sync(0xffffffffu, last, 0);
            }
            if (last) {
                issue_group(a, grp, q + kStages, st, bar, tile, p0, rowb, lane, row);
                if (lane == 0) hd.issued = q + kStages + 1;
            }
        }
        ring.stage = ring.stage + 1 == kStages ? 0u : ring.stage + 1;
    }
    if (__syncthreads_or(!ok)) {
        // A wait gave up: wait, with the default bound, for the copies still
        // in flight into the ring, so that none lands after the CTA has left.
        if (tid == 0) {
            const unsigned n = hd.issued;
            for (unsigned q = n > kStages ? n - kStages : 0; q < n; ++q) {
                const unsigned st = (start.stage + q) % kStages;
                mbar_wait_bounded(&hd.full[st], ((start.phase >> st) ^ (q / kStages)) & 1u);
            }
        }
        return false;
    }

    if (a.no_root) return true;
    // Root aggregation (CxLik.c:598-632): L = sum_k sum_i pn[k][i] root.
    if (!a.root_last && on) {
        load_l2<KT>(static_cast<const V *>(a.root) + (size_t)w.k0 * U * w.ppad + p, w.ppad, acc);
        lns = static_cast<const S *>(a.rootsc)[p];
    }
    T x[KT * 4];
#pragma unroll
    for (int k = 0; k < KT; ++k) unquad(acc.q[k], x + 4 * k);
    // Lsum = sum over components and states in one sequential order; every
    // lane of the group gathers the others' entries and sums them all.
    double Lsum = 0.0;
    const unsigned lead = lane - g;
#pragma unroll
    for (int gg = 0; gg < G; ++gg) {
#pragma unroll
        for (int q = 0; q < KT * 4; ++q) {
            const T y = G > 1 ? __shfl_sync(0xffffffffu, x[q], lead + gg) : x[q];
            Lsum = fma(__ldg(a.pn + gg * KT * 4 + q), (double)y, Lsum);
        }
    }
    double v = 0.0;
    bool ninf = false;
    if (g == 0 && p < a.npat) {
        const double lsc = (sizeof(T) == 8) ? (double)lns
                                           : (double)lns * 0.69314718055994530942;
        v = (log(Lsum) + lsc) * (double)a.freqs[p];
        if (isnan(v)) v = -INFINITY;
        if (a.site) a.site[p] = v;
        if (isinf(v)) {
            ninf = (v < 0.0);
            v = 0.0;
        }
    }
    if (G > 1) {
        // Pattern pl's value moves to thread pl, so the tile reduces in the
        // one-thread-per-pattern order (the extra threads add exact zeros).
        __shared__ double s_v[kBlock];
        __shared__ unsigned char s_inf[kBlock];
        if (g == 0) {
            s_v[w.pl] = v;
            s_inf[w.pl] = ninf;
        }
        __syncthreads();
        v = tid < tile ? s_v[tid] : 0.0;
        ninf = tid < tile ? s_inf[tid] != 0 : false;
    }
    reduce_sites(a, tile_idx, v, ninf);
    return true;
}
// The walker with two op lanes (FP32, one thread per pattern, staged
// leaves): the CTA is two groups of `tile` threads over the same patterns.
// The host schedules the plan in steps of two mutually independent ops (a
// record with no children fills an empty lane) and a ring stage holds one
// step's two records; lane l runs the step's l-th op.  A result one lane
// writes is read by the other only in a later step, after the block barrier
// between steps.  The root is the last step's lane-0 op, so lane 0
// aggregates it and the other adds exact zeros to the tile sum: the bits are
// those of walk_tile.  `phase` holds, per ring stage, the parity of the next
// completion to wait for.  Returns false if a bounded wait gave up.
template <int KT>
__device__ bool walk_tile_lanes(const PlanArgs &a, unsigned tile_idx, const SmemLayout &Lay,
                                unsigned ring_depth, uint32_t &phase) {
    typedef float T;
    constexpr unsigned L = 2;
    extern __shared__ __align__(128) unsigned char smem[];
    const unsigned nthr = blockDim.x;
    const unsigned tile = nthr / L;
    const unsigned tid = threadIdx.x;
    const unsigned lane = tid / tile;  // op lane of this thread
    const unsigned pl = tid % tile;    // pattern within the tile
    const unsigned p = tile_idx * tile + pl;
    const size_t ppad = a.ppad;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + Lay.bars);
    unsigned char *ring = smem + Lay.ring;
    float4 *slots = reinterpret_cast<float4 *>(smem + Lay.slots);
    int *slot_sc = reinterpret_cast<int *>(smem + Lay.slot_sc);
    const size_t sstride = (size_t)a.rstride * L;
    uint8_t *masks = smem + Lay.masks;
    const unsigned R = ring_depth;
    const unsigned nsteps = a.nops / L;  // the host pads nops to a multiple

    pdl_wait();  // the records hold the P kernel's matrices
    // Start streaming the job's first R steps of op records.
    if (tid == 0) {
        fence_proxy_async();
        for (unsigned o = 0; o < R && o < nsteps; ++o) {
            mbar_expect_tx(&bars[o], (uint32_t)sstride);
            bulk_g2s(ring + (size_t)o * sstride, a.rec + (size_t)o * sstride,
                     (uint32_t)sstride, &bars[o]);
        }
    }
    // Stage this tile's leaf masks with 16-byte loads.
    const unsigned chunks = tile / 16;
    for (unsigned i = tid; i < a.nleaf * chunks; i += nthr) {
        const unsigned l = i / chunks, c = i % chunks;
        const uint4 *src =
            reinterpret_cast<const uint4 *>(a.leaves[l] + (size_t)tile_idx * tile) + c;
        reinterpret_cast<uint4 *>(masks + (size_t)l * tile)[c] = __ldg(src);
    }
    __syncthreads();

    T acc[KT * 4];
    int lns = 0;
    const uint32_t spin = g_spin_limit;
    for (unsigned o = 0, stage = 0; o < nsteps;
         ++o, stage = (stage + 1 == R) ? 0u : stage + 1) {
        // Every thread waits for the step's records itself (one block
        // barrier per step, the hand-off below); a warp computes only if all
        // its threads saw the records arrive.
        const bool ok =
            __all_sync(0xffffffffu, mbar_wait_bounded(&bars[stage], (phase >> stage) & 1u,
                                                      spin));
        phase ^= 1u << stage;
        void *ydata = nullptr, *yscaler = nullptr;
        int yslot = -1;
        bool yhbm = false;
        unsigned nchild = 0;
        if (ok) {
            const unsigned char *rec =
                ring + (size_t)stage * sstride + (size_t)lane * a.rstride;
            const RecHead *hd = reinterpret_cast<const RecHead *>(rec);
            const RecChild *kids = reinterpret_cast<const RecChild *>(rec + sizeof(RecHead));
            nchild = hd->nchild;
            lns = 0;
            // A child's inputs: its state rows (internal) with its scaler, or
            // its leaf's state mask.  Loading them is split from computing
            // the message so that an op with two children issues both
            // children's loads before it waits on either.
            struct In {
                T x[KT * 4];
                int l;
                unsigned m;
            };
            auto load_in = [&](const RecChild &ch, In &in) {
                in.m = 0u;
                if (ch.src == SRC_LEAF)
                    in.m = masks[(size_t)ch.idx * tile + pl];
                else
                    in.l = load_internal<KT>(ch, slots, slot_sc, tile, pl, p, ppad, in.x);
            };
            auto message = [&](const RecChild &ch, const In &in, T *msg) {
                const float4 *P = reinterpret_cast<const float4 *>(rec + ch.off);
#pragma unroll
                for (int k = 0; k < KT; ++k) {
                    if (ch.src == SRC_LEAF) {
                        unpack(P[k * 16 + in.m], msg + 4 * k);
                    } else {
                        const float4 c[4] = {P[k * 4], P[k * 4 + 1], P[k * 4 + 2],
                                             P[k * 4 + 3]};
                        pcol(c, in.x + 4 * k, msg + 4 * k);
                    }
                }
            };
            auto fold = [&](unsigned ci, const RecChild &ch, const In &in, const T *msg) {
                if (ch.src != SRC_LEAF) lns = lns + in.l;
#pragma unroll
                for (int q = 0; q < KT * 4; ++q) acc[q] = ci == 0 ? msg[q] : acc[q] * msg[q];
            };
            T msg[KT * 4];
            if (nchild == 2) {
                const RecChild c0 = kids[0], c1 = kids[1];
                In in0, in1;
                load_in(c0, in0);
                load_in(c1, in1);
                message(c0, in0, msg);
                fold(0, c0, in0, msg);
                message(c1, in1, msg);
                fold(1, c1, in1, msg);
            } else {
                for (unsigned ci = 0; ci < nchild; ++ci) {
                    const RecChild ch = kids[ci];
                    In in;
                    load_in(ch, in);
                    message(ch, in, msg);
                    fold(ci, ch, in, msg);
                }
            }
            ydata = hd->data;
            yscaler = hd->scaler;
            yslot = hd->slot;
            yhbm = !(hd->flags & REC_NO_HBM);
        }
        // Every thread has read the stage: hand it to step o + R.  A record
        // wait that gave up in any warp ends the tile for all: thread 0
        // waits for the copies still in flight into the ring.
        if (!cta_hand_off(ok, nthr)) {
            if (tid == 0) {
                atomicOr(a.err, 1u);
                drain_ring(bars, phase ^ (1u << stage), o, nsteps, R);
            }
            return false;
        }
        if (tid == 0 && o + R < nsteps) {
            fence_proxy_async();
            mbar_expect_tx(&bars[stage], (uint32_t)sstride);
            bulk_g2s(ring + (size_t)stage * sstride, a.rec + (size_t)(o + R) * sstride,
                     (uint32_t)sstride, &bars[stage]);
        }
        // An empty lane of a step (no children) computes and stores nothing.
        if (nchild == 0) continue;
        const T mx = fmax(T(0), tree_max<KT * 4>(acc));
        // The rescale rule of walk_tile (same bits).
        if (mx > T(0) && mx <= (T)3.0e38 && (nchild > 2 || mx < (T)1.52587890625e-05f)) {
            int e;
            frexpf(mx, &e);
            const int n = -e, n1 = n / 2, n2 = n - n1;
            const float s1 = pow2f(n1), s2 = pow2f(n2);
#pragma unroll
            for (int q = 0; q < KT * 4; ++q) acc[q] = (acc[q] * s1) * s2;
            lns = lns + e;
        }
        if (yhbm) {
            float4 *y = static_cast<float4 *>(ydata) + p;
#pragma unroll
            for (int k = 0; k < KT; ++k) y[(size_t)k * ppad] = pack4(acc + k * 4);
            static_cast<int *>(yscaler)[p] = lns;
        }
        if (yslot >= 0) {
            float4 *ys = slots + (size_t)yslot * KT * tile + pl;
#pragma unroll
            for (int k = 0; k < KT; ++k) ys[(size_t)k * tile] = pack4(acc + k * 4);
            slot_sc[(size_t)yslot * tile + pl] = lns;
        }
    }

    if (a.no_root) {
        __syncthreads();
        return true;
    }
    // Root aggregation (CxLik.c:598-632), lane 0's.
    if (!a.root_last) {
        const float4 *r = static_cast<const float4 *>(a.root) + p;
#pragma unroll
        for (int k = 0; k < KT; ++k) unpack(r[(size_t)k * ppad], acc + k * 4);
        lns = static_cast<const int *>(a.rootsc)[p];
    }
    double Lsum = 0.0;
#pragma unroll
    for (int q = 0; q < KT * 4; ++q) Lsum = fma(__ldg(a.pn + q), (double)acc[q], Lsum);
    double v = 0.0;
    bool ninf = false;
    if (lane == 0 && p < a.npat) {
        v = (log(Lsum) + (double)lns * 0.69314718055994530942) * (double)a.freqs[p];
        if (isnan(v)) v = -INFINITY;
        if (a.site) a.site[p] = v;
        if (isinf(v)) {
            ninf = (v < 0.0);
            v = 0.0;
        }
    }
    reduce_sites(a, tile_idx, v, ninf);
    return true;
}

// The FP32 walker with two patterns per thread (one thread per pattern
// pair, components not split): thread t owns patterns t and t + blockDim
// of the tile, so loads stay coalesced, and every P row, record field and
// loop step serves both.  The arithmetic of each pattern is that of
// walk_tile<float, K, 1, STAGED>, and the tile reduction runs in its order,
// so the bits are the same.
template <int K, bool STAGED>
__device__ bool walk_tile2(const PlanArgs &a, unsigned tile_idx, const SmemLayout &Lay,
                           unsigned ring_depth, uint32_t &phase) {
    typedef float T;
    extern __shared__ __align__(128) unsigned char smem[];
    const unsigned nthr = blockDim.x;
    const unsigned tile = 2 * nthr;
    const unsigned tid = threadIdx.x;
    const unsigned pl[2] = {tid, tid + nthr};
    const unsigned p[2] = {tile_idx * tile + tid, tile_idx * tile + tid + nthr};
    const size_t ppad = a.ppad;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + Lay.bars);
    unsigned char *ring = smem + Lay.ring;
    float4 *slots = reinterpret_cast<float4 *>(smem + Lay.slots);
    int *slot_sc = reinterpret_cast<int *>(smem + Lay.slot_sc);
    const size_t sstride = STAGED ? (size_t)a.rstride : Lay.stage;
    uint8_t *masks = smem + Lay.masks;
    const unsigned R = ring_depth;

    if (STAGED) {
        pdl_wait();
        if (tid == 0) {
            fence_proxy_async();
            for (unsigned o = 0; o < R && o < a.nops; ++o) {
                mbar_expect_tx(&bars[o], a.rstride);
                bulk_g2s(ring + (size_t)o * a.rstride, a.rec + (size_t)o * a.rstride,
                         a.rstride, &bars[o]);
            }
        }
        const unsigned chunks = tile / 16;
        for (unsigned i = tid; i < a.nleaf * chunks; i += nthr) {
            const unsigned l = i / chunks, c = i % chunks;
            const uint4 *src =
                reinterpret_cast<const uint4 *>(a.leaves[l] + (size_t)tile_idx * tile) + c;
            reinterpret_cast<uint4 *>(masks + (size_t)l * tile)[c] = __ldg(src);
        }
        __syncthreads();
    } else {
        pdl_wait();
        if (tid == 0)
            for (unsigned o = 0; o < R && o < a.nops; ++o) {
                const uint8_t *rows0[kLeafPre];
                read_rows(a, o, rows0);
                issue_stage(a, o, ring + (size_t)o * sstride, &bars[o], tile_idx, tile, rows0);
            }
    }

    T acc[2][K * 4];
    int lns[2] = {0, 0};
    const uint32_t spin = g_spin_limit;
    for (unsigned o = 0, stage = 0; o < a.nops;
         ++o, stage = (stage + 1 == R) ? 0u : stage + 1) {
        const uint8_t *pre[kLeafPre] = {nullptr, nullptr, nullptr, nullptr};
        if (!STAGED && tid == 0 && o + R < a.nops) read_rows(a, o + R, pre);
        // Every thread waits for the record (walk_tile's hand-off).
        const bool ok =
            __all_sync(0xffffffffu, mbar_wait_bounded(&bars[stage], (phase >> stage) & 1u,
                                                      spin));
        phase ^= 1u << stage;
        void *ydata = nullptr, *yscaler = nullptr;
        int yslot = -1;
        bool yhbm = false;
        unsigned nchild = 0;
        uint32_t nbytes = (uint32_t)sstride;
        if (ok) {
        const unsigned char *rec = ring + (size_t)stage * sstride;
        const uint8_t *lrow = rec + a.rstride;
        unsigned nlk = 0;
        const RecHead *hd = reinterpret_cast<const RecHead *>(rec);
        const RecChild *kids = reinterpret_cast<const RecChild *>(rec + sizeof(RecHead));
        nchild = hd->nchild;
        const uint32_t fl = hd->flags;
        uint32_t kind = (fl >> kOpKindShift) & 7u;
        if ((kind == OPK_FL || kind == OPK_FI) && o == 0) kind = OPK_GENERIC;
        if (kind != OPK_GENERIC) {
            op2_kind<K, STAGED, 2>(kind, rec, kids, (fl & kOpKindA) ? 1u : 0u, acc, lns, masks,
                                   lrow, slots, slot_sc, tile, pl, p, ppad);
        } else {
        lns[0] = lns[1] = 0;
        for (unsigned ci = 0; ci < nchild; ++ci) {
            const RecChild ch = kids[ci];
            const float *area = reinterpret_cast<const float *>(rec + ch.off);
            T msg[2][K * 4];
            if (ch.src == SRC_LEAF) {
                unsigned m[2];
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    m[h] = STAGED ? masks[(size_t)ch.idx * tile + pl[h]]
                                  : lrow[(size_t)nlk * tile + pl[h]];
                if (!STAGED) ++nlk;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float4 *t = reinterpret_cast<const float4 *>(area) + m[h];
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        const float4 v = t[k * 16];
                        msg[h][k * 4 + 0] = v.x;
                        msg[h][k * 4 + 1] = v.y;
                        msg[h][k * 4 + 2] = v.z;
                        msg[h][k * 4 + 3] = v.w;
                    }
                }
            } else {
                const bool in_slot = (ch.src == SRC_SLOT);
                const float4 *P = reinterpret_cast<const float4 *>(area);
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    const float4 c[4] = {P[k * 4], P[k * 4 + 1], P[k * 4 + 2], P[k * 4 + 3]};
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const float4 v =
                            in_slot ? slots[((size_t)ch.idx * K + k) * tile + pl[h]]
                                    : static_cast<const float4 *>(ch.data)[(size_t)k * ppad + p[h]];
                        float x[4];
                        unpack(v, x);
                        pcol(c, x, msg[h] + k * 4);
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    lns[h] += in_slot ? slot_sc[(size_t)ch.idx * tile + pl[h]]
                                      : static_cast<const int *>(ch.scaler)[p[h]];
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (ci == 0) {
#pragma unroll
                    for (int q = 0; q < K * 4; ++q) acc[h][q] = msg[h][q];
                } else {
#pragma unroll
                    for (int q = 0; q < K * 4; ++q) acc[h][q] *= msg[h][q];
                }
            }
        }
        }  // generic
        ydata = hd->data;
        yscaler = hd->scaler;
        yslot = hd->slot;
        yhbm = !(fl & REC_NO_HBM);
        nbytes = (hd->next_bytes != 0u && hd->next_bytes <= (uint32_t)sstride)
                     ? hd->next_bytes : (uint32_t)sstride;
        }  // ok
        if (!cta_hand_off(ok, nthr)) {
            if (tid == 0) {
                atomicOr(a.err, 1u);
                drain_ring(bars, phase ^ (1u << stage), o, a.nops, R);
            }
            return false;
        }
        if (tid == 0 && o + R < a.nops) {
            if (STAGED) {
                fence_proxy_async();
                mbar_expect_tx(&bars[stage], nbytes);
                bulk_g2s(ring + (size_t)stage * a.rstride,
                         a.rec + (size_t)(o + R) * a.rstride, nbytes, &bars[stage]);
            } else {
                issue_stage(a, o + R, ring + (size_t)stage * sstride, &bars[stage], tile_idx,
                            tile, pre);
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            T mx = T(0);
#pragma unroll
            for (int q = 0; q < K * 4; ++q) mx = fmax(mx, acc[h][q]);
            // The rescale rule of walk_tile (same bits).
            if (mx > T(0) && mx <= (T)3.0e38 && (nchild > 2 || mx < 1.52587890625e-05f)) {
                int e;
                frexpf(mx, &e);
                const int n = -e;
                if (n >= -126 && n <= 127) {
                    const float s1 = pow2f(n);
#pragma unroll
                    for (int q = 0; q < K * 4; ++q) acc[h][q] *= s1;
                } else {
                    const int n1 = n / 2, n2 = n - n1;
                    const float s1 = pow2f(n1), s2 = pow2f(n2);
#pragma unroll
                    for (int q = 0; q < K * 4; ++q) acc[h][q] = (acc[h][q] * s1) * s2;
                }
                lns[h] += e;
            }
            if (yhbm) {
                float4 *y = static_cast<float4 *>(ydata) + p[h];
#pragma unroll
                for (int k = 0; k < K; ++k) y[(size_t)k * ppad] = pack4(acc[h] + k * 4);
                static_cast<int *>(yscaler)[p[h]] = lns[h];
            }
            if (yslot >= 0) {
                float4 *ys = slots + (size_t)yslot * K * tile + pl[h];
#pragma unroll
                for (int k = 0; k < K; ++k) ys[(size_t)k * tile] = pack4(acc[h] + k * 4);
                slot_sc[(size_t)yslot * tile + pl[h]] = lns[h];
            }
        }
    }

    if (a.no_root) {
        __syncthreads();
        return true;
    }
    double v[2] = {0.0, 0.0};
    bool ninf[2] = {false, false};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if (!a.root_last) {
            const float4 *r = static_cast<const float4 *>(a.root) + p[h];
#pragma unroll
            for (int k = 0; k < K; ++k) unpack(r[(size_t)k * ppad], acc[h] + k * 4);
            lns[h] = static_cast<const int *>(a.rootsc)[p[h]];
        }
        double L = 0.0;
#pragma unroll
        for (int q = 0; q < K * 4; ++q) L = fma(__ldg(a.pn + q), (double)acc[h][q], L);
        if (p[h] < a.npat) {
            v[h] = (log(L) + (double)lns[h] * 0.69314718055994530942) * (double)a.freqs[p[h]];
            if (isnan(v[h])) v[h] = -INFINITY;
            if (a.site) a.site[p[h]] = v[h];
            if (isinf(v[h])) {
                ninf[h] = (v[h] < 0.0);
                v[h] = 0.0;
            }
        }
    }
    reduce_sites_n<2>(a, tile_idx, v, ninf);
    return true;
}

// A batched job's arguments, copied into shared memory when a CTA's next
// item belongs to another job: read through a pointer into global memory,
// every field would be reloaded after each store the walker makes.  The
// previous item ended with a block barrier, so no thread still reads the
// old copy.
static_assert(sizeof(PlanArgs) % 8 == 0, "PlanArgs is copied in 8-byte words");
__device__ __forceinline__ void load_job(PlanArgs &dst, const PlanArgs *src) {
    const unsigned long long *s = reinterpret_cast<const unsigned long long *>(src);
    unsigned long long *d = reinterpret_cast<unsigned long long *>(&dst);
    for (unsigned i = threadIdx.x; i < sizeof(PlanArgs) / 8; i += blockDim.x) d[i] = s[i];
    __syncthreads();
}

__device__ __forceinline__ void init_ring(const SmemLayout &Lay, unsigned R) {
    extern __shared__ __align__(128) unsigned char smem[];
    if (threadIdx.x == 0) {
        uint64_t *bars = reinterpret_cast<uint64_t *>(smem + Lay.bars);
        for (unsigned r = 0; r < R; ++r) mbar_init(&bars[r], 1);
        fence_mbar_init();
    }
    __syncthreads();
}

__device__ __forceinline__ void init_lean() {
    extern __shared__ __align__(128) unsigned char smem[];
    if (threadIdx.x == 0) {
        LeanHead &hd = *reinterpret_cast<LeanHead *>(smem);
        for (unsigned r = 0; r < kStages; ++r) {
            mbar_init(&hd.full[r], 1);
            hd.done[r] = 0;
        }
        hd.issued = 0;
        hd.abort = 0;
        fence_mbar_init();
    }
    __syncthreads();
}

// Launch bounds of the walkers (see walker_threads).
template <typename T, int KT, int G>
struct CtaOf {
    static constexpr int threads =
        walker_threads(sizeof(T) == 4 ? CXG_FP32 : CXG_FP64, KT, G);
    static constexpr int per_sm = threads > 512 ? 1 : 2;
};

// One plan: one CTA per tile.
template <typename T, int KT, int G>
__global__ void __launch_bounds__(CtaOf<T, KT, G>::threads, CtaOf<T, KT, G>::per_sm)
    walk_kernel(PlanArgs a) {
    const LeanLayout Lay = lean_layout(sizeof(T) == 4 ? CXG_FP32 : CXG_FP64, KT * G,
                                       blockDim.x / G, a.nslot, a.ring, a.rstride, a.lmax);
    init_lean();
    RingPos ring{0, 0};
    walk_tile<T, KT, G>(a, blockIdx.x, Lay, a.ring, ring);
}

// One plan with L = 2 op lanes (FP32, one thread per pattern, staged
// leaves): one CTA of NT = 2 x tile threads per tile, tile <= 64.  The
// bounds keep a 70,000-pattern tree (1,100 tiles of 64, 2,200 of 32) in one
// wave on 152 SMs: eight 128-thread CTAs per SM (64 registers) or fifteen
// 64-thread CTAs (68 registers).
template <int K, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) walk_kernel_lanes(PlanArgs a) {
    const SmemLayout Lay = smem_layout(CXG_FP32, K, blockDim.x / 2, a.nslot, a.ring,
                                       a.rstride * 2, 0, a.nleaf);
    init_ring(Lay, a.ring);
    uint32_t phase = 0;
    walk_tile_lanes<K>(a, blockIdx.x, Lay, a.ring, phase);
}

// Many jobs: a persistent grid claims (job, tile) items in the host's order
// (longest first).
template <typename T, int KT, int G>
__global__ void __launch_bounds__(CtaOf<T, KT, G>::threads, CtaOf<T, KT, G>::per_sm)
    walk_batch_kernel(BatchArgs b) {
    __shared__ unsigned s_item;
    __shared__ __align__(16) PlanArgs s_job;
    const LeanLayout Lay = lean_layout(sizeof(T) == 4 ? CXG_FP32 : CXG_FP64, KT * G,
                                       blockDim.x / G, b.max_nslot, b.ring, b.max_rstride,
                                       b.max_lmax);
    init_lean();
    RingPos ring{0, 0};
    unsigned job = ~0u;
    for (unsigned n = 0;; ++n) {
        unsigned item;
        if (b.direct) {
            item = n == 0 ? blockIdx.x : b.nitems;
        } else {
            if (threadIdx.x == 0) s_item = atomicAdd(b.counter, 1u);
            __syncthreads();
            item = s_item;
            __syncthreads();
        }
        if (item >= b.nitems) break;
        const WalkItem it = b.items[item];
        if (it.job != job) {
            load_job(s_job, b.jobs + it.job);
            job = it.job;
        }
        if (!walk_tile<T, KT, G>(s_job, it.tile, Lay, b.ring, ring)) break;
    }
}

// Two patterns per thread (FP32, one thread per pattern pair).
template <int K, bool STAGED>
__global__ void __launch_bounds__(kBlock) walk_kernel2(PlanArgs a) {
    const SmemLayout Lay = smem_layout(CXG_FP32, K, blockDim.x * 2, a.nslot, a.ring,
                                       a.rstride, a.lmax, a.nleaf);
    init_ring(Lay, a.ring);
    uint32_t phase = 0;
    walk_tile2<K, STAGED>(a, blockIdx.x, Lay, a.ring, phase);
}

template <int K, bool STAGED>
__global__ void __launch_bounds__(kBlock) walk_batch_kernel2(BatchArgs b) {
    __shared__ unsigned s_item;
    __shared__ __align__(16) PlanArgs s_job;
    unsigned job = ~0u;
    const SmemLayout Lay = smem_layout(CXG_FP32, K, blockDim.x * 2, b.max_nslot, b.ring,
                                       b.max_rstride, b.max_lmax, b.max_nleaf);
    init_ring(Lay, b.ring);
    uint32_t phase = 0;
    for (unsigned n = 0;; ++n) {
        unsigned item;
        if (b.direct) {
            item = n == 0 ? blockIdx.x : b.nitems;
        } else {
            if (threadIdx.x == 0) s_item = atomicAdd(b.counter, 1u);
            __syncthreads();
            item = s_item;
            __syncthreads();
        }
        if (item >= b.nitems) break;
        const WalkItem it = b.items[item];
        if (it.job != job) {
            load_job(s_job, b.jobs + it.job);
            job = it.job;
        }
        if (!walk_tile2<K, STAGED>(s_job, it.tile, Lay, b.ring, phase)) break;
    }
}

unsigned plan_blocks(unsigned ppad, unsigned tile) { return (ppad + tile - 1) / tile; }

template <typename Kern>
static cudaError_t ensure_smem(Kern k, size_t sm, size_t &optin) {
    // Raised on every new maximum, not only above 48 KiB: the default limit
    // counts static and dynamic shared memory together, so a dynamic size
    // just under 48 KiB plus the walker's static arrays would not launch.
    // Several host threads launch walkers (the server's workers): the
    // attribute only grows, under one lock.
    static std::mutex mu;
    std::lock_guard<std::mutex> g(mu);
    if (sm > optin) {
        cudaError_t e = cudaFuncSetAttribute(
            k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return e;
        optin = sm;
    }
    return cudaSuccess;
}

// Instantiated walker shapes (per-thread components KT, threads per
// pattern G): every kact with G = 1, and a pattern's components split over 2
// or 4 threads (walker_shape_ok).
#define CXG_SHAPES_G1(X) X(1, 1) X(2, 1) X(3, 1) X(4, 1) X(5, 1) X(6, 1) X(7, 1) X(8, 1)
#define CXG_SHAPES_GN(X) X(1, 2) X(2, 2) X(3, 2) X(4, 2) X(1, 4) X(2, 4)

template <typename T, int KT, int G>
static cudaError_t walk_fn(size_t sm, void (**fn)(PlanArgs)) {
    static size_t optin = 0;
    *fn = walk_kernel<T, KT, G>;
    return ensure_smem(walk_kernel<T, KT, G>, sm, optin);
}
template <typename T, int KT, int G>
static cudaError_t batch_fn(size_t sm, void (**fn)(BatchArgs)) {
    static size_t optin = 0;
    *fn = walk_batch_kernel<T, KT, G>;
    return ensure_smem(walk_batch_kernel<T, KT, G>, sm, optin);
}
template <int K, int NT, int MINB>
static cudaError_t lanes_fn(size_t sm, void (**fn)(PlanArgs)) {
    static size_t optin = 0;
    *fn = walk_kernel_lanes<K, NT, MINB>;
    return ensure_smem(walk_kernel_lanes<K, NT, MINB>, sm, optin);
}
template <int K, bool ST>
static cudaError_t walk2_fn(size_t sm, void (**fn)(PlanArgs)) {
    static size_t optin = 0;
    *fn = walk_kernel2<K, ST>;
    return ensure_smem(walk_kernel2<K, ST>, sm, optin);
}
template <int K, bool ST>
static cudaError_t batch2_fn(size_t sm, void (**fn)(BatchArgs)) {
    static size_t optin = 0;
    *fn = walk_batch_kernel2<K, ST>;
    return ensure_smem(walk_batch_kernel2<K, ST>, sm, optin);
}

// The two-patterns-per-thread walker for kact (FP32), with its dynamic
// shared memory limit raised to `sm` bytes.
template <typename Fn>
static cudaError_t pick_walker2(unsigned kact, bool staged, size_t sm, Fn *fn, bool batch) {
#define CXG_X2(K)                                                                       \
    if (kact == (K)) {                                                                  \
        if (batch)                                                                      \
            return staged ? batch2_fn<K, true>(sm, reinterpret_cast<void (**)(BatchArgs)>(fn)) \
                          : batch2_fn<K, false>(sm, reinterpret_cast<void (**)(BatchArgs)>(fn)); \
        return staged ? walk2_fn<K, true>(sm, reinterpret_cast<void (**)(PlanArgs)>(fn))       \
                      : walk2_fn<K, false>(sm, reinterpret_cast<void (**)(PlanArgs)>(fn));     \
    }
    CXG_X2(1) CXG_X2(2) CXG_X2(3) CXG_X2(4) CXG_X2(5)
#undef CXG_X2
    return cudaErrorInvalidValue;
}

// The walker for (kact, G), with its dynamic shared memory limit raised to
// `sm` bytes.
template <typename T, typename Fn>
static cudaError_t pick_walker(unsigned kact, unsigned G, size_t sm, Fn *fn, bool batch) {
#define CXG_X(KT, GG)                                                                     \
    if (kact == (KT) * (GG) && G == (GG))                                                 \
        return batch ? batch_fn<T, KT, GG>(sm, reinterpret_cast<void (**)(BatchArgs)>(fn)) \
                     : walk_fn<T, KT, GG>(sm, reinterpret_cast<void (**)(PlanArgs)>(fn));
    CXG_SHAPES_G1(CXG_X)
    CXG_SHAPES_GN(CXG_X)
#undef CXG_X
    return cudaErrorInvalidValue;
}

// The op-lane walker for kact (FP32), with its dynamic shared memory limit
// raised to `sm` bytes.
static cudaError_t pick_walker_lanes(unsigned kact, unsigned tile, size_t sm,
                                     void (**fn)(PlanArgs)) {
#define CXG_XL(K) \
    if (kact == (K))                                                      \
        return tile == 64 ? lanes_fn<K, 128, 8>(sm, fn) : lanes_fn<K, 64, 15>(sm, fn);
    CXG_XL(1) CXG_XL(2) CXG_XL(3) CXG_XL(4) CXG_XL(5)
#undef CXG_XL
    return cudaErrorInvalidValue;
}

// Dynamic shared memory of a walker launch: the lean layout (its ring counts
// ops per stage) for one pattern per thread and one op lane, else the layout
// of the two-pattern and op-lane walkers (its ring counts records).
size_t walk_smem_bytes(const WalkShape &w, unsigned nslot, unsigned rstride, unsigned lmax,
                       unsigned nleaf) {
    return w.lean() ? lean_smem_bytes(w.precision, w.kact, w.tile, nslot, w.ring, rstride, lmax)
                    : plan_smem_bytes(w.precision, w.kact, w.tile, nslot, w.ring,
                                      rstride * w.lanes, lmax, nleaf);
}

static bool shape_launches(const WalkShape &w) {
    return w.tile != 0 && w.tile % 32 == 0 && w.ring != 0 &&
           walker_shape_ok(w.precision, w.kact, w.tpp, w.ppt) &&
           (w.lean() ? w.tile * w.tpp <= walker_threads(w.precision, w.kact / w.tpp, w.tpp) &&
                           (w.tpp == 1 || w.tile <= kBlock)
                     : w.tile <= kBlock && w.tile / w.ppt >= 32 && w.ring <= 8);
}

static WalkShape shape_of(int precision, unsigned kact, unsigned tile, unsigned tpp,
                          unsigned ppt, unsigned lanes, unsigned ring) {
    WalkShape w;
    w.precision = precision;
    w.kact = kact;
    w.tile = tile;
    w.tpp = tpp ? tpp : 1;
    w.ppt = ppt ? ppt : 1;
    w.lanes = lanes;
    w.ring = ring;
    return w;
}

cudaError_t launch_plan(int precision, const PlanArgs &a, cudaStream_t s, unsigned lanes,
                        bool pdl) {
    const WalkShape w = shape_of(precision, a.kact, a.tile, a.tpp, a.ppt, lanes, a.ring);
    if (!shape_launches(w) || a.rstride % 16 || a.rstride == 0 ||
        a.ntiles != plan_blocks(a.ppad, a.tile) || (!w.lean() && a.ppad % a.tile) ||
        (w.lean() && w.ring * a.lmax > 32))
        return cudaErrorInvalidValue;
    if (lanes != 1 && !(lanes == 2 && lanes_shape_ok(precision, a.kact, w.tpp, w.ppt) &&
                        a.lmax == 0 && a.tile * lanes <= kLaneThreads &&
                        a.nops % lanes == 0))
        return cudaErrorInvalidValue;
    const size_t sm = walk_smem_bytes(w, a.nslot, a.rstride, a.lmax, a.nleaf);
    void (*fn)(PlanArgs) = nullptr;
    cudaError_t e = lanes == 2      ? pick_walker_lanes(a.kact, a.tile, sm, &fn)
                    : w.ppt == 2    ? pick_walker2(a.kact, a.lmax == 0, sm, &fn, false)
                    : precision == CXG_FP32
                        ? pick_walker<float>(a.kact, w.tpp, sm, &fn, false)
                        : pick_walker<double>(a.kact, w.tpp, sm, &fn, false);
    if (e != cudaSuccess) return e;
    const unsigned nb = a.ntiles, nt = a.tile * w.tpp * lanes / w.ppt;
    if (pdl) {
        // A dependent of the P kernel just before it on the stream.
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(nb);
        cfg.blockDim = dim3(nt);
        cfg.dynamicSmemBytes = sm;
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        return cudaLaunchKernelEx(&cfg, fn, a);
    }
    fn<<<nb, nt, sm, s>>>(a);
    return cudaGetLastError();
}

static cudaError_t pick_batch(const WalkShape &w, bool staged, size_t sm,
                              void (**fn)(BatchArgs)) {
    return w.ppt == 2 ? pick_walker2(w.kact, staged, sm, fn, true)
           : w.precision == CXG_FP32 ? pick_walker<float>(w.kact, w.tpp, sm, fn, true)
                                     : pick_walker<double>(w.kact, w.tpp, sm, fn, true);
}

cudaError_t launch_batch(int precision, const BatchArgs &b_in, unsigned grid,
                         cudaStream_t s) {
    // Items that fit one persistent grid get one CTA each: the hardware
    // spreads those CTAs over the SMs evenly, where persistent CTAs that
    // claim items first would crowd onto some SMs.
    BatchArgs b = b_in;
    if (b.nitems > 0 && b.nitems <= grid) {
        b.direct = 1;
        grid = b.nitems;
    }
    const WalkShape w = shape_of(precision, b.kact, b.tile, b.tpp, b.ppt, 1, b.ring);
    if (!shape_launches(w) || b.max_rstride % 16 || b.max_rstride == 0 || grid == 0 ||
        (w.lean() && w.ring * b.max_lmax > 32))
        return cudaErrorInvalidValue;
    const size_t sm = walk_smem_bytes(w, b.max_nslot, b.max_rstride, b.max_lmax, b.max_nleaf);
    void (*fn)(BatchArgs) = nullptr;
    const cudaError_t e = pick_batch(w, b.max_lmax == 0, sm, &fn);
    if (e != cudaSuccess) return e;
    fn<<<grid, b.tile * w.tpp / w.ppt, sm, s>>>(b);
    return cudaGetLastError();
}

int batch_ctas_per_sm(const WalkShape &w, bool staged, size_t smem) {
    if (!shape_launches(w)) return 0;
    void (*fn)(BatchArgs) = nullptr;
    cudaError_t e = pick_batch(w, staged, smem, &fn);
    int n = 0;
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, (int)(w.tile * w.tpp / w.ppt),
                                                          smem);
    return e == cudaSuccess ? n : 0;
}

__global__ void qdecomp_kernel(const double *rtri, const double *pi,
                               double *out) {
    if (blockIdx.x == 0 && threadIdx.x < 4) qdecomp4_warp(rtri, pi, out, 0);
}

cudaError_t launch_qdecomp(const double *rtri, const double *pi, double *out,
                           cudaStream_t s) {
    qdecomp_kernel<<<1, 32, 0, s>>>(rtri, pi, out);
    return cudaGetLastError();
}

}  // namespace cxg
