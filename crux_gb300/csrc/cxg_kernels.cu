// Device kernels of the pruning likelihood on sm_103a.
//
// Layout in HBM: a CL buffer of K active components over ppad patterns is
// [K][U][ppad] 16-byte units (FP32: U = 1, components in pairs, see Rows;
// FP64: U = 2, two double2), so that the threads of a warp, one pattern
// each, move 512 contiguous bytes per instruction.  Leaves are one uint8
// state mask per pattern.  Scalers are one FP64 log scale (plain form) or
// one int32 power-of-two exponent (FP32 form) per pattern.
//
// Kernels:
//   pmat_kernel     P(t) = V diag(exp(lambda r t)) V^-1 per (child edge,
//                   component), FP64, clipped at 0 (CxLik.c:258-292), plus
//                   the 16-entry message table of every leaf child.
//   walk_kernel     one CTA per tile of patterns walks the whole node-update
//                   list (patterns are independent through the entire
//                   post-order, CxLik.c:314-596, so no grid-wide sync is
//                   needed): records and leaf masks come in groups through a
//                   ring in shared memory, the previous op's result stays in
//                   registers, every parent is written through to HBM.  Then
//                   it aggregates the root (CxLik.c:598-632) and adds the
//                   weighted site lnLs in fixed point.
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

// Lanes per (child edge, component): a warp's FP64 instruction takes its SM
// quarter 64 cycles whatever its lanes do, and sixteen lanes need 39 of them
// where four need 73.  So sixteen while the warps have the chip's 608 quarters
// almost to themselves and the edges are few (an evaluation of one path on 64
// taxa: 3 us less; 250 taxa, two components: 135 -> 131; 300: 152 -> 157; 509
// taxa, one component: 200 -> 209).
__host__ __device__ inline unsigned pmat_lanes(const PmatArgs &a) {
    return a.nchild <= 512 && a.nchild * a.kact <= 1024 ? 16 : 4;
}
__host__ __device__ inline unsigned pmat_blocks(const PmatArgs &a) {
    return (a.nchild * a.kact * pmat_lanes(a) + 127) / 128;
}
__host__ __device__ inline unsigned image_units(const PmatArgs &a) {
    return a.nrec * a.img_units + a.img_tail;
}

// Unit t of a plan's program image, read from pinned host memory.  (A copy
// and an event before the P kernel took 2 us more of every evaluation whose
// path is new.)
__device__ inline void copy_image(const PmatArgs &a, unsigned t) {
    if (t >= image_units(a)) return;
    size_t off = 0;
    bool mine = true;
    if (t < a.nrec * a.img_units) {
        const unsigned u = t % a.img_units;
        const size_t rec = (size_t)(t / a.img_units) * a.rstride;
        // (The areas behind a record's children are the P blocks' to write.)
        const uint32_t nchild =
            reinterpret_cast<const RecHead *>(a.img_src + rec)->nchild;
        mine = u < 2 + 2 * nchild;
        off = rec + u * 16;
    } else {
        off = a.img_off + (size_t)(t - a.nrec * a.img_units) * 16;
    }
    const uint4 v = *reinterpret_cast<const uint4 *>(a.img_src + off);
    if (mine) *reinterpret_cast<uint4 *>(a.img_dst + off) = v;
}

__global__ void pmat_kernel(PmatArgs a) {
    pdl_launch_dependents();
    // The walker adds to its result only after this grid has completed
    // (stream order, or griddepcontrol.wait).
    if (a.zero != nullptr && blockIdx.x == 0 && threadIdx.x < sizeof(WalkResult) / 8)
        reinterpret_cast<uint64_t *>(a.zero)[threadIdx.x] = 0;
    if (a.pn_src != nullptr && blockIdx.x == 0 && threadIdx.x < a.kact * 4)
        a.pn_dst[threadIdx.x] = a.pn_src[threadIdx.x];
    const unsigned nblk = pmat_blocks(a);
    if (blockIdx.x >= nblk) {
        copy_image(a, (blockIdx.x - nblk) * blockDim.x + threadIdx.x);
        return;
    }
    const unsigned lanes = pmat_lanes(a);
    const unsigned idx = (blockIdx.x * blockDim.x + threadIdx.x) / lanes;
    if (idx >= a.nchild * a.kact) return;  // the same for all its lanes
    if (lanes == 16)
        pmat_one16(a, idx, threadIdx.x & 15u);
    else
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
    if (a.nchild * a.kact == 0) return cudaSuccess;
    const unsigned copies = a.img_src != nullptr ? (image_units(a) + 127) / 128 : 0;
    pmat_kernel<<<pmat_blocks(a) + copies, 128, 0, s>>>(a);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// The sum of a job's site lnLs, in 128-bit fixed point with 64 fraction
// bits.  Integer addition is associative, so the sum is the same for every
// tile and launch shape, and it is exact but for what each value has below
// 2^-64.  (The FP64 unit adds one warp instruction in 64 cycles: a
// compensated FP64 sum, six dependent adds a step, took 3 to 8 us at the end
// of every walk -- shuffles, a serial fold per CTA and one per job.)
// ---------------------------------------------------------------------------
typedef unsigned __int128 fixed128;

// |v| < 2^63; NaN and infinities do not come here.
__device__ __forceinline__ fixed128 to_fixed(double v) {
    const uint64_t bits = (uint64_t)__double_as_longlong(v);
    const int e = (int)(bits >> 52) & 0x7ff;
    uint64_t m = bits & 0xfffffffffffffull;
    if (e != 0) m |= 1ull << 52;
    const int sh = (e != 0 ? e : 1) - 1075 + 64;  // v = m 2^(sh - 64)
    fixed128 f = 0;
    if (sh >= 0)
        f = (fixed128)m << (sh < 127 ? sh : 127);
    else if (sh > -64)
        f = m >> -sh;
    return (long long)bits < 0 ? (fixed128)0 - f : f;
}

__device__ __forceinline__ fixed128 warp_sum(fixed128 f) {
    uint64_t lo = (uint64_t)f, hi = (uint64_t)(f >> 64);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const uint64_t l = __shfl_xor_sync(0xffffffffu, lo, off);
        const uint64_t h = __shfl_xor_sync(0xffffffffu, hi, off);
        const fixed128 t = (((fixed128)hi << 64) | lo) + (((fixed128)h << 64) | l);
        lo = (uint64_t)t;
        hi = (uint64_t)(t >> 64);
    }
    return ((fixed128)hi << 64) | lo;
}

// Add the CTA's site values (finite ones; -inf sites are counted) to the
// job's result.  No tile waits to be the last: whoever reads the result puts
// the limbs together.
template <int NV>
__device__ void reduce_sites(const PlanArgs &a, const double (&v)[NV],
                             const bool (&neg_inf)[NV]) {
    __shared__ uint64_t s_limb[kMaxThreads / 32][4];
    __shared__ unsigned s_ninf[kMaxThreads / 32];
    const unsigned nwarp = blockDim.x / 32;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    fixed128 f = 0;
    unsigned ninf = 0;
#pragma unroll
    for (int h = 0; h < NV; ++h) {
        f += to_fixed(v[h]);
        ninf += __popc(__ballot_sync(0xffffffffu, neg_inf[h]));
    }
    f = warp_sum(f);
    // The top limb keeps the sign.
    const uint64_t w = (uint64_t)(f >> (32 * (lane & 3u)));
    uint64_t limb = lane == 3 ? (uint64_t)(long long)(int)(uint32_t)w : (uint32_t)w;
    if (nwarp > 1) {
        if (lane < 4) s_limb[warp][lane] = limb;
        if (lane == 4) s_ninf[warp] = ninf;
        __syncthreads();
        if (warp == 0 && lane < 4)
            for (unsigned q = 1; q < nwarp; ++q) limb += s_limb[q][lane];
        if (warp == 0 && lane == 4)
            for (unsigned q = 1; q < nwarp; ++q) ninf += s_ninf[q];
    }
    if (warp == 0) {
        if (lane < 4)
            atomicAdd(reinterpret_cast<unsigned long long *>(a.res->acc) + lane, limb);
        if (lane == 4 && ninf) atomicAdd(&a.res->ninf, ninf);
    }
    __syncthreads();  // s_limb is reused by the next item
}

// ---------------------------------------------------------------------------
// Plan walker.  T = double: plain form; T = float: FP32 form.  Both scale by
// powers of two (rescale), where the reference divides by the largest child
// message (CxLik.c:390-403 and 577-588).
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

__device__ __forceinline__ float pow2f(int n) {  // n in [-126, 127]
    return __int_as_float((n + 127) << 23);
}

// Shared memory of an op-lane CTA: mbarriers [ring]; the stage ring [ring] of
// `stage` bytes, each the op records of a step; stack slots
// [nslot][K][U][tile] units; slot scalers [nslot][tile]; and every leaf's
// mask row [nleaf][tile], loaded once per tile.
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
    // (An op reads the next one's header and two mask rows ahead; past the
    // last stage those lie in this gap.)
    L.slots = L.stage0 + kStages * L.stage + ((64 + 2 * (size_t)tile + 15) & ~(size_t)15);
    L.slot_sc = L.slots + (size_t)nslot * kact * U * tile * 16;
    L.total = L.slot_sc + (((size_t)nslot * tile * sc + 15) & ~(size_t)15);
    return L;
}

// A header's slot in the word the walker keeps of it: above the flags, plus
// one.
constexpr unsigned kSlotShift = 16;
// Set where a result is not simply written to HBM (kept in a slot, or not
// written).
constexpr uint32_t kPlainMask = 0xffffu << kSlotShift | REC_NO_HBM;

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

// Two packed FP32 values (a register pair): the FP32 products run on two of
// a pattern's components at a time (fma.rn.f32x2, each half rounded as a
// scalar fused multiply-add).
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
// base + a * b bytes, one instruction; 16-byte loads through L2 (rows may
// have been written by this walk) and stores, at global addresses.
__device__ __forceinline__ uint64_t addr_at(uint64_t base, uint32_t a, uint32_t b) {
    uint64_t r;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(base));
    return r;
}
// Unit u of a CL row at `at`; its units are `pitch` patterns apart (counted in
// patterns: the bytes pass 32 bits from 2^28 patterns on).
__device__ __forceinline__ uint64_t unit_at(uint64_t at, uint32_t pitch, uint32_t u) {
    return addr_at(at, pitch, u * 16u);
}
template <typename X>
__device__ __forceinline__ X ld_l2(uint64_t at) {
    return __ldcg(reinterpret_cast<const X *>(at));
}
// (Units of packed pairs move as two 64-bit words: taken apart to four
// floats and packed again, each pair cost two register moves.)
typedef ulonglong2 pairs;
__device__ __forceinline__ void st_global(uint64_t at, const pairs v) {
    asm volatile("st.global.v2.b64 [%0], {%1, %2};" ::"l"(at), "l"(v.x), "l"(v.y) : "memory");
}
__device__ __forceinline__ void st_global(uint64_t at, const float4 v) {
    asm volatile("st.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(at), "f"(v.x), "f"(v.y),
                 "f"(v.z), "f"(v.w)
                 : "memory");
}
__device__ __forceinline__ void st_global(uint64_t at, const double2 v) {
    asm volatile("st.global.v2.f64 [%0], {%1, %2};" ::"l"(at), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ void st_global(uint64_t at, float v) {
    asm volatile("st.global.f32 [%0], %1;" ::"l"(at), "f"(v) : "memory");
}
__device__ __forceinline__ void st_global(uint64_t at, int v) {
    asm volatile("st.global.s32 [%0], %1;" ::"l"(at), "r"(v) : "memory");
}
__device__ __forceinline__ void st_global(uint64_t at, double v) {
    asm volatile("st.global.f64 [%0], %1;" ::"l"(at), "d"(v) : "memory");
}
__device__ __forceinline__ float vmax(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ int vmax(int a, int b) { return max(a, b); }

// ---------------------------------------------------------------------------
// One pattern's rows: the KT components (of KT * G) that a thread holds, the
// first being component k0, a multiple of KT.
//
// FP32 layouts (CL rows in HBM and in the stack, P matrices and leaf tables
// in the op records): components go in pairs, 2m and 2m + 1, the two values
// of a state side by side, so that a 16-byte unit is two register pairs and
// the packed products need no moves; the last of an odd number of components
// stands alone.
//   CL row     unit 2m + h: (s = 2h: k = 2m, 2m + 1; s = 2h + 1: same)
//              unit of a lone component: its four states
//   P          pair block at m * 128 bytes: column j, row i: two floats
//              lone block at k * 64 bytes, by columns
//   leaf table pair block at m * 512 bytes: [h][16 masks] units as a CL row's
//              lone block at k * 256 bytes: [16 masks] of its four states
// A thread whose odd KT splits pairs between threads (G > 1) holds single
// components and reads and writes single floats of those units.
//
// FP64: component by component, two units (double2) of a CL row each; P by
// rows; leaf tables in HBM, [16 masks][K][4].
// ---------------------------------------------------------------------------
template <typename T, int KT, int G>
struct Rows;

template <int KT, int G>
struct Rows<float, KT, G> {
    typedef float4 V;
    static constexpr int NP = (G == 1 || KT % 2 == 0) ? KT / 2 : 0;  // pairs
    static constexpr int NS = KT - 2 * NP;                           // single components
    static constexpr bool split = NS > 0 && G > 1;  // singles are halves of pairs
    f32x2 pr[NP ? NP : 1][4];
    float sg[NS ? NS : 1][4];

    // A row's units in HBM (`at`: the pattern's place in unit 0; units are
    // `pitch` bytes apart) and in shared memory (`stride` units apart).  A
    // split single's state s is one float of unit (k & ~1) + s / 2.
    __device__ static __forceinline__ unsigned part(unsigned k, int s) {
        return ((s & 1) * 2 + (k & 1u)) * 4;
    }
    __device__ __forceinline__ void set(int u, const pairs x) {
        pr[u / 2][(u & 1) * 2] = x.x;
        pr[u / 2][(u & 1) * 2 + 1] = x.y;
    }
    __device__ __forceinline__ pairs unit(int u) const {
        return pairs{pr[u / 2][(u & 1) * 2], pr[u / 2][(u & 1) * 2 + 1]};
    }
    __device__ __forceinline__ void load_l2(uint64_t at, uint32_t pitch, unsigned k0) {
#pragma unroll
        for (int u = 0; u < 2 * NP; ++u) set(u, ld_l2<pairs>(unit_at(at, pitch, k0 + u)));
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            const unsigned k = k0 + 2 * NP + i;
            if (split) {
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    sg[i][s] = __ldcg(reinterpret_cast<const float *>(
                        unit_at(at, pitch, (k & ~1u) + (s >> 1)) + part(k, s)));
            } else {
                unpack(ld_l2<float4>(unit_at(at, pitch, k)), sg[i]);
            }
        }
    }
    __device__ __forceinline__ void store_global(uint64_t at, uint32_t pitch,
                                                 unsigned k0) const {
#pragma unroll
        for (int u = 0; u < 2 * NP; ++u) st_global(unit_at(at, pitch, k0 + u), unit(u));
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            const unsigned k = k0 + 2 * NP + i;
            if (split) {
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    st_global(unit_at(at, pitch, (k & ~1u) + (s >> 1)) + part(k, s), sg[i][s]);
            } else {
                st_global(unit_at(at, pitch, k),
                          make_float4(sg[i][0], sg[i][1], sg[i][2], sg[i][3]));
            }
        }
    }
    __device__ __forceinline__ void load_smem(const float4 *p, unsigned stride, unsigned k0) {
#pragma unroll
        for (int u = 0; u < 2 * NP; ++u)
            set(u, *reinterpret_cast<const pairs *>(p + (k0 + u) * stride));
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            const unsigned k = k0 + 2 * NP + i;
            if (split) {
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    sg[i][s] = reinterpret_cast<const float *>(
                        p + ((k & ~1u) + (s >> 1)) * stride)[part(k, s) / 4];
            } else {
                unpack(p[k * stride], sg[i]);
            }
        }
    }
    __device__ __forceinline__ void store_smem(float4 *p, unsigned stride, unsigned k0) const {
#pragma unroll
        for (int u = 0; u < 2 * NP; ++u)
            *reinterpret_cast<pairs *>(p + (k0 + u) * stride) = unit(u);
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            const unsigned k = k0 + 2 * NP + i;
            if (split) {
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    reinterpret_cast<float *>(p + ((k & ~1u) + (s >> 1)) *
                                                      stride)[part(k, s) / 4] = sg[i][s];
            } else {
                p[k * stride] = make_float4(sg[i][0], sg[i][1], sg[i][2], sg[i][3]);
            }
        }
    }
    // Component q of this thread's, state s.
    __device__ __forceinline__ float get(int q, int s) const {
        if (q >= 2 * NP) return sg[q - 2 * NP][s];
        float a, b;
        unpack2f(pr[q / 2][s], a, b);
        return (q & 1) ? b : a;
    }
    // Largest entry (operands that are NaN are passed over, as fmax does).
    __device__ __forceinline__ float top() const {
        float m = 0.0f;
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            float a[4], b[4];
#pragma unroll
            for (int s = 0; s < 4; ++s) unpack2f(pr[i][s], a[s], b[s]);
            m = max3f(max3f(max3f(a[0], b[0], a[1]), b[1], a[2]), max3f(b[2], a[3], b[3]), m);
        }
#pragma unroll
        for (int i = 0; i < NS; ++i)
            m = max3f(max3f(sg[i][0], sg[i][1], sg[i][2]), sg[i][3], m);
        return m;
    }
    __device__ __forceinline__ void scale(float f) {
        const f32x2 ff = pack2f(f, f);
#pragma unroll
        for (int i = 0; i < NP; ++i)
#pragma unroll
            for (int s = 0; s < 4; ++s) pr[i][s] = mul2(pr[i][s], ff);
#pragma unroll
        for (int i = 0; i < NS; ++i)
#pragma unroll
            for (int s = 0; s < 4; ++s) sg[i][s] *= f;
    }
    __device__ __forceinline__ void mul(const Rows &b) {
#pragma unroll
        for (int i = 0; i < NP; ++i)
#pragma unroll
            for (int s = 0; s < 4; ++s) pr[i][s] = mul2(pr[i][s], b.pr[i][s]);
#pragma unroll
        for (int i = 0; i < NS; ++i)
#pragma unroll
            for (int s = 0; s < 4; ++s) sg[i][s] *= b.sg[i][s];
    }
};

template <int KT, int G>
struct Rows<double, KT, G> {
    typedef double2 V;
    double v[KT][4];

    __device__ __forceinline__ void set(int u, const double2 x) {
        v[u / 2][(u & 1) * 2] = x.x;
        v[u / 2][(u & 1) * 2 + 1] = x.y;
    }
    __device__ __forceinline__ double2 unit(int u) const {
        return make_double2(v[u / 2][(u & 1) * 2], v[u / 2][(u & 1) * 2 + 1]);
    }
    __device__ __forceinline__ void load_l2(uint64_t at, uint32_t pitch, unsigned k0) {
#pragma unroll
        for (int u = 0; u < 2 * KT; ++u)
            set(u, ld_l2<double2>(unit_at(at, pitch, 2 * k0 + u)));
    }
    __device__ __forceinline__ void store_global(uint64_t at, uint32_t pitch,
                                                 unsigned k0) const {
#pragma unroll
        for (int u = 0; u < 2 * KT; ++u) st_global(unit_at(at, pitch, 2 * k0 + u), unit(u));
    }
    __device__ __forceinline__ void load_smem(const double2 *p, unsigned stride, unsigned k0) {
#pragma unroll
        for (int u = 0; u < 2 * KT; ++u) set(u, p[(2 * k0 + u) * stride]);
    }
    __device__ __forceinline__ void store_smem(double2 *p, unsigned stride, unsigned k0) const {
#pragma unroll
        for (int u = 0; u < 2 * KT; ++u) p[(2 * k0 + u) * stride] = unit(u);
    }
    __device__ __forceinline__ double get(int q, int s) const { return v[q][s]; }
    // Exponent word of the largest of entries that are >= 0: the sign bit is
    // clear, so the high words order as the values (a NaN above infinity),
    // on the integer pipe.
    __device__ __forceinline__ int top() const {
        int m = 0;
#pragma unroll
        for (int k = 0; k < KT; ++k) {
            const int a = max(__double2hiint(v[k][0]), __double2hiint(v[k][1]));
            const int b = max(__double2hiint(v[k][2]), __double2hiint(v[k][3]));
            m = max(m, max(a, b));
        }
        return m;
    }
    // High word of the smallest entry that is not 0 (negative if one is).
    __device__ __forceinline__ int low() const {
        int m = 0x7fffffff;
#pragma unroll
        for (int k = 0; k < KT; ++k)
#pragma unroll
            for (int s = 0; s < 4; ++s)
                m = min(m, __double_as_longlong(v[k][s]) ? __double2hiint(v[k][s]) : 0x7fffffff);
        return m;
    }
    // Times 2^n: zeros stay, the caller keeps the other exponents within the
    // normal range.
    __device__ __forceinline__ void shift(int n) {
#pragma unroll
        for (int k = 0; k < KT; ++k)
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const int h = __double2hiint(v[k][s]), l = __double2loint(v[k][s]);
                v[k][s] = __hiloint2double((h | l) ? h + (n << 20) : 0, l);
            }
    }
    __device__ __forceinline__ void scale(double f) {
#pragma unroll
        for (int k = 0; k < KT; ++k)
#pragma unroll
            for (int s = 0; s < 4; ++s) v[k][s] *= f;
    }
    __device__ __forceinline__ void mul(const Rows &b) {
#pragma unroll
        for (int k = 0; k < KT; ++k)
#pragma unroll
            for (int s = 0; s < 4; ++s) v[k][s] *= b.v[k][s];
    }
};

// r[h] = P r[h] for the NP patterns of a thread (each unit of P, at `area` in
// the record, is read once for all of them): every entry a product and
// three fused adds, in column order.
template <int KT, int G, int N>
__device__ __forceinline__ void apply_p(const unsigned char *area, unsigned k0,
                                        Rows<float, KT, G> (&r)[N]) {
    typedef Rows<float, KT, G> R;
#pragma unroll
    for (int i = 0; i < R::NP; ++i) {
        const pairs *P = reinterpret_cast<const pairs *>(area + (k0 / 2 + i) * 128);
        f32x2 y[N][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const pairs a = P[2 * j], b = P[2 * j + 1];
            const f32x2 c[4] = {a.x, a.y, b.x, b.y};
#pragma unroll
            for (int h = 0; h < N; ++h)
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    y[h][s] = j == 0 ? mul2(c[s], r[h].pr[i][0])
                                     : fma2(c[s], r[h].pr[i][j], y[h][s]);
        }
#pragma unroll
        for (int h = 0; h < N; ++h)
#pragma unroll
            for (int s = 0; s < 4; ++s) r[h].pr[i][s] = y[h][s];
    }
#pragma unroll
    for (int i = 0; i < R::NS; ++i) {
        float y[N][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float c[4];
            if (R::split) {
                const unsigned k = k0 + i;
                const float *f = reinterpret_cast<const float *>(area + (k / 2) * 128) + (k & 1u);
#pragma unroll
                for (int s = 0; s < 4; ++s) c[s] = f[(j * 4 + s) * 2];
            } else {
                unpack(reinterpret_cast<const float4 *>(area + (k0 + 2 * R::NP) * 64)[j], c);
            }
#pragma unroll
            for (int h = 0; h < N; ++h)
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    y[h][s] = j == 0 ? c[s] * r[h].sg[i][0]
                                     : fmaf(c[s], r[h].sg[i][j], y[h][s]);
        }
#pragma unroll
        for (int h = 0; h < N; ++h)
#pragma unroll
            for (int s = 0; s < 4; ++s) r[h].sg[i][s] = y[h][s];
    }
}
template <int KT, int G, int N>
__device__ __forceinline__ void apply_p(const unsigned char *area, unsigned k0,
                                        Rows<double, KT, G> (&r)[N]) {
#pragma unroll
    for (int k = 0; k < KT; ++k) {
        const double2 *P = reinterpret_cast<const double2 *>(area) + (k0 + k) * 8;
        double y[N][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const double2 a = P[2 * i], b = P[2 * i + 1];
#pragma unroll
            for (int h = 0; h < N; ++h) {
                const double *x = r[h].v[k];
                y[h][i] = fma(b.y, x[3], fma(b.x, x[2], fma(a.y, x[1], a.x * x[0])));
            }
        }
#pragma unroll
        for (int h = 0; h < N; ++h)
#pragma unroll
            for (int i = 0; i < 4; ++i) r[h].v[k][i] = y[h][i];
    }
}

// The message of a leaf child with state mask m: r = it, or r *= it.  FP32:
// from the table in the record at `area`; FP64: from table `tab` of `ltab`.
template <bool MUL, int KT, int G>
__device__ __forceinline__ void leaf_message(const unsigned char *area, unsigned,
                                             const double *, unsigned m, unsigned k0,
                                             Rows<float, KT, G> &r) {
    typedef Rows<float, KT, G> R;
#pragma unroll
    for (int i = 0; i < R::NP; ++i) {
        const pairs *t = reinterpret_cast<const pairs *>(area + (k0 / 2 + i) * 512) + m;
        const pairs a = t[0], b = t[16];
        const f32x2 c[4] = {a.x, a.y, b.x, b.y};
#pragma unroll
        for (int s = 0; s < 4; ++s) r.pr[i][s] = MUL ? mul2(r.pr[i][s], c[s]) : c[s];
    }
#pragma unroll
    for (int i = 0; i < R::NS; ++i) {
        float c[4];
        if (R::split) {
            const unsigned k = k0 + i;
            const float *f =
                reinterpret_cast<const float *>(area + (k / 2) * 512) + m * 4 + (k & 1u);
#pragma unroll
            for (int s = 0; s < 4; ++s) c[s] = f[(s >> 1) * 64 + (s & 1) * 2];
        } else {
            unpack(reinterpret_cast<const float4 *>(area + (k0 + 2 * R::NP) * 256)[m], c);
        }
#pragma unroll
        for (int s = 0; s < 4; ++s) r.sg[i][s] = MUL ? r.sg[i][s] * c[s] : c[s];
    }
}
template <bool MUL, int KT, int G>
__device__ __forceinline__ void leaf_message(const unsigned char *, unsigned tab,
                                             const double *ltab, unsigned m, unsigned k0,
                                             Rows<double, KT, G> &r) {
    const double2 *t =
        reinterpret_cast<const double2 *>(ltab + (((size_t)tab * 16 + m) * (KT * G) + k0) * 4);
#pragma unroll
    for (int k = 0; k < KT; ++k) {
        const double2 a = __ldg(t + 2 * k), b = __ldg(t + 2 * k + 1);
        r.v[k][0] = MUL ? r.v[k][0] * a.x : a.x;
        r.v[k][1] = MUL ? r.v[k][1] * a.y : a.y;
        r.v[k][2] = MUL ? r.v[k][2] * b.x : b.x;
        r.v[k][3] = MUL ? r.v[k][3] * b.y : b.y;
    }
}

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
// FP32: when the largest entry of any of eight consecutive patterns has left
// [2^-16, 2^44), all eight go to [2^19, 2^20), the exponent added to the
// integer scaler.  So patterns of a warp fall together, where pattern by
// pattern, at below 2^-16 to [0.5, 1), nearly every op had some lane in the
// branch.  Eight are what a warp holds with four threads a pattern: the
// groups are the same in every shape, and with them the bits also of rows with
// subnormal entries.  (Groups of a warp's 32, 16 or 8 gave other bits there
// and rescaled less: 128 taxa x 81,664 patterns, eight proposals 1,837 us and
// 1,846 now.)  P has entries of at most 1, so a product of two rows stays far
// inside the FP32 range, and the scaling of normal entries is exact.  Called
// by whole warps.
template <int KT, int G>
__device__ __forceinline__ void rescale(Rows<float, KT, G> &r, int &lns, bool always) {
    constexpr uint32_t kLow = (127 - 16) << 23, kHigh = (127 + 44) << 23;
    const float mx = group_max<G>(r.top());
    const bool out = (__float_as_uint(mx) - kLow >= kHigh - kLow) | always;
    if (!__any_sync(0xffffffffu, out)) return;
    if (G < 4) {
        const unsigned group = ((1u << (8 * G % 32)) - 1u) << (threadIdx.x & (32u - 8 * G));
        if ((__ballot_sync(0xffffffffu, out) & group) == 0) return;
    }
    // From its exponent field, 126 more than frexp's exponent; rows below
    // 2^-108 need two factors, zeros and what is not a number none.
    const uint32_t b = __float_as_uint(mx) >> 23;
    if (b - 19u < 255u - 19u) {
        r.scale(pow2f(146 - (int)b));
        lns -= 146 - (int)b;
    } else if (b < 19u && mx > 0.0f) {
        int e;
        frexpf(mx, &e);
        r.scale(pow2f(127));
        if (20 - e > 127) r.scale(pow2f(20 - e - 127));
        lns -= 20 - e;
    }
}

// FP64: below 2^-32 (or at 2^511), to [1, 2), and its exponent times ln 2
// joins the log scaler. The reference divides by the largest child message and
// adds its log on every op (CxLik.c:390-403, 577-588); the product of rows and
// scale is the same, the power of two is exact, and the FP64 pipe, which
// bounds this form, is spared a reciprocal, 4 K products and a log per op (134
// to about 80 FP64 instructions per update). The largest entries of two
// messages multiply to at least 2^-64 or so, and an entry is a normal number
// down to 2^-958 of their product: a component that one child favours and the
// other does not keeps its rows, as it does where rows stay near 1. (Scaled
// only below 2^-256, such sites came out wrong or -inf. That low a bound saves
// 0.2 % of four proposals on 128 taxa x 81,664 patterns, 6,770 us, and 0.7 %
// of eight branches on 49,000, 2,702 us. To 2^200, and so less often, is no
// faster, and a scaler far from the site's lnL costs it digits.) Two rows
// below 2^511 do not overflow. Rows of zeros stay zeros, and a pattern with an
// infinite entry ends with NaN rows, as dividing by an infinite scaler leaves
// it: its site lnL is -inf either way.
template <int KT, int G>
__device__ __forceinline__ void rescale(Rows<double, KT, G> &r, double &lns, bool) {
    const int hi = group_max<G>(r.top());
    constexpr int kLow = (1023 - 32) << 20, kHigh = (1023 + 511) << 20;
    if (hi >= kLow && hi < kHigh) return;
    double s;
    if (hi >= 0x7ff00000) {
        s = 0.0;  // infinity times 0: NaN
        lns = INFINITY;
    } else {
        // (Subnormal rows, zeros among them, take 2^1000.)
        int e = hi < (1 << 20) ? -1000 : (hi >> 20) - 1023;
        e = max(e, -1000);
        lns = fma((double)e, 0.69314718055994530942, lns);
        // On the integer pipe where every entry is 0 or a normal number before
        // and after: eight products of two components take their SM quarter 512
        // cycles (branches 2,832 -> 2,735 us, proposals 6,869 -> 6,800).
        if (r.low() >= max(e + 1, 1) << 20) {
            r.shift(-e);
            return;
        }
        s = __hiloint2double((1023 - e) << 20, 0);
    }
    r.scale(s);
}

// ln(L 2^e): the exponent of L joins e, so that the sum does not depend on
// how rows and scaler shared it.
__device__ __forceinline__ double site_log(double L, int e) {
    int f;
    const double m = frexp(L, &f);
    return log(m) + (double)(e + f) * 0.69314718055994530942;
}

// A thread's view of the tile it walks: N patterns `nthr` apart (G = 1), the
// first at pl in the tile and p in the CL buffers.
template <typename T>
struct TileView {
    typedef typename Prec<T>::V V;
    typedef typename Prec<T>::S S;
    V *slots;
    S *slot_sc;
    const double *ltab;  // FP64: leaf-message tables
    uint32_t pitch;      // patterns between a CL's units
    unsigned tile, pl, p, k0;
};

// An internal child's rows and scaler: from its stack slot, or from HBM
// through L2 (rows this same thread wrote earlier in the walk, or an
// earlier launch did).  `cr` is the child's descriptor in the record.
template <typename T, int KT, int G, int N>
__device__ __forceinline__ void child_rows(const unsigned char *cr, const TileView<T> &w,
                                           Rows<T, KT, G> (&x)[N],
                                           typename Prec<T>::S (&l)[N]) {
    typedef typename Prec<T>::V V;
    typedef typename Prec<T>::S S;
    constexpr unsigned U = Prec<T>::U;
    const ulonglong2 ptr = *reinterpret_cast<const ulonglong2 *>(cr);
    const uint2 si = *reinterpret_cast<const uint2 *>(cr + 16);  // src, idx
    const unsigned step = w.tile / N;
    if (si.x == SRC_SLOT) {
        const V *q = w.slots + si.y * (KT * G * U) * w.tile + w.pl;
#pragma unroll
        for (int h = 0; h < N; ++h) {
            x[h].load_smem(q + h * step, w.tile, w.k0);
            l[h] = w.slot_sc[si.y * w.tile + w.pl + h * step];
        }
    } else {
        const uint64_t q = addr_at(ptr.x, w.p, sizeof(V)), ql = addr_at(ptr.y, w.p, sizeof(S));
#pragma unroll
        for (int h = 0; h < N; ++h) {
            x[h].load_l2(q + h * step * sizeof(V), w.pitch, w.k0);
            l[h] = __ldcg(reinterpret_cast<const S *>(ql + h * step * sizeof(S)));
        }
    }
}

// One op.  `acc` and `lns` hold the previous op's result on entry and this
// op's on return; m0 and m1 are the state masks of its first two leaf
// children, `rows` this pattern's masks of the op's leaf children (one row
// per `tile` bytes).  Two-child ops run the code of their kind (an op's kind
// and the child that plays A are in its flags), others a loop over children.
// The product of two messages and the sum of two scalers are the same in
// either order, so every path gives the same bits.
template <typename T, int KT, int G, int N>
__device__ __forceinline__ void walk_op(const unsigned char *rec, uint32_t flags, bool first,
                                        const unsigned (&m0)[N], const unsigned (&m1)[N],
                                        const uint8_t *rows, const TileView<T> &w,
                                        Rows<T, KT, G> (&acc)[N],
                                        typename Prec<T>::S (&lns)[N]) {
    typedef typename Prec<T>::S S;
    typedef Rows<T, KT, G> R;
    constexpr unsigned KA = KT * G;
    constexpr unsigned PB = KA * 16 * sizeof(T);                    // bytes of a P area
    constexpr unsigned LB = sizeof(T) == 4 ? KA * 16 * 4 * 4 : PB;  // of a leaf's area
    const unsigned char *kid0 = rec + sizeof(RecHead);
    const unsigned char *area = kid0 + 2 * sizeof(RecChild);
    const unsigned ia = (flags & kOpKindA) ? 1u : 0u;
    uint32_t kind = (flags >> kOpKindShift) & 7u;
    // A walk that starts inside a plan (one launch per node) holds no
    // previous result.
    if (first && (kind == OPK_FL || kind == OPK_FI)) kind = OPK_GENERIC;
    auto tab_of = [&](unsigned c) -> unsigned {
        return sizeof(T) == 8 ? reinterpret_cast<const RecChild *>(kid0)[c].tab : 0u;
    };
    if (kind == OPK_FL || kind == OPK_IL) {
        if (kind == OPK_IL)
            child_rows<T, KT, G, N>(kid0 + ia * sizeof(RecChild), w, acc, lns);
        const unsigned tab = tab_of(ia ^ 1u);
        apply_p<KT, G, N>(area + (ia ? LB : 0u), w.k0, acc);
#pragma unroll
        for (int h = 0; h < N; ++h)
            leaf_message<true, KT, G>(area + (ia ? 0u : PB), tab, w.ltab, m0[h], w.k0, acc[h]);
    } else if (kind == OPK_LL) {
        const unsigned t0 = tab_of(0), t1 = tab_of(1);
#pragma unroll
        for (int h = 0; h < N; ++h) {
            leaf_message<false, KT, G>(area, t0, w.ltab, m0[h], w.k0, acc[h]);
            leaf_message<true, KT, G>(area + LB, t1, w.ltab, m1[h], w.k0, acc[h]);
            lns[h] = S(0);
        }
    } else if (kind == OPK_FI || kind == OPK_II) {
        R xb[N];
        S lb[N];
        child_rows<T, KT, G, N>(kid0 + (ia ^ 1u) * sizeof(RecChild), w, xb, lb);
        if (kind == OPK_II)
            child_rows<T, KT, G, N>(kid0 + ia * sizeof(RecChild), w, acc, lns);
        // (A's products come first: B's rows are on their way from L2.)
        apply_p<KT, G, N>(area + (ia ? PB : 0u), w.k0, acc);
        apply_p<KT, G, N>(area + (ia ? 0u : PB), w.k0, xb);
#pragma unroll
        for (int h = 0; h < N; ++h) {
            acc[h].mul(xb[h]);
            lns[h] = lns[h] + lb[h];
        }
    } else {
        // Any number of children, each read from where its record says.
        const unsigned nchild = reinterpret_cast<const RecHead *>(rec)->nchild;
        unsigned nl = 0;
#pragma unroll 1
        for (unsigned ci = 0; ci < nchild; ++ci) {
            const unsigned char *cr = kid0 + ci * sizeof(RecChild);
            const uint4 d = *reinterpret_cast<const uint4 *>(cr + 16);  // src idx tab off
            R x[N];
            S l[N];
            if (d.x == SRC_LEAF) {
#pragma unroll
                for (int h = 0; h < N; ++h) {
                    const unsigned m = rows[nl * w.tile + h * (w.tile / N)];
                    leaf_message<false, KT, G>(rec + d.w, d.z, w.ltab, m, w.k0, x[h]);
                    l[h] = S(0);
                }
                ++nl;
            } else {
                child_rows<T, KT, G, N>(cr, w, x, l);
                apply_p<KT, G, N>(rec + d.w, w.k0, x);
            }
#pragma unroll
            for (int h = 0; h < N; ++h) {
                if (ci == 0) {
                    acc[h] = x[h];
                    lns[h] = l[h];
                } else {
                    acc[h].mul(x[h]);
                    lns[h] = lns[h] + l[h];
                }
                // A long product stays inside the range.
                if (ci >= 1 && ci + 1 < nchild) rescale<KT, G>(acc[h], lns[h], true);
            }
        }
    }
}

// Walk every op of job `a` for tile `tile_idx`, aggregate the root and
// reduce.  G consecutive threads share a pattern, each holding KT of its
// KT*G components; with G = 1 a thread owns N patterns, blockDim apart.
// Every G, N and tile gives the same bits: scalers are maxima over the
// group, the root sum runs in one order and the sum over sites in any.
// Returns false if a bounded wait gave up.
template <typename T, int KT, int G, int N>
__device__ bool walk_tile(const PlanArgs &a, unsigned tile_idx, const LeanLayout &Lay,
                          unsigned grp, RingPos &ring) {
    static_assert(G == 1 || N == 1, "several threads a pattern or several patterns a thread");
    typedef typename Prec<T>::S S;
    typedef typename Prec<T>::V V;
    typedef Rows<T, KT, G> R;
    extern __shared__ __align__(128) unsigned char smem[];
    LeanHead &hd = *reinterpret_cast<LeanHead *>(smem);
    const unsigned nthr = blockDim.x, nwarp = nthr / 32;
    const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const unsigned tile = nthr / G * N;
    const unsigned p0 = tile_idx * tile;
    const unsigned g = tid % G;
    TileView<T> w;
    w.slots = reinterpret_cast<V *>(smem + Lay.slots);
    w.slot_sc = reinterpret_cast<S *>(smem + Lay.slot_sc);
    w.ltab = a.ltab;
    w.pitch = a.ppad;
    w.tile = tile;
    w.pl = tid / G;
    w.p = p0 + w.pl;
    w.k0 = g * KT;
    // The last tile of a job may pass its padded patterns by whole warps
    // (32 / G patterns each, and the padding is to 128); a tile of the
    // two-pattern walker divides them.
    const bool on = w.p < a.ppad;
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

    R acc[N];
    S lns[N];
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
                atomicOr(&a.res->err, 1u);
                *(volatile uint32_t *)&hd.abort = 1u;
            }
            break;
        }
        if (on) {
            const unsigned n = min(grp, a.nops - q * grp);
            const unsigned char *rec = st;
            const uint8_t *rows = st + (size_t)grp * a.rstride + w.pl;
            // What an op needs from its header, and its first two leaf
            // children's masks, are read while the op before it runs (past
            // a group's last op the words read are not used).
            uint64_t y, ysc;
            uint32_t word;
            unsigned m0[N], m1[N];
            auto head = [&](const unsigned char *r, uint64_t &hy, uint64_t &hs, uint32_t &hw) {
                const ulonglong2 h0 = *reinterpret_cast<const ulonglong2 *>(r);
                const uint4 h1 = *reinterpret_cast<const uint4 *>(r + 16);
                hy = addr_at(h0.x, w.p, sizeof(V));
                hs = addr_at(h0.y, w.p, sizeof(S));
                // (In a uniform register: the branches on it are the warp's.)
                hw = __reduce_or_sync(0xffffffffu, h1.z | (h1.y + 1u) << kSlotShift);
            };
            auto masks = [&](const uint8_t *rw, unsigned (&a0)[N], unsigned (&a1)[N]) {
#pragma unroll
                for (int h = 0; h < N; ++h) {
                    a0[h] = rw[h * nthr];
                    a1[h] = rw[tile + h * nthr];
                }
            };
            head(rec, y, ysc, word);
            masks(rows, m0, m1);
            for (unsigned b = 0; b < n; ++b) {
                walk_op<T, KT, G, N>(rec, word, (q | b) == 0u, m0, m1, rows, w, acc, lns);
                rec += a.rstride;
                rows += lmax * tile;
                uint64_t ny, nysc;
                uint32_t nword;
                unsigned nm0[N], nm1[N];
                head(rec, ny, nysc, nword);
                masks(rows, nm0, nm1);
#pragma unroll
                for (int h = 0; h < N; ++h) rescale<KT, G>(acc[h], lns[h], false);
                if ((word & kPlainMask) == 0) {
#pragma unroll
                    for (int h = 0; h < N; ++h) {
                        acc[h].store_global(y + h * nthr * sizeof(V), w.pitch, w.k0);
                        if (g == 0) st_global(ysc + h * nthr * sizeof(S), lns[h]);
                    }
                } else {
                    const unsigned slot = word >> kSlotShift;
#pragma unroll
                    for (int h = 0; h < N; ++h) {
                        if (!(word & REC_NO_HBM)) {
                            acc[h].store_global(y + h * nthr * sizeof(V), w.pitch, w.k0);
                            if (g == 0) st_global(ysc + h * nthr * sizeof(S), lns[h]);
                        }
                        if (slot != 0) {
                            const unsigned at = (slot - 1) * tile, q0 = w.pl + h * nthr;
                            acc[h].store_smem(w.slots + at * (KT * G * Prec<T>::U) + q0, tile,
                                              w.k0);
                            if (g == 0) w.slot_sc[at + q0] = lns[h];
                        }
                    }
                }
                if (G > 1) __syncwarp();  // lane g = 0's scaler is read by the group
                y = ny;
                ysc = nysc;
                word = nword;
#pragma unroll
                for (int h = 0; h < N; ++h) {
                    m0[h] = nm0[h];
                    m1[h] = nm1[h];
                }
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
    double v[N];
    bool ninf[N];
#pragma unroll
    for (int h = 0; h < N; ++h) {
        const unsigned p = w.p + h * nthr;
        // Root aggregation (CxLik.c:598-632): L = sum_k sum_i pn[k][i] root.
        if (!a.root_last && on) {
            acc[h].load_l2(addr_at(reinterpret_cast<uint64_t>(a.root), p, sizeof(V)), w.pitch,
                           w.k0);
            lns[h] = static_cast<const S *>(a.rootsc)[p];
        }
        // L = sum over components and states in one sequential order; every
        // lane of the group gathers the others' entries and sums them all.
        double L = 0.0;
        const unsigned lead = lane - g;
#pragma unroll
        for (int gg = 0; gg < G; ++gg) {
#pragma unroll
            for (int i = 0; i < KT * 4; ++i) {
                T x = acc[h].get(i / 4, i % 4);
                if (G > 1) x = __shfl_sync(0xffffffffu, x, lead + gg);
                L = fma(__ldcg(a.pn + gg * KT * 4 + i), (double)x, L);
            }
        }
        v[h] = 0.0;
        ninf[h] = false;
        if (g == 0 && p < a.npat) {
            v[h] = (sizeof(T) == 8 ? log(L) + (double)lns[h] : site_log(L, (int)lns[h])) *
                   (double)a.freqs[p];
            // (NaN, or +inf from rows that left the range: no likelihood.)
            if (!(v[h] < INFINITY)) v[h] = -INFINITY;
            if (a.site) a.site[p] = v[h];
            ninf[h] = isinf(v[h]);
            if (ninf[h]) v[h] = 0.0;
        }
    }
    reduce_sites<N>(a, v, ninf);
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
    constexpr unsigned L = 2;
    extern __shared__ __align__(128) unsigned char smem[];
    const unsigned nthr = blockDim.x;
    const unsigned tile = nthr / L;
    const unsigned tid = threadIdx.x;
    const unsigned lane = tid / tile;  // op lane of this thread
    const unsigned pl = tid % tile;    // pattern within the tile
    const unsigned p = tile_idx * tile + pl;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + Lay.bars);
    unsigned char *ring = smem + Lay.ring;
    float4 *slots = reinterpret_cast<float4 *>(smem + Lay.slots);
    int *slot_sc = reinterpret_cast<int *>(smem + Lay.slot_sc);
    const size_t sstride = (size_t)a.rstride * L;
    uint8_t *masks = smem + Lay.masks;
    const unsigned R_ = ring_depth;
    const unsigned nsteps = a.nops / L;  // the host pads nops to a multiple

    pdl_wait();  // the records hold the P kernel's matrices
    // Start streaming the job's first R steps of op records.
    if (tid == 0) {
        fence_proxy_async();
        for (unsigned o = 0; o < R_ && o < nsteps; ++o) {
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

    typedef Rows<float, KT, 1> R;
    R acc[1];
    int lns[1] = {0};
    const TileView<float> w{slots, slot_sc, nullptr, a.ppad, tile, pl, p, 0u};
    const uint32_t spin = g_spin_limit;
    for (unsigned o = 0, stage = 0; o < nsteps;
         ++o, stage = (stage + 1 == R_) ? 0u : stage + 1) {
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
            // A child's message: the rows of an internal child (a leaf has
            // none) are loaded first, so that an op with two children issues
            // both children's loads before it waits on either.
            auto load_in = [&](unsigned c, R (&x)[1], int (&l)[1]) {
                l[0] = 0;
                if (kids[c].src != SRC_LEAF)
                    child_rows<float, KT, 1, 1>(reinterpret_cast<const unsigned char *>(kids + c),
                                                w, x, l);
            };
            auto message = [&](unsigned c, R (&x)[1]) {
                if (kids[c].src == SRC_LEAF)
                    leaf_message<false, KT, 1>(rec + kids[c].off, 0u, nullptr,
                                               masks[(size_t)kids[c].idx * tile + pl], 0u, x[0]);
                else
                    apply_p<KT, 1, 1>(rec + kids[c].off, 0u, x);
            };
            R x[1];
            int l[1];
            if (nchild == 2) {
                load_in(0, acc, lns);
                load_in(1, x, l);
                message(0, acc);
                message(1, x);
                acc[0].mul(x[0]);
                lns[0] += l[0];
            } else {
                for (unsigned ci = 0; ci < nchild; ++ci) {
                    load_in(ci, x, l);
                    message(ci, x);
                    if (ci == 0) {
                        acc[0] = x[0];
                        lns[0] = l[0];
                    } else {
                        acc[0].mul(x[0]);
                        lns[0] += l[0];
                    }
                    // (As in walk_op: a long product stays inside the range.)
                    if (ci >= 1 && ci + 1 < nchild) rescale<KT, 1>(acc[0], lns[0], true);
                }
            }
            ydata = hd->data;
            yscaler = hd->scaler;
            yslot = hd->slot;
            yhbm = !(hd->flags & REC_NO_HBM);
        }
        // Every thread has read the stage: hand it to the step a ring on.  A record
        // wait that gave up in any warp ends the tile for all: thread 0
        // waits for the copies still in flight into the ring.
        if (!cta_hand_off(ok, nthr)) {
            if (tid == 0) {
                atomicOr(&a.res->err, 1u);
                drain_ring(bars, phase ^ (1u << stage), o, nsteps, R_);
            }
            return false;
        }
        if (tid == 0 && o + R_ < nsteps) {
            fence_proxy_async();
            mbar_expect_tx(&bars[stage], (uint32_t)sstride);
            bulk_g2s(ring + (size_t)stage * sstride, a.rec + (size_t)(o + R_) * sstride,
                     (uint32_t)sstride, &bars[stage]);
        }
        // (An empty lane of a step, with no children, stores nothing.)
        if (nchild != 0) {
            rescale<KT, 1>(acc[0], lns[0], false);
            if (yhbm) {
                acc[0].store_global(reinterpret_cast<uint64_t>(static_cast<float4 *>(ydata) + p),
                                    w.pitch, 0u);
                static_cast<int *>(yscaler)[p] = lns[0];
            }
            if (yslot >= 0) {
                acc[0].store_smem(slots + (unsigned)yslot * KT * tile + pl, tile, 0u);
                slot_sc[(unsigned)yslot * tile + pl] = lns[0];
            }
        }
        __syncthreads();  // the other lane may read these results next step
    }

    if (a.no_root) {
        __syncthreads();
        return true;
    }
    // Root aggregation (CxLik.c:598-632), lane 0's.
    if (!a.root_last) {
        acc[0].load_l2(reinterpret_cast<uint64_t>(static_cast<const float4 *>(a.root) + p),
                       w.pitch, 0u);
        lns[0] = static_cast<const int *>(a.rootsc)[p];
    }
    double Lsum = 0.0;
#pragma unroll
    for (int q = 0; q < KT * 4; ++q)
        Lsum = fma(__ldcg(a.pn + q), (double)acc[0].get(q / 4, q % 4), Lsum);
    double v[1] = {0.0};
    bool ninf[1] = {false};
    if (lane == 0 && p < a.npat) {
        v[0] = site_log(Lsum, lns[0]) * (double)a.freqs[p];
        if (!(v[0] < INFINITY)) v[0] = -INFINITY;  // as in walk_tile
        if (a.site) a.site[p] = v[0];
        ninf[0] = isinf(v[0]);
        if (ninf[0]) v[0] = 0.0;
    }
    reduce_sites<1>(a, v, ninf);
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

// Launch bounds of the walkers (see walker_threads): up to five components a
// thread fit 128 registers (two CTAs of 256), the others take what they need.
template <typename T, int KT, int G, int N, bool WIDE>
struct CtaOf {
    static constexpr int threads = WIDE ? kMaxThreads : kTuneThreads;
    static constexpr int per_sm = !WIDE && sizeof(T) == 4 && KT * N <= 5 ? 2 : 1;
};

// One plan: one CTA per tile.
template <typename T, int KT, int G, int N, bool WIDE>
__global__ void __launch_bounds__(CtaOf<T, KT, G, N, WIDE>::threads,
                                  CtaOf<T, KT, G, N, WIDE>::per_sm)
    walk_kernel(PlanArgs a) {
    const LeanLayout Lay = lean_layout(sizeof(T) == 4 ? CXG_FP32 : CXG_FP64, KT * G,
                                       blockDim.x / G * N, a.nslot, a.ring, a.rstride,
                                       a.lmax);
    init_lean();
    RingPos ring{0, 0};
    walk_tile<T, KT, G, N>(a, blockIdx.x, Lay, a.ring, ring);
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
template <typename T, int KT, int G, int N>
__global__ void __launch_bounds__(CtaOf<T, KT, G, N, false>::threads,
                                  CtaOf<T, KT, G, N, false>::per_sm)
    walk_batch_kernel(BatchArgs b) {
    __shared__ unsigned s_item;
    __shared__ __align__(16) PlanArgs s_job;
    const LeanLayout Lay = lean_layout(sizeof(T) == 4 ? CXG_FP32 : CXG_FP64, KT * G,
                                       blockDim.x / G * N, b.max_nslot, b.ring, b.max_rstride,
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
        const WalkItem it = b.order != nullptr
                                ? WalkItem{b.order[item / b.ntiles], item % b.ntiles}
                                : b.items[item];
        if (it.job != job) {
            load_job(s_job, b.jobs + it.job);
            job = it.job;
        }
        if (!walk_tile<T, KT, G, N>(s_job, it.tile, Lay, b.ring, ring)) break;
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
// pattern G, patterns per thread N): every kact with one of each, a
// pattern's components split over 2 or 4 threads, and the FP32 form with two
// patterns a thread (walker_shape_ok).
#define CXG_SHAPES_1(X) \
    X(1, 1, 1) X(2, 1, 1) X(3, 1, 1) X(4, 1, 1) X(5, 1, 1) X(6, 1, 1) X(7, 1, 1) X(8, 1, 1)
#define CXG_SHAPES_G(X) X(1, 2, 1) X(2, 2, 1) X(3, 2, 1) X(4, 2, 1) X(1, 4, 1) X(2, 4, 1)
#define CXG_SHAPES_N(X) X(1, 1, 2) X(2, 1, 2) X(3, 1, 2) X(4, 1, 2) X(5, 1, 2)

template <typename T, int KT, int G, int N, bool WIDE>
static cudaError_t walk_fn(size_t sm, void (**fn)(PlanArgs)) {
    static size_t optin = 0;
    *fn = walk_kernel<T, KT, G, N, WIDE>;
    return ensure_smem(walk_kernel<T, KT, G, N, WIDE>, sm, optin);
}
template <typename T, int KT, int G, int N>
static cudaError_t batch_fn(size_t sm, void (**fn)(BatchArgs)) {
    static size_t optin = 0;
    *fn = walk_batch_kernel<T, KT, G, N>;
    return ensure_smem(walk_batch_kernel<T, KT, G, N>, sm, optin);
}
template <int K, int NT, int MINB>
static cudaError_t lanes_fn(size_t sm, void (**fn)(PlanArgs)) {
    static size_t optin = 0;
    *fn = walk_kernel_lanes<K, NT, MINB>;
    return ensure_smem(walk_kernel_lanes<K, NT, MINB>, sm, optin);
}
// The walkers of shape w, with their dynamic shared memory limit raised to
// `sm` bytes.
template <typename T>
static cudaError_t pick_walker(const WalkShape &w, size_t sm, void (**fn)(PlanArgs)) {
#define CXG_X(KT, GG, NN)                                             \
    if (w.kact == (KT) * (GG) && w.tpp == (GG) && w.ppt == (NN))      \
        return walk_fn<T, KT, GG, NN, false>(sm, fn);
#define CXG_W(KT) \
    if (w.kact == (KT)) return walk_fn<T, KT, 1, 1, true>(sm, fn);
    if constexpr (sizeof(T) == 4) {
        if (w.wide) {
            CXG_W(1) CXG_W(2) CXG_W(3) CXG_W(4) CXG_W(5)
            return cudaErrorInvalidValue;
        }
        CXG_SHAPES_N(CXG_X)
    }
    CXG_SHAPES_1(CXG_X)
    CXG_SHAPES_G(CXG_X)
#undef CXG_W
    return cudaErrorInvalidValue;
#undef CXG_X
}
template <typename T>
static cudaError_t pick_batch_walker(const WalkShape &w, size_t sm, void (**fn)(BatchArgs)) {
#define CXG_X(KT, GG, NN)                                             \
    if (w.kact == (KT) * (GG) && w.tpp == (GG) && w.ppt == (NN))      \
        return batch_fn<T, KT, GG, NN>(sm, fn);
    if constexpr (sizeof(T) == 4) {
        CXG_SHAPES_N(CXG_X)
    }
    CXG_SHAPES_1(CXG_X)
    CXG_SHAPES_G(CXG_X)
    return cudaErrorInvalidValue;
#undef CXG_X
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
// ops per stage), or that of the op-lane walker (its ring counts steps).
size_t walk_smem_bytes(const WalkShape &w, unsigned nslot, unsigned rstride, unsigned lmax,
                       unsigned nleaf) {
    return w.lanes == 1
               ? lean_layout(w.precision, w.kact, w.tile, nslot, w.ring, rstride, lmax).total
               : smem_layout(w.precision, w.kact, w.tile, nslot, w.ring, rstride * w.lanes, lmax,
                             nleaf).total;
}

static bool shape_launches(const WalkShape &w) {
    if (w.tile == 0 || w.tile % 32 || w.ring == 0 ||
        !walker_shape_ok(w.precision, w.kact, w.tpp, w.ppt))
        return false;
    if (w.lanes == 2)
        return lanes_shape_ok(w.precision, w.kact, w.tpp, w.ppt) && w.ring <= 8 &&
               w.tile * 2 <= kLaneThreads;
    // (Only whole warps of a tile may pass a job's patterns: two patterns a
    // thread need tiles that divide them.)
    return w.lanes == 1 && w.tile / w.ppt >= 32 && w.threads() <= walker_threads(w) &&
           (!w.wide || wide_shape_ok(w)) &&
           (w.ppt == 1 || kPatternQuantum % w.tile == 0);
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
    WalkShape w = shape_of(precision, a.kact, a.tile, a.tpp, a.ppt, lanes, a.ring);
    w.wide = a.wide;
    if (!shape_launches(w) || a.rstride % 16 || a.rstride == 0 ||
        a.ntiles != plan_blocks(a.ppad, a.tile) || (lanes == 1 && w.ring * a.lmax > 32) ||
        (lanes == 2 && (a.lmax != 0 || a.nops % 2 || a.ppad % a.tile)))
        return cudaErrorInvalidValue;
    const size_t sm = walk_smem_bytes(w, a.nslot, a.rstride, a.lmax, a.nleaf);
    void (*fn)(PlanArgs) = nullptr;
    cudaError_t e = lanes == 2              ? pick_walker_lanes(a.kact, a.tile, sm, &fn)
                    : precision == CXG_FP32 ? pick_walker<float>(w, sm, &fn)
                                            : pick_walker<double>(w, sm, &fn);
    if (e != cudaSuccess) return e;
    const unsigned nb = a.ntiles, nt = w.threads() * lanes;
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

static cudaError_t pick_batch(const WalkShape &w, size_t sm, void (**fn)(BatchArgs)) {
    if (w.wide) return cudaErrorInvalidValue;
    return w.precision == CXG_FP32 ? pick_batch_walker<float>(w, sm, fn)
                                   : pick_batch_walker<double>(w, sm, fn);
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
        w.ring * b.max_lmax > 32)
        return cudaErrorInvalidValue;
    const size_t sm = walk_smem_bytes(w, b.max_nslot, b.max_rstride, b.max_lmax, 0);
    void (*fn)(BatchArgs) = nullptr;
    const cudaError_t e = pick_batch(w, sm, &fn);
    if (e != cudaSuccess) return e;
    fn<<<grid, w.threads(), sm, s>>>(b);
    return cudaGetLastError();
}

int batch_ctas_per_sm(const WalkShape &w, size_t smem) {
    if (!shape_launches(w)) return 0;
    void (*fn)(BatchArgs) = nullptr;
    cudaError_t e = pick_batch(w, smem, &fn);
    int n = 0;
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, (int)w.threads(),
                                                          smem);
    return e == cudaSuccess ? n : 0;
}

__global__ void qdecomp_kernel(const __grid_constant__ QModel m, double *out) {
    if (blockIdx.x == 0) qdecomp_warp(m.rtri, m.pi, out);
}

cudaError_t launch_qdecomp(const QModel &m, double *out, cudaStream_t s) {
    qdecomp_kernel<<<1, 32, 0, s>>>(m, out);
    return cudaGetLastError();
}

}  // namespace cxg
