// hj_join_tc.cu -- tensor-core forms (HJ_FORM_TC_TF32, HJ_FORM_TC_BF16X3, HJ_FORM_TC_FP16).
//
// Replaces the same block-pair kernel as hj_join_fp64.cu (the reference's
// EGO_LOOP_TRAN[_NOSELF], hilbertjoin/egojoin.h:311-392, :482-553), but with
// the norm expansion the reference itself uses,
//     |a - b|^2 = |a|^2 + |b|^2 - 2 a.b      (egojoin.h:182-195, :329-381),
// and the a.b tile on the 5th-generation tensor cores:
//
//   * one persistent CTA per SM, 12 warps, warp-specialised:
//       warp 0   TMA producer: the A tile (128 EGO ranks x K) once per work
//                item into one of two A buffers, then the B tiles (256 ranks)
//                one 128-byte K atom (32 KB) at a time into a ring of stages;
//       warp 1   MMA issuer (one elected lane): tcgen05.mma, M=128, N=256,
//                operands from shared memory (128-byte swizzled, K-major),
//                accumulator in tensor memory, two accumulators (512 columns);
//       warps 2, 3  near warps: classify the queued rows that may hold near
//                pairs, 32 at a time (warp 2 instead completes the A tiles of
//                joins with folded norms);
//       warps 4-11 epilogue: tcgen05.ld of the accumulator rows (TMEM lane
//                quadrant = warp % 4, two warps per quadrant on 128 columns
//                each), dist^2 estimate, near rows found and queued;
//   * TF32: operands rounded to TF32 on the device (round to nearest), one
//     MMA per K step; BF16X3: a = a_hi + a_lo in BF16, a.b =
//     a_hi.b_hi + a_lo.b_hi + a_hi.b_lo (three MMAs per K step); FP16: the
//     operands scaled by a power of two into FP16's range and rounded once
//     (the precision of TF32 at twice its MMA rate), one MMA per K step, the
//     norms, eps^2 and the bound in the same scaled units;
//   * exact count: with s = |a|^2 + |b|^2 - 2 v (v the tensor-core dot product),
//     every error of v, of the FP32 norms and of the FP32 epilogue is bounded
//     by c_rel * (|a|^2 + |b|^2) + c_abs (tc_band_constants). A pair with
//     s + bound <= eps^2 is certainly inside, one with s - bound > eps^2 is
//     certainly outside, and every other pair (the band) is queued and
//     re-evaluated by k_recheck with the FP64 pair test. So the count equals
//     the plain FP64 form's, bit for bit.
//   * fast path: per row and 32-column group the epilogue takes the minimum of
//     |b|^2 - 2 v (of -2 v where the norms are folded into the accumulator); only
//     if that can still reach eps^2 + bound (rare: neighbours are a small fraction
//     of the candidates) is the row queued for the near warps, or, where several
//     rows of the group are near, the group classified by the warp itself,
//     branch-free from its registers.
//
// What bounds it (one B200, distance kernel alone, before -> after the epilogue took
// this form; SM clock 1.965 GHz, in the two longest 1.8 under the power limit): one
// global centre, 1M x 64 FP16, 32 neighbours: 83.7 -> 76.4 ms; 600k x 64: 29.3 -> 27.7;
// 200k x 64: 4.33 -> 3.46; 200k x 200k x 20 (folded norms): 15.1 -> 6.2; 30k x 70k x 100:
// 1.18 -> 0.51; 150k x 128 BF16x3: 6.3 -> 5.2. Block centres, 4M x 28 clustered FP16:
// 33.9 -> 27.1; 300k x 32 TF32: 1.63 -> 1.26 to 1.50. At K = 64 a tile's MMAs
// take 512 clocks and a tile without near rows about 1100: the chain MMA -> commit
// -> TMEM load -> release -> MMA over two accumulators. Near rows add the rest. An
// instruction of the epilogue costs its warp four to six clocks and a ready barrier,
// a vote or a tcgen05 fence 30 to 50, with two epilogue warps per scheduler; so the
// tile loop is kept short: 64 columns per TMEM load, two votes per load, item data
// one item ahead, group minima in registers (one load per 32 tiles). Measured and
// dropped: 32-column loads double-buffered (more votes and waits: +25%), 128
// columns at once (spills), two issuing warps, each set of four epilogue warps on
// one accumulator, near rows worked off by the epilogue warps between tiles.
//
// Every mbarrier wait is bounded in time (hj_common.cuh); on a timeout the
// kernel raises kErrTimeout (with the number of the wait that gave up in bits
// 8..15 of the error word), every role stops at its next wait, the copies and
// MMAs already issued are drained, the tensor memory is freed and the kernel
// returns. hj_debug_set_wait_gate makes the epilogue's first wait one that
// nothing ends, so that tests run this path.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cmath>
#include <mutex>
#include <string>
#include <type_traits>

#include "../../include/hj.h"
#include "hj_common.cuh"
#include "hj_internal.h"

namespace hj {

// Epilogue warps: two per TMEM lane quadrant, each on kEpiCols of the 256
// accumulator columns, read kChunkCols at a time.
constexpr int kEpiWarps = 8;
constexpr int kEpiCols = 128;
constexpr int kChunkCols = 64;
// Band slots are reserved by each warp in chunks (one atomic, whose latency the warp
// waits for, per chunk); slots a warp leaves unused are marked with ia = kBandHole.
// Block centring, where near pairs are common, takes larger chunks.
constexpr uint32_t kBandChunk = 256, kBandChunkRare = 32;
constexpr uint32_t kBandHole = 0xffffffffu;
static_assert(kEpiWarps * kEpiCols == 4 * kTcTileB && kEpiCols == 2 * kChunkCols && kChunkCols == 64,
              "the shared-memory plan and the epilogue assume 8 warps of two chunks");
// Warpgroup 0 holds the control and near warps, warpgroups 1 and 2 the epilogue. The
// block launches with 168 registers a thread (64512); warpgroup 0 gives part of its
// share to the epilogue: 128 x 88 + 256 x 208 = 64512.
constexpr int kFoldWarp = 2;
constexpr int kEpiWarp0 = 4;
constexpr int kTcThreads = 32 * (kEpiWarp0 + kEpiWarps);
constexpr int kCtlRegs = 88, kEpiRegs = 208;
static_assert(128 * kCtlRegs + 32 * kEpiWarps * kEpiRegs <= kTcThreads * 168, "register split");
constexpr uint32_t kAtomBytes = 128;                  // bytes of K per row per swizzle atom
constexpr uint32_t kAStageBytes = kTcTileA * kAtomBytes;  // 16 KB per A atom
constexpr uint32_t kBStageBytes = kTcTileB * kAtomBytes;  // 32 KB per B atom
constexpr uint32_t kTmemCols = 512;

// Near rows are not classified where they are found. A lane whose 32 columns may
// hold a pair that is not certainly outside copies them, with what classifies
// them, into its warp's queue in shared memory, and the near warps work the queues
// off beside the epilogue, up to 32 rows at a time (lane = row). A row's
// classification takes one to two thousand clocks of latency (the B norms, a slot in
// the band queue), and one near row in a tile used to hold the accumulator of all
// eight warps for it; at 1M x 64 and 32 neighbours six tiles in ten have one.
// An entry: 32 values | |a|^2, thr_in, thr_out, A rank | first B rank, job, norms
// folded, 0 | 4 unused words (an odd number of 16-byte units, so that lanes
// reading their rows do not meet in a bank).
constexpr uint32_t kNearWords = 44;
constexpr uint32_t kNearCap = 24;    // entries per warp, at most
// A group with more near rows is classified by the epilogue warp (lane = row): about
// 1000 clocks however many rows, against the queue's per-row cost. With one centre, 30k x
// 70k x 100: 0.54 ms at 0, 0.50 at 1, 0.49 at 2, 0.54 at 3, 0.62 at 6; 1M x 64: 80, 70,
// 69, 69, 68 ms. Block centres, 4M x 28: 38.8 ms at 2, 37.7 at 3, 37.3 at 4, 37.9 at 6,
// 40.5 at 8.
constexpr int kNearDenseBc = 4, kNearDenseOne = 2;
// Fewer entries than this are not worth a B stage, and so small a queue is not used:
// where three B stages and the A tile leave no room (BF16x3 from d = 193, block-centred
// from 62; TF32 from 225), rows would wait for one another's place, and a tile's MMAs
// take 3700 clocks and more, behind which the warp classifies all near rows itself. One
// entry -> none, 60k points, 8 and 64 neighbours: BF16x3 d = 256 2.11 -> 1.77 and 2.52 ->
// 1.80 ms, TF32 256 1.67 -> 1.20 and 2.37 -> 1.33; block-centred BF16x3, 150k x 64
// clustered 2.16 -> 1.31.
constexpr uint32_t kNearMinCap = 8;
// Rows that a near warp waits for before it starts on a batch, unless a queue is half
// full, instead of at the first row: 200k x 200k x 20 6.7 -> 6.35 ms, 1M x 64 72 -> 69.6;
// at 12 rows half of that.
constexpr uint32_t kNearBatch = 24;
constexpr uint32_t kNearDone = 0x80000000u;  // in a queue's tail: its warp has finished

struct BandEntry {
    uint32_t ia, jb;  // EGO ranks in A and B
    float s_hat;      // one centre: the pair's accumulator value, from which the recheck forms the
                      // estimate of dist^2; block centring: the estimate, NaN where not kept
    uint32_t pad;
};

struct TcArgs {
    uint32_t ka;        // K atoms per operand buffer, the largest of the jobs' (TF32: kpad/32; BF16, FP16: kpad16/64)
                        // (each job multiplies only its own ksteps)
    uint32_t a_bufs;    // 1 or 2 A buffers
    uint32_t nst;       // B ring stages
    uint32_t near_cap;  // entries of each epilogue warp's near queue (>= 1)
    int near_rows;      // most near rows of a group that go to the queue (0: it is not used)
    const WorkItem *items;
    uint64_t n_items;
    const float *norm_a, *norm_b;   // FP32 |x|^2 per EGO rank (padding: kPadNorm)
    const float *tmax_b;            // per 256-rank B tile: max |x|^2
    const float *gmin_b;            // per 32-rank B group: min |x|^2
    const TcJob *jobs;              // per job: counted rows, thresholds, count (item.pad = job)
    uint64_t na, nb;                // job 0's counted ranks (debug output only)
    BandEntry *band;
    uint64_t band_cap;
    unsigned long long *band_total;  // slots reserved (chunks of kBandChunk or kBandChunkRare)
    unsigned long long *band_holes;  // reserved slots left unused (marked kBandHole); may be null
    uint32_t *err;
    float *dbg;                     // optional: s_hat for every pair, input order [na][nb] (tests)
    const uint32_t *perm_a, *perm_b;  // EGO rank -> input index (for dbg)
    uint32_t a_xoff;                // first column of the A operand in its rows (block centring: dp)
    uint32_t fold;                  // some job's norms are folded: the fold warp completes every A tile
    uint64_t gate_ns;               // test hook: > 0 makes the epilogue wait this long on a barrier
                                    // that nothing arrives on, then raise kErrTimeout
    uint64_t near_ns;               // the near warps' limit for the queues to end after an error
    // per-block centring (BC kernels): norm_a is then q of the A rows (norm_b and
    // gmin_b unused: the accumulator holds w = v - q_j / 2); |h| of the A rows,
    // block summaries and centres of both sets
    const float *xn_a;
    const float4 *blk_a, *blk_b;
    const float *cent_a, *cent_b;
    BcConsts bc;
};

// ---------------------------------------------------------------- PTX helpers

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t *dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// Register share of a warpgroup: all its warps execute the same one of these, once.
template <int R>
__device__ __forceinline__ void reg_dec() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R));
}
template <int R>
__device__ __forceinline__ void reg_inc() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R));
}

__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}
__device__ __forceinline__ void mma_commit(bool issue, uint64_t *bar) {
    if (!issue) return;
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// This and mma_commit act in the warp's elected lane only (`issue`).
template <int FORM>
__device__ __forceinline__ void mma_issue(bool issue, uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
    if (!issue) return;
    if constexpr (FORM == HJ_FORM_TC_TF32) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
            "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
            "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    }
}

// 64 consecutive accumulator columns of this thread's TMEM lane: the load is
// issued here and its registers may be read after tmem_wait on them.
__device__ __forceinline__ void tmem_ld(uint32_t taddr, float (&v)[64]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x64.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, "
        "%20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32, %33, %34, %35, %36, %37, "
        "%38, %39, %40, %41, %42, %43, %44, %45, %46, %47, %48, %49, %50, %51, %52, %53, %54, %55, "
        "%56, %57, %58, %59, %60, %61, %62, %63}, [%64]; "
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]),
          "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]), "=f"(v[16]),
          "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]), "=f"(v[24]),
          "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31]), "=f"(v[32]),
          "=f"(v[33]), "=f"(v[34]), "=f"(v[35]), "=f"(v[36]), "=f"(v[37]), "=f"(v[38]), "=f"(v[39]), "=f"(v[40]),
          "=f"(v[41]), "=f"(v[42]), "=f"(v[43]), "=f"(v[44]), "=f"(v[45]), "=f"(v[46]), "=f"(v[47]), "=f"(v[48]),
          "=f"(v[49]), "=f"(v[50]), "=f"(v[51]), "=f"(v[52]), "=f"(v[53]), "=f"(v[54]), "=f"(v[55]), "=f"(v[56]),
          "=f"(v[57]), "=f"(v[58]), "=f"(v[59]), "=f"(v[60]), "=f"(v[61]), "=f"(v[62]), "=f"(v[63])
        : "r"(taddr)
        : "memory");
}

// Waits for the warp's outstanding TMEM loads. The registers are operands, so
// that no use of them is scheduled before the wait.
__device__ __forceinline__ void tmem_wait(float (&v)[64]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7]),
                   "+f"(v[8]), "+f"(v[9]), "+f"(v[10]), "+f"(v[11]), "+f"(v[12]), "+f"(v[13]), "+f"(v[14]),
                   "+f"(v[15]), "+f"(v[16]), "+f"(v[17]), "+f"(v[18]), "+f"(v[19]), "+f"(v[20]), "+f"(v[21]),
                   "+f"(v[22]), "+f"(v[23]), "+f"(v[24]), "+f"(v[25]), "+f"(v[26]), "+f"(v[27]), "+f"(v[28]),
                   "+f"(v[29]), "+f"(v[30]), "+f"(v[31]), "+f"(v[32]), "+f"(v[33]), "+f"(v[34]), "+f"(v[35]),
                   "+f"(v[36]), "+f"(v[37]), "+f"(v[38]), "+f"(v[39]), "+f"(v[40]), "+f"(v[41]), "+f"(v[42]),
                   "+f"(v[43]), "+f"(v[44]), "+f"(v[45]), "+f"(v[46]), "+f"(v[47]), "+f"(v[48]), "+f"(v[49]),
                   "+f"(v[50]), "+f"(v[51]), "+f"(v[52]), "+f"(v[53]), "+f"(v[54]), "+f"(v[55]), "+f"(v[56]),
                   "+f"(v[57]), "+f"(v[58]), "+f"(v[59]), "+f"(v[60]), "+f"(v[61]), "+f"(v[62]), "+f"(v[63])::"memory");
}

// max(a, b, c) in one instruction (three-input max.f32, sm_100).
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// The largest of the 32 values from v: 16 instructions in a tree of depth 4.
__device__ __forceinline__ float max32(const float *v) {
    float t[10];
#pragma unroll
    for (int i = 0; i < 10; ++i) t[i] = fmax3(v[3 * i], v[3 * i + 1], v[3 * i + 2]);
    const float u0 = fmax3(t[0], t[1], t[2]), u1 = fmax3(t[3], t[4], t[5]);
    const float u2 = fmax3(t[6], t[7], t[8]), u3 = fmax3(t[9], v[30], v[31]);
    return fmaxf(fmax3(u0, u1, u2), u3);
}

// v[j] of 32 values in registers: a tree of selects (31; an index would put v in local
// memory).
__device__ __forceinline__ float pick32(const float *v, int j) {
    float t[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) t[i] = (j & 16) ? v[16 + i] : v[i];
#pragma unroll
    for (int h = 8; h > 0; h >>= 1)
#pragma unroll
        for (int i = 0; i < h; ++i) t[i] = (j & h) ? t[h + i] : t[i];
    return t[0];
}

// Shared-memory matrix descriptor: K-major operand in 128-byte swizzle atoms
// (8 rows x 128 B, atoms stacked along M/N every 1024 B).
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

// Instruction descriptor: D = F32, A/B K-major, M = 128, N = 256.
template <int FORM>
__device__ __forceinline__ constexpr uint32_t instr_desc() {
    constexpr uint32_t ab = FORM == HJ_FORM_TC_TF32 ? 2u : (FORM == HJ_FORM_TC_BF16X3 ? 1u : 0u);  // TF32, BF16, F16
    return (1u << 4) | (ab << 7) | (ab << 10) | ((uint32_t)(kTcTileB >> 3) << 17) | ((uint32_t)(kTcTileA >> 4) << 24);
}

// Whether the phase has completed, without waiting.
__device__ __forceinline__ bool mbar_test(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Waits for a phase regardless of the error word, until `deadline`
// (%globaltimer): the drain of copies and MMAs already issued.
__device__ __forceinline__ void drain_until(uint64_t *bar, uint32_t parity, uint64_t deadline) {
    while (!mbar_try_wait(bar, parity)) {
        if (globaltimer_ns() > deadline) break;
    }
}

// A warp's slots in the band queue, taken in chunks (one atomic per chunk; all
// state warp-uniform).
struct BandSlots {
    unsigned long long k0, nb;
    uint32_t rem;
    // the slot of the entry of rank r: r < rem ? k0 + r : nb + (r - rem)
    __device__ unsigned long long at(uint32_t r) const { return r < rem ? k0 + r : nb + (r - rem); }
};
struct BandWriter {
    const TcArgs &p;
    uint32_t lane, chunk;
    unsigned long long slot = 0, end = 0;  // the current chunk
    __device__ BandWriter(const TcArgs &p_, uint32_t lane_, uint32_t chunk_) : p(p_), lane(lane_), chunk(chunk_) {}
    // c new slots: the rest of the chunk first, then a new one
    __device__ BandSlots reserve(uint32_t c) {
        BandSlots b{slot, 0, (uint32_t)(end - slot)};
        if (c <= b.rem) {
            slot += c;
            return b;
        }
        const uint32_t need = c - b.rem, size = need > chunk ? need : chunk;
        unsigned long long nb = 0;
        if (lane == 0) nb = atomicAdd(p.band_total, (unsigned long long)size);
        b.nb = __shfl_sync(0xffffffffu, nb, 0);
        slot = b.nb + need;
        end = b.nb + size;
        return b;
    }
    __device__ void store(unsigned long long k, uint32_t ia, uint32_t jb, float s_hat, uint32_t job) const {
        if (k >= p.band_cap) return;
        BandEntry e;
        e.ia = ia;
        e.jb = jb;
        e.s_hat = s_hat;
        e.pad = job;
        p.band[k] = e;
    }
    // the unused rest of the chunk: marked for the recheck to skip
    __device__ void finish() {
        for (unsigned long long k = slot + lane; k < end; k += 32) store(k, kBandHole, 0, 0.f, 0);
        if (lane == 0 && end > slot && p.band_holes) atomicAdd(p.band_holes, end - slot);
        slot = end;
    }
};

__device__ __forceinline__ uint32_t lds_acquire(const uint32_t *a) {
    uint32_t v;
    asm volatile("ld.acquire.cta.shared.u32 %0, [%1];" : "=r"(v) : "r"(smem_u32(a)) : "memory");
    return v;
}
__device__ __forceinline__ void sts_release(uint32_t *a, uint32_t v) {
    asm volatile("st.release.cta.shared.u32 [%0], %1;" ::"r"(smem_u32(a)), "r"(v) : "memory");
}

// Columns of the 32 from rank gj that row gi may count: below b_end, and above its own
// rank for a self-join.
__device__ __forceinline__ uint32_t count_mask(uint32_t gi, uint32_t gj, uint32_t b_end, bool self) {
    const int hi = (int)b_end - (int)gj, lo = self ? (int)gi + 1 - (int)gj : 0;
    const uint32_t mh = hi >= 32 ? 0xffffffffu : (hi <= 0 ? 0u : (1u << hi) - 1u);
    const uint32_t ml = lo <= 0 ? 0xffffffffu : (lo >= 32 ? 0u : ~((1u << lo) - 1u));
    return mh & ml;
}

// ---------------------------------------------------------------- the kernel

template <int FORM, bool BC>
__global__ void __launch_bounds__(kTcThreads, 1)
    k_join_tc(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_a2,
              const __grid_constant__ CUtensorMap tm_b, const __grid_constant__ CUtensorMap tm_b2, TcArgs p) {
    // A atoms per buffer: TF32 ka; BF16 2*ka (hi atoms, then lo atoms). B atoms
    // per tile, in ring order: TF32 q = 0..ka-1; BF16 (hi q, lo q) for each q.
    constexpr bool kBf = FORM == HJ_FORM_TC_BF16X3;
    constexpr int32_t kAtomElems = FORM == HJ_FORM_TC_TF32 ? 32 : 64;  // K elements per 128-byte atom
    const uint32_t a_atoms = kBf ? 2 * p.ka : p.ka;
    const uint32_t a_buf_bytes = a_atoms * kAStageBytes;

    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar_afull[2], bar_aempty[2], bar_aready[2], bar_accfull[2], bar_accempty[2];
    __shared__ __align__(8) uint64_t bar_drain, bar_gate;
    __shared__ __align__(8) uint64_t bar_bfull[8], bar_bempty[8];
    __shared__ uint32_t tmem_base_sh;
    __shared__ uint32_t near_tail[kEpiWarps], near_head[kEpiWarps];  // entries queued (| kNearDone), worked off

    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t a_base = smem_base;
    const uint32_t b_base = smem_base + p.a_bufs * a_buf_bytes;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    volatile uint32_t *err = p.err;

    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bar_afull[i], 1);
            mbar_init(&bar_aempty[i], 1);
            mbar_init(&bar_aready[i], 1);
            mbar_init(&bar_accfull[i], 1);
            mbar_init(&bar_accempty[i], kEpiWarps);
        }
        for (uint32_t i = 0; i < p.nst; ++i) {
            mbar_init(&bar_bfull[i], 1);
            mbar_init(&bar_bempty[i], 1);
        }
        mbar_init(&bar_drain, 1);
        for (int i = 0; i < kEpiWarps; ++i) near_tail[i] = near_head[i] = 0;
        mbar_init(&bar_gate, 1);
        fence_barrier_init();
    }
    if (warp == 0) {
        tmem_alloc(&tmem_base_sh, kTmemCols);
        if (lane == 0) {
            prefetch_tmap(&tm_a);
            prefetch_tmap(&tm_b);
            if (kBf) {
                prefetch_tmap(&tm_a2);
                prefetch_tmap(&tm_b2);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_sh;
    const uint64_t stride = gridDim.x;
    float *near_base = reinterpret_cast<float *>(smem_raw + (b_base + p.nst * kBStageBytes - smem_u32(smem_raw)));
    const uint32_t near_ring = p.near_cap * kNearWords;  // floats per epilogue warp
    // item `i` of the list, an empty one past its end
    auto item_at = [&](uint64_t i) { return i < p.n_items ? p.items[i] : WorkItem{0, 0, 0, 0}; };

    // every warp of a warpgroup executes the same setmaxnreg
    if (warp < kEpiWarp0) {
        reg_dec<kCtlRegs>();
        if (warp == 0) {
            // ------------------------------------------------ TMA producer
            if (lane == 0) {
                uint32_t a_cnt = 0, b_cnt = 0;
                uint32_t abuf = 0, aph = 1;  // A buffer of the next item, parity of its last release
                uint32_t s = 0, sph = 1;     // B stage of the next atom, parity of its last release
                bool ok = true;
                WorkItem w = item_at(blockIdx.x);
                for (uint64_t it = blockIdx.x; ok && it < p.n_items; it += stride) {
                    const WorkItem wn = item_at(it + stride);
                    const uint32_t ka = p.jobs[w.pad].ka;  // this job's K atoms (<= p.ka)
                    const uint32_t ja_atoms = kBf ? 2 * ka : ka;
                    // parity 1 of a barrier that never completed a phase counts as passed: the first uses do not wait
                    if (!mbar_wait(&bar_aempty[abuf], aph, err, 1)) break;
                    mbar_arrive_expect_tx(&bar_afull[abuf], ja_atoms * kAStageBytes);
                    const uint32_t adst = a_base + abuf * a_buf_bytes;
                    for (uint32_t q = 0; q < ja_atoms; ++q) {
                        const bool lo = kBf && q >= ka;
                        const uint32_t kq = kBf ? (lo ? q - ka : q) : q;
                        tma_load_2d(smem_raw + (adst + q * kAStageBytes - smem_u32(smem_raw)), lo ? &tm_a2 : &tm_a,
                                    (int32_t)(kq * kAtomElems + p.a_xoff), (int32_t)(w.a * kTcTileA), &bar_afull[abuf]);
                    }
                    ++a_cnt;
                    if (++abuf == p.a_bufs) abuf = 0, aph ^= 1u;
                    for (uint32_t bt = w.b0; ok && bt < w.b1; ++bt) {
                        for (uint32_t q = 0; q < ja_atoms; ++q) {
                            if (!mbar_wait(&bar_bempty[s], sph, err, 2)) {
                                ok = false;
                                break;
                            }
                            mbar_arrive_expect_tx(&bar_bfull[s], kBStageBytes);
                            const bool lo = kBf && (q & 1u);
                            const uint32_t kq = kBf ? (q >> 1) : q;
                            tma_load_2d(smem_raw + (b_base + s * kBStageBytes - smem_u32(smem_raw)), lo ? &tm_b2 : &tm_b,
                                        (int32_t)(kq * kAtomElems), (int32_t)(bt * kTcTileB), &bar_bfull[s]);
                            ++b_cnt;
                            if (++s == p.nst) s = 0, sph ^= 1u;
                        }
                    }
                    w = wn;
                }
                // Drain: on the normal path every copy has been consumed; after an
                // error (the loops stop at the first failed wait) every copy issued
                // has landed before the CTA leaves (its full barrier's phase).
                if (*err) {
                    const uint64_t deadline = globaltimer_ns() + kWaitLimitNs;
                    for (uint32_t k = 0; k < p.nst && k < b_cnt; ++k) {
                        const uint32_t j = b_cnt - 1 - k;
                        drain_until(&bar_bfull[j % p.nst], (j / p.nst) & 1u, deadline);
                    }
                    for (uint32_t k = 0; k < p.a_bufs && k < a_cnt; ++k) {
                        const uint32_t j = a_cnt - 1 - k;
                        drain_until(&bar_afull[j % p.a_bufs], (j / p.a_bufs) & 1u, deadline);
                    }
                }
            }
        } else if (warp == 1) {
            // ------------------------------------------------ MMA issuer
            // An MMA is accepted about when the one before it ends (128 clocks at N =
            // 256), so what the thread does between two MMAs beyond that adds to the
            // tile: the next stage and the next accumulator are looked at before the
            // current stage's MMAs are issued, descriptors advance by additions, and the
            // whole warp runs the loop with one elected lane issuing (a lane running it
            // alone took a third longer per tile).
            {
                const bool el = elect_one();
                constexpr uint32_t idesc = instr_desc<FORM>();
                uint64_t *bar_a = p.fold ? bar_aready : bar_afull;
                uint32_t abuf = 0, aph = 0;      // A buffer of the item, its phase
                uint32_t s = 0, sph = 0;         // B stage of the next atom, its phase
                uint32_t acc = 0, accph = 1;     // accumulator of the next tile, parity of its last release
                bool acc_ready = true, b_ready = false;
                bool issued_any = false, ok = true;
                const uint64_t b_desc0 = sw128_desc(b_base);
                WorkItem w = item_at(blockIdx.x);
                for (uint64_t it = blockIdx.x; ok && it < p.n_items; it += stride) {
                    const WorkItem wn = item_at(it + stride);
                    const uint32_t ka = p.jobs[w.pad].ka, ksteps = p.jobs[w.pad].ksteps;
                    const uint32_t jb_atoms = kBf ? 2 * ka : ka;
                    if (!mbar_wait(&bar_a[abuf], aph, err, 3)) break;
                    tc_fence_after();
                    const uint64_t a_desc0 = sw128_desc(a_base + abuf * a_buf_bytes);
                    for (uint32_t n = w.b1 - w.b0; ok && n > 0; --n) {
                        if (!acc_ready && !mbar_wait(&bar_accempty[acc], accph, err, 4)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t dcol = tmem + acc * kTcTileB;
                        uint64_t *bar_full = &bar_accfull[acc];
                        acc ^= 1u;
                        accph ^= acc ^ 1u;
                        uint32_t accumulate = 0;
                        for (uint32_t q = 0; q < jb_atoms; ++q) {
                            if (!b_ready && !mbar_wait(&bar_bfull[s], sph, err, 5)) {
                                ok = false;
                                break;
                            }
                            const uint64_t bdesc = b_desc0 + s * (kBStageBytes / 16);
                            uint64_t *bar_release = &bar_bempty[s];
                            if (++s == p.nst) s = 0, sph ^= 1u;
                            b_ready = mbar_test(&bar_bfull[s], sph);
                            if (q + 1 == jb_atoms) acc_ready = mbar_test(&bar_accempty[acc], accph);
                            // a K step advances both descriptors by 32 bytes (2 in their 16-byte units)
                            if constexpr (!kBf) {
                                const uint64_t adesc = a_desc0 + q * (kAStageBytes / 16);
                                // 4 K steps per atom, fewer in the last (zero columns not multiplied)
                                const uint32_t kk_end = ksteps - 4 * q < 4 ? ksteps - 4 * q : 4;
                                if (kk_end == 4) {
#pragma unroll
                                    for (uint32_t kk = 0; kk < 4; ++kk) {
                                        mma_issue<FORM>(el, dcol, adesc + 2 * kk, bdesc + 2 * kk, idesc, accumulate);
                                        accumulate = 1;
                                    }
                                } else {
#pragma unroll
                                    for (uint32_t kk = 0; kk < 3; ++kk) {
                                        if (kk < kk_end) {
                                            mma_issue<FORM>(el, dcol, adesc + 2 * kk, bdesc + 2 * kk, idesc, accumulate);
                                            accumulate = 1;
                                        }
                                    }
                                }
                            } else {
                                const uint32_t kq = q >> 1;
                                const uint32_t kk_end = ksteps - 4 * kq < 4 ? ksteps - 4 * kq : 4;
                                const uint64_t a_hi = a_desc0 + kq * (kAStageBytes / 16);
                                const uint64_t a_lo = a_desc0 + (ka + kq) * (kAStageBytes / 16);
                                if ((q & 1u) == 0) {  // B_hi atom: A_hi.B_hi + A_lo.B_hi
#pragma unroll
                                    for (uint32_t kk = 0; kk < 4; ++kk) {
                                        if (kk >= kk_end) break;
                                        mma_issue<FORM>(el, dcol, a_hi + 2 * kk, bdesc + 2 * kk, idesc, accumulate);
                                        accumulate = 1;
                                        mma_issue<FORM>(el, dcol, a_lo + 2 * kk, bdesc + 2 * kk, idesc, 1);
                                    }
                                } else {  // B_lo atom: A_hi.B_lo
#pragma unroll
                                    for (uint32_t kk = 0; kk < 4; ++kk)
                                        if (kk < kk_end) mma_issue<FORM>(el, dcol, a_hi + 2 * kk, bdesc + 2 * kk, idesc, 1);
                                }
                            }
                            mma_commit(el, bar_release);  // stage free once these MMAs have read it
                            issued_any = true;
                        }
                        if (!ok) break;
                        mma_commit(el, bar_full);
                    }
                    mma_commit(el, &bar_aempty[abuf]);
                    if (++abuf == p.a_bufs) abuf = 0, aph ^= 1u;
                    w = wn;
                }
                // all MMAs complete before the tensor memory is released
                if (issued_any) {
                    mma_commit(el, &bar_drain);
                    drain_until(&bar_drain, 0, globaltimer_ns() + kWaitLimitNs);
                }
            }
        } else if (!kBf && warp == kFoldWarp && p.fold) {
            // ------------------------------------------------ A side of folded norms
            // A folded row holds the pieces of |x|^2 / 2 in its columns d .. d + 2.
            // As a B operand they meet the A side's constants; here those replace
            // the pieces of the A tile that has landed (once per item, 128 rows of
            // 3 columns), before the MMA warp is told that the tile is ready.
            uint32_t abuf = 0, aph = 0;
            for (uint64_t it = blockIdx.x; it < p.n_items; it += stride) {
                const TcJob &J = p.jobs[p.items[it].pad];
                const bool fold = J.fold != 0;
                const uint32_t d = J.d;
                const bool landed = mbar_wait(&bar_afull[abuf], aph, err, 7);
                if (!__all_sync(0xffffffffu, landed)) break;
                if (fold) {
                    const uint32_t abase = a_base + abuf * a_buf_bytes;
                    for (uint32_t r = lane; r < (uint32_t)kTcTileA; r += 32) {
#pragma unroll
                        for (uint32_t m = 0; m < 3; ++m) {
                            const uint32_t col = d + m, q = col / kAtomElems;
                            const uint32_t byte = (col % kAtomElems) * (kAtomBytes / kAtomElems);
                            const uint32_t off = q * kAStageBytes + r * kAtomBytes + (((byte >> 4) ^ (r & 7u)) << 4) +
                                                 (byte & 15u);
                            if constexpr (FORM == HJ_FORM_TC_TF32) {
                                asm volatile("st.shared.b32 [%0], %1;" ::"r"(abase + off), "r"(0xBF800000u) : "memory");
                            } else {  // -2^15, -2^4, -2^-7
                                const uint16_t c = m == 0 ? 0xF800 : (m == 1 ? 0xCC00 : 0xA000);
                                asm volatile("st.shared.b16 [%0], %1;" ::"r"(abase + off), "h"(c) : "memory");
                            }
                        }
                    }
                    fence_proxy_async();
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar_aready[abuf]);
                if (++abuf == p.a_bufs) abuf = 0, aph ^= 1u;
            }
        } else {
            // ------------------------------------------------ near warps
            // Warp 3, and warp 2 where no job folds its norms: each works off the queues
            // of its share of the epilogue warps. Lane r < kEpiWarps keeps queue r.
            const bool mine = lane < (uint32_t)kEpiWarps && (p.fold || (lane & 1u) == (warp & 1u));
            uint32_t head = 0, slot = 0;  // entries worked off, and the next one's slot
            uint32_t job = 0xffffffffu;
            unsigned long long cnt = 0;
            BandWriter band(p, lane, BC ? kBandChunk : kBandChunkRare);
            auto flush = [&]() {
                const unsigned long long wc = warp_sum_u64(cnt);
                if (lane == 0 && wc) atomicAdd(p.jobs[job].count, wc);
                cnt = 0;
            };
            // Every epilogue warp ends its queue: its own waits are bounded, and it stops
            // at the next one once the error word is set. So the loop ends, however long
            // the join; its own limit, a second line, runs from the first sight of an error.
            uint64_t t_err = 0;
            for (uint32_t idle = 0;;) {
                const uint32_t tail = mine ? lds_acquire(&near_tail[lane]) : kNearDone;
                __syncwarp();  // the acquiring lanes' view becomes the warp's
                const uint32_t avail = mine ? (tail - head) & ~kNearDone : 0u;
                // a batch costs the same for one row and for 32, and its instructions
                // compete with the epilogue's: it waits for rows, or a queue half full
                const uint32_t rows = __reduce_add_sync(0xffffffffu, avail);
                const bool last = __all_sync(0xffffffffu, (tail & kNearDone) != 0);
                if (last && rows == 0) break;
                if (!last && rows < kNearBatch && 2 * __reduce_max_sync(0xffffffffu, avail) < p.near_cap) {
                    if ((++idle & 1023u) == 0 && __any_sync(0xffffffffu, *err != 0)) {
                        const uint64_t now = __shfl_sync(0xffffffffu, globaltimer_ns(), 0);
                        if (t_err == 0) t_err = now;
                        if (now - t_err > p.near_ns) break;
                    }
                    __nanosleep(200);
                    continue;
                }
                // lane i takes row i of the queues in order
                uint32_t my_q = 0, my_i = 0, taken = 0, took = 0;
#pragma unroll
                for (uint32_t r = 0; r < (uint32_t)kEpiWarps; ++r) {
                    const uint32_t have = __shfl_sync(0xffffffffu, avail, r), n = have < 32 - taken ? have : 32 - taken;
                    if (lane >= taken && lane < taken + n) my_q = r, my_i = lane - taken;
                    if (lane == r) took = n;
                    taken += n;
                }
                const bool row = lane < taken;
                uint32_t at = __shfl_sync(0xffffffffu, slot, my_q) + my_i;
                if (at >= p.near_cap) at -= p.near_cap;
                const float *ent = near_base + my_q * near_ring + at * kNearWords;
                float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                uint4 u = make_uint4(0u, 0u, 0u, 0u);
                uint32_t g_in = 0, bbits = 0, ejob = 0;
                if (row) {
                    q = *reinterpret_cast<const float4 *>(ent + 32);
                    u = *reinterpret_cast<const uint4 *>(ent + 36);
                    ejob = u.y;
                    const TcJob &J = p.jobs[ejob];
                    const uint32_t mask = count_mask(__float_as_uint(q.w), u.x, (uint32_t)J.b_end, J.self != 0);
                    const float4 *nrm = reinterpret_cast<const float4 *>(BC || u.z ? nullptr : p.norm_b + u.x);
                    float4 nb[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) nb[k] = nrm ? __ldg(nrm + k) : make_float4(0.f, 0.f, 0.f, 0.f);
                    uint32_t g_out = 0;
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const float4 v = *reinterpret_cast<const float4 *>(ent + 4 * k);
                        const float t[4] = {fmaf(-2.0f, v.x, nb[k].x), fmaf(-2.0f, v.y, nb[k].y),
                                            fmaf(-2.0f, v.z, nb[k].z), fmaf(-2.0f, v.w, nb[k].w)};
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            g_in |= t[j] <= q.y ? 1u << (4 * k + j) : 0u;
                            g_out |= t[j] <= q.z ? 1u << (4 * k + j) : 0u;
                        }
                    }
                    g_in &= mask;
                    bbits = g_out & mask & ~g_in;
                }
                // counts, into the job that every row of the batch belongs to as a rule
                const uint32_t j0 = __shfl_sync(0xffffffffu, ejob, 0);
                if (__all_sync(0xffffffffu, !row || ejob == j0)) {
                    if (j0 != job) {
                        if (job != 0xffffffffu) flush();
                        job = j0;
                    }
                    cnt += __popc(g_in);
                } else if (g_in) {
                    atomicAdd(p.jobs[ejob].count, (unsigned long long)__popc(g_in));
                }
                if (__any_sync(0xffffffffu, bbits != 0)) {
                    const uint32_t nbits = __popc(bbits);
                    uint32_t incl = nbits;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                        if (lane >= (uint32_t)o) incl += y;
                    }
                    const BandSlots sl = band.reserve(__shfl_sync(0xffffffffu, incl, 31));
                    uint32_t rank = incl - nbits;
                    while (bbits) {
                        const int j = __ffs(bbits) - 1;
                        bbits &= bbits - 1;
                        const float w = ent[j];
                        band.store(sl.at(rank++), __float_as_uint(q.w), u.x + j,
                                   BC ? fmaf(-2.0f, w, q.x) * p.jobs[ejob].s_unscale : w, ejob);
                    }
                }
                __syncwarp();  // the rows have been read
                if (took) {
                    head = (head + took) & ~kNearDone;
                    slot = slot + took < p.near_cap ? slot + took : slot + took - p.near_cap;
                    sts_release(&near_head[lane], head);
                }
            }
            if (job != 0xffffffffu) flush();
            band.finish();
        }
    } else {
        // ------------------------------------------------ epilogue
        reg_inc<kEpiRegs>();
        const uint32_t quad = warp & 3u;
        const uint32_t half = (warp - kEpiWarp0) >> 2;  // columns [kEpiCols half, kEpiCols (half + 1))
        const uint32_t lane_base = (quad * 32u) << 16;
        // this warp's near queue: entries queued, the next one's slot, and the entries
        // worked off when last looked at (warp-uniform)
        const uint32_t ew = warp - kEpiWarp0;
        float *near = near_base + ew * near_ring;
        uint32_t n_tail = 0, n_slot = 0, n_head = 0;
        unsigned long long cnt = 0;
        uint32_t acc = 0, accph = 0;
        bool run = true;
        if (p.gate_ns) {  // test hook: a wait that nothing ends
            const uint64_t t0 = globaltimer_ns();
            while (!mbar_try_wait(&bar_gate, 0)) {
                if (globaltimer_ns() - t0 > p.gate_ns) {
                    atomicOr((uint32_t *)err, kErrTimeout | (9u << 8));
                    break;
                }
            }
            run = false;
        }
        // All classification is in FP32 with eps^2 rounded outward (T_lo, T_hi)
        // and the bound rounded up; the FP32 rounding of the epilogue itself is
        // part of c_rel. A pair is inside if s + tau <= T_lo, outside if
        // s - tau > T_hi, and in the band otherwise.
        // Per item: this lane's row (A rank), its norm and the classification
        // thresholds, taken against the largest B-tile norm of the item (a band at
        // least as wide as any tile's: still exact). The next item's rows and the
        // item after it are loaded one item ahead, so that a change of item waits
        // for no memory. Per tile only the group minima are needed on the fast
        // path (none when the norms are folded); they are loaded one tile ahead. B
        // norms and column bounds are read on the slow path.
        WorkItem w = run ? item_at(blockIdx.x) : WorkItem{0, 0, 0, 0};
        WorkItem wn = item_at(blockIdx.x + stride), wnn = item_at(blockIdx.x + 2 * stride);
        // per-block centring: the row's p, |h| and |p|, its block's |c| and centre
        // coordinates (lane, lane + 32), the job's eps^2 bounds; per tile the B
        // block's summary and centre, prefetched one tile ahead with the minima
        float p_row = 0.f, xa = 0.f, pa = 0.f, cna = 0.f, t_lo = 0.f, t_hi = 0.f;
        float ca[2] = {0.f, 0.f}, pf_cb[2] = {0.f, 0.f};
        float4 pf_blk = make_float4(0.f, 0.f, 0.f, 0.f);
        bool fold = false;  // the current item's column norms are in the accumulator
        // block centring: the B block of the kEpiCols columns from rank g
        auto prefetch = [&](uint32_t g) {
            if constexpr (BC) {
                const uint32_t blkb = g / kBcBlock;
                pf_blk = __ldg(p.blk_b + blkb);
                pf_cb[0] = __ldg(p.cent_b + blkb * kBcCentStride + lane);
                pf_cb[1] = __ldg(p.cent_b + blkb * kBcCentStride + 32 + lane);
            }
        };
        // one centre: the group minima of the warp's columns in tile b + lane (a load
        // per 32 tiles; a tile's four are read from its lane)
        auto load_gmin = [&](uint32_t b, uint32_t b1) {
            return b + lane < b1
                       ? __ldg(reinterpret_cast<const float4 *>(p.gmin_b + (b + lane) * (kTcTileB / 32) + half * (kEpiCols / 32)))
                       : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        // an item's row data, loaded one item ahead (norm arrays cover the padded ranks)
        struct Rows {
            float n, x, c0, c1, cn;
            float4 gmin;
        };
        auto load_rows = [&](const WorkItem &ww) {
            Rows r;
            const uint64_t g = (uint64_t)ww.a * kTcTileA + quad * 32 + lane;
            r.n = __ldg(p.norm_a + g);
            if constexpr (BC) {
                r.x = __ldg(p.xn_a + g);
                const uint64_t blka = (uint64_t)ww.a * kTcTileA / kBcBlock;
                r.cn = __ldg(&p.blk_a[blka].y);
                r.c0 = __ldg(p.cent_a + blka * kBcCentStride + lane);
                r.c1 = __ldg(p.cent_a + blka * kBcCentStride + 32 + lane);
            } else {
                // the largest B-tile norm of the item: this lane's share
                r.x = 0.f;
                for (uint32_t b = ww.b0 + lane; b < ww.b1; b += 32) r.x = fmaxf(r.x, __ldg(p.tmax_b + b));
                r.cn = r.c0 = r.c1 = 0.f;
                r.gmin = load_gmin(ww.b0, ww.b1);
            }
            return r;
        };
        // per-item row state, and the job whose count the warp is accumulating
        uint32_t gi = 0, b_end = 0;  // ranks are below 2^31
        bool row_ok = false, self = false;
        float na = kPadNorm, thr_out = -3.0e38f, thr_in = -3.0e38f, s_unscale = 1.f;
        uint32_t job = 0xffffffffu;
        BandWriter band(p, lane, BC ? kBandChunk : kBandChunkRare);
        auto flush = [&]() {
            const unsigned long long wc = warp_sum_u64(cnt);
            if (lane == 0 && wc) atomicAdd(p.jobs[job].count, wc);
            cnt = 0;
        };
        auto item_rows = [&](const WorkItem &ww, const Rows &r) {
            if (ww.pad != job) {
                if (job != 0xffffffffu) flush();
                job = ww.pad;
            }
            const TcJob &J = p.jobs[job];
            const float T_lo = J.T_lo, T_hi = J.T_hi, crel = J.c_rel_f, cabs = J.c_abs_f;
            b_end = (uint32_t)J.b_end;
            self = J.self != 0;
            s_unscale = J.s_unscale;
            gi = ww.a * kTcTileA + quad * 32 + lane;
            row_ok = gi >= J.a_row0 && gi < J.a_end;
            if constexpr (BC) {
                // thresholds per tile (they depend on the B block): see the tile loop
                p_row = row_ok ? r.n : 0.f;
                xa = row_ok ? r.x : 0.f;
                pa = fabsf(p_row);
                cna = r.cn;
                ca[0] = r.c0;
                ca[1] = r.c1;
                t_lo = T_lo;
                t_hi = T_hi;
                na = p_row;
                thr_out = thr_in = -3.0e38f;
                (void)crel;
                (void)cabs;
                return;
            }
            fold = J.fold != 0;
            na = row_ok ? r.n : kPadNorm;
            float tmaxb = r.x;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) tmaxb = fmaxf(tmaxb, __shfl_xor_sync(0xffffffffu, tmaxb, o));
            // With tau_max = c_rel (|a|^2 + max |b|^2) + c_abs >= tau of every pair
            // of the item, and t_j = |b_j|^2 - 2 v_j, s_j = |a|^2 + t_j:
            //   t_j <= thr_in  => s_j + tau <= eps^2  (certainly inside),
            //   t_j >  thr_out => s_j - tau >  eps^2  (certainly outside),
            // anything between is a band pair. Both thresholds carry margins
            // for their own FP32 rounding (rounded inward / outward). With folded
            // norms the accumulator holds w_j = v_j - |b_j|^2 / 2 and t_j = -2 w_j.
            const float tau_max = fmaf(crel, na + tmaxb, cabs) * 1.001f;
            const float marg = 8.0f * 5.9604645e-8f * (fabsf(T_hi) + fabsf(na) + tmaxb + tau_max);
            thr_out = (T_hi + tau_max) - na + marg;
            thr_in = (T_lo - tau_max) - na - marg;
            if (!row_ok) thr_out = thr_in = -3.0e38f;
        };
        // Band entries of a lane's row: the columns `bbits` of the 32 from rank gj, whose
        // values are v. Ranks by a warp prefix sum, slots from one warp-wide reservation.
        // The error statistic reads the estimates: with one centre the pair's value is
        // kept, and the recheck forms the estimate from it. With block centres the value
        // alone would not do, and keeping the estimate took 2M x 28 clustered from 7.3 to
        // 8.1 ms: NaN there.
        auto put_band_bits = [&](const float *v, uint32_t bbits, uint32_t gj) {
            if (!__any_sync(0xffffffffu, bbits != 0)) return;
            const uint32_t nbits = __popc(bbits);
            uint32_t incl = nbits;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= (uint32_t)o) incl += y;
            }
            const BandSlots sl = band.reserve(__shfl_sync(0xffffffffu, incl, 31));
            uint32_t rank = incl - nbits;
            while (bbits) {
                const int j = __ffs(bbits) - 1;
                bbits &= bbits - 1;
                band.store(sl.at(rank++), gi, gj + j, BC ? __int_as_float(0x7fc00000) : pick32(v, j), job);
            }
        };
        // Groups of 32 columns in which many rows are near: every lane classifies its
        // own row from its registers. With one centre, where hardly any of the rows has
        // band pairs, those rows are left to the queue (the rows returned), which is
        // cheaper than picking the values by their column. Values dropped -> all picked
        // -> this: 200k x 20 3.20 -> 3.31 -> 3.24 ms, 150k x 8 0.635 -> 0.678 -> 0.656,
        // 150k x 4 0.193 -> 0.225 -> 0.229, 20k x 32 with eps at the median 0.180 -> 0.193
        // -> 0.200. With up to 4 or 6 rows left to the queue the last two take 0.25 and
        // 0.22, and 0.26 and 0.35.
        auto dense_rows = [&](const float *v, bool need, uint32_t gj) -> uint32_t {
            const uint32_t colmask = need && row_ok ? count_mask(gi, gj, b_end, self) : 0u;
            uint32_t g_in = 0, g_out = 0;
            if (BC || fold) {
                // t = -2 w, so t <= thr  <=>  w >= -thr / 2 (exact scaling)
                const float w_in = -0.5f * thr_in, w_out = -0.5f * thr_out;
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    g_in |= v[j] >= w_in ? (1u << j) : 0u;
                    g_out |= v[j] >= w_out ? (1u << j) : 0u;
                }
            } else {
                const float4 *nrm = reinterpret_cast<const float4 *>(p.norm_b + gj);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const float4 nb = __ldg(nrm + k);
                    const float t[4] = {fmaf(-2.0f, v[4 * k], nb.x), fmaf(-2.0f, v[4 * k + 1], nb.y),
                                        fmaf(-2.0f, v[4 * k + 2], nb.z), fmaf(-2.0f, v[4 * k + 3], nb.w)};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        g_in |= t[j] <= thr_in ? (1u << (4 * k + j)) : 0u;
                        g_out |= t[j] <= thr_out ? (1u << (4 * k + j)) : 0u;
                    }
                }
            }
            g_in &= colmask;
            const uint32_t bbits = g_out & colmask & ~g_in;
            if constexpr (!BC) {
                const uint32_t rows = __ballot_sync(0xffffffffu, bbits != 0);
                if (__popc(rows) <= p.near_rows) {
                    cnt += bbits ? 0 : __popc(g_in);
                    return rows;
                }
            }
            cnt += __popc(g_in);
            put_band_bits(v, bbits, gj);
            return 0;
        };
        // waits until the near queue has room for a row; false: the error word is set
        auto wait_room = [&]() -> bool {
            const uint64_t t0 = globaltimer_ns();
            for (uint32_t i = 1;; ++i) {
                n_head = __shfl_sync(0xffffffffu, lds_acquire(&near_head[ew]), 0);
                if (((n_tail - n_head) & ~kNearDone) < p.near_cap) return true;
                if ((i & 255u) == 0) {
                    const bool late = globaltimer_ns() - t0 > kWaitLimitNs;
                    if (__any_sync(0xffffffffu, *err != 0 || late)) {
                        if (lane == 0 && *err == 0) atomicOr((uint32_t *)err, kErrTimeout | (8u << 8));
                        return false;
                    }
                }
            }
        };
        auto put_row = [&](const float *v, uint32_t rank, uint32_t gj) {
            const uint32_t at = n_slot + rank < p.near_cap ? n_slot + rank : n_slot + rank - p.near_cap;
            float4 *ent = reinterpret_cast<float4 *>(near + at * kNearWords);
#pragma unroll
            for (int q = 0; q < 8; ++q) ent[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
            ent[8] = make_float4(na, thr_in, thr_out, __uint_as_float(gi));
            *reinterpret_cast<uint4 *>(ent + 9) = make_uint4(gj, job, BC || fold ? 1u : 0u, 0u);
        };
        auto publish = [&](uint32_t k) {
            n_slot = n_slot + k < p.near_cap ? n_slot + k : n_slot + k - p.near_cap;
            n_tail = (n_tail + k) & ~kNearDone;
            __syncwarp();
            if (lane == 0) sts_release(&near_tail[ew], n_tail);
        };
        // The near rows of a chunk's two groups (bits of r0, r1; the columns from rank
        // gj, their values in v) into the near queue.
        auto queue_rows = [&](const float *v, uint32_t r0, uint32_t r1, uint32_t gj) {
            const uint32_t lt = (1u << lane) - 1u, k0 = __popc(r0), k = k0 + __popc(r1);
            if (((n_tail + k - n_head) & ~kNearDone) > p.near_cap)
                n_head = __shfl_sync(0xffffffffu, lds_acquire(&near_head[ew]), 0);
            if (((n_tail + k - n_head) & ~kNearDone) <= p.near_cap) {
                if ((r0 >> lane) & 1u) put_row(v, __popc(r0 & lt), gj);
                if ((r1 >> lane) & 1u) put_row(v + 32, k0 + __popc(r1 & lt), gj + 32);
                publish(k);
                return;
            }
            // no room for all of them: one by one
            while (r0 | r1) {
                if (!wait_room()) return;  // (the count is void)
                const uint32_t first = r0 ? r0 & (0u - r0) : r1 & (0u - r1);
                if (r0) {
                    if ((first >> lane) & 1u) put_row(v, 0, gj);
                    r0 ^= first;
                } else {
                    if ((first >> lane) & 1u) put_row(v + 32, 0, gj + 32);
                    r1 ^= first;
                }
                publish(1);
            }
        };
        Rows rn{};
        if (w.b0 < w.b1) {
            rn = load_rows(w);
            prefetch(w.b0 * kTcTileB + half * kEpiCols);
        }
        for (uint64_t it = blockIdx.x; run && it < p.n_items; it += stride) {
            item_rows(w, rn);
            float4 gmin32 = rn.gmin;
            const bool more = it + stride < p.n_items;
            if (more) rn = load_rows(wn);
            // rows that are not counted compare false (NaN); testing hook: every pair
            // is estimated
            const float thr_none = __int_as_float(0x7fc00000);
            float thr_fast = !row_ok ? thr_none : (p.dbg != nullptr ? 3.0e38f : thr_out);
            uint32_t gj = w.b0 * kTcTileB + half * kEpiCols;
            const uint32_t gj_end = w.b1 * kTcTileB;
            // after the item's last tile, the next item's first (prefetch)
            const uint32_t gj_next = more ? wn.b0 * kTcTileB + half * kEpiCols : gj;
            for (; gj < gj_end; gj += kTcTileB) {
                if constexpr (BC) {
                    // the half's B block: D = |c_A - c_B|^2 (FP32, lanes over the
                    // dims), the band half-width of the lane's row against the block,
                    // and the thresholds on t = -2 w (s = q_row + D + t; |w| <= S)
                    float D = 0.f;
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        const float df = ca[m] - pf_cb[m];
                        D = fmaf(df, df, D);
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) D += __shfl_xor_sync(0xffffffffu, D, o);
                    float S;
                    const float tau = bc_tau(xa, cna, pa, pf_blk.x, pf_blk.y, pf_blk.z, D, p.bc, &S);
                    const float marg = 8.0f * 5.9604645e-8f * (fabsf(t_hi) + pa + pf_blk.z + D + tau + 2.0f * S);
                    na = p_row + D;
                    thr_out = row_ok ? (t_hi + tau) - p_row - D + marg : -3.0e38f;
                    thr_in = row_ok ? (t_lo - tau) - p_row - D - marg : -3.0e38f;
                    thr_fast = !row_ok ? thr_none : (p.dbg != nullptr ? 3.0e38f : thr_out);
                    prefetch(gj + kTcTileB < gj_end ? gj + kTcTileB : gj_next);
                }
                float gmin[4] = {0.f, 0.f, 0.f, 0.f};
                if (!BC && !fold) {
                    const uint32_t k = (gj / kTcTileB - w.b0) & 31u;
                    if (k == 0 && gj / kTcTileB != w.b0) gmin32 = load_gmin(gj / kTcTileB, w.b1);
                    gmin[0] = __shfl_sync(0xffffffffu, gmin32.x, k), gmin[1] = __shfl_sync(0xffffffffu, gmin32.y, k);
                    gmin[2] = __shfl_sync(0xffffffffu, gmin32.z, k), gmin[3] = __shfl_sync(0xffffffffu, gmin32.w, k);
                }
                if (!mbar_wait(&bar_accfull[acc], accph, err, 6)) {
                    run = false;
                    break;
                }
                tc_fence_after();
                // The warp's columns in two chunks. With two accumulators a tile's period
                // is half the chain MMA -> commit -> load -> release -> MMA, so the
                // accumulator goes back as soon as the second chunk is in registers,
                // before it is reduced.
                const uint32_t taddr = tmem + lane_base + acc * kTcTileB + half * kEpiCols;
#pragma unroll 1
                for (uint32_t c = 0; c < (uint32_t)kEpiCols; c += kChunkCols) {
                    float v[kChunkCols];
                    tmem_ld(taddr + c, v);
                    tmem_wait(v);
                    if (c) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&bar_accempty[acc]);
                    }
                    // min_j (|b_j|^2 - 2 v_j) >= gmin - 2 max_j v_j per 32-column group, gmin
                    // the group's minimum norm (0 where the norms are in the accumulator:
                    // exact); a vote per group, both taken before any branch
                    const float m0 = fmaf(-2.0f, max32(v), c ? gmin[2] : gmin[0]);
                    const float m1 = fmaf(-2.0f, max32(v + 32), c ? gmin[3] : gmin[1]);
                    const uint32_t r0 = __ballot_sync(0xffffffffu, m0 <= thr_fast);
                    const uint32_t r1 = __ballot_sync(0xffffffffu, m1 <= thr_fast);
                    if ((r0 | r1) == 0) continue;
                    // groups of a few near rows go to the queue
                    const bool dense0 = __popc(r0) > p.near_rows, dense1 = __popc(r1) > p.near_rows;
                    const uint32_t q0 = dense0 ? dense_rows(v, (r0 >> lane) & 1u, gj + c) : r0;
                    const uint32_t q1 = dense1 ? dense_rows(v + 32, (r1 >> lane) & 1u, gj + c + 32) : r1;
                    if (q0 | q1) queue_rows(v, q0, q1, gj + c);
                    if (p.dbg != nullptr && gi < p.na) {  // testing hook: every estimate
#pragma unroll
                        for (int j = 0; j < kChunkCols; ++j)
                            if (gj + c + j < p.nb)
                                p.dbg[(uint64_t)p.perm_a[gi] * p.nb + p.perm_b[gj + c + j]] =
                                    (na + fmaf(-2.0f, v[j], BC || fold ? 0.f : p.norm_b[gj + c + j])) * s_unscale;
                    }
                }
                acc ^= 1u;
                accph ^= acc ^ 1u;
            }
            w = wn;
            wn = wnn;
            wnn = item_at(it + 3 * stride);
        }
        if (job != 0xffffffffu) flush();
        band.finish();
        __syncwarp();
        if (lane == 0) sts_release(&near_tail[ew], n_tail | kNearDone);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, kTmemCols);

}

// ---------------------------------------------------------------- recheck

// FP64 pair test (the oracle's) on every band pair, against the pair's job
// (BandEntry.pad); also the largest |estimate - dist2| seen, as FP32 bits in
// max_err_bits. norm_a, norm_b: the squared norms per rank with one centre, whose
// entries hold accumulator values (the column norm is in those of folded jobs); null
// with block centres.
// 16-byte loads of both rows where the rows allow it (every job's d * sizeof(TIn)
// a multiple of 16: `vec`); the FP64 sum runs over the dims in order either way.
template <typename TIn>
__device__ __forceinline__ double pair_dist2(const TIn *a, const TIn *b, uint32_t d, bool vec) {
    double acc = 0.0;
    if (vec) {
        constexpr uint32_t V = 16 / sizeof(TIn);
        using Vec = typename std::conditional<sizeof(TIn) == 4, float4, double2>::type;
        const Vec *av = reinterpret_cast<const Vec *>(a), *bv = reinterpret_cast<const Vec *>(b);
        for (uint32_t k = 0; k < d / V; ++k) {
            const Vec x = __ldg(av + k), y = __ldg(bv + k);
            TIn xs[V], ys[V];
            memcpy(xs, &x, 16);
            memcpy(ys, &y, 16);
#pragma unroll
            for (uint32_t j = 0; j < V; ++j) {
                const double df = __dsub_rn((double)xs[j], (double)ys[j]);
                acc = __fma_rn(df, df, acc);
            }
        }
        return acc;
    }
    for (uint32_t k = 0; k < d; ++k) {
        const double df = __dsub_rn((double)a[k], (double)b[k]);
        acc = __fma_rn(df, df, acc);
    }
    return acc;
}

template <typename TIn>
__global__ void k_recheck(const TcJob *__restrict__ jobs, const BandEntry *__restrict__ band,
                          const unsigned long long *band_total, uint64_t cap, unsigned int *max_err_bits, bool vec,
                          const float *__restrict__ norm_a, const float *__restrict__ norm_b) {
    const uint64_t n = min((unsigned long long)cap, *band_total);
    const uint32_t lane = threadIdx.x & 31u;
    float emax = 0.f;
    // counts accumulate per thread while its entries stay in one job (a launch of
    // one join: always), flushed when the job changes and once at the end
    unsigned long long c_acc = 0;
    uint32_t cur = 0xffffffffu;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const BandEntry e = band[i];
        if (e.ia == kBandHole) continue;  // a slot reserved and left unused
        const TcJob &J = jobs[e.pad];
        const TIn *a = static_cast<const TIn *>(J.rows_a) + (uint64_t)(e.ia - J.a_row0) * J.d;
        const TIn *b = static_cast<const TIn *>(J.rows_b) + (uint64_t)(e.jb - J.b_row0) * J.d;
        const double acc = pair_dist2(a, b, J.d, vec);
        if (e.pad != cur) {
            if (c_acc) atomicAdd(jobs[cur].count, c_acc);
            cur = e.pad;
            c_acc = 0;
        }
        c_acc += acc <= J.T ? 1ull : 0ull;
        float s = e.s_hat;
        if (norm_a) s = (__ldg(norm_a + e.ia) + fmaf(-2.0f, s, J.fold ? 0.f : __ldg(norm_b + e.jb))) * J.s_unscale;
        emax = fmaxf(emax, (float)fabs((double)s - acc));  // NaN estimates (not kept) are skipped
    }
    // one atomic per warp when the warp's lanes end in the same job (the usual case)
    const uint32_t j0 = __shfl_sync(0xffffffffu, cur, 0);
    if (__all_sync(0xffffffffu, cur == j0 || c_acc == 0)) {
        const unsigned long long c = warp_sum_u64(c_acc);
        if (lane == 0 && c) atomicAdd(jobs[j0].count, c);
    } else if (c_acc) {
        atomicAdd(jobs[cur].count, c_acc);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) emax = fmaxf(emax, __shfl_xor_sync(0xffffffffu, emax, o));
    if (lane == 0) atomicMax(max_err_bits, __float_as_uint(emax));
}

// ---------------------------------------------------------------- host side

// Error bound of the tensor-core estimate s = |a|^2 + |b|^2 - 2 v against the
// FP64 pair test, |s - dist2| <= c_rel (|a|^2 + |b|^2) + c_abs, built from:
//   operand rounding (TF32: 2 * 2^-11 relative per product; BF16 split:
//   a = a_hi + a_lo + r with |r| <= 2^-16 |a|, dropped a_lo b_lo and r terms
//   <= 3.1 * 2^-16 |a_k b_k|), FP32 rounding of FP64 inputs (2 * 2^-24),
//   tensor-core FP32 accumulation budgeted at 2^-22 of S = sum |a_k b_k| per
//   product term (K terms TF32, 3K BF16). The budget follows the model that
//   Fasi, Higham, Mikaitis and Pranesh (Numerical behavior of NVIDIA tensor
//   cores, PeerJ Computer Science 7:e330, 2021) measured for earlier tensor
//   cores: each hardware step adds k products (exact) to the accumulator after
//   aligning all k + 1 terms to the largest exponent and truncating them to
//   FP32's 24 bits, then truncates the sum to FP32. Each truncation loses less
//   than 2^-23 of the largest term, which is at most S, so a step loses less
//   than (k + 2) 2^-23 S and the K / k steps less than K (1 + 2/k) 2^-23 S,
//   within K 2^-22 S for every k >= 2. tests/test_gpu_tc.py checks the whole
//   bound on adversarial cancellation at K = 256 (running sums far above the
//   result) for every form. |a.b| <= sum |a_k b_k| <=
//   (|a|^2 + |b|^2) / 2 (Cauchy-Schwarz, AM-GM) -- the dot error enters s
//   twice; FP32 norms (2^-24 each) and the FP32 epilogue (three roundings of
//   values up to 2 (|a|^2 + |b|^2), 6 * 2^-24, budgeted 10 * 2^-24); the FP64
//   direct difference's own rounding (d * 2^-50).
// A margin factor 1.25 covers the bookkeeping in between. c_abs covers
// subnormal operands (TF32/BF16 keep the FP32 exponent range; values below
// 2^-100 times the largest coordinate are the only ones that can lose
// relative accuracy) and is negligible for data of ordinary scale.
//
// FP16 (in units scaled by op_scale^2, where the largest centred coordinate
// is below 2^15): operands rounded once from FP64, 2^-11 relative each, so
// products as TF32's; FP16 subnormals (|v| < 2^-14) carry an absolute error up
// to 2^-25 instead, at most 2 * 2^-25 * 2^15 per product term, d terms, twice
// in s: c_abs = 1.25 * d * 2^-8.
//
// Folded norms (tc_fold): the accumulator sums the products and the pieces of
// -|b|^2 / 2, so its terms sum to at most (|a|^2 + |b|^2) / 2 + |b|^2 / 2, within
// twice the dot product's: the accumulation budget doubles, over K = d + 3
// columns. The split of the norm is off by 2^-33 |b|^2 + 2^-32, far inside the
// FP32 rounding of |b|^2 that it replaces; its absolute part (2^-31 in s) joins
// c_abs. FP16 coordinates are below 2^10 there: subnormals cost 2 * 2^-25 *
// 2^10 per product term, d terms, twice: c_abs = 1.25 * (d * 2^-13 + 2^-31).
void tc_band_constants(int form, uint32_t d, double maxabs, bool fold, double *c_rel, double *c_abs) {
    const double u24 = std::ldexp(1.0, -24), acc = std::ldexp(1.0, -22);
    // product terms summed (zero columns are not multiplied)
    const double kpad = fold ? 2.0 * (double)tc_kterms(form, d + 3) : (double)tc_kterms(form, d);
    double dot;
    if (form == HJ_FORM_TC_TF32 || form == HJ_FORM_TC_FP16) {
        const double u = std::ldexp(1.0, -11);
        dot = 2 * u + u * u + 2 * u24 + kpad * acc;
    } else {
        dot = 3.1 * std::ldexp(1.0, -16) + 2 * u24 + 3 * kpad * acc;
    }
    *c_rel = 1.25 * (dot + 12 * u24 + (double)d * std::ldexp(1.0, -50));
    if (form == HJ_FORM_TC_FP16)
        *c_abs = fold ? 1.25 * ((double)d * std::ldexp(1.0, -13) + std::ldexp(1.0, -31))
                      : 1.25 * (double)d * std::ldexp(1.0, -8);
    else
        *c_abs = 1e-30 + 4.0 * (double)d * std::ldexp(std::fmax(maxabs, 1e-30), -100) * std::fmax(maxabs, 1.0);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn(std::string *err) {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
        else
            cudaGetLastError();
    });
    if (!fn) *err = "cuTensorMapEncodeTiled unavailable";
    return fn;
}

// 2D map over a row-major [rows][kp] matrix, box = one 128-byte K atom x box_rows.
static bool make_map(CUtensorMap *m, const void *base, CUtensorMapDataType type, uint64_t rows, uint32_t kp,
                     uint32_t box_rows, std::string *err) {
    EncodeTiledFn fn = encode_fn(err);
    if (!fn) return false;
    const uint32_t esz = type == CU_TENSOR_MAP_DATA_TYPE_FLOAT32 ? 4 : 2;
    cuuint64_t gdim[2] = {kp, rows};
    cuuint64_t gstride[1] = {(cuuint64_t)kp * esz};
    cuuint32_t box[2] = {kAtomBytes / esz, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(m, type, 2,
                    const_cast<void *>(base), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        *err = "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")";
        return false;
    }
    return true;
}

struct TcLayout {
    uint32_t ka, a_bufs, nst, near_cap;
    size_t smem;
};

constexpr int kTcSmemMax = 225 * 1024 + kEpiWarps * kNearWords * 4;  // 224 KB + 1 KB + one near entry per warp
static TcLayout tc_layout(int form, uint32_t d) {
    TcLayout L;
    L.ka = form == HJ_FORM_TC_TF32 ? (d + 31) / 32 : (d + 63) / 64;
    const uint32_t a_atoms = form == HJ_FORM_TC_BF16X3 ? 2 * L.ka : L.ka;
    const size_t a_bytes = (size_t)a_atoms * kAStageBytes;
    // + 1 KB alignment and 0.3 KB static <= 227 KB per block
    const size_t budget = 224 * 1024;
    const size_t near_entry = (size_t)kEpiWarps * kNearWords * 4;
    // the near queues take the place of a B stage where three stages remain, or of
    // the second A buffer (an item's tiles then wait for its A tile) where four do
    L.a_bufs = 2 * a_bytes + 3 * kBStageBytes + kNearMinCap * near_entry <= budget ? 2 : 1;
    const size_t left = budget - L.a_bufs * a_bytes;
    L.nst = (uint32_t)(left / kBStageBytes);
    if (L.nst > 8) L.nst = 8;
    if (left - (size_t)L.nst * kBStageBytes < kNearMinCap * near_entry && L.nst > 3) --L.nst;
    const size_t cap = (left - (size_t)L.nst * kBStageBytes) / near_entry;
    L.near_cap = (uint32_t)(cap < 1 ? 1 : (cap < kNearCap ? cap : kNearCap));
    L.smem = L.a_bufs * a_bytes + (size_t)L.nst * kBStageBytes + L.near_cap * near_entry + 1024;
    return L;
}

bool tc_fold(int form, uint32_t d) {
    return form != HJ_FORM_TC_BF16X3 && tc_layout(form, d + 3).ka == tc_layout(form, d).ka;
}
uint32_t tc_atoms(int form, uint32_t kcols) { return tc_layout(form, kcols).ka; }
uint32_t tc_ksteps(int form, uint32_t kcols) {
    const uint32_t k = form == HJ_FORM_TC_TF32 ? 8u : 16u;
    return (kcols + k - 1) / k;
}
uint32_t tc_kterms(int form, uint32_t kcols) { return tc_ksteps(form, kcols) * (form == HJ_FORM_TC_TF32 ? 8u : 16u); }

// Per-block centring constants (operand units, FP16 form):
//   kp21: the accumulation model above, K = 3d + 3 rounded up to the MMA's 16
//     (the product terms summed) of magnitude sum <= S per dot, the dot
//     entering s twice: 2 K 2^-22;
//   rho_u: |fl16(h) - h| <= 2^-11 |h| per coordinate (normal range), with
//     |h| <= |fl16(h)| (1 + 2^-10): 1.001 * 2^-11 per unit of the stored |h|;
//   rho_c: subnormal FP16 (|h| < 2^-14) is off by at most 2^-25 per
//     coordinate, and the FP64 shift (x - center) * scale by 2^-52 of 2^15:
//     sqrt(d) (2^-25 + 2^-37), doubled;
//   u_norm: q rounded once from FP64 to FP32 (2^-24 relative), doubled, and
//     the split of q / 2 into FP16 pieces (2^-34 relative);
//   u_d: D in FP32, two FMAs per lane and a five-step sum of the lanes, with
//     the differences of FP16 values exact or rounded once: 16 * 2^-24;
//   theta_t: the FP64 pair test sums d squares of exact differences with FMAs,
//     relative error below (d + 2) 2^-53 of dist2 ~ eps^2: 2 (d + 2) 2^-53 T.
BcConsts bc_constants(int form, uint32_t d, double T, double op_scale) {
    // BF16x3: three MMAs per K step. A BF16 value has 8 significant bits, so
    // |lo| <= 2^-8 |v| and the dropped lo.lo products stay below 2^-16 S
    // (1.001 covers S being taken over the stored hi + lo), doubled for s.
    const double s2 = op_scale * op_scale,
                 kpad = (double)tc_kterms(form, bc_cols(d, form)) * (form == HJ_FORM_TC_BF16X3 ? 3.0 : 1.0);
    auto up = [](double v) {
        const float f = (float)v;
        return (double)f >= v ? f : std::nextafter(f, INFINITY);
    };
    BcConsts k;
    k.kp21 = up(2.0 * kpad * std::ldexp(1.0, -22) +
                (form == HJ_FORM_TC_BF16X3 ? 2.0 * 1.001 * std::ldexp(1.0, -16) : 0.0));
    k.eps = up(std::sqrt(T * s2) * (1.0 + 1e-12));
    // FP16 / TF32 round once to 11 significant bits; the BF16 hi + lo pair keeps v
    // to 2^-17 (hi to 2^-8 |v|, and lo to half a unit of the last of its 8 bits)
    k.rho_u = up(1.001 * std::ldexp(1.0, form == HJ_FORM_TC_BF16X3 ? -17 : -11));
    // the subnormal spacing of the operand type (half of it per rounding: FP16
    // 2^-25, BF16 2^-134, TF32 2^-150, taken as 2^-140) and the FP64 shift of
    // coordinates below 2^10 (2^-52 of 2^10, generously 2^-37)
    const double sub = form == HJ_FORM_TC_FP16     ? std::ldexp(1.0, -25)
                       : form == HJ_FORM_TC_BF16X3 ? std::ldexp(1.0, -134)
                                                   : std::ldexp(1.0, -140);
    const double floor_abs = sub + std::ldexp(1.0, -37);
    k.rho_c = up(2.0 * std::sqrt((double)d) * floor_abs);
    k.u_norm = up(std::ldexp(1.0, -23) + std::ldexp(1.0, -33));
    k.u_d = up(16.0 * std::ldexp(1.0, -24));
    // + the absolute floor of the q / 2 split (2^-32 in w, 2^-31 in s, twice in tau)
    k.theta_t = up(2.0 * (d + 2.0) * std::ldexp(1.0, -53) * T * s2 + std::ldexp(1.0, -29));
    return k;
}

static float *g_dbg_out = nullptr;  // set by tests through hj_debug_tc_estimates
static uint64_t g_gate_ns = 0;      // set by tests through hj_debug_set_wait_gate
static uint64_t g_near_ns = kWaitLimitNs;  // set by tests through hj_debug_set_near_limit

void fill_tc_job(TcJob *j, int form, uint32_t d, double T, double op_scale, double maxabs, uint64_t a_row0,
                 uint64_t na_eff, uint64_t b_row0, uint64_t nb_eff, bool self, unsigned long long *count,
                 const void *rows_a, const void *rows_b, bool fold, double *c_rel_out, double *c_abs_out) {
    double c_rel = 0, c_abs = 0;
    tc_band_constants(form, d, maxabs, fold, &c_rel, &c_abs);
    const double s2 = op_scale * op_scale;  // FP16: the units of the norms; 1 otherwise
    const double T_tc = T * s2;
    memset(j, 0, sizeof(*j));
    j->a_row0 = a_row0;
    j->a_end = a_row0 + na_eff;
    j->b_row0 = b_row0;
    j->b_end = b_row0 + nb_eff;
    j->T = T;
    j->count = count;
    j->rows_a = rows_a;
    j->rows_b = rows_b;
    const float t = (float)T_tc;  // outward rounding of eps^2 and upward rounding of the bound
    j->T_lo = (double)t <= T_tc ? t : std::nextafter(t, -INFINITY);
    j->T_hi = (double)t >= T_tc ? t : std::nextafter(t, INFINITY);
    const float cr = (float)c_rel, ca = (float)c_abs;
    j->c_rel_f = (double)cr >= c_rel ? cr : std::nextafter(cr, INFINITY);
    j->c_abs_f = (double)ca >= c_abs ? ca : std::nextafter(ca, INFINITY);
    j->s_unscale = (float)(1.0 / s2);  // a power of two: exact
    j->self = self ? 1u : 0u;
    j->ka = tc_layout(form, d).ka;
    j->ksteps = tc_ksteps(form, fold ? d + 3 : d);
    j->d = d;
    j->fold = fold ? 1u : 0u;
    if (c_rel_out) *c_rel_out = c_rel;
    if (c_abs_out) *c_abs_out = c_abs;
}

int launch_join_tc(const SortedSet &A, const SortedSet &B, int form, const TcJob *d_jobs, uint64_t na0, uint64_t nb0,
                   const IndexResult &idx, uint2 *band, uint64_t band_cap, unsigned long long *d_band_total,
                   uint32_t *d_err, int num_sms, cudaStream_t st, std::string *err, const BcConsts *bc,
                   unsigned long long *d_band_holes) {
    if (idx.n_items == 0) return 0;
    if (bc && (A.d > kBcMaxDim || !A.bc_op || !B.bc_op || A.bc_dp != B.bc_dp || A.bc_form != form ||
               B.bc_form != form || (form == HJ_FORM_TC_BF16X3 && (!A.bc_op_lo || !B.bc_op_lo)))) {
        *err = "per-block centring needs d <= 64 and the centred layouts of the form";
        return 1;
    }
    const TcLayout L = tc_layout(form, bc ? bc_cols(A.d, form) : A.d);
    if (L.nst < 2) {
        *err = "dimension too large for the tensor-core kernel";
        return 1;
    }
    CUtensorMap ma, ma2, mb, mb2;
    if (bc) {
        // rows of 4 dp columns; A reads the window from column dp (the producer's
        // x offset), B from column 0; past the row end the copy fills zeros
        const CUtensorMapDataType ty = form == HJ_FORM_TC_TF32    ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                       : form == HJ_FORM_TC_BF16X3 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                                                   : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
        if (!make_map(&ma, A.bc_op, ty, A.npad_tc, 4 * A.bc_dp, kTcTileA, err)) return 1;
        if (!make_map(&mb, B.bc_op, ty, B.npad_tc, 4 * B.bc_dp, kTcTileB, err)) return 1;
        ma2 = ma;
        mb2 = mb;
        if (form == HJ_FORM_TC_BF16X3) {
            if (!make_map(&ma2, A.bc_op_lo, ty, A.npad_tc, 4 * A.bc_dp, kTcTileA, err)) return 1;
            if (!make_map(&mb2, B.bc_op_lo, ty, B.npad_tc, 4 * B.bc_dp, kTcTileB, err)) return 1;
        }
    } else if (form == HJ_FORM_TC_TF32) {
        if (!make_map(&ma, A.tf32, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, A.npad_tc, A.kpad_tf32, kTcTileA, err)) return 1;
        if (!make_map(&mb, B.tf32, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, B.npad_tc, B.kpad_tf32, kTcTileB, err)) return 1;
        ma2 = ma;
        mb2 = mb;
    } else if (form == HJ_FORM_TC_FP16) {
        if (!make_map(&ma, A.bf_hi, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, A.npad_tc, A.kpad_bf16, kTcTileA, err)) return 1;
        if (!make_map(&mb, B.bf_hi, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, B.npad_tc, B.kpad_bf16, kTcTileB, err)) return 1;
        ma2 = ma;
        mb2 = mb;
    } else {
        const CUtensorMapDataType t = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
        if (!make_map(&ma, A.bf_hi, t, A.npad_tc, A.kpad_bf16, kTcTileA, err)) return 1;
        if (!make_map(&ma2, A.bf_lo, t, A.npad_tc, A.kpad_bf16, kTcTileA, err)) return 1;
        if (!make_map(&mb, B.bf_hi, t, B.npad_tc, B.kpad_bf16, kTcTileB, err)) return 1;
        if (!make_map(&mb2, B.bf_lo, t, B.npad_tc, B.kpad_bf16, kTcTileB, err)) return 1;
    }
    TcArgs a;
    memset(&a, 0, sizeof(a));
    a.ka = L.ka;
    a.a_bufs = L.a_bufs;
    a.nst = L.nst;
    a.near_cap = L.near_cap;
    a.near_rows = L.near_cap < kNearMinCap ? 0 : (bc ? kNearDenseBc : kNearDenseOne);
    a.items = idx.items;
    a.n_items = idx.n_items;
    a.norm_a = A.norms;
    a.norm_b = B.norms;
    a.tmax_b = B.tile_maxnorm_b;
    a.gmin_b = B.group_minnorm;
    a.jobs = d_jobs;
    a.na = na0;
    a.nb = nb0;
    a.band = reinterpret_cast<BandEntry *>(band);
    a.band_cap = band_cap;
    a.band_total = d_band_total;
    a.band_holes = d_band_holes;
    a.err = d_err;
    a.dbg = g_dbg_out;
    a.perm_a = A.perm;
    a.perm_b = B.perm;
    a.gate_ns = g_gate_ns;
    a.near_ns = g_near_ns;
    a.fold = !bc && A.fold ? 1u : 0u;
    if (bc) {
        a.norm_a = A.bc_norms;
        a.norm_b = nullptr;  // q_j / 2 is folded into the accumulator
        a.gmin_b = nullptr;
        a.tmax_b = nullptr;
        a.xn_a = A.bc_xn;
        a.blk_a = A.bc_blk;
        a.blk_b = B.bc_blk;
        a.cent_a = A.bc_cent;
        a.cent_b = B.bc_cent;
        a.bc = *bc;
        a.a_xoff = A.bc_dp;
    }
    uint64_t grid = (uint64_t)num_sms;
    if (grid > idx.n_items) grid = idx.n_items;
    if (bc && form == HJ_FORM_TC_TF32) {
        ensure_max_dynamic_smem((const void *)k_join_tc<HJ_FORM_TC_TF32, true>, kTcSmemMax);
        k_join_tc<HJ_FORM_TC_TF32, true><<<(unsigned)grid, kTcThreads, L.smem, st>>>(ma, ma2, mb, mb2, a);
    } else if (bc && form == HJ_FORM_TC_BF16X3) {
        ensure_max_dynamic_smem((const void *)k_join_tc<HJ_FORM_TC_BF16X3, true>, kTcSmemMax);
        k_join_tc<HJ_FORM_TC_BF16X3, true><<<(unsigned)grid, kTcThreads, L.smem, st>>>(ma, ma2, mb, mb2, a);
    } else if (bc) {
        ensure_max_dynamic_smem((const void *)k_join_tc<HJ_FORM_TC_FP16, true>, kTcSmemMax);
        k_join_tc<HJ_FORM_TC_FP16, true><<<(unsigned)grid, kTcThreads, L.smem, st>>>(ma, ma2, mb, mb2, a);
    } else if (form == HJ_FORM_TC_TF32) {
        ensure_max_dynamic_smem((const void *)k_join_tc<HJ_FORM_TC_TF32, false>, kTcSmemMax);
        k_join_tc<HJ_FORM_TC_TF32, false><<<(unsigned)grid, kTcThreads, L.smem, st>>>(ma, ma2, mb, mb2, a);
    } else if (form == HJ_FORM_TC_FP16) {
        ensure_max_dynamic_smem((const void *)k_join_tc<HJ_FORM_TC_FP16, false>, kTcSmemMax);
        k_join_tc<HJ_FORM_TC_FP16, false><<<(unsigned)grid, kTcThreads, L.smem, st>>>(ma, ma2, mb, mb2, a);
    } else {
        ensure_max_dynamic_smem((const void *)k_join_tc<HJ_FORM_TC_BF16X3, false>, kTcSmemMax);
        k_join_tc<HJ_FORM_TC_BF16X3, false><<<(unsigned)grid, kTcThreads, L.smem, st>>>(ma, ma2, mb, mb2, a);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        *err = std::string("tensor-core kernel launch: ") + cudaGetErrorString(e);
        return 1;
    }
    return 0;
}

uint64_t band_slack(int num_sms, bool bc) {
    return (uint64_t)num_sms * (kEpiWarps + 2) * (bc ? kBandChunk : kBandChunkRare);
}

void launch_recheck(const TcJob *d_jobs, int dtype_bytes, const uint2 *band, const unsigned long long *d_band_total,
                    uint64_t band_cap, unsigned int *d_max_err_bits, cudaStream_t st, bool vec_rows,
                    const float *norm_a, const float *norm_b) {
    const BandEntry *b = reinterpret_cast<const BandEntry *>(band);
    if (dtype_bytes == 8)
        k_recheck<double><<<1184, 256, 0, st>>>(d_jobs, b, d_band_total, band_cap, d_max_err_bits, vec_rows, norm_a,
                                                norm_b);
    else
        k_recheck<float><<<1184, 256, 0, st>>>(d_jobs, b, d_band_total, band_cap, d_max_err_bits, vec_rows, norm_a,
                                               norm_b);
}

void set_tc_debug_output(float *dbg) { g_dbg_out = dbg; }

void set_tc_wait_gate(uint64_t ns) { g_gate_ns = ns; }

void set_tc_near_limit(uint64_t ns) { g_near_ns = ns ? ns : kWaitLimitNs; }

}  // namespace hj
