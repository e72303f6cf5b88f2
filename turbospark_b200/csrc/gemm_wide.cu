// Quantized matmul for 24..128 token rows per pass on the fifth-generation tensor cores: y[t, r] = W[r, :] . x[t, :].
//
// One CTA per SM walks 128-row tiles of a Q4_K matrix.  Roles, a warpgroup or a thread of their own so that each one's
// latencies hide behind the others' work:
//   warp 0       one thread copies the raw blocks (cp.async.bulk.tensor, 128 rows x 144 bytes each) into a ring
//   warp 1       one thread copies the activation chunks of each 256-column block into another
//   warps 4-11   dequantisation: a warpgroup per half of a block; thread = row.  It turns its 128 nibbles into the
//                integers q * sc (exact in f16) and writes them straight into tensor memory (tcgen05.st) as the A
//                operand of the half's eight K=16 steps; the sub-block mins m go to a small shared-memory tile
//                that a seventeenth step multiplies with the activation's 32-column sums (hi + lo f16 split) into
//                a second accumulator
//   warp 2       one thread issues tcgen05.mma (A from tensor memory, or from shared memory for the mins step; B from
//                shared memory through a matrix descriptor; fp32 accumulators in tensor memory) and commits
//                completions onto the barriers
//   warps 12-19  fold: a warpgroup per half of the token columns; thread = row.  A block's two accumulators are read back
//                (tcgen05.ld) and folded into registers as acc += d * D1 - dmin * D2, so the per-block f16 scales d
//                and dmin never lose a bit; then the epilogue, f16 or f32
// Every weight byte is dequantised once per tile whatever the token count.
//
// What bounds it: the MMA thread and the tensor pipe behind it.  Seventeen MMAs with A in tensor memory take 1000 cycles at 32
// token rows and 1750 at 128; a block takes 1400 and 1950 in all.  When the whole MMA warp walked the blocks with the instruction
// predicated on one lane, issuing alone took 75-90 cycles an MMA and a block 2500; with sixteen warps that dequantised and
// folded in turn, in step with one another, a block took 3400 and 4700.  Measured, 57344 x 4096: 96 -> 58 us at 32 token
// rows, 138 -> 80 at 128; 4096 x 4096: 30 -> 20 at 128.
//
// Tensor memory (512 columns): the mins' accumulators, two of the quants', then the A slots.  Up to 64 token rows two blocks'
// A operands fit and two accumulators of the mins; up to 96 one block's and two accumulators; above that one of either.
//
// Shared-memory B operand (K-major, 128-byte swizzle): 64 columns of a token are a row of 128 bytes whose eight 16-byte
// chunks are XORed with the token's index mod 8; a 64-column block is n_pad such rows, the chunks of sums (no swizzle)
// follow the four blocks.  Within a chunk the K order is x0,x2,x1,x3,x4,x6,x5,x7 - the order in which one LOP3 pulls nibble
// pairs out of a 32-bit word of quants - so no byte shuffle is needed on the weight side.  The global copy of the activations
// is laid out exactly like a stage of that ring, which makes the load of a block one bulk copy.  The mins tile: chunk c of
// row r at c * 2048 + r * 16.
#include <cuda.h>

#include <atomic>
#include <map>
#include <mutex>

#include "gemm_quant.cuh"
#include "tc05.cuh"

namespace {

constexpr int WM = 128;              // weight rows per tile (UMMA M)
constexpr int WIDE_WARP_RAW = 0, WIDE_WARP_ACT = 1, WIDE_WARP_MMA = 2;  // and one idle warp, then 8 dequantising and 8 folding ones
constexpr int WIDE_THREADS = 640;
constexpr int WIDE_RAW_STAGES = 4;   // raw blocks in flight (one 128-row x 144-byte box each)
constexpr int WIDE_RAW_BYTES = WM * 144;
constexpr int WIDE_B_STAGES = 3;     // activation ring: 3 stages up to 64 token rows, 2 above (a stage doubles)
constexpr int WIDE_NMAX = 128;       // token rows per pass
constexpr int WIDE_NDUAL = 64;       // up to here two blocks' A operands fit beside the accumulators, and three activation stages
constexpr int WIDE_NTWO = 96;        // up to here two accumulators of the mins' products fit tensor memory
constexpr int WIDE_A_COLS = 64;      // tensor-memory columns of one A slot: 128 f16 K positions, half a block
constexpr int WIDE_MIN_BYTES = WM * 16 * 2;  // the mins step's A operand: 128 rows x 16 K positions of f16
constexpr int WIDE_SCALE_SLOTS = 8;  // a block's scales are written at most four blocks before it is folded
constexpr int WIDE_TMEM_COLS = 512;
constexpr int WIDE_SINK_BYTES = 256 * 4;
constexpr int WIDE_RING_AT = (1024 + WIDE_SINK_BYTES + WIDE_SCALE_SLOTS * WM * 4 + 2 * WIDE_MIN_BYTES + WIDE_RAW_STAGES * WIDE_RAW_BYTES + 1023) & ~1023;
// activation stages start on the 1024-byte boundaries that the 128-byte swizzle counts from
__host__ __device__ constexpr int wide_stage_stride(int n_pad) { return (WIDE_CHUNKS * n_pad * 16 + 1023) & ~1023; }

__device__ __forceinline__ uint32_t hmul2_bits(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t hsub2_bits(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
struct WideBars {
    uint64_t raw_full[WIDE_RAW_STAGES], raw_empty[WIDE_RAW_STAGES];
    uint64_t b_full[WIDE_B_STAGES], b_empty[WIDE_B_STAGES];
    // a block's two halves may be multiplied: their A operand is written and the accumulator that the half starts on -
    // the quants' with the first, the mins' with the second - is folded; the halves' slots are free again
    uint64_t a_full[2][2], a_empty[2][2];
    uint64_t d_full[2];  // a block's accumulators are complete
    uint64_t scale_full[WIDE_SCALE_SLOTS];
    uint64_t mma_over;   // every MMA that was issued has finished
    uint32_t tmem_base;
    uint32_t failed;
    uint32_t ticket;
};

// x natural [tokens, cols] f16 -> for every pass of `per_pass` token rows and every 256-column block, n_pad tokens x 34 chunks
// of 16 bytes (see the file header); n_pad is per_pass for every pass, the last one's missing rows being zeros, so that pass p
// starts at p * units * 34 * per_pass chunks.  A CTA takes eight tokens of one block: warp = token, lane = 16-byte chunk; the
// 32-column sums come from two shuffles over the four lanes of a sub-block; the CTA's 34 x 8 chunks go out through
// shared memory as 128-byte runs.
__global__ void __launch_bounds__(256) wide_prepare_kernel(const __half* __restrict__ x, int64_t x_stride, int tokens, int per_pass, int units,
                                                           uint4* __restrict__ xw) {
    __shared__ uint4 tile[WIDE_CHUNKS][8];
    pdl_wait();
    const int blk = blockIdx.x;
    const int pass = blockIdx.y / (per_pass >> 3), grp = blockIdx.y % (per_pass >> 3);
    const int nt = min(per_pass, tokens - pass * per_pass);  // token rows of this pass; the others are zeros
    const int n_pad = per_pass;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = grp * 8 + w;  // token row within the pass
    uint4 o = make_uint4(0, 0, 0, 0);
    float sum = 0.f;
    if (n < nt) {
        const uint4 raw = *reinterpret_cast<const uint4*>(x + (size_t)(pass * per_pass + n) * x_stride + (size_t)blk * 256 + 8 * lane);
        __half h[8];
        *reinterpret_cast<uint4*>(h) = raw;
#pragma unroll
        for (int i = 0; i < 8; i++) sum += __half2float(h[i]);
        o = act_pack8(h);
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    tile[lane][w] = o;
    if ((lane & 3) == 0) {  // sub-block lane / 4: (hi, lo) halves at chunk 32 + sub / 4, pair sub % 4
        const int sub = lane >> 2;
        const __half hi = __float2half_rn(sum);
        const __half2 hl = __halves2half2(hi, __float2half_rn(sum - __half2float(hi)));
        reinterpret_cast<__half2*>(&tile[32 + (sub >> 2)][w])[sub & 3] = hl;
    }
    __syncthreads();
    uint4* dst = xw + (size_t)(pass * units + blk) * WIDE_CHUNKS * n_pad;
    // eight tokens are one swizzle group: 1024 bytes per 64-column block, then the sums of the whole pass
    for (int i = threadIdx.x; i < 32 * 8; i += 256) {
        const int cb = i >> 6, t = (i >> 3) & 7, c = i & 7;
        dst[(size_t)(cb * n_pad + grp * 8 + t) * 8 + c] = tile[cb * 8 + (c ^ t)][t];
    }
    if (threadIdx.x < 16) {
        const int c = threadIdx.x >> 3, t = threadIdx.x & 7;
        dst[(size_t)(32 + c) * n_pad + grp * 8 + t] = tile[32 + c][t];
    }
}

// One box of the weight matrix (128 rows x one 144-byte block) lands as 128 consecutive 144-byte rows: a lane stride
// of nine 16-byte units, so the 128-bit loads of 32 consecutive rows do not collide.
__device__ __forceinline__ void tensor_g2s_2d(void* dst_smem, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                     smem_u32(dst_smem)),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
                 : "memory");
}

// A warpgroup's share of the register file.  The shares may not exceed what the block is launched with (WIDE_THREADS x
// WIDE_LAUNCH_REGS), which launch_gemm_wide_q4k checks against the compiled kernel: the increase waits until the others
// have given theirs up.
constexpr int WIDE_LAUNCH_REGS = 96;
template <bool MANY>
struct WideRegs {
    static constexpr int FEED = MANY ? 32 : 64, DEQ = MANY ? 72 : 80, FOLD = MANY ? 152 : 128;
    static_assert(FEED + 2 * DEQ + 2 * FOLD <= WIDE_THREADS / 128 * WIDE_LAUNCH_REGS, "register shares");
};
template <int N>
__device__ __forceinline__ void regs_take() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void regs_give() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// ROUNDS: how many 16-column read-backs cover a warp's share of the accumulator columns (n_pad / 2 <= 16 * ROUNDS).
// MANY: several passes of n_pad token rows in one launch (see launch_gemm_wide_q4k)
template <int ROUNDS, bool MANY>
__global__ void __launch_bounds__(WIDE_THREADS, 1)
    gemm_wide_q4k_kernel(const __grid_constant__ CUtensorMap wmap, int64_t rows, int units, const uint4* __restrict__ xw, int n_pad,
                         int all_tokens, int passes, void* __restrict__ y, int64_t y_stride, int y_f32, int n_whole, int ksplit, float* __restrict__ part,
                         uint32_t* __restrict__ err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    WideBars* bars = reinterpret_cast<WideBars*>(smem);
    volatile uint32_t* sink = reinterpret_cast<uint32_t*>(smem + 1024);  // one word per dequantising thread, never read
    __half2* scale_ring = reinterpret_cast<__half2*>(smem + 1024 + WIDE_SINK_BYTES);  // (d, dmin) of every row of a block
    uint8_t* min_ring = smem + 1024 + WIDE_SINK_BYTES + WIDE_SCALE_SLOTS * WM * 4;
    uint8_t* raw_ring = min_ring + 2 * WIDE_MIN_BYTES;
    uint8_t* b_ring = smem + WIDE_RING_AT;
    // the depths of the operand rings and the accumulators' copies follow the pass's width (see the file header)
    const uint32_t n_bst = n_pad <= WIDE_NDUAL ? 3u : 2u;
    const uint32_t a_depth = n_pad <= WIDE_NDUAL ? 2u : 1u;  // blocks in the tensor-memory A slots
    const uint32_t d2_sets = n_pad <= WIDE_NTWO ? 2u : 1u;
    const int b_stage_bytes = WIDE_CHUNKS * n_pad * 16, b_stride = wide_stage_stride(n_pad);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // Work items, dealt round-robin to the CTAs: the first n_whole tiles (a multiple of the grid) go whole; each of the
    // remaining tiles - fewer than CTAs - is cut into `ksplit` runs of its blocks so that the last wave fills the
    // device too.  A run leaves its partial sums in `part` (after 1024 ticket words); the CTA that finishes a tile's last
    // run adds them in run order and writes the tile.
    // MANY: an item is a whole tile for one of the passes, the passes of a tile side by side so that its weights come from
    // memory once; the runs of a tile that a single pass would cut are added in the same order, in registers.
    const int n_tiles = (int)(rows / WM);
    const int n_items = MANY ? n_tiles * passes : n_whole + (n_tiles - n_whole) * ksplit;
    const int upk = (units + ksplit - 1) / ksplit;  // blocks per run
    struct Item {
        int tile, b0, nblk, ks;  // ks < 0: a whole tile
        int pass;
    };
    auto item_of = [&](int item) {
        Item it;
        it.pass = 0;
        if (MANY) {
            it.tile = item / passes, it.pass = item % passes, it.b0 = 0, it.nblk = units, it.ks = -1;
        } else if (item < n_whole) {
            it.tile = item, it.b0 = 0, it.nblk = units, it.ks = -1;
        } else {
            const int t = item - n_whole;
            it.tile = n_whole + t / ksplit, it.ks = ksplit > 1 ? t % ksplit : -1;
            it.b0 = (t % ksplit) * upk;
            it.nblk = max(0, min(units, it.b0 + upk) - it.b0);
        }
        return it;
    };

    if (threadIdx.x == 0) {
        for (int i = 0; i < WIDE_RAW_STAGES; i++) mbar_init(&bars->raw_full[i], 1), mbar_init(&bars->raw_empty[i], 8);
        for (int i = 0; i < WIDE_B_STAGES; i++) mbar_init(&bars->b_full[i], 1), mbar_init(&bars->b_empty[i], 1);
        for (int i = 0; i < 2; i++) {
            for (int h = 0; h < 2; h++) mbar_init(&bars->a_full[i][h], 4 + 8), mbar_init(&bars->a_empty[i][h], 1);
            mbar_init(&bars->d_full[i], 1);
        }
        for (int i = 0; i < WIDE_SCALE_SLOTS; i++) mbar_init(&bars->scale_full[i], 4);
        mbar_init(&bars->mma_over, 1);
        bars->failed = 0;
        mbar_fence_init();
    }
    if (warp == WIDE_WARP_MMA) {  // the MMA warp owns the tensor-memory allocation
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)),
                     "r"((uint32_t)WIDE_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // accumulators of the mins' products, two of the quants', then 2 * a_depth A slots (a read-back that reaches past the
    // last accumulator stays inside the allocation)
    const uint32_t tmem_d2 = bars->tmem_base;
    const uint32_t tmem_d1 = tmem_d2 + d2_sets * (uint32_t)n_pad;
    const uint32_t tmem_a = tmem_d1 + 2 * (uint32_t)n_pad;

    if (warp < 4) {
        regs_give<WideRegs<MANY>::FEED>();
        if (warp == WIDE_WARP_RAW) {
            // ---- producer of the raw blocks: one tensor copy (128 rows x 144 bytes) per block.  Weights come from no
            // kernel that this launch may overlap, so the ring fills before the activations are there.
            if (lane == 0) {
                uint32_t nb = 0;
                bool ok = true;
                for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
                    const Item wi = item_of(item);
                    for (int blk = 0; blk < wi.nblk && ok; blk++, nb++) {
                        const uint32_t s = nb % WIDE_RAW_STAGES;
                        if (nb >= WIDE_RAW_STAGES) ok = mbar_wait(&bars->raw_empty[s], ((nb / WIDE_RAW_STAGES) - 1) & 1, err);
                        if (!ok) break;
                        mbar_expect_tx(&bars->raw_full[s], (uint32_t)WIDE_RAW_BYTES);
                        tensor_g2s_2d(raw_ring + s * WIDE_RAW_BYTES, &wmap, (wi.b0 + blk) * 36, wi.tile * WM, &bars->raw_full[s]);
                    }
                }
                if (!ok) bars->failed = 1;
                // no copy is in flight when the CTA leaves, also when another role has given up
                for (uint32_t k = nb > WIDE_RAW_STAGES ? nb - WIDE_RAW_STAGES : 0; k < nb; k++)
                    mbar_wait(&bars->raw_full[k % WIDE_RAW_STAGES], (k / WIDE_RAW_STAGES) & 1, err);
            }
        } else if (warp == WIDE_WARP_ACT) {
            // ---- producer of the activation chunks: its own warp, so a full activation ring never holds up the weights
            if (lane == 0) {
                pdl_wait();
                uint32_t nb = 0;
                bool ok = true;
                for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
                    const Item wi = item_of(item);
                    for (int blk = 0; blk < wi.nblk && ok; blk++, nb++) {
                        const uint32_t bs = nb % n_bst;
                        if (nb >= n_bst) ok = mbar_wait(&bars->b_empty[bs], ((nb / n_bst) - 1) & 1, err);
                        if (!ok) break;
                        mbar_expect_tx(&bars->b_full[bs], (uint32_t)b_stage_bytes);
                        bulk_g2s(b_ring + bs * b_stride, xw + (size_t)(wi.pass * units + wi.b0 + blk) * WIDE_CHUNKS * n_pad, (uint32_t)b_stage_bytes, &bars->b_full[bs]);
                    }
                }
                if (!ok) bars->failed = 1;
                for (uint32_t k = nb > n_bst ? nb - n_bst : 0; k < nb; k++) mbar_wait(&bars->b_full[k % n_bst], (k / n_bst) & 1, err);
            }
        } else if (warp == WIDE_WARP_MMA) {
            // ---- MMA issue: one thread walks the blocks
            if (tc_elect()) {
                // instruction descriptor: f32 accumulate, f16 A and B, both K-major, N = n_pad, M = 128
                const uint32_t idesc = (1u << 4) | ((uint32_t)(n_pad >> 3) << 17) | ((uint32_t)(WM >> 4) << 24);
                // shared-memory matrix descriptors without the start address (descriptor version 1).  Activations: 128-byte
                // swizzle, eight-token groups 1024 bytes apart; sums: no swizzle, leading-byte-offset = chunk stride,
                // stride-byte-offset = 128 (eight tokens of 16 bytes)
                const uint64_t desc_hi = ((uint64_t)1u << 16) | ((uint64_t)(1024u >> 4) << 32) | (1ull << 46) | (2ull << 61);
                const uint64_t desc_sum_hi = ((uint64_t)((uint32_t)(n_pad * 16) >> 4) << 16) | ((uint64_t)(128u >> 4) << 32) | (1ull << 46);
                // the mins tile: chunk stride 128 rows x 16 bytes, eight rows of 16 bytes per row group
                const uint64_t desc_min_hi = ((uint64_t)((uint32_t)(WM * 16) >> 4) << 16) | ((uint64_t)(128u >> 4) << 32) | (1ull << 46);
                uint32_t nb = 0;
                bool ok = true;
                for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
                    const int nblk = item_of(item).nblk;
                    for (int blk = 0; blk < nblk && ok; blk++, nb++) {
                        const uint32_t bs = nb % n_bst, set = nb & 1, slot = (nb % a_depth) * 2, par = (nb >> 1) & 1;
                        ok = mbar_wait(&bars->b_full[bs], (nb / n_bst) & 1, err);
                        if (ok) ok = mbar_wait(&bars->a_full[set][0], par, err);
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t a_col = tmem_a + slot * WIDE_A_COLS;
                        const uint32_t d1 = tmem_d1 + set * (uint32_t)n_pad;
                        // the descriptor's address field (16-byte units): 32 bytes per K step, n_pad rows of 128 bytes per 64 columns
                        const uint32_t b_at = (smem_u32(b_ring + bs * b_stride) >> 4) & 0x3FFFu;
                        const uint64_t desc0 = desc_hi | (uint64_t)b_at;
                        auto step_at = [&](int j) { return desc0 + (uint64_t)((uint32_t)(j >> 2) * (uint32_t)(8 * n_pad) + (uint32_t)(j & 3) * 2u); };
                        tc_issue_ts<false>(d1, a_col, desc0, idesc);
#pragma unroll
                        for (int j = 1; j < 8; j++) tc_issue_ts<true>(d1, a_col + 8 * j, step_at(j), idesc);
                        ok = mbar_wait(&bars->a_full[set][1], par, err);
                        if (!ok) break;
                        tc_fence_after();
                        // the mins step before the first half's slot is given back: that half's writers also write the mins
                        tc_issue_ss<false>(tmem_d2 + (nb % d2_sets) * (uint32_t)n_pad,
                                           desc_min_hi | (uint64_t)((smem_u32(min_ring + set * WIDE_MIN_BYTES) >> 4) & 0x3FFFu),
                                           desc_sum_hi | (uint64_t)(b_at + 32u * (uint32_t)n_pad), idesc);
                        tc_commit(&bars->a_empty[nb % a_depth][0]);
#pragma unroll
                        for (int j = 8; j < 16; j++) tc_issue_ts<true>(d1, a_col + 8 * j, step_at(j), idesc);
                        tc_commit(&bars->a_empty[nb % a_depth][1]);
                        tc_commit(&bars->b_empty[bs]);
                        tc_commit(&bars->d_full[set]);
                    }
                }
                if (!ok) bars->failed = 1;
                tc_commit(&bars->mma_over);  // nor is an MMA when tensor memory is given back
                mbar_wait(&bars->mma_over, 0, err);
            }
            __syncwarp();
        }
    } else if (warp < 12) {
        // ---- dequantisation: a warpgroup takes one half (sub-blocks 4h .. 4h + 3) of every block, thread = row of the tile
        regs_give<WideRegs<MANY>::DEQ>();
        const int h = (warp >> 2) - 1, q4 = warp & 3;
        const int row = q4 * 32 + lane;
        const uint32_t lane_base = (uint32_t)(q4 * 32) << 16;
        uint32_t nb = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
            const int nblk = item_of(item).nblk;
            for (int blk = 0; blk < nblk && ok; blk++, nb++) {
                const uint32_t s = nb % WIDE_RAW_STAGES, slot = (nb % a_depth) * 2 + h;
                ok = __all_sync(0xffffffffu, mbar_wait(&bars->raw_full[s], (nb / WIDE_RAW_STAGES) & 1, err));
                if (!ok) break;
                const uint8_t* bp = raw_ring + s * WIDE_RAW_BYTES + row * 144;
                const uint4 hdr = *reinterpret_cast<const uint4*>(bp);
                uint32_t w[16];
#pragma unroll
                for (int i = 0; i < 4; i++) *reinterpret_cast<uint4*>(w + 4 * i) = *reinterpret_cast<const uint4*>(bp + 16 + 64 * h + 16 * i);
                // 6-bit scales and mins of the half's four sub-blocks, a byte each (crates/compute/src/quant_gguf/q4_k.rs:43-54)
                const uint32_t sc4 = h == 0 ? hdr.y & 0x3F3F3F3Fu : (hdr.w & 0x0F0F0F0Fu) | ((hdr.y >> 2) & 0x30303030u);
                const uint32_t mn4 = h == 0 ? hdr.z & 0x3F3F3F3Fu : ((hdr.w >> 4) & 0x0F0F0F0Fu) | ((hdr.z >> 2) & 0x30303030u);
                const uint32_t k1024 = 0x64006400u;  // integers up to 63 as f16 pairs: (0x6400 | v) is 1024 + v
                auto pair_of = [&](uint32_t four, int i) { return hsub2_bits(__byte_perm(four, 0x64646464u, 0x4040u + 0x0101u * i), k1024); };
                // The stage is given back when the block sits in registers.  An arrival alone does not wait for loads in flight
                // (the copy that refilled the stage was seen to overtake them while the tensor core kept shared memory
                // busy); a store of something computed from all of them does.
                sink[threadIdx.x - 128] = w[0] ^ w[4] ^ w[8] ^ w[12] ^ hdr.x;
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->raw_empty[s]);
                if (nb >= a_depth) ok = mbar_wait(&bars->a_empty[nb % a_depth][h], ((nb / a_depth) - 1) & 1, err);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                if (h == 0) scale_ring[(nb % WIDE_SCALE_SLOTS) * WM + row] = *reinterpret_cast<const __half2*>(&hdr.x);
                // K positions 8h .. 8h + 7 of the mins step: (m, m) against the (hi, lo) sums of sub-blocks 4h .. 4h + 3
                *reinterpret_cast<uint4*>(min_ring + (nb & 1) * WIDE_MIN_BYTES + h * (WM * 16) + row * 16) =
                    make_uint4(pair_of(mn4, 0), pair_of(mn4, 1), pair_of(mn4, 2), pair_of(mn4, 3));
#pragma unroll
                for (int g = 0; g < 2; g++) {
                    const uint32_t s0 = pair_of(sc4, 2 * g), s1 = pair_of(sc4, 2 * g + 1);
                    const uint32_t off0 = hmul2_bits(s0, 0xE400E400u);  // -1024 * sc, exact
                    const uint32_t off1 = hmul2_bits(s1, 0xD400D400u);  // -64 * sc, exact
                    uint32_t r[32];
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const uint32_t v = w[8 * g + i], v8 = v >> 8;
                        r[2 * i] = hfma2_u32(lop3_and_or(v, 0x000F000Fu, 0x64006400u), s0, off0);  // q * sc, exact
                        r[2 * i + 1] = hfma2_u32(lop3_and_or(v8, 0x000F000Fu, 0x64006400u), s0, off0);
                        r[16 + 2 * i] = hfma2_u32(lop3_and_or(v, 0x00F000F0u, 0x54005400u), s1, off1);
                        r[16 + 2 * i + 1] = hfma2_u32(lop3_and_or(v8, 0x00F000F0u, 0x54005400u), s1, off1);
                    }
                    tc_st32(tmem_a + slot * WIDE_A_COLS + lane_base + 32 * g, r);
                }
                tc_wait_st();
                tc_fence_before();
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    if (h == 0) mbar_arrive(&bars->scale_full[nb % WIDE_SCALE_SLOTS]);
                    mbar_arrive(&bars->a_full[nb & 1][h]);
                }
            }
        }
        if (!ok && lane == 0) bars->failed = 1;
    } else {
        // ---- fold and epilogue: a warpgroup takes half of the token columns, thread = row of the tile
        regs_take<WideRegs<MANY>::FOLD>();
        const int g = (warp >> 2) - 3, q4 = warp & 3;
        const int row = q4 * 32 + lane;
        const int cpw = n_pad >> 1;
        const uint32_t col0 = ((uint32_t)(q4 * 32) << 16) + (uint32_t)(g * cpw);
        uint32_t nb = 0;
        bool ok = true;
        if (lane == 0) {  // the accumulators start out free
            mbar_arrive(&bars->a_full[0][0]), mbar_arrive(&bars->a_full[1][0]), mbar_arrive(&bars->a_full[0][1]);
            if (d2_sets == 2) mbar_arrive(&bars->a_full[1][1]);
        }
        pdl_wait();
        for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
            const Item wi = item_of(item);
            const int nblk = wi.nblk, tile = wi.tile, ks = wi.ks;
            const bool runs = MANY && ksplit > 1 && tile >= n_whole;
            int run_left = upk;
            float acc[16 * ROUNDS], total[MANY ? 16 * ROUNDS : 1];
#pragma unroll
            for (int i = 0; i < 16 * ROUNDS; i++) acc[i] = 0.f;
            if (MANY) {
#pragma unroll
                for (int i = 0; i < 16 * ROUNDS; i++) total[i] = 0.f;
            }
            auto end_run = [&]() {
#pragma unroll
                for (int i = 0; i < 16 * ROUNDS; i++) total[MANY ? i : 0] += acc[i], acc[i] = 0.f;
                run_left = upk;
            };
            // acc += by * (this warp's share of an accumulator); 32 columns per round trip, columns past the share are read
            // and dropped
            auto fold = [&](uint32_t from, float by) {
                if constexpr (MANY) {  // the sums of finished runs leave room for sixteen
#pragma unroll
                    for (int c = 0; c < ROUNDS; c++)
                        if (16 * c < cpw) {
                            uint32_t v[16];
                            tc_ld16(from + col0 + 16 * c, v);
                            tc_wait_ld(v);
#pragma unroll
                            for (int i = 0; i < 16; i++) acc[16 * c + i] = fmaf(by, __uint_as_float(v[i]), acc[16 * c + i]);
                        }
                } else {
#pragma unroll
                    for (int c = 0; c < ROUNDS; c += 2)
                        if (16 * c < cpw) {
                            uint32_t v0[16], v1[16];
                            tc_ld16(from + col0 + 16 * c, v0);
                            tc_ld16(from + col0 + 16 * c + 16, v1);
                            tc_wait_ld(v0, v1);
#pragma unroll
                            for (int i = 0; i < 16; i++) {
                                acc[16 * c + i] = fmaf(by, __uint_as_float(v0[i]), acc[16 * c + i]);
                                acc[16 * c + 16 + i] = fmaf(by, __uint_as_float(v1[i]), acc[16 * c + 16 + i]);
                            }
                        }
                }
                tc_fence_before();
                __syncwarp();
            };
            for (int blk = 0; blk < nblk && ok; blk++, nb++) {
                // acc += d * D1 - dmin * D2
                const uint32_t set = nb & 1;
                ok = mbar_wait(&bars->scale_full[nb % WIDE_SCALE_SLOTS], (nb / WIDE_SCALE_SLOTS) & 1, err) &&
                     mbar_wait(&bars->d_full[set], (nb >> 1) & 1, err);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                const __half2 dd = scale_ring[(nb % WIDE_SCALE_SLOTS) * WM + row];
                const float d = __low2float(dd), neg_dmin = -__high2float(dd);
                // the mins' products first: of their accumulators there may be only one
                fold(tmem_d2 + (nb % d2_sets) * (uint32_t)n_pad, neg_dmin);
                if (lane == 0) mbar_arrive(&bars->a_full[(nb + d2_sets) & 1][1]);
                fold(tmem_d1 + set * (uint32_t)n_pad, d);
                if (lane == 0) mbar_arrive(&bars->a_full[set][0]);
                if (MANY && runs && --run_left == 0) end_run();
            }
            if (MANY && runs) {
                if (run_left != upk) end_run();
#pragma unroll
                for (int i = 0; i < 16 * ROUNDS; i++) acc[i] = total[MANY ? i : 0];
            }
            const int64_t orow = (int64_t)tile * WM + row;
            // this thread's share of the token columns: cpw of them from n0 on, the ones behind the last token left out.
            // (Short code on purpose: unrolled over the accumulators, it runs once per tile out of a cold instruction cache.)
            const int tok0 = MANY ? wi.pass * n_pad : 0, tokens = MANY ? min(n_pad, all_tokens - tok0) : all_tokens;
            const int n0 = g * cpw, n_mine = max(0, min(cpw, tokens - n0));
            auto put16 = [&](const float* v, int first) {  // sixteen columns from n0 + first on
                const int64_t at = (int64_t)(tok0 + n0 + first) * y_stride + orow;
                if (y_f32) {
                    float* p = reinterpret_cast<float*>(y) + at;
#pragma unroll
                    for (int i = 0; i < 16; i++, p += y_stride)
                        if (first + i < n_mine) *p = v[i];
                } else {
                    __half* p = reinterpret_cast<__half*>(y) + at;
#pragma unroll
                    for (int i = 0; i < 16; i++, p += y_stride)
                        if (first + i < n_mine) *p = __float2half_rn(v[i]);
                }
            };
            if (MANY || ks < 0) {
                if (ok) {
#pragma unroll
                    for (int c = 0; c < ROUNDS; c++) put16(acc + 16 * c, 16 * c);
                }
            } else {
                // a run of a cut tile: leave the partial sums, take a ticket; whoever holds the last one adds the runs in
                // run order (so the result does not depend on who that is) and puts the counter back to zero.  A run's sums
                // lie as the threads hold them: four columns of a thread are 16 bytes, a warp's are 512.
                uint32_t* tickets = reinterpret_cast<uint32_t*>(part);
                float4* pdata = reinterpret_cast<float4*>(part + 1024) + (size_t)(tile - n_whole) * ksplit * (WM * WIDE_NMAX / 4) + (warp - 12) * 32 + lane;
                {
                    float4* p = pdata + (size_t)ks * (WM * WIDE_NMAX / 4);
#pragma unroll
                    for (int i = 0; i < 4 * ROUNDS; i++)
                        if (4 * i < n_mine) p[i * 256] = ok ? make_float4(acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
                __threadfence();
                asm volatile("bar.sync 1, 256;" ::: "memory");
                if (warp == 12 && lane == 0) {
                    const uint32_t t = atomicAdd(&tickets[tile - n_whole], 1u);
                    if (t == (uint32_t)ksplit - 1) tickets[tile - n_whole] = 0;
                    bars->ticket = t;
                }
                asm volatile("bar.sync 1, 256;" ::: "memory");
                if (bars->ticket == (uint32_t)ksplit - 1) {
                    __threadfence();
                    // sixteen columns at a time, run by run: the loads of four runs are in flight together
                    for (int c = 0; 16 * c < n_mine; c++) {
                        float sum[16];
#pragma unroll
                        for (int i = 0; i < 16; i++) sum[i] = 0.f;
                        for (int k0 = 0; k0 < ksplit; k0 += 4) {
                            float4 v[4][4];
#pragma unroll
                            for (int k = 0; k < 4; k++)
#pragma unroll
                                for (int i = 0; i < 4; i++)
                                    v[k][i] = k0 + k < ksplit && 16 * c + 4 * i < n_mine ? __ldcg(pdata + (size_t)(k0 + k) * (WM * WIDE_NMAX / 4) + (4 * c + i) * 256)
                                                                                         : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                            for (int k = 0; k < 4; k++)
                                if (k0 + k < ksplit)
#pragma unroll
                                    for (int i = 0; i < 4; i++) sum[4 * i] += v[k][i].x, sum[4 * i + 1] += v[k][i].y, sum[4 * i + 2] += v[k][i].z, sum[4 * i + 3] += v[k][i].w;
                        }
                        put16(sum, 16 * c);
                    }
                }
                asm volatile("bar.sync 1, 256;" ::: "memory");  // the ticket word is reused by the next cut tile
            }
        }
        if (!ok && lane == 0) bars->failed = 1;
        pdl_launch_dependents();  // by the warps that have waited: who starts then may rely on everything before this launch
    }
    tc_fence_before();
    __syncthreads();
    if (warp == WIDE_WARP_MMA) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(bars->tmem_base), "r"((uint32_t)WIDE_TMEM_COLS) : "memory");
    }
}

}  // namespace

bool gemm_wide_supported(int qtype, int64_t rows, int64_t cols, int tokens) {
    return qtype == TSB_Q4_K && rows % WM == 0 && cols % 256 == 0 && tokens >= 1;
}

// How a matrix's 128-row tiles are dealt to the CTAs: whole tiles while they fill complete waves, the rest cut into
// `ksplit` runs of blocks.  ksplit minimises the longest CTA's time in units of one block (18 KB of weights): a run
// of a cut tile also writes its 128 x n_pad partial sums and the tile's last run reads them all back, which at 128
// token rows costs as much as seven blocks, plus one block's worth of fixed work.  The plan must not depend on the
// token count - the order in which a row's sums are added, and so its bits, would change with its batch mates - so
// the cost is taken at 96 token rows whatever the pass carries.
struct WidePlan {
    int n_whole, ksplit;
    int64_t tail_rows;
};
static WidePlan wide_plan(int sm_count, int64_t rows, int units) {
    constexpr int n_pad = 96;
    const int tiles = (int)(rows / WM), grid = sm_count;
    WidePlan p;
    p.n_whole = tiles / grid * grid;
    const int tail = tiles - p.n_whole;
    p.ksplit = 1;
    p.tail_rows = (int64_t)tail * WM;
    if (tail == 0) return p;
    const float per_run = 1.f + (float)n_pad / 18.f;
    float best = (float)((tail + grid - 1) / grid) * (float)units;
    for (int k = 2; k <= units && k <= 16; k++) {
        const int upk = (units + k - 1) / k;
        const float load = (float)((tail * k + grid - 1) / grid) * ((float)upk + per_run);
        if (load < best - 1e-3f) best = load, p.ksplit = k;
    }
    if (const char* env = getenv("TSB_WIDE_KSPLIT")) p.ksplit = std::max(1, std::min(units, atoi(env)));  // experiments
    const int upk = (units + p.ksplit - 1) / p.ksplit;
    p.ksplit = (units + upk - 1) / upk;  // no empty runs: every run of a tile takes a ticket
    return p;
}
// Several passes in one launch when whole tiles of all of them fill the device about as well as one pass after the other with its
// cut tiles does: the launch saves the passes' prologues and the traffic of their partial sums, and reads the weights once.
static bool wide_takes_many(const WidePlan& p, int sm_count, int n_tiles, int units, int passes) {
    if (passes < 2) return false;
    const int tail = n_tiles - p.n_whole, upk = (units + p.ksplit - 1) / p.ksplit;
    const int64_t one = (int64_t)p.n_whole / sm_count * units + (tail ? (int64_t)((tail * p.ksplit + sm_count - 1) / sm_count) * upk : 0) + (p.ksplit > 1 ? 5 : 1);
    const int64_t many = ((int64_t)n_tiles * passes + sm_count - 1) / sm_count * units;
    return many <= passes * one;
}
static int wide_pass_rows(int tokens) {
    const int passes = (tokens + WIDE_NMAX - 1) / WIDE_NMAX;
    return ((tokens + passes - 1) / passes + 15) / 16 * 16;
}
// (rows behind the last token are left as they are: a token row's products do not meet another's)
ActOut wide_operand(void* workspace, int tokens) { return ActOut{static_cast<uint4*>(workspace), nullptr, wide_pass_rows(tokens), 0}; }
// the operand copy of every pass of a call with `tokens` token rows
size_t gemm_wide_workspace_bytes(int64_t cols, int tokens) {
    const int passes = (tokens + WIDE_NMAX - 1) / WIDE_NMAX;
    return (size_t)(passes < 1 ? 1 : passes) * (size_t)(cols / 256) * WIDE_CHUNKS * WIDE_NMAX * 16;
}
size_t gemm_wide_partial_bytes_for(int sm_count, int64_t rows, int64_t cols) {
    const WidePlan p = wide_plan(sm_count, rows, (int)(cols / 256));
    return p.ksplit > 1 ? 4096 + (size_t)p.ksplit * WIDE_NMAX * p.tail_rows * sizeof(float) : 0;
}
size_t gemm_wide_partial_bytes(const tsb_ctx* ctx, int64_t rows, int64_t cols) {
    return gemm_wide_partial_bytes_for(ctx->sm_count, rows, cols);
}

static size_t wide_smem_bytes(int n_pad) {
    const size_t b_stages = n_pad <= WIDE_NDUAL ? 3 : 2;
    return (size_t)WIDE_RING_AT + b_stages * (size_t)wide_stage_stride(n_pad);
}

// The tensor map of a weight matrix: 2-D over 32-bit words, [rows][units * 36], box 128 rows x 36 words (one block).
// Encoding goes through the driver entry point (no link against libcuda); maps are kept per (address, shape).
static cudaError_t wide_weight_map(const uint8_t* w, int64_t rows, int units, CUtensorMap* out) {
    typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                 const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static std::mutex mu;
    static EncodeFn encode = nullptr;
    struct Key {
        const void* p;
        int64_t rows;
        int units;
        bool operator<(const Key& o) const { return p != o.p ? p < o.p : rows != o.rows ? rows < o.rows : units < o.units; }
    };
    static std::map<Key, CUtensorMap> cache;
    std::lock_guard<std::mutex> lock(mu);
    if (!encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres);
        if (e != cudaSuccess) return e;
        if (!fn || qres != cudaDriverEntryPointSuccess) return cudaErrorNotSupported;
        encode = reinterpret_cast<EncodeFn>(fn);
    }
    const Key key{w, rows, units};
    auto it = cache.find(key);
    if (it == cache.end()) {
        if (cache.size() > 8192) cache.clear();
        CUtensorMap m;
        const cuuint64_t gdim[2] = {(cuuint64_t)units * 36, (cuuint64_t)rows};
        const cuuint64_t gstride[1] = {(cuuint64_t)units * 144};
        const cuuint32_t box[2] = {36, (cuuint32_t)WM};
        const cuuint32_t estride[2] = {1, 1};
        if (encode(&m, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<uint8_t*>(w), gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
        it = cache.emplace(key, m).first;
    }
    *out = it->second;
    return cudaSuccess;
}

cudaError_t launch_gemm_wide_q4k(tsb_ctx* ctx, cudaStream_t st, const uint8_t* w, int64_t rows, int64_t cols, const __half* x,
                                 int64_t x_stride, int tokens, void* y, int64_t y_stride, bool y_f32, void* workspace, void* partials) {
    const int units = (int)(cols / 256);
    static SmemOptIn configured1, configured2, configured3;
    const size_t smem_max = std::max(wide_smem_bytes(WIDE_NDUAL), wide_smem_bytes(WIDE_NMAX));
    if (cudaError_t e = tsb_opt_in_smem(ctx, gemm_wide_q4k_kernel<2, false>, smem_max, configured1); e != cudaSuccess) return e;
    if (cudaError_t e = tsb_opt_in_smem(ctx, gemm_wide_q4k_kernel<4, false>, smem_max, configured2); e != cudaSuccess) return e;
    if (cudaError_t e = tsb_opt_in_smem(ctx, gemm_wide_q4k_kernel<4, true>, smem_max, configured3); e != cudaSuccess) return e;
    static std::atomic<int> launch_regs{0};  // what the register shares are drawn on
    if (launch_regs.load() == 0) {
        cudaFuncAttributes a1, a2, a3;
        if (cudaError_t e = cudaFuncGetAttributes(&a1, gemm_wide_q4k_kernel<2, false>); e != cudaSuccess) return e;
        if (cudaError_t e = cudaFuncGetAttributes(&a2, gemm_wide_q4k_kernel<4, false>); e != cudaSuccess) return e;
        if (cudaError_t e = cudaFuncGetAttributes(&a3, gemm_wide_q4k_kernel<4, true>); e != cudaSuccess) return e;
        launch_regs = std::min(a1.numRegs, std::min(a2.numRegs, a3.numRegs));
    }
    if (launch_regs.load() < WIDE_LAUNCH_REGS) return cudaErrorLaunchOutOfResources;
    CUtensorMap wmap;
    if (cudaError_t e = wide_weight_map(w, rows, units, &wmap); e != cudaSuccess) return e;
    // token rows go through in equal passes of at most WIDE_NMAX; one launch lays out the operand of every pass
    const int passes = (tokens + WIDE_NMAX - 1) / WIDE_NMAX, n_pad = wide_pass_rows(tokens);
    const size_t pass_chunks = (size_t)units * WIDE_CHUNKS * n_pad;
    uint4* xw = static_cast<uint4*>(workspace);
    if (!workspace)
        if (cudaError_t e = cudaMallocAsync((void**)&xw, pass_chunks * passes * 16, st); e != cudaSuccess) return e;
    cudaError_t e = cudaSuccess;
    if (x)
        e = tsb_launch(ctx, wide_prepare_kernel, dim3((unsigned)units, (unsigned)(passes * (n_pad >> 3))), dim3(256), 0, st, true, x, x_stride, tokens, n_pad,
                       units, xw);
    const WidePlan plan = wide_plan(ctx->sm_count, rows, units);
    const int n_tiles = (int)(rows / WM), ksplit = plan.ksplit;
    const size_t smem = wide_smem_bytes(n_pad);
    if (wide_takes_many(plan, ctx->sm_count, n_tiles, units, passes)) {
        // one CTA per SM: the kernel wants the whole tensor memory and most of the shared memory
        const dim3 grid((unsigned)min(n_tiles * passes, ctx->sm_count));
        if (e == cudaSuccess)
            e = tsb_launch(ctx, gemm_wide_q4k_kernel<4, true>, grid, dim3(WIDE_THREADS), smem, st, true, wmap, rows, units, (const uint4*)xw, n_pad, tokens, passes, y,
                           y_stride, (int)(y_f32 ? 1 : 0), plan.n_whole, ksplit, (float*)nullptr, ctx->dev_error);
    } else {
        float* part = static_cast<float*>(partials);
        const bool own_part = ksplit > 1 && !part;
        if (own_part && e == cudaSuccess) {
            e = cudaMallocAsync((void**)&part, 4096 + (size_t)ksplit * WIDE_NMAX * plan.tail_rows * sizeof(float), st);
            if (e == cudaSuccess) e = cudaMemsetAsync(part, 0, 4096, st);  // the ticket words start at zero
        }
        const dim3 grid((unsigned)min(plan.n_whole + (n_tiles - plan.n_whole) * ksplit, ctx->sm_count));
        for (int pass = 0; pass < passes && e == cudaSuccess; pass++) {
            const int t0 = pass * n_pad, nt = min(n_pad, tokens - t0);
            if (nt <= 0) break;
            uint8_t* yp = static_cast<uint8_t*>(y) + (size_t)t0 * y_stride * (y_f32 ? 4 : 2);
            auto kernel = n_pad <= WIDE_NDUAL ? gemm_wide_q4k_kernel<2, false> : gemm_wide_q4k_kernel<4, false>;
            e = tsb_launch(ctx, kernel, grid, dim3(WIDE_THREADS), smem, st, true, wmap, rows, units, (const uint4*)(xw + pass * pass_chunks), n_pad, nt, 1, (void*)yp,
                           y_stride, (int)(y_f32 ? 1 : 0), plan.n_whole, ksplit, part, ctx->dev_error);
        }
        if (own_part && part) cudaFreeAsync(part, st);
    }
    if (!workspace) cudaFreeAsync(xw, st);
    return e;
}
