// A few to a few hundred activation rows: y[M][N] = x[M][K] * W[N][K]^T straight from the NF4 units,
// one pass over the weights, no bf16 copy of W in memory. Two forms of one kernel:
//   NS = 0   (49 rows and more) operand bf16(code_book[nibble] * absmax), sums over K in tensor memory: the
//            weights of the dequantise + GEMM route
//   NS > 0   (up to 16, 32 or 48 rows) block-scaled: operand bf16(code_book[nibble]), every 64-block's sum by
//            itself in tensor memory, times the fp32 absmax added up in registers: the arithmetic of the
//            small-batch decode kernels. A decode thread adds up a quarter of its row's columns (the group's),
//            so it needs the absmax of all four blocks of a chunk: through the unused half of the table's
//            lines. Block sums have two sets of tensor-memory columns up to 32 rows, one at 48. (With all
//            columns of the group's own block per thread the loop spilled, and 33..48 rows took two passes:
//            twelve layers at 32 rows 643 us against 584, down at 40 rows 24.5 against 13.4.)
//
// The weight is the A operand of tcgen05.mma and lives in TENSOR MEMORY: a decode thread owns one
// output row of a 128-row tile, reads the row's 32 nibble bytes of a 64-wide block (coalesced: a
// unit keeps the rows of a block back to back), rebuilds the 64 weights as
// bf16(code_book[nibble] * absmax) - the same two fp32 operations and one rounding as
// dequantize_weight - and writes them with tcgen05.st as one row of the operand. There is no swizzle
// to respect. The activations (at most 256 rows a launch) are the B operand, fetched by TMA into a
// shared-memory ring; the accumulator is [128 weight rows][activation rows] fp32 in tensor memory.
//
//   warp 0       TMA producer (x blocks of 64 columns)
//   warp 1       tensor-memory allocation, one thread issues the MMAs
//   warps 2, 3   idle (a warp reaches the tensor-memory lanes 32 * (warp % 4) only)
//   warps 4..19  four groups of four: the CTA's (row tile, 64-block) items go in chunks of up to four
//                consecutive blocks of a tile, group g decodes the g-th block of a chunk into slot g of one
//                of two operand sets; all sixteen drain the accumulator
//
// Bound: shared-memory bandwidth of the decode (a byte, two weights, is one 8-byte load from a
// bank-private table of fp32 pairs: 1024 cycles a chunk) beside x arriving and being read by the tensor
// core, and the fixed cost of a launch: about 2 us of set-up, 1.5 us until the first x block, 3 us to
// finish a tile. One wait and one commit of the issuing thread serve a whole chunk: a barrier test (about
// 150 cycles), a commit (200) and four MMAs (130) are what an item costs that thread; item by item the
// loop ran at 0.45 us per item, chunk by chunk at 0.30 us. The weights arrive by cp.async, 32 contiguous
// pieces per instruction, three items ahead (loads into registers did not stay in flight: 0.5 us per item).
//
// Linears of a 2560-wide layer (o 2560x4096, down 2560x9728, gate|up 19456x2560), us per call, against
// the batched decode kernels (32 rows) and dequantise + GEMM (77 rows and more):
//   rows   o            down          gate|up
//     32    8.6 (14.1)  12.3 (21.0)   20.7 (32.0)
//     77    9.2 (27.7)  13.1 (58.3)   23.8 (45.0)
//    256   14.1 (28.8)  19.8 (59.5)   37.2 (52.1)
//
// Two splits of the (row tile, 64-block) items, chosen by choose_split():
//   cluster  a row tile belongs to a cluster of 1..8 CTAs, each with an equal part of K; the partial
//            tiles meet through distributed shared memory, every CTA finishing a share of the columns.
//            For outputs of few tiles (o, down, qkv).
//   stream   items in tile-major order are cut into equal contiguous ranges, one per CTA, one CTA per SM,
//            through tiles and K alike. A tile that one CTA holds completely is finished from tensor
//            memory; otherwise each CTA writes its fp32 partial tile to the scratch and the LAST to
//            arrive (a counter per tile, nobody waits) adds the parts in CTA order. For tall outputs
//            (gate|up), whose tiles are shared by two CTAs at most.
// Either way every sum has a fixed order: the results are bit-reproducible.
#include <cooperative_groups.h>
#include <cuda.h>

#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "nf4_internal.h"
#include "nf4_tma.h"

namespace nf4 {

namespace {

constexpr int kTileM = 128;        // weight rows of a tile (tensor-memory lanes)
constexpr int kGroups = 4;         // decode groups of four warps
constexpr int kDecodeWarps = 4 * kGroups;
constexpr int kFirstDecodeWarp = 4;
constexpr int kThreads = 32 * (kFirstDecodeWarp + kDecodeWarps);
constexpr int kSets = 2;                 // operand sets of kGroups slots in tensor memory
constexpr int kSlotCols = kUnitK / 2;    // 64 bf16 per lane = 32 columns
constexpr int kSlotCol0 = 256;           // accumulators below, operand slots from here
constexpr int kMaxX = kSets * kGroups;   // blocks of x in the ring at most
constexpr uint32_t kLutBytes = 65536u;   // look-up table, at the first shared address that is a multiple of 64 KB
constexpr uint32_t kXRing = 131072u;     // the x ring behind it starts here at the latest, counted from the CTA's first byte
constexpr uint32_t kPart = 65536u;       // a cluster's partial tiles, at the same place in every CTA
constexpr uint32_t kPartScaled = 131072u;  // the same in the block-scaled form (the table's lines hold absmax values)
constexpr int kSmem = 227 * 1024;
constexpr int kHeadBytes = 2048;         // barriers, code books
constexpr int kDepth = 3;                // items a decode warp has in flight
constexpr int kSlotBytes = 2 * kUnitStrideF32;  // one warp's part of an item: two units at most
constexpr uint32_t kRingEnd = kHeadBytes + kDecodeWarps * kDepth * kSlotBytes;
static_assert(2048 + kRingEnd <= 65536, "weight ring below the table");
static_assert(kPart + kTileM * 256 * 4 <= kSmem, "a partial tile of 256 columns");

struct MidParams {
    const uint8_t* units;
    const float* qmap;
    const float* nmap;
    const float4* row_scales;
    const uint16_t* residual;
    uint16_t* y;
    float* partials;  // two tiles of [NB/4][128][4] floats per CTA
    int* counters;    // per tile, zero between launches
    int* status;
    long long limit;
    int KU, RT, n_rows, unit_stride, kind;
    int M, NB;        // activation rows; rounded up to 16
    int n_out;        // row pitch of y
    int ff;           // 0, or gate|up rows of each half
    int n_tiles;
    int x_stages;
    int x_per_item;   // 0: an x stage holds a chunk's kGroups blocks; 1: stages of one block (wide x)
    int split;        // 0: stream; else CTAs per tile (cluster size)
    uint32_t idesc;
};

__device__ __forceinline__ uint64_t x_desc(uint32_t saddr) {  // K-major, 128-byte swizzle
    return (uint64_t)((saddr & 0x3FFFF) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ void commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

// Four or eight columns without a wait: the values are there after tmem_landed() on them.
__device__ __forceinline__ void tmem_ld_start(uint32_t addr, uint32_t* r, std::integral_constant<int, 4>) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void tmem_ld_start(uint32_t addr, uint32_t* r, std::integral_constant<int, 8>) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(addr) : "memory");
}
__device__ __forceinline__ void tmem_ld_start(uint32_t addr, uint32_t* r, std::integral_constant<int, 12>) {
    tmem_ld_start(addr, r, std::integral_constant<int, 8>{});
    tmem_ld_start(addr + 8, r + 8, std::integral_constant<int, 4>{});
}
template <int N>
__device__ __forceinline__ void tmem_landed(uint32_t (&r)[N]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < N; ++i) asm volatile("" : "+r"(r[i]));  // (no use before the wait)
}

__device__ __forceinline__ void tmem_ld8(uint32_t addr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
        : "r"(addr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// Bounded wait without back-off: the chain decode -> MMA -> free slot is latency-critical. The limit counts
// from the end of the launch before, which this kernel is resident beside (x cannot arrive earlier): a wait
// that runs out waits for that launch once and starts its clock again.
__device__ __forceinline__ bool wait_spin(uint64_t* bar, uint32_t parity, long long limit, volatile int* abort_flag) {
    if (mbar_try_wait(bar, parity)) return true;
    long long t0 = clock64();
    bool alone = false;
    const int tries = limit < 100000 ? 4 : 256;  // between two looks at the clock: a fraction of the limit
    while (true) {
#pragma unroll 1
        for (int i = 0; i < tries; ++i)
            if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (clock64() - t0 > limit) {
            if (alone) return false;
            asm volatile("griddepcontrol.wait;" ::: "memory");
            alone = true;
            t0 = clock64();
        }
    }
}

// Two weights: byte `I` of `word` through the lane's column of the table, times absmax, one rounding.
template <int I>
__device__ __forceinline__ uint32_t decode2(uint32_t word, uint32_t lut_lane, uint64_t am2) {
    uint32_t addr;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(addr) : "r"(word), "r"(lut_lane), "n"(0x7604 | (I << 4)));
    uint64_t q;
    asm("ld.shared.b64 %0, [%1];" : "=l"(q) : "r"(addr));
    asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(q) : "l"(am2));
    uint32_t r;
    asm("{\n\t.reg .f32 a, b;\n\tmov.b64 {a, b}, %1;\n\tcvt.rn.bf16x2.f32 %0, b, a;\n\t}" : "=r"(r) : "l"(q));
    return r;
}

// The same byte as two code-book values rounded to bf16 (block-scaled form).
template <int I>
__device__ __forceinline__ uint32_t lookup2(uint32_t word, uint32_t lut_lane) {
    uint32_t addr, r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(addr) : "r"(word), "r"(lut_lane), "n"(0x7604 | (I << 4)));
    asm("ld.shared.u32 %0, [%1];" : "=r"(r) : "r"(addr));
    return r;
}

__device__ __forceinline__ uint4 lds_v4(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}

// Finished sums of one accumulator lane (columns m0 .. m0 + C - 1) to the output.
template <int C>
__device__ __forceinline__ void emit(const MidParams& p, int tile, int quarter, int lane, int m0, const float (&v)[C]) {
    const int upper = lane >> 4;
    if (p.ff > 0) {
        // lanes 0..15 hold gate rows, 16..31 the matching up rows: of each pair of columns the lower
        // half-warp finishes the first, the upper half-warp the second
        const int nn = tile * 64 + quarter * 16 + (lane & 15);
#pragma unroll
        for (int k = 0; k < C; k += 2) {
            const float other = __shfl_xor_sync(0xffffffffu, upper ? v[k] : v[k + 1], 16);
            const float gate = upper ? other : v[k], up = upper ? v[k + 1] : other;
            // gate and up pass through bf16 first, like a bf16 gate_up buffer
            const float g = bf16_bits_to_f32(f32_to_bf16_bits(gate));
            const float u = bf16_bits_to_f32(f32_to_bf16_bits(up));
            const int m = m0 + k + upper;
            if (m < p.M && nn < p.ff)
                p.y[(size_t)m * p.n_out + nn] = f32_to_bf16_bits(__fdividef(g, 1.0f + __expf(-g)) * u);
        }
    } else {
        // (the residual by a plain load: the launch before is visible behind griddepcontrol.wait, to coherent loads)
        const int nn = tile * kTileM + quarter * 32 + lane;
        if (nn >= p.n_out) return;
#pragma unroll
        for (int k = 0; k < C; ++k) {
            if (m0 + k < p.M) {
                const size_t at = (size_t)(m0 + k) * p.n_out + nn;
                p.y[at] = f32_to_bf16_bits(p.residual ? v[k] + bf16_bits_to_f32(p.residual[at]) : v[k]);
            }
        }
    }
}

// NS = 0: operands bf16(code_book[nibble] * absmax), summed over K in tensor memory. NS = 16, 32 or 48 (the
// activation rows, rounded up): block-scaled, see the head of the file.
template <int NS>
__global__ void __launch_bounds__(kThreads, 1)
gemm_midrows_kernel(const __grid_constant__ CUtensorMap map_x, const MidParams p) {
    extern __shared__ __align__(1024) uint8_t mid_smem[];
    constexpr int kSumSets = NS <= 32 ? 2 : 1;  // sets of block sums in tensor memory (256 columns)
    constexpr int C = NS > 0 ? NS / kGroups : 8;  // block-scaled: columns of a row that a decode thread adds up
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t base = smem_u32(mid_smem);
    // The table's lines are found by inserting a byte into an address, so it starts at a multiple of 64 KB of
    // the address itself, whatever the upper bits of a CTA's shared addresses are in a cluster; everything
    // else is counted from the CTA's first byte.
    const uint32_t lut = (base + 0xffffu) & ~0xffffu;
    const uint32_t lut_off = lut - base;
    uint64_t* x_full = reinterpret_cast<uint64_t*>(mid_smem);
    uint64_t* x_empty = x_full + kMaxX;
    uint64_t* a_full = x_empty + kMaxX;     // [kSets]
    uint64_t* done = a_full + kSets;        // [kSets] the MMAs of the set's chunk are through
    uint64_t* acc_full = done + kSets;    // [2]
    uint64_t* acc_empty = acc_full + 2;     // [2]
    uint64_t* drain = acc_empty + 2;
    uint64_t* join_bar = drain + 1;         // [2] every decode warp has written its part; s_last is known
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(join_bar + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* s_last = abort_flag + 1;
    float* s_nmap = reinterpret_cast<float*>(mid_smem + 1024);  // [256]

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int KB = p.KU;
    // (requested first, used when the tables are built)
    const float q_lane = __ldg(p.qmap + (lane & 15));
    const float n_mine = p.kind == kAbsmaxCodes && tid < 256 ? __ldg(p.nmap + tid) : 0.0f;
    const uint32_t x_bytes = (uint32_t)p.NB * 128u;
    auto x_stage = [&](int s) { return lut_off + kLutBytes + (uint32_t)s * x_bytes; };
    // (the dynamic shared memory starts at most 2 KB behind a multiple of 64 KB)
    if (lut_off < kRingEnd || lut_off + kLutBytes + (uint32_t)p.x_stages * x_bytes > kSmem) {
        if (tid == 0) atomicExch(p.status, kStatusBadArgument);
        if (p.split > 1) {  // (the rest of the cluster may look at this CTA's memory)
            cooperative_groups::this_cluster().sync();
            cooperative_groups::this_cluster().sync();
        }
        return;
    }
    // this CTA's items [i0, i0 + n)
    const int c = blockIdx.x;
    int q = 0, r = 0, i0, n;
    if (p.split > 0) {
        const int tile = c / p.split, rank = c - tile * p.split;
        const int k0 = KB * rank / p.split;
        i0 = tile * KB + k0;
        n = KB * (rank + 1) / p.split - k0;
    } else {
        const int total = p.n_tiles * KB, G = gridDim.x;
        q = total / G;
        r = total - q * G;
        i0 = c * q + min(c, r);
        n = q + (c < r ? 1 : 0);
    }

    // ---- decode warps: weights through a private ring of asynchronous copies ----
    const int dw = max(warp - kFirstDecodeWarp, 0), quarter = dw & 3, grp = dw >> 2;
    const int row16 = lane & 15, upper = lane >> 4;
    const int ff_rt = p.ff / kTileRows;
    // 16-row unit of this lane in tile `t`, clamped (rows past the weight are never written back)
    auto unit_rt = [&](int t) {
        if (p.ff > 0) return min(t * 4 + quarter, ff_rt - 1) + (upper ? ff_rt : 0);
        return min(t * 8 + quarter * 2 + upper, p.RT - 1);
    };
    const size_t ST = (size_t)p.unit_stride;
    const uint32_t ring = base + kHeadBytes + (uint32_t)(dw * kDepth * kSlotBytes);
    // A warp's item is two units (its lanes' rows 0..15 and 16..31): each copied as 32 contiguous pieces of
    // 16 bytes and, behind both, one piece (codes) or four (fp32) of absmax a unit. The two pieces of a row
    // change places in every other group of four rows, so that eight rows' pieces fall into different banks.
    const int scale_bytes = p.kind == kAbsmaxCodes ? kTileRows : 4 * kTileRows;
    const uint32_t piece = (uint32_t)((lane & ~1) + ((lane & 1) ^ ((lane >> 3) & 1))) * 16u;
    auto unit0_rt = [&](int t) { return p.ff > 0 ? min(t * 4 + quarter, ff_rt - 1) : min(t * 8 + quarter * 2, p.RT - 1); };
    auto unit1_rt = [&](int t) {
        return p.ff > 0 ? min(t * 4 + quarter, ff_rt - 1) + ff_rt : min(t * 8 + quarter * 2 + 1, p.RT - 1);
    };
    // the next block this warp fetches: block pf_kb of tile pf_tile, of this CTA's part [.., pf_end) of the
    // tile; pf_left items of the CTA lie in later tiles
    int pf_tile = i0 / KB, pf_kb = i0 - pf_tile * KB, pf_slot = 0;
    int pf_end = min(KB, pf_kb + n), pf_left = n - (pf_end - pf_kb);
    pf_kb += grp;
    const uint8_t* pf_u0 = p.units + (size_t)unit0_rt(pf_tile) * KB * ST;
    size_t pf_u1 = (size_t)(unit1_rt(pf_tile) - unit0_rt(pf_tile)) * KB * ST;  // from unit 0 to unit 1
    auto row_scale = [&](int tile) {
        return p.kind == kAbsmaxCodes ? __ldg(p.row_scales + min(unit_rt(tile) * kTileRows + row16, p.n_rows - 1))
                                      : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    };
    float4 e_next = row_scale(pf_tile);
    auto cp16 = [](uint32_t dst, const uint8_t* src) {
        asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    };
    auto fetch = [&]() {  // this warp's next item into its next ring slot; one commit group either way
        while (pf_kb >= pf_end && pf_left > 0) {
            ++pf_tile;
            pf_kb = grp;
            pf_end = min(KB, pf_left);
            pf_left -= pf_end;
            pf_u0 = p.units + (size_t)unit0_rt(pf_tile) * KB * ST;
            pf_u1 = (size_t)(unit1_rt(pf_tile) - unit0_rt(pf_tile)) * KB * ST;
        }
        if (pf_kb < pf_end) {
            const uint8_t* u = pf_u0 + (size_t)pf_kb * ST;
            const uint32_t dst = ring + (uint32_t)(pf_slot * kSlotBytes);
            cp16(dst + piece, u + lane * 16);
            cp16(dst + 512 + piece, u + pf_u1 + lane * 16);
            const int at = lane * 16;  // of both units' absmax bytes
            if (at < 2 * scale_bytes)
                cp16(dst + 1024 + at, u + kUnitNibbleBytes + (at < scale_bytes ? at : pf_u1 + at - scale_bytes));
            pf_kb += kGroups;
        }
        pf_slot = pf_slot == kDepth - 1 ? 0 : pf_slot + 1;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (warp >= kFirstDecodeWarp)
        for (int b = 0; b < kDepth; ++b) fetch();  // in flight before anything else

    if (tid == 0) {
        for (int s = 0; s < kMaxX; ++s) {
            mbar_init(&x_full[s], 1);
            mbar_init(&x_empty[s], 1);
        }
        for (int s = 0; s < kSets; ++s) {
            mbar_init(&a_full[s], kDecodeWarps);
            mbar_init(&done[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], kDecodeWarps);
        }
        mbar_init(drain, 1);
        mbar_init(&join_bar[0], kDecodeWarps);
        mbar_init(&join_bar[1], 1);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid < 256) s_nmap[tid] = n_mine;
    if constexpr (NS > 0) {
        // look-up table: entry e of lane l at e * 256 + l * 4 = bf16 {value of e's high nibble, of its low nibble}
        for (int i = tid; i < 256 * 8; i += kThreads) {  // (whole warps)
            const int e = i >> 3;
            const float hi = __shfl_sync(0xffffffffu, q_lane, e >> 4), lo = __shfl_sync(0xffffffffu, q_lane, e & 15);
            const uint32_t w = f32x2_to_bf16x2_bits(hi, lo);
            *reinterpret_cast<uint4*>(mid_smem + lut_off + (uint32_t)e * 256u + (uint32_t)(i & 7) * 16u) =
                make_uint4(w, w, w, w);
        }
    } else {
        // look-up table: entry e of lane l at e * 256 + l * 8 = {value of e's high nibble, of its low nibble}
        for (int i = tid; i < 256 * 16; i += kThreads) {  // (whole warps)
            const int e = i >> 4;
            const float hi = __shfl_sync(0xffffffffu, q_lane, e >> 4), lo = __shfl_sync(0xffffffffu, q_lane, e & 15);
            *reinterpret_cast<float4*>(mid_smem + lut_off + (uint32_t)i * 16u) = make_float4(hi, lo, hi, lo);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    const int bufs = p.NB <= 128 ? 2 : 1;  // accumulator buffers of 128 (or one of 256) columns

    auto give_up = [&](int code) {
        if (!*abort_flag) atomicExch(p.status, code);
        *abort_flag = 1;
    };

    if (warp == 0) {
        if (elect_one()) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            int kb = i0 % KB;
            bool ok = true;
            if (p.x_per_item) {
                int s = 0, i = 0;
                uint32_t ph = 0;
                for (; i < n && ok; ++i) {
                    if (i >= p.x_stages) ok = wait_spin(&x_empty[s], ph, p.limit, abort_flag);
                    if (!ok) break;
                    mbar_expect_tx(&x_full[s], x_bytes);
                    tma_load_2d(mid_smem + x_stage(s), &map_x, kb * kUnitK, 0, &x_full[s]);
                    if (++kb == KB) kb = 0;
                    if (++s == p.x_stages) {
                        s = 0;
                        if (i >= p.x_stages) ph ^= 1u;
                    }
                }
                // copies issued by this thread must have landed before the CTA exits
                for (int g = max(0, i - p.x_stages); g < i; ++g)
                    mbar_wait_bounded(&x_full[g % p.x_stages], (g / p.x_stages) & 1);
            } else {
                int ch = 0;
                for (int left = n; left > 0; ++ch) {
                    const int set = ch & 1, size = min(min(kGroups, KB - kb), left);
                    if (ch >= kSets) ok = wait_spin(&done[set], ((ch >> 1) - 1) & 1, p.limit, abort_flag);
                    if (!ok) break;
                    mbar_expect_tx(&x_full[set], (uint32_t)size * x_bytes);
                    for (int k = 0; k < size; ++k)
                        tma_load_2d(mid_smem + x_stage(set * kGroups + k), &map_x, (kb + k) * kUnitK, 0, &x_full[set]);
                    left -= size;
                    kb = kb + size == KB ? 0 : kb + size;
                }
                for (int g = max(0, ch - kSets); g < ch; ++g) mbar_wait_bounded(&x_full[g & 1], (g >> 1) & 1);
            }
            if (!ok) give_up(kStatusTimeoutEmpty);
        }
        __syncwarp();
    } else if (warp == 1) {
        if (elect_one()) {
            int s = 0, seg = 0, ch = 0, kb = i0 % KB;
            uint32_t xph = 0;
            bool ok = true;
            for (int left = n; left > 0 && ok; ++seg) {
                const int b = seg % bufs;
                const uint32_t d = tmem + (uint32_t)(b * 128);
                if (NS == 0 && seg >= bufs && !wait_spin(&acc_empty[b], ((seg / bufs) - 1) & 1, p.limit, abort_flag)) {
                    give_up(kStatusTimeoutTmem);
                    break;
                }
                int len = min(left, KB - kb);  // this CTA's part of the tile
                left -= len;
                kb = 0;
                uint32_t acc = 0;
                for (; len > 0; len -= kGroups, ++ch) {
                    const int set = ch & 1;
                    const uint32_t ph = (ch >> 1) & 1;
                    if (p.x_per_item) {
                        ok = wait_spin(&a_full[set], ph, p.limit, abort_flag);
                    } else {  // (both tests in flight together)
                        const bool ra = mbar_try_wait(&a_full[set], ph), rx = mbar_try_wait(&x_full[set], ph);
                        ok = (ra || wait_spin(&a_full[set], ph, p.limit, abort_flag)) &&
                             (rx || wait_spin(&x_full[set], ph, p.limit, abort_flag));
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int k = 0; k < kGroups; ++k) {
                        if (k < len && ok) {
                            const int st = p.x_per_item ? s : set * kGroups + k;
                            if (p.x_per_item) ok = wait_spin(&x_full[s], xph, p.limit, abort_flag);
                            if (ok) {
                                const uint64_t bd = x_desc(base + x_stage(st));
                                const uint32_t a = tmem + kSlotCol0 + (uint32_t)((set * kGroups + k) * kSlotCols);
                                if constexpr (NS > 0) {  // a sum of its own for every block
                                    const uint32_t db = tmem + (uint32_t)(((kSumSets == 2 ? set : 0) * kGroups + k) * NS);
#pragma unroll
                                    for (int j = 0; j < 4; ++j) mma_ts(db, a + 8 * j, bd + 2 * j, p.idesc, j > 0);
                                } else {
#pragma unroll
                                    for (int j = 0; j < 4; ++j) {
                                        mma_ts(d, a + 8 * j, bd + 2 * j, p.idesc, acc);
                                        acc = 1u;
                                    }
                                }
                                if (p.x_per_item) {
                                    commit(&x_empty[s]);
                                    if (++s == p.x_stages) {
                                        s = 0;
                                        xph ^= 1u;
                                    }
                                }
                            }
                        }
                    }
                    if (!ok) {
                        give_up(kStatusTimeoutFull);
                        break;
                    }
                    commit(&done[set]);
                }
                if (NS == 0 && ok) commit(&acc_full[b]);
            }
            // no MMA is in flight when tensor and shared memory are given up
            commit(drain);
            mbar_wait_bounded(drain, 0);
        }
        __syncwarp();
    } else if (warp >= kFirstDecodeWarp) {
        const uint32_t lut_lane = lut + (uint32_t)lane * (NS > 0 ? 4u : 8u);
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        bool ok = true;
        float4 e = e_next;
        int ch = 0;      // chunk
        int c_slot = 0;  // ring slot of the next item
        // Block-scaled: the lane's row of the CTA's part of the tile, the group's columns; how many blocks the
        // chunk before has (1) and the one before that (2), where their sums are still to be added.
        float acc[C];
        int len1 = 0, len2 = 0;
        // absmax of block k of chunk c, in the unused half of the table's lines: four chunks deep, a warp that
        // writes chunk c has seen every warp through with chunk c - 4
        auto am_at = [&](int c, int k) { return lut + (uint32_t)((((c & 3) * kGroups + k) * 4 + quarter) * 256 + 128 + lane * 4); };
        auto add_blocks = [&](int c, int len) {  // absmax times block sum, blocks in order
            ok = wait_spin(&done[c & 1], (c >> 1) & 1, p.limit, abort_flag) &&
                 wait_spin(&a_full[c & 1], (c >> 1) & 1, p.limit, abort_flag);  // (over: orders the absmax values)
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) return;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t src = tmem + lane_off + (uint32_t)((kSumSets == 2 ? c & 1 : 0) * kGroups * NS + grp * C);
#pragma unroll
            for (int k0 = 0; k0 < kGroups; k0 += 2) {
                uint32_t v[2 * C];
                tmem_ld_start(src + (uint32_t)(k0 * NS), v, std::integral_constant<int, C>{});
                tmem_ld_start(src + (uint32_t)((k0 + 1) * NS), v + C, std::integral_constant<int, C>{});
                float am[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(am[k]) : "r"(am_at(c, k0 + k)));
                tmem_landed(v);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    if (k0 + k < len) {
#pragma unroll
                        for (int i = 0; i < C; ++i) acc[i] = fmaf(am[k], __uint_as_float(v[k * C + i]), acc[i]);
                    }
                }
            }
        };
        auto give_up_decoding = [&]() {
            if (lane == 0) give_up(kStatusTimeoutEmpty);
        };
        // the warp's part of one chunk of `len` blocks: block kb, or nothing (the chunk is short)
        auto chunk = [&](int kb, bool have, int len) {
            const int set = ch & 1;
            // the set's previous operands have been used; block-scaled: and their sums added, so that all of the
            // set is free when this warp arrives
            auto free_set = [&]() {
                if (NS > 0 && kSumSets == 2) {
                    if (len2 > 0) add_blocks(ch - 2, len2);
                } else if (NS > 0) {  // one set of sums: those of the chunk before
                    if (len1 > 0) add_blocks(ch - 1, len1);
                } else if (ch >= kSets) {
                    ok = wait_spin(&done[set], ((ch >> 1) - 1) & 1, p.limit, abort_flag);
                    ok = __all_sync(0xffffffffu, ok);
                }
                if (!ok) give_up_decoding();
                return ok;
            };
            if (kSumSets == 2 && !free_set()) return;
            if (NS == 0 && !have) {  // (nothing to publish)
                ++ch;
                if (lane == 0) mbar_arrive(&a_full[set]);
                return;
            }
            const uint32_t dst = tmem + lane_off + kSlotCol0 + (uint32_t)((set * kGroups + grp) * kSlotCols);
            if (have) {
                asm volatile("cp.async.wait_group %0;" ::"n"(kDepth - 1) : "memory");
                __syncwarp();  // (every lane's copies have landed)
                const uint32_t src = ring + (uint32_t)(c_slot * kSlotBytes);
                c_slot = c_slot == kDepth - 1 ? 0 : c_slot + 1;
                const uint32_t mine = src + (uint32_t)(lane * 32), flip = (uint32_t)((row16 >> 2) & 1) * 16u;
                const uint4 wa = lds_v4(mine + flip), wb = lds_v4(mine + (16u - flip));
                float am;
                if (p.kind == kAbsmaxCodes) {
                    uint32_t code;
                    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(code) : "r"(src + 1024 + lane));
                    am = __fadd_rn(__fmul_rn(s_nmap[code], kb >= __float_as_int(e.z) ? e.y : e.x), e.w);
                } else {
                    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(am) : "r"(src + 1024 + 4 * lane));
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                // stored byte 8 t + 2 j + e covers k = 16 j + 4 t + 2 e: operand column 8 j + 2 t + e
                const uint32_t ws[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
                uint64_t am_pair;
                asm("mov.b64 %0, {%1, %1};" : "=l"(am_pair) : "f"(am));
                if constexpr (NS > 0) asm volatile("st.shared.f32 [%0], %1;" ::"r"(am_at(ch, grp)), "f"(am) : "memory");
                auto pair = [&](auto byte, uint32_t word) {
                    if constexpr (NS > 0) return lookup2<decltype(byte)::value>(word, lut_lane);
                    else return decode2<decltype(byte)::value>(word, lut_lane, am_pair);
                };
                using B0 = std::integral_constant<int, 0>;
                using B1 = std::integral_constant<int, 1>;
                using B2 = std::integral_constant<int, 2>;
                using B3 = std::integral_constant<int, 3>;
                uint32_t o[16];
#pragma unroll
                for (int t = 0; t < 4; ++t) {  // j = 0, 1: the low words of the 8-byte chunks
                    o[2 * t + 0] = pair(B0{}, ws[2 * t]);
                    o[2 * t + 1] = pair(B1{}, ws[2 * t]);
                    o[8 + 2 * t + 0] = pair(B2{}, ws[2 * t]);
                    o[8 + 2 * t + 1] = pair(B3{}, ws[2 * t]);
                }
                tmem_st16(dst, o);
                uint32_t o2[16];
#pragma unroll
                for (int t = 0; t < 4; ++t) {  // j = 2, 3: the high words
                    o2[2 * t + 0] = pair(B0{}, ws[2 * t + 1]);
                    o2[2 * t + 1] = pair(B1{}, ws[2 * t + 1]);
                    o2[8 + 2 * t + 0] = pair(B2{}, ws[2 * t + 1]);
                    o2[8 + 2 * t + 1] = pair(B3{}, ws[2 * t + 1]);
                }
                tmem_st16(dst + 16, o2);
                fetch();  // (every lane has used the slot's words: tcgen05.st is warp-wide)
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            }
            if (kSumSets == 1 && !free_set()) return;
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&a_full[set]);
            ++ch;
            len2 = kSumSets == 2 ? len1 : 0;
            len1 = NS > 0 ? len : 0;
        };

        const int chunks = (p.M + 7) >> 3;    // accumulator columns in use, in eights
        const int row = quarter * 32 + lane;  // lane of the accumulator
        int seg = 0;
        bool waited = false;
        uint32_t joins = 0;
        for (int ls = 0; ls < n && ok; ++seg) {
            const int tile = (i0 + ls) / KB;
            const int kb0 = (i0 + ls) - tile * KB;
            const int le = min(n, ls + KB - kb0);  // this CTA's part of the tile: local items [ls, le)
            e = e_next;
            if (le < n) e_next = row_scale(tile + 1);
            if constexpr (NS > 0) {
#pragma unroll
                for (int i = 0; i < C; ++i) acc[i] = 0.0f;
            }
            for (int j = 0; j < le - ls && ok; j += kGroups) chunk(kb0 + j + grp, j + grp < le - ls, min(kGroups, le - ls - j));
            if (!ok) break;
            // ---- the tile's sums: the last blocks', or the accumulator ----
            const int b = seg % bufs;
            if constexpr (NS > 0) {
                if (len2 > 0) add_blocks(ch - 2, len2);
                if (ok && len1 > 0) add_blocks(ch - 1, len1);
                len1 = len2 = 0;
            } else {
                ok = wait_spin(&acc_full[b], (seg / bufs) & 1, p.limit, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
            }
            if (!ok) {
                if (lane == 0) give_up(kStatusTimeoutTmem);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (!waited) {
                // the previous launch may still read what is written from here on (y, scratch)
                asm volatile("griddepcontrol.wait;" ::: "memory");
                waited = true;
            }
            const uint32_t dcol = tmem + lane_off + (uint32_t)(b * 128);
            // this thread's columns of the row, C at a time
            auto for_sums = [&](auto use) {
                if constexpr (NS > 0) {
                    use(grp * C, acc);
                } else {
                    for (int ch = grp; ch < chunks; ch += kGroups) {
                        float v[C];
                        tmem_ld8(dcol + (uint32_t)(ch * 8), v);
                        use(ch * 8, v);
                        __syncwarp();  // (lanes past the output left early; the next load is warp-wide)
                    }
                }
            };
            const bool whole = kb0 == 0 && le - ls == KB;
            const size_t part = (size_t)kTileM * p.NB;
            if (p.split <= 1 && whole) {
                for_sums([&](int m0, float (&v)[C]) { emit(p, tile, quarter, lane, m0, v); });
            } else {
                // partial tile, to shared memory (every copy, look-up and MMA of this CTA is through with
                // it) or to the scratch
                float4* o = p.split > 1 ? reinterpret_cast<float4*>(mid_smem + (NS > 0 ? kPartScaled : kPart))
                                        : reinterpret_cast<float4*>(p.partials + ((size_t)c * 2 + (kb0 == 0 ? 1 : 0)) * part);
                for_sums([&](int m0, float (&v)[C]) {
#pragma unroll
                    for (int i = 0; i < C; i += 4)
                        o[(size_t)(m0 + i) / 4 * kTileM + row] = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                });
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (NS == 0 && lane == 0) mbar_arrive(&acc_empty[b]);
            if (p.split == 0 && !whole) {
                const int t0 = tile * KB, t1 = t0 + KB - 1;  // first and last item of the tile
                const int big = r * (q + 1);
                const int c0 = t0 < big ? t0 / (q + 1) : r + (t0 - big) / q;
                const int c1 = t1 < big ? t1 / (q + 1) : r + (t1 - big) / q;
                __threadfence();
                __syncwarp();
                if (lane == 0) mbar_arrive(&join_bar[0]);
                // (bounded, unlike a named barrier: a warp that gave up does not come)
                if (dw == 0 && wait_spin(&join_bar[0], joins & 1, p.limit, abort_flag) && lane == 0) {
                    int old;
                    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;"
                                 : "=r"(old) : "l"(p.counters + tile) : "memory");
                    const int last = old == c1 - c0;
                    if (last) p.counters[tile] = 0;
                    *s_last = last;
                    mbar_arrive(&join_bar[1]);
                }
                __syncwarp();
                ok = wait_spin(&join_bar[1], joins & 1, p.limit, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                ++joins;
                if (!ok) {
                    if (lane == 0) give_up(kStatusTimeoutTmem);
                    break;
                }
                if (*s_last) {
                    __threadfence();
                    for (int ch = grp; ch < chunks; ch += kGroups) {
                        float v[8];
#pragma unroll
                        for (int k = 0; k < 8; ++k) v[k] = 0.0f;
                        const float* src = p.partials + (size_t)ch * 8 * kTileM + (size_t)row * 4;
#pragma unroll 4
                        for (int cc = c0; cc <= c1; ++cc) {
                            // the CTA that holds the tile's first item wrote its second slot
                            const float* s = src + ((size_t)cc * 2 + (cc == c0 ? 1 : 0)) * part;
                            const float4 a = __ldcg(reinterpret_cast<const float4*>(s));
                            const float4 d = __ldcg(reinterpret_cast<const float4*>(s + 4 * kTileM));
                            v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
                            v[4] += d.x; v[5] += d.y; v[6] += d.z; v[7] += d.w;
                        }
                        emit(p, tile, quarter, lane, ch * 8, v);
                    }
                    __syncwarp();  // (lanes past the output left early; the next tile's loads are warp-wide)
                }
            }
            ls = le;
        }
        if (!waited) asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
    }

    if (p.split > 1) {  // every thread of every CTA of the cluster gets here, after a failed wait too
        namespace cg = cooperative_groups;
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        const int S = p.split, rank = (int)cluster.block_rank(), tile = c / S;
        const int row = quarter * 32 + lane;
        // The CTAs' warps take the columns four at a time; parts are added in rank order, all loads first.
        // Only the last read holds the other CTAs up.
        const int fours = warp >= kFirstDecodeWarp && !*abort_flag ? (p.M + 3) >> 2 : 0;
        bool arrived = false;
        for (int c4 = rank * kGroups + grp; c4 < fours; c4 += S * kGroups) {
            float4* mine = reinterpret_cast<float4*>(mid_smem + (NS > 0 ? kPartScaled : kPart)) + (size_t)c4 * kTileM + row;
            float4 a[8];
#pragma unroll
            for (int s = 0; s < 8; ++s) a[s] = s < S ? *cluster.map_shared_rank(mine, s) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            float v[4] = {a[0].x, a[0].y, a[0].z, a[0].w};
#pragma unroll
            for (int s = 1; s < 8; ++s) {
                if (s < S) {
                    v[0] += a[s].x; v[1] += a[s].y; v[2] += a[s].z; v[3] += a[s].w;
                }
            }
            if (c4 + S * kGroups >= fours) {
                __syncwarp();
                asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
                arrived = true;
            }
            emit(p, tile, quarter, lane, c4 * 4, v);
        }
        __syncwarp();
        if (!arrived) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // nobody leaves while its part is read
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

using MidKernel = void (*)(const CUtensorMap, const MidParams);

// What the launches on one device need to know, found out once.
struct MidDevice {
    cudaError_t err = cudaSuccess;
    int clusters[9] = {0};  // clusters of 1..8 CTAs of this kernel that run at the same time
};

const MidDevice& mid_device(int dev) {
    static MidDevice devs[64];
    static std::once_flag once[64];
    MidDevice& d = devs[dev];
    std::call_once(once[dev], [&] {
        for (MidKernel k : {gemm_midrows_kernel<0>, gemm_midrows_kernel<16>, gemm_midrows_kernel<32>, gemm_midrows_kernel<48>})
            if (d.err == cudaSuccess)
                d.err = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
        for (int s = 1; s <= 8 && d.err == cudaSuccess; ++s) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((unsigned)(s * 148));
            cfg.blockDim = dim3(kThreads);
            cfg.dynamicSmemBytes = kSmem;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = (unsigned)s;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            d.err = cudaOccupancyMaxActiveClusters(&d.clusters[s], gemm_midrows_kernel<0>, &cfg);
        }
    });
    return d;
}

// Time of a launch among others in us, by split: constants of a straight-line fit to 31 shapes (256x512 to
// 151936x1024, 5120x8192, gate|up up to 51200x5120) times 13 row counts, every split forced, on 148 SMs.
// `col` constants are per 100 activation rows (rounded up to 16); a chunk is up to four 64-blocks.
struct SplitCost {
    // clusters: per chunk of a CTA, per wave of tiles (whole tiles; shared by a cluster), launches that
    // cannot share the chip with the next one, waves behind the first
    double chunk, chunk_col, one, one_col, many, many_col, alone, wave;
    // stream: per chunk, per tile of a CTA, per CTA of a tile behind the second, launch, not shared
    double s_chunk, s_chunk_col, tile, tile_col, join, join_col, launch, launch_col, s_alone;
};
constexpr SplitCost kCostScaled = {0.66, 0.68, 2.08, 1.40, 2.97, 2.77, 1.63, 1.77,
                                   0.97, 1.69, 0.74, 0.23, 0.15, 0.07, 2.05, 2.26, 3.92};
constexpr SplitCost kCostPlain = {0.78, 0.21, 1.29, 1.66, 2.51, 1.84, 1.83, 2.17,
                                  1.00, 0.57, 0.68, 0.53, 0.00, 0.57, 0.52, 2.50, 5.48};

// 0: the stream split (where there are partial tiles for it); else CTAs per tile. On the measured shapes the choice is 0.4 % behind the best split on
// average and 10 % at worst (10 % on average and 57 % at worst by the model of one layer's width before it:
// 6144x2560 at 32 rows 14.9 -> 9.5 us, 30000x512 at 256 rows 30.2 -> 20.4 us).
int choose_split(const MidDevice& d, int n_tiles, int KB, int NB, bool block_scaled, bool stream, int sm_count) {
    static const int forced = [] {  // for measurements: AILA_NF4_MID_SPLIT=0..8
        const char* e = std::getenv("AILA_NF4_MID_SPLIT");
        return e && *e ? std::atoi(e) : -1;
    }();
    if (forced >= (stream ? 0 : 1) && forced <= 8 && forced <= KB) return forced;
    const SplitCost& c = block_scaled ? kCostScaled : kCostPlain;
    const double cols = NB / 100.0;
    const int64_t total = (int64_t)n_tiles * KB;
    const int64_t ctas = (total + 7) / 8 < sm_count ? (total + 7) / 8 : sm_count;
    const double items = (double)total / ctas, tiles = items / KB;
    double best = 1e30;
    int split = stream ? 0 : 1;
    if (stream && ctas <= 8 * (int64_t)n_tiles)  // (a tile's last CTA adds all parts: not more than a cluster has)
        best = items / 4 * (c.s_chunk + c.s_chunk_col * cols) + tiles * (c.tile + c.tile_col * cols) +
               (1 / tiles > 2 ? (1 / tiles - 2) * (c.join + c.join_col * cols) : 0) + c.launch + c.launch_col * cols +
               (2 * ctas > sm_count ? c.s_alone : 0);
    for (int s = 1; s <= 8 && s <= KB; ++s) {
        if (d.clusters[s] <= 0) continue;
        const int waves = (n_tiles + d.clusters[s] - 1) / d.clusters[s];
        const int chunks = ((KB + s - 1) / s + kGroups - 1) / kGroups;
        const double cost = waves * (chunks * (c.chunk + c.chunk_col * cols) +
                                     (s == 1 ? c.one + c.one_col * cols : c.many + c.many_col * cols)) +
                            (2 * n_tiles > d.clusters[s] ? c.alone : 0) + (waves - 1) * c.wave;
        if (cost < best) {
            best = cost;
            split = s;
        }
    }
    return split;
}

}  // namespace

int gemm_midrows_tiles(const AilaNf4Linear& w, int64_t swiglu_ff) {
    return (int)(swiglu_ff > 0 ? (swiglu_ff + 63) / 64 : (w.N + kTileM - 1) / kTileM);
}

bool gemm_midrows_supported(const AilaNf4Linear& w, int64_t swiglu_ff) {
    if (w.absmax_kind == kAbsmaxCodes && !w.d_row_scales) return false;
    if (swiglu_ff > 0 && (swiglu_ff % kTileRows != 0 || w.N != 2 * swiglu_ff)) return false;
    return (int64_t)gemm_midrows_tiles(w, swiglu_ff) * w.KU < ((int64_t)1 << 30);
}

size_t gemm_midrows_partial_bytes(int ctas, int rows) {
    return (size_t)ctas * 2 * kTileM * (size_t)((rows + 15) / 16 * 16) * sizeof(float);
}

// x is 16-byte aligned; rows <= kMidRowsMax; counters hold a zero per tile.
AilaNf4Status launch_gemm_midrows(const AilaNf4Linear& w, AilaNf4Scratch& sc, const void* x, void* y,
                                  const void* residual, int rows, int64_t swiglu_ff, bool block_scaled, cudaStream_t s) {
    if (rows < 1 || rows > (block_scaled ? kMidRowsScaled : kMidRowsMax))
        return fail(AILA_NF4_ERR_INVALID_ARGUMENT, "gemm_midrows: row count");
    MidParams p = {};
    const ScaleParams sp = w.scale_params();
    p.units = w.d_units;
    p.qmap = w.d_qmap;
    p.nmap = sp.nmap;
    p.row_scales = static_cast<const float4*>(w.d_row_scales);
    p.residual = static_cast<const uint16_t*>(residual);
    p.y = static_cast<uint16_t*>(y);
    p.counters = sc.d_counters;
    p.status = sc.d_status;
    p.limit = sc.wait_limit_cycles;
    p.KU = w.KU;
    p.RT = w.RT;
    p.n_rows = (int)w.N;
    p.unit_stride = w.unit_stride;
    p.kind = w.absmax_kind;
    p.M = rows;
    p.NB = (rows + 15) / 16 * 16;
    p.ff = (int)swiglu_ff;
    p.n_out = (int)(swiglu_ff > 0 ? swiglu_ff : w.N);
    p.n_tiles = gemm_midrows_tiles(w, swiglu_ff);
    const int x_fit = (kSmem - (int)kXRing) / (p.NB * 128);
    p.x_stages = x_fit < kMaxX ? x_fit : kMaxX;
    p.x_per_item = p.x_stages < kMaxX;
    // instruction descriptor: D = f32, A = B = bf16, both K-major, N >> 3, M >> 4
    p.idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.NB >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
    CUtensorMap map_x;
    if (!encode_map(&map_x, x, (uint64_t)rows, (uint64_t)w.K, (uint32_t)p.NB))
        return fail(AILA_NF4_ERR_CUDA, "cuTensorMapEncodeTiled failed for the activation tensor");
    int dev = 0;
    cudaGetDevice(&dev);
    const MidDevice& md = mid_device(dev & 63);
    if (md.err != cudaSuccess) return cuda_fail(md.err, "cudaFuncSetAttribute(gemm_midrows)");
    p.split = choose_split(md, p.n_tiles, p.KU, p.NB, block_scaled, sc.d_mid_partials != nullptr, sc.sm_count);
    const int64_t total = (int64_t)p.n_tiles * p.KU;
    const int64_t want = p.split > 0 ? (int64_t)p.n_tiles * p.split : (total + 7) / 8;  // stream: eight items per CTA at least
    const int grid = (int)(p.split > 0 || want < sc.sm_count ? want : sc.sm_count);
    p.partials = sc.d_mid_partials;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    cfg.attrs = attr;
    if (overlapped_launches()) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (p.split > 1) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = (unsigned)p.split;
        attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
        ++cfg.numAttrs;
    }
    const MidKernel kernel = !block_scaled ? gemm_midrows_kernel<0>
                             : p.NB == 16  ? gemm_midrows_kernel<16>
                             : p.NB == 32  ? gemm_midrows_kernel<32>
                                           : gemm_midrows_kernel<48>;
    const cudaError_t le = cudaLaunchKernelEx(&cfg, kernel, map_x, p);
    if (le != cudaSuccess) return cuda_fail(le, "gemm_midrows_kernel launch");
    return AILA_NF4_OK;
}

}  // namespace nf4
