// Grouped dequant GEMM on the 5th-generation tensor cores (tcgen05 + TMEM) for the wide MoE path.
//
// Problem: for every expert group g with n_g token rows, OUT[row][m] = sum_k W_g[m][k] * X[row][k],
// W_g stored as GGUF superblocks. Weights sit on the MMA M side (128-row tiles), tokens on N; a group's
// rows are cut into column blocks of equal width (a multiple of 16), because tensor time follows the
// width while every block decodes the same weights again.
//
// Exactness: the A operand carries EXACT small integers in fp16 (IQ2_XXS: +-{8,25,43}*(2*sub+1);
// Q4_K / Q2_K: code * sub-scale), the B operand the fp16 image of bf16-exact activations, so
// every product is exact and only the f32 accumulation in TMEM rounds. The per-superblock f16
// scale d cannot ride inside the MMA; the accumulator is therefore drained once per 256 K by the
// epilogue warps (acc[row][n] += d[row][block] * tmem[row][n]) while the other TMEM buffer is
// being filled. Affine qtypes add one more K=16/32 MMA per superblock: A' = integer mins,
// B' = per-sub-block activation sums (hi/lo fp16 split), drained as acc -= dmin * tmem'.
//
// Where the operands live, and why. Shared memory is the unit this kernel runs out of: with A in shared
// memory a 64-K chunk cost 16 KiB of tile stores, 16 KiB of A and up to 32 KiB of B operand reads,
// 32 KiB of TMA writes and the bank conflicts of 64 table lookups per row - about 930 cycles of
// its 128 bytes per cycle against 512 cycles of MMA. So the decoded A operand goes to TENSOR memory
// (tcgen05.st from the decoding warps, tcgen05.mma with A in TMEM): neither its stores nor its reads
// touch shared memory any more, and the room it leaves holds the IQ2_XXS tables replicated per lane
// (64 KiB, no conflicts). The price is the columns: 224 instead of 256 per IQ2_XXS tile, and one
// min-term accumulator instead of two.
//
// CTA = 28 warps, persistent over a device-built tile list:
//   warp 0      TMA producer: activation tiles [N x 64] fp16, 128-byte swizzle, mbarrier tx; B' tiles of the
//               min term (the sub-block sums, 64-byte swizzle); the lookup tables once
//   warp 1      MMA issuer: per 64-K chunk 4 x tcgen05.mma (K=16), superblocks alternating between two accumulators
//   warp 2      TMA producer: the raw weight superblocks of the tile's 128 rows (u8 boxes, four or five in flight)
//   warp 3      looks the tiles up ahead of the other roles
//   then the dequant producers: thread = (row, half of a 64-K chunk) decodes 32 weights of the staged
//               superblock to fp16 and stores them into its row's lane of the A ring; the same warps write the A'
//               rows and the per-row block scales for the epilogue
//   and the epilogue warps, one per (32 TMEM lanes, 32 or 64 columns): TMEM -> registers (tcgen05.ld), scale,
//               accumulate, final store
// Single-lane roles are chosen with elect.sync. Every mbarrier wait is bounded; on expiry the CTA sets
// status 3, unwinds and frees its TMEM.
//
// Two forms. The plain one multiplies by ONE matrix and stores bf16 rows (down projection). The
// fused one computes gate and up together: a tile's 128 A rows are 64 gate rows and the 64 up rows
// of the same intermediates, interleaved (A row 2i = gate row i, 2i + 1 = up row i; the producers
// are free to choose which weight row feeds which tile row). Gate and up of an intermediate then
// sit in neighbouring TMEM lanes, i.e. in neighbouring threads of an epilogue warp, which pairs
// them with one shuffle, applies the clamps, SiLU, the route weight and the single bf16 rounding
// (src/graph/moe.c:605-613) and stores the fp16 image the down GEMM reads. Neither projection is
// ever written to memory.
#pragma once
#include <type_traits>

#include "gemv_stream.cuh"
#include "moe_common.cuh"
#include "tcgen05.cuh"

namespace yb {

constexpr int kTileStep = YVEX_B200_MOE_TILE_STEP;               // columns a group's last tile is padded to
static_assert(kTileStep == 16, "the N of tcgen05.mma kind::f16 at M = 128 is a multiple of 16");
constexpr int kTileM = 128, kBoxN = 64, kMinTileN = 128, kChunkK = 64;
constexpr uint32_t kBoxBytes = kBoxN * kChunkK * 2;          // activations arrive in boxes of 64 rows: a ragged tile fetches what it needs
constexpr uint32_t kMinTileBytes = kTileM * 64;               // 8 KiB: A' or B' of the min term, 32 fp16 per row, 64-byte swizzle
constexpr uint32_t kTmemCols = 512;
constexpr int kScaleRing = 4;                               // superblocks of per-row scales kept for the epilogue

// <= kTileN token rows of one expert (expert < 0: the shared expert). Column blocks of the same expert
// form groups of consecutive entries [first, first + count) covering <= kGroupRows rows: the tiles of a
// group are walked weight tile by weight tile, so the CTAs running side by side share one weight
// tile (read from DRAM once) while the group's activation rows stay in L2.
struct ColBlock { int row0, ncols, expert, first, count, pad; };
constexpr int kGroupRows = 1024;

// Tensor maps of one launch. A weight pack is described as u8 [rows / fuse][fuse * row_bytes] with
// `fuse` consecutive rows joined into one tensor row, so that the row pitch is a multiple of 16
// bytes whatever the block size (66-byte IQ2_XXS blocks give pitches that are only multiples of 2).
struct GemmMaps {
    CUtensorMap act, act_tail;                  // activation rows in boxes of 64 and of 32 rows
    CUtensorMap sums;                           // affine qtypes: [rows][K/256][32] hi/lo sub-block sums
    CUtensorMap w_routed[2], w_shared[2];
};

struct GemmParams {
    uint32_t row_bytes;
    int fuse;                                   // rows per tensor row of the weight maps: 1, 2, 4 or 8
    int M, K;
    const ColBlock *colblocks;
    const int *num_colblocks;
    uint16_t *out_bf16;                         // [rows][M] bf16 bits (plain kernel: down results) ...
    const int *out_rows;                        // optional: result row of sorted row r is out_rows[r]
    // optional: sorted row r is stored at this byte address instead, which may lie in ANOTHER GPU's memory
    // (plain peer stores over NVLink: an expert-parallel rank returns a pair's row straight to its home
    // rank from the epilogue, so no separate exchange carries it back); 0 = the row is dropped
    const unsigned long long *out_addr;
    __half *mid;                                // ... or [rows][M] SwiGLU intermediates as fp16 (fused gate/up kernel)
    const float *col_weight;                    // route weight of sorted row r (fused kernel)
    float limit;                                // SwiGLU clamp (fused kernel)
    int *status;
};

constexpr int kTileRing = 4;                                // tiles looked up ahead of the roles

struct GemmSmem {
    uint64_t a_full[4], a_empty[4], b_full[5], b_empty[5], tab_full;
    uint64_t raw_full[5], raw_empty[5];
    uint64_t acc_full[2], acc_empty[2], min_full[2], min_empty[2];
    uint64_t tile_full[kTileRing], tile_empty[kTileRing];
    int4 tile[kTileRing];                                   // {first row, columns, expert, m tile} of the tiles ahead
    uint32_t tmem_base;
    int abort;
};

// A ring position: stage and the parity of its current use.
struct RingAt {
    uint32_t s = 0, ph = 0;
    template <int kDepth> __device__ __forceinline__ void next() { if (++s == (uint32_t)kDepth) { s = 0; ph ^= 1u; } }
};

// ---- per-qtype decoders -----------------------------------------------------------------------------
// A decoder sees one superblock of one weight row in its slot of a raw stage. kBoxBytes is the pitch of the slots and the
// width of the TMA box that fetches one: the block plus the most its start can lie above a 16-byte boundary
// (block sizes are multiples of 2, 4 or 16 bytes), rounded up to 16 and, for Q2_K, to a pitch without bank conflicts.
// Two threads share a row: thread h decodes weights 64 c + 32 h .. + 31 of 64-K chunk c.
//   open       the block that starts `off` bytes into its slot; what of it is wanted in registers
//   fetch      the words, table entries and integer scale of half h of chunk c (read before the wait for the chunk's stage)
//   convert    sixteen of its weights (q = 0, 1) as eight words of two fp16
//   scales     {d, dmin} of the block, and whether they are acceptable
//   mins       this thread's share of the A' row (affine qtypes)
//   kTableBytes, kMinSlots   shared-memory tables the decoder reads; K slots of the min term's MMA (0: none)
// prmt.b32 with a run-time selector. (__byte_perm masks the selector with 0x7777 first; the decoders'
// selectors never have bit 3 of a nibble set, and the instruction reads only the low 16 bits.)
__device__ __forceinline__ uint32_t prmt_raw(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

// Eight codes (bytes) -> eight fp16 (code + bias - bias) * scale in K order, exact: 0x6400 | b is 1024 + b, and the product with
// the integer scale and the subtraction round once.
__device__ __forceinline__ void scaled8(uint32_t bytes_lo, uint32_t bytes_hi, uint32_t sc2, uint32_t nb2, uint32_t *v) {
    v[0] = prmt_raw(bytes_lo, 0x64646464u, 0x4140); v[1] = prmt_raw(bytes_lo, 0x64646464u, 0x4342);
    v[2] = prmt_raw(bytes_hi, 0x64646464u, 0x4140); v[3] = prmt_raw(bytes_hi, 0x64646464u, 0x4342);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __half2 h = __hfma2(*reinterpret_cast<__half2 *>(&v[i]), *reinterpret_cast<const __half2 *>(&sc2), *reinterpret_cast<const __half2 *>(&nb2));
        v[i] = *reinterpret_cast<const uint32_t *>(&h);
    }
}
// An integer scale s < 64 as half2(s, s), and half2(-bias * s) (exact: bias is 1024 or 1152).
__device__ __forceinline__ void scale_pair(uint32_t s, float bias, uint32_t &sc2, uint32_t &nb2) {
    const uint32_t dup = prmt_raw(s, 0x64646464u, 0x4040);
    const __half2 v = __hsub2(*reinterpret_cast<const __half2 *>(&dup), __float2half2_rn(1024.0f));
    const __half2 n = __hmul2(v, __float2half2_rn(-bias));
    sc2 = *reinterpret_cast<const uint32_t *>(&v);
    nb2 = *reinterpret_cast<const uint32_t *>(&n);
}

// Four bytes (each < 1024) -> four exact fp16 values: 0x6400 | b is 1024 + b, minus 1024.
__device__ __forceinline__ uint2 bytes_to_half4(uint32_t b4) {
    uint32_t lo = __byte_perm(b4, 0x64646464u, 0x4140), hi = __byte_perm(b4, 0x64646464u, 0x4342);
    const __half2 k = __floats2half2_rn(1024.0f, 1024.0f);
    const __half2 a = __hsub2(*reinterpret_cast<__half2 *>(&lo), k), b = __hsub2(*reinterpret_cast<__half2 *>(&hi), k);
    return make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
}

__device__ __forceinline__ float2 checked_scales(uint32_t d_bits, uint32_t dmin_bits, float d_mul, bool &bad) {
    const float d = f16_bits_to_float((uint16_t)d_bits), dmin = f16_bits_to_float((uint16_t)dmin_bits);
    bad = !isfinite(d) || !isfinite(dmin) || d < 0.0f || dmin < 0.0f;
    return make_float2(d * d_mul, dmin);
}

struct GemmIq2 {
    static constexpr int kBlockBytes = 66, kMinSlots = 0, kBoxBytes = 80;     // 66 bytes from a 2-byte aligned start
    static constexpr uint32_t kTableBytes = gs::kTableBytes;
    struct Block { const uint32_t *raw; uint32_t mis; };
    struct Half { uint32_t sel[4], sc2, nb2; };
    __device__ static void open(const uint8_t *slot, uint32_t off, Block &b) { b.raw = reinterpret_cast<const uint32_t *>(slot + (off & ~3u)); b.mis = off & 3u; }
    __device__ static void fetch(const Block &b, int c, int h, const uint8_t *tab, uint32_t lane4, Half &p) {
        const uint32_t o = b.mis + 2u + 8u * (2 * c + h), sh = 8u * (o & 3u);
        const uint32_t *w = b.raw + (o >> 2);
        const uint32_t w1 = w[1];
        const uint32_t grids = __funnelshift_r(w[0], w1, sh), ss = __funnelshift_r(w1, w[2], sh);
        // index byte into byte 1 of the table offset, the lane's column into byte 0 (each lane has its own bank)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            p.sel[j] = *reinterpret_cast<const uint32_t *>(tab + prmt_raw(grids, lane4, 0x5504u | ((uint32_t)j << 4))) |
                       *reinterpret_cast<const uint32_t *>(tab + 128 + prmt_raw(ss >> (7 * j), lane4, 0x5504u));
        scale_pair((ss >> 27) | 1u, 1152.0f, p.sc2, p.nb2);                                      // 2 * sub + 1
    }
    // weights 64 c + 32 h + 16 q .. + 15 as eight words of two fp16
    __device__ static void convert(const Half &p, int q, uint32_t (&v)[8]) {
        constexpr uint32_t kLo = (8u + 128u) | ((25u + 128u) << 8) | ((43u + 128u) << 16);
        constexpr uint32_t kHi = (128u - 8u) | ((128u - 25u) << 8) | ((128u - 43u) << 16);
#pragma unroll
        for (int j = 0; j < 2; ++j)
            scaled8(prmt_raw(kLo, kHi, p.sel[2 * q + j]), prmt_raw(kLo, kHi, p.sel[2 * q + j] >> 16), p.sc2, p.nb2, v + 4 * j);
    }
    __device__ static float2 scales(const Block &b, bool &bad) { return checked_scales(b.raw[0] >> (8u * b.mis), 0u, 0.125f, bad); }
    __device__ static void mins(const Block &, int, uint8_t *, uint32_t) {}
};

struct GemmQ4k {
    static constexpr int kBlockBytes = 144, kMinSlots = 16, kBoxBytes = 144;   // 8 mins x (hi, lo); blocks are 16-byte aligned
    static constexpr uint32_t kTableBytes = 0;
    struct Block { const uint4 *raw; uint4 head; };
    struct Half { uint4 q[2]; uint32_t sc2, nb2, shift; };
    __device__ static void open(const uint8_t *slot, uint32_t, Block &b) { b.raw = reinterpret_cast<const uint4 *>(slot); b.head = b.raw[0]; }   // d, dmin and the 12 scale bytes
    // sub-block 2c + h: the low (h = 0) or high nibbles of the chunk's 32 bytes. Its 6-bit scale: byte k of the first four
    // scale bytes, or (c >= 2) the low nibble of byte k of the last four under the top two bits of the first's.
    __device__ static void fetch(const Block &b, int c, int h, const uint8_t *, uint32_t, Half &p) {
        p.q[0] = b.raw[1 + 2 * c];
        p.q[1] = b.raw[2 + 2 * c];
        const uint32_t k8 = 8u * (uint32_t)(2 * (c & 1) + h);
        const uint32_t sc = c < 2 ? (b.head.y >> k8) & 63u : ((b.head.w >> k8) & 15u) | (((b.head.y >> (k8 + 6u)) & 3u) << 4);
        p.shift = 4u * (uint32_t)h;
        scale_pair(sc, 1024.0f, p.sc2, p.nb2);
    }
    __device__ static void convert(const Half &p, int q, uint32_t (&v)[8]) {
        scaled8((p.q[q].x >> p.shift) & 0x0f0f0f0fu, (p.q[q].y >> p.shift) & 0x0f0f0f0fu, p.sc2, p.nb2, v);
        scaled8((p.q[q].z >> p.shift) & 0x0f0f0f0fu, (p.q[q].w >> p.shift) & 0x0f0f0f0fu, p.sc2, p.nb2, v + 4);
    }
    __device__ static float2 scales(const Block &b, bool &bad) { return checked_scales(b.head.x, b.head.x >> 16, 1.0f, bad); }
    // A' row: slots 0..7 = the eight mins (paired with the hi sums), 8..15 = the same mins (lo sums); thread h writes
    // 16-byte part h. (four bytes at a time: mins 0..3 are bytes 4..7 & 63, mins 4..7 the high nibbles of bytes 8..11 with
    // the top two bits of bytes 4..7 above them)
    __device__ static void mins(const Block &b, int h, uint8_t *tile, uint32_t row) {
        const uint32_t s1 = b.head.z, s2 = b.head.w;
        const uint2 lo = bytes_to_half4(s1 & 0x3f3f3f3fu);
        const uint2 hi = bytes_to_half4(((s2 >> 4) & 0x0f0f0f0fu) | (((s1 >> 6) & 0x03030303u) << 4));
        *reinterpret_cast<uint4 *>(tile + sm100::sw64_offset(row, h)) = make_uint4(lo.x, lo.y, hi.x, hi.y);
    }
};

struct GemmQ2k {
    // 16 mins x (hi, lo); 4-byte aligned start. The box is 112 bytes, not the 96 that hold a block: rows seven 16-byte units
    // apart meet no two on the same banks in 16-byte reads.
    static constexpr int kBlockBytes = 84, kMinSlots = 32, kBoxBytes = 112;
    static constexpr uint32_t kTableBytes = 0;
    struct Block { uint32_t w[24]; };           // w[0..3] scales and mins, w[4..19] codes, w[20] d and dmin
    struct Half { uint32_t q[8], s, plane2; };
    // The whole block in six 16-byte reads, then moved down to word 0 by the start's offset (word reads at a 112-byte pitch
    // would be four to a bank, and a thread needs every word of the block).
    __device__ static void open(const uint8_t *slot, uint32_t off, Block &b) {
        const uint4 *raw = reinterpret_cast<const uint4 *>(slot);
#pragma unroll
        for (int i = 0; i < 6; ++i) { const uint4 v = raw[i]; b.w[4 * i] = v.x; b.w[4 * i + 1] = v.y; b.w[4 * i + 2] = v.z; b.w[4 * i + 3] = v.w; }
#pragma unroll
        for (int i = 0; i < 23; ++i) b.w[i] = (off & 4u) ? b.w[i + 1] : b.w[i];
#pragma unroll
        for (int i = 0; i < 21; ++i) b.w[i] = (off & 8u) ? b.w[i + 2] : b.w[i];
    }
    // plane 2 (c & 1) + h of the 32 bytes of half c >> 1: two 16-weight sub-blocks, scale bytes 8 (c >> 1) + 2 plane + (0, 1)
    __device__ static void fetch(const Block &b, int c, int h, const uint8_t *, uint32_t, Half &p) {
        p.plane2 = 2u * (uint32_t)(2 * (c & 1) + h);
#pragma unroll
        for (int i = 0; i < 8; ++i) p.q[i] = b.w[4 + 8 * (c >> 1) + i];
        p.s = b.w[2 * (c >> 1) + (c & 1)] >> (16 * h);
    }
    __device__ static void convert(const Half &p, int q, uint32_t (&v)[8]) {
        uint32_t sc2, nb2;
        scale_pair((p.s >> (8 * q)) & 15u, 1024.0f, sc2, nb2);
        scaled8((p.q[4 * q] >> p.plane2) & 0x03030303u, (p.q[4 * q + 1] >> p.plane2) & 0x03030303u, sc2, nb2, v);
        scaled8((p.q[4 * q + 2] >> p.plane2) & 0x03030303u, (p.q[4 * q + 3] >> p.plane2) & 0x03030303u, sc2, nb2, v + 4);
    }
    __device__ static float2 scales(const Block &b, bool &bad) { return checked_scales(b.w[20], b.w[20] >> 16, 1.0f, bad); }
    // A' row: slots 0..15 = the sixteen mins (hi sums), 16..31 = the same mins (lo sums); thread h converts mins 8h..8h+7
    // and writes them to parts h and h + 2.
    __device__ static void mins(const Block &b, int h, uint8_t *tile, uint32_t row) {
        const uint2 lo = bytes_to_half4(((h ? b.w[2] : b.w[0]) >> 4) & 0x0f0f0f0fu), hi = bytes_to_half4(((h ? b.w[3] : b.w[1]) >> 4) & 0x0f0f0f0fu);
        const uint4 v = make_uint4(lo.x, lo.y, hi.x, hi.y);
        *reinterpret_cast<uint4 *>(tile + sm100::sw64_offset(row, h)) = v;
        *reinterpret_cast<uint4 *>(tile + sm100::sw64_offset(row, h + 2)) = v;
    }
};

// ---- shared-memory plan -----------------------------------------------------------------------------
// tiles (1024-byte aligned; the kernel refuses to run if the dynamic shared memory does not start on
// such a boundary): B ring, [min tiles: two A', two B'], then the raw superblock ring (kRawStages x 128 rows x
// kBoxBytes, plus a pad: the decoders' funnel reads run one word over), the scale ring, the lookup tables and the barriers.
template <class Dec> struct GemmPlan {
    static constexpr bool kHasMin = Dec::kMinSlots > 0;
    // Tensor memory: two accumulators of kTileN columns that alternate by superblock, one min-term accumulator (affine), and
    // the A ring: 32 columns (two fp16 each) per 64-K chunk. 224 + 224 + 2 x 32, or 128 + 128 + 128 + 4 x 32.
    static constexpr int kTileN = kHasMin ? 128 : 224;                              // columns per tile
    static constexpr int kAStages = kHasMin ? 4 : 2, kBStages = kHasMin ? 5 : 4;
    static constexpr int kRawStages = kHasMin ? 5 : 4;                      // raw weight superblocks in flight
    static constexpr uint32_t kMinCol = 2 * kTileN, kACol = kTmemCols - kAStages * (kChunkK / 2);
    static_assert(kMinCol + (kHasMin ? kTileN : 0) <= kACol, "tensor memory columns");
    // 8 producer and 16 epilogue warps: an epilogue warp owns 32 TMEM lanes x kColsPerWarp columns
    static constexpr int kEpilogueWarps = 16, kColsPerWarp = kHasMin ? 32 : 64;
    static constexpr int kProducerWarps = 8;
    static constexpr int kThreads = 32 * (4 + kProducerWarps + kEpilogueWarps);
    // registers per thread of each role (setmaxnreg)
    static constexpr int kCtlRegs = kHasMin ? 48 : 40;
    static constexpr int kProdRegs = kHasMin ? 72 : 56, kEpiRegs = kHasMin ? 72 : 88;
    static constexpr uint32_t kBTileBytes = kTileN * kChunkK * 2;
    static constexpr uint32_t kRawStageBytes = kTileM * Dec::kBoxBytes;
    using Scale = typename std::conditional<kHasMin, float2, float>::type;          // {d, dmin} or d per row and superblock
    static constexpr size_t kTilesBytes = (size_t)kBStages * kBTileBytes + (kHasMin ? 4 : 0) * (size_t)kMinTileBytes;
    static constexpr size_t kRawBytes = (size_t)kRawStages * kRawStageBytes + 128;
    static constexpr size_t kScaleBytes = (size_t)kScaleRing * kTileM * sizeof(Scale);
    static constexpr size_t kBytes = kTilesBytes + kRawBytes + kScaleBytes + Dec::kTableBytes + sizeof(GemmSmem);
    static_assert(kBytes <= 227 * 1024, "shared memory plan exceeds the 227 KiB a CTA can have");
    static_assert(kBTileBytes % 1024 == 0 && kTilesBytes % 1024 == 0, "swizzled tiles start on 1024-byte boundaries");
    static_assert(kRawStageBytes % 128 == 0 && (kTileM / 16) * Dec::kBoxBytes % 128 == 0,
                  "TMA destinations are 128-byte aligned (boxes of 64 rows, up to 8 rows fused)");
};

// Sets this warpgroup's registers per thread to N, given the count the kernel was launched with. An
// increase waits until other warpgroups of the CTA have handed enough registers back.
template <int N, int kLaunched> __device__ __forceinline__ void set_registers() {
    if constexpr (N > kLaunched) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
    else if constexpr (N < kLaunched) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

// a0 = d * v0 + a0, a1 = d * v1 + a1 in one instruction (each rounded like fmaf)
__device__ __forceinline__ void fma2(float &a0, float &a1, float d, uint32_t v0, uint32_t v1) {
    asm("{\n\t.reg .b64 a, v, s;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 v, {%2, %3};\n\tmov.b64 s, {%4, %4};\n\t"
        "fma.rn.f32x2 a, s, v, a;\n\tmov.b64 {%0, %1}, a;\n\t}"
        : "+f"(a0), "+f"(a1) : "r"(v0), "r"(v1), "f"(d));
}

template <class Dec, bool kFused>
__global__ void __launch_bounds__(GemmPlan<Dec>::kThreads, 1)
moe_grouped_gemm_kernel(const __grid_constant__ GemmMaps maps, GemmParams p) {
    using namespace sm100;
    using Plan = GemmPlan<Dec>;
    constexpr bool kHasMin = Plan::kHasMin;
    constexpr int kTileN = Plan::kTileN;
    constexpr uint32_t kBTileBytes = Plan::kBTileBytes;
    constexpr int kProducerWarps = Plan::kProducerWarps, kAStages = Plan::kAStages, kBStages = Plan::kBStages, kRawStages = Plan::kRawStages;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    if (smem_u32(smem_raw) & 1023u) {                           // uniform: nothing has been set up yet
        pdl_wait();
        if (threadIdx.x == 0) raise(p.status, YVEX_B200_STATUS_TIMEOUT);
        return;
    }
    uint8_t *tiles = smem_raw;
    uint8_t *b_tiles = tiles;                                   // [kBStages][kTileN rows x 128 bytes]
    uint8_t *min_a = b_tiles + kBStages * kBTileBytes, *min_b = min_a + 2 * kMinTileBytes;      // [2][8 KiB] each when the qtype has mins
    uint8_t *raw_stage = tiles + Plan::kTilesBytes;             // [kRawStages][fuse][128 / fuse rows][kBoxBytes]
    typename Plan::Scale *dscale = reinterpret_cast<typename Plan::Scale *>(raw_stage + Plan::kRawBytes);
    uint8_t *tab = reinterpret_cast<uint8_t *>(dscale) + Plan::kScaleBytes;
    GemmSmem *sm = reinterpret_cast<GemmSmem *>(tab + Dec::kTableBytes);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kAStages; ++s) { mbar_init(&sm->a_full[s], kProducerWarps); mbar_init(&sm->a_empty[s], 1); }
        for (int s = 0; s < kBStages; ++s) { mbar_init(&sm->b_full[s], 1); mbar_init(&sm->b_empty[s], 1); }
        mbar_init(&sm->tab_full, 1);
        for (int s = 0; s < kRawStages; ++s) { mbar_init(&sm->raw_full[s], 1); mbar_init(&sm->raw_empty[s], kProducerWarps); }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&sm->acc_full[b], 1); mbar_init(&sm->acc_empty[b], Plan::kEpilogueWarps);
            mbar_init(&sm->min_full[b], kProducerWarps + 1); mbar_init(&sm->min_empty[b], 1);
        }
        // readers of a tile's entry: the three single-lane roles and every epilogue warp
        for (int i = 0; i < kTileRing; ++i) { mbar_init(&sm->tile_full[i], 1); mbar_init(&sm->tile_empty[i], 3 + Plan::kEpilogueWarps); }
        sm->abort = 0;
        fence_barrier_init();
    }
    if (warp == 0) tmem_alloc(&sm->tmem_base, kTmemCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sm->tmem_base;
    volatile int *abort = &sm->abort;
    pdl_wait();                                                 // tile list, activations and sums come from the kernels before
    pdl_trigger();

    const int ncb = *p.num_colblocks;
    constexpr int kRowsPerMat = kFused ? kTileM / 2 : kTileM;      // weight rows of one matrix in a tile
    const int mtiles = p.M / kRowsPerMat, nsb = p.K / 256;
    const uint32_t tiles_total = (uint32_t)ncb * (uint32_t)mtiles;

    // Every role walks the same tile sequence: group of column blocks -> m tile -> column block. Warp 3 looks the tiles up
    // ahead of the roles (two dependent loads and a few divisions are about a microsecond, which every role used to spend at
    // each tile's start with the pipeline standing still) and leaves them in a ring. Tile counts fit 32 bits: 2^31 tiles
    // would need activations of more than 2^43 bytes.
    struct Tile { int row0, ncols, expert, mt; };
    auto next_tile = [&](uint32_t n, Tile &tl) -> bool {            // single-lane roles: entry n of this CTA's sequence
        const uint32_t i = n % kTileRing;
        if (!mbar_wait(&sm->tile_full[i], (n / kTileRing) & 1u, abort)) return false;
        const int4 v = sm->tile[i];
        tl.row0 = v.x; tl.ncols = v.y; tl.expert = v.z; tl.mt = v.w;
        mbar_arrive(&sm->tile_empty[i]);
        return true;
    };
    // Weight map of matrix `mat` and first tensor row of a tile. (Selects, not maps.w_routed[mat]: a dynamically
    // indexed parameter array makes the compiler copy the parameter block to local memory.)
    auto weights_of = [&](const Tile &tl, int mat, int &y) {
        y = ((tl.expert < 0 ? 0 : tl.expert * p.M) + tl.mt * kRowsPerMat) / p.fuse;
        return mat ? (tl.expert < 0 ? &maps.w_shared[1] : &maps.w_routed[1]) : (tl.expert < 0 ? &maps.w_shared[0] : &maps.w_routed[0]);
    };

    const uint32_t my_tiles = tiles_total > blockIdx.x ? (tiles_total - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;

    // Register budget per role: 28 warps leave 72 registers per thread, and the epilogue's 64 partial sums per thread
    // do not fit in that: the control warps and producers hand registers back and the epilogue warpgroups take them.
    // Warps 0-3, 4-11 and 12+ are whole warpgroups, and each sets its count as the first thing on its own branch, where
    // the compiler can hold the role to it (behind a common if/else it allocated all roles for the launch's 72 and spilled).
    constexpr int kLaunched = (65536 / Plan::kThreads) & ~7;
    static_assert(4 * Plan::kCtlRegs + kProducerWarps * Plan::kProdRegs + Plan::kEpilogueWarps * Plan::kEpiRegs <= kLaunched * (Plan::kThreads / 32),
                  "the role budgets must fit in the registers the CTA was launched with, or the increase never returns");
    if (warp < 4) {
    set_registers<Plan::kCtlRegs, kLaunched>();
    if (warp == 0) {
        // ---------------- TMA producer: activation tiles (and the B' tiles of the min term) ----------------
        if (elect_one()) {
            prefetch_tensormap(&maps.act);
            if (kHasMin) prefetch_tensormap(&maps.sums);
            if (Dec::kTableBytes && my_tiles) {
                mbar_expect_tx(&sm->tab_full, Dec::kTableBytes);
                bulk_load(tab, &gs::kIq2StreamTable, Dec::kTableBytes, &sm->tab_full);
            }
            RingAt b;
            uint32_t sb_it = 0;
            bool ok = true;
            uint32_t tn = 0;
            Tile tl;
            for (; tn < my_tiles && ok; ++tn) {
                if (!next_tile(tn, tl)) break;
                // boxes of 64 rows, the last one of 32 where that is enough: a ragged tile fetches what it needs
                const int rem = tl.ncols & 63;
                const uint32_t boxes = (uint32_t)(tl.ncols >> 6) + (rem > 32 ? 1u : 0u);
                const bool tail = rem > 0 && rem <= 32;
                for (int sb = 0; sb < nsb && ok; ++sb, ++sb_it) {
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
                        if (!mbar_wait(&sm->b_empty[b.s], b.ph ^ 1u, abort)) { ok = false; break; }
                        mbar_expect_tx(&sm->b_full[b.s], boxes * kBoxBytes + (tail ? kBoxBytes / 2 : 0u));
                        const int x = (4 * sb + c) * kChunkK;
                        uint8_t *dst = b_tiles + b.s * kBTileBytes;
                        for (uint32_t i = 0; i < boxes; ++i) tma_load_2d(dst + i * kBoxBytes, &maps.act, x, tl.row0 + (int)(i * kBoxN), &sm->b_full[b.s]);
                        if (tail) tma_load_2d(dst + boxes * kBoxBytes, &maps.act_tail, x, tl.row0 + (int)(boxes * kBoxN), &sm->b_full[b.s]);
                        b.next<kBStages>();
                    }
                    if (kHasMin && ok) {
                        // (rows past the block's last one bring a neighbour's sums, past the last row of all zeros: columns never stored)
                        const uint32_t buf = sb_it & 1u, bph = (sb_it >> 1) & 1u;
                        if (!mbar_wait(&sm->min_empty[buf], bph ^ 1u, abort)) { ok = false; break; }
                        mbar_expect_tx(&sm->min_full[buf], kMinTileBytes);
                        tma_load_2d(min_b + buf * kMinTileBytes, &maps.sums, 32 * sb, tl.row0, &sm->min_full[buf]);
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        // One thread issues every MMA in chunk order; superblocks alternate between two TMEM accumulators.
        if (elect_one()) {
            const uint64_t bdesc0 = smem_desc_sw128(smem_u32(b_tiles));
            const uint64_t amin0 = smem_desc_sw64(smem_u32(min_a)), bmin0 = smem_desc_sw64(smem_u32(min_b));
            RingAt a, b;
            uint32_t sb_it = 0;
            bool ok = true;
            uint32_t tn = 0;
            Tile tl;
            for (; tn < my_tiles && ok; ++tn) {
                if (!next_tile(tn, tl)) break;
                const uint32_t idesc = idesc_f16((uint32_t)((tl.ncols + 15) & ~15));
                for (int sb = 0; sb < nsb && ok; ++sb, ++sb_it) {
                    const uint32_t buf = sb_it & 1u, bph = (sb_it >> 1) & 1u, acc = tmem + buf * kTileN;
                    if (!mbar_wait(&sm->acc_empty[buf], bph ^ 1u, abort)) { ok = false; break; }
                    tc_fence_after();
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
                        if (!mbar_wait(&sm->b_full[b.s], b.ph, abort) || !mbar_wait(&sm->a_full[a.s], a.ph, abort)) { ok = false; break; }
                        tc_fence_after();
                        // descriptors differ from the stage-0 one only in the start-address field (16-byte units)
                        const uint64_t bd = bdesc0 + (uint64_t)(b.s * (kBTileBytes >> 4));
                        const uint32_t at = tmem + Plan::kACol + a.s * (kChunkK / 2);
#pragma unroll
                        for (int k = 0; k < 4; ++k) umma_f16_ts(acc, at + 8 * k, bd + 2 * k, idesc, (c | k) ? 1u : 0u);
                        umma_commit(&sm->a_empty[a.s]);
                        umma_commit(&sm->b_empty[b.s]);
                        a.next<kAStages>();
                        b.next<kBStages>();
                    }
                    if (!ok) break;
                    if (kHasMin) {
                        // there is one min-term accumulator: the superblock before must have been drained
                        if (sb_it && !mbar_wait(&sm->acc_empty[buf ^ 1u], ((sb_it - 1u) >> 1) & 1u, abort)) { ok = false; break; }
                        if (!mbar_wait(&sm->min_full[buf], bph, abort)) { ok = false; break; }
                        tc_fence_after();
                        const uint64_t ad = amin0 + (uint64_t)(buf * (kMinTileBytes >> 4)), bd = bmin0 + (uint64_t)(buf * (kMinTileBytes >> 4));
#pragma unroll
                        for (int k = 0; k < Dec::kMinSlots / 16; ++k) umma_f16(tmem + Plan::kMinCol, ad + 2 * k, bd + 2 * k, idesc, k ? 1u : 0u);
                        umma_commit(&sm->min_empty[buf]);
                    }
                    umma_commit(&sm->acc_full[buf]);
                }
            }
        }
    } else if (warp == 2) {
        // ---------------- TMA producer: raw weight superblocks ----------------
        // One box per fused row r, [rows / fuse tensor rows] x [kBoxBytes from the 16-byte boundary at or below the block]
        // (the fused form: the same from each of the two matrices), up to kRawStages superblocks ahead of the producers.
        if (elect_one()) {
            uint32_t n = 0;
            bool ok = true;
            uint32_t tn = 0;
            Tile tl;
            for (; tn < my_tiles && ok; ++tn) {
                if (!next_tile(tn, tl)) break;
                int y;
                const CUtensorMap *map = weights_of(tl, 0, y), *map2 = kFused ? weights_of(tl, 1, y) : nullptr;
                for (int sb = 0; sb < nsb && ok; ++sb, ++n) {
                    const uint32_t s = n % kRawStages, ph = (n / kRawStages) & 1u;
                    if (!mbar_wait(&sm->raw_empty[s], ph ^ 1u, abort)) { ok = false; break; }
                    mbar_expect_tx(&sm->raw_full[s], Plan::kRawStageBytes);
                    const int rows = kRowsPerMat / p.fuse;
                    for (int r = 0; r < p.fuse; ++r) {
                        const int x = (int)(r * p.row_bytes + sb * Dec::kBlockBytes) & ~15;
                        uint8_t *dst = raw_stage + s * Plan::kRawStageBytes + r * rows * Dec::kBoxBytes;
                        tma_load_2d(dst, map, x, y, &sm->raw_full[s]);
                        if constexpr (kFused) tma_load_2d(dst + kRowsPerMat * Dec::kBoxBytes, map2, x, y, &sm->raw_full[s]);
                    }
                }
            }
        }
    } else if (elect_one()) {
        // ---------------- warp 3: tile look-ups ----------------
        for (uint32_t n = 0; n < my_tiles; ++n) {
            const uint32_t t = blockIdx.x + n * gridDim.x, i = n % kTileRing;
            const ColBlock *g0 = p.colblocks + t / (uint32_t)mtiles;    // any block of the group names the group
            const uint32_t first = (uint32_t)g0->first, count = (uint32_t)g0->count;
            const uint32_t local = t - first * (uint32_t)mtiles, mt = local / count;
            const ColBlock *cb = p.colblocks + first + (local - mt * count);
            const int4 v = make_int4(cb->row0, cb->ncols, cb->expert, (int)mt);
            if (!mbar_wait(&sm->tile_empty[i], ((n / kTileRing) & 1u) ^ 1u, abort)) break;
            sm->tile[i] = v;
            mbar_arrive(&sm->tile_full[i]);
        }
    }
    } else if (warp < 4 + kProducerWarps) {
        set_registers<Plan::kProdRegs, kLaunched>();
        if (Dec::kTableBytes && my_tiles && !mbar_wait_warp(&sm->tab_full, 0u, abort)) goto done;
        // ---------------- dequant producers ----------------
        // warps w and w + 4 own the 32 TMEM lanes (A rows) of w % 4: thread = (row, 32-weight half of a 64-K chunk)
        const int h = (warp - 4) >> 2;
        const uint32_t row = (uint32_t)(32 * (warp & 3) + lane);
        const uint32_t a_at = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + Plan::kACol + 16u * (uint32_t)h, lane4 = 4u * (uint32_t)lane;
        RingAt a;
        // where the row's bytes land in a raw stage, and where its superblock 0 starts in the tensor row
        // (fused form: tile row 2i is row i of the first matrix, 2i + 1 row i of the second, whose boxes follow)
        const uint32_t wrow = kFused ? row >> 1 : row, wmat = kFused ? row & 1u : 0u;
        const uint32_t sub = wrow % (uint32_t)p.fuse;
        const uint32_t slot = ((wmat * (uint32_t)p.fuse + sub) * (uint32_t)(kRowsPerMat / p.fuse) + wrow / (uint32_t)p.fuse) * Dec::kBoxBytes;
        const uint32_t x_row = sub * p.row_bytes;
        uint32_t sb_it = 0;
        for (uint32_t tile = 0; tile < my_tiles && !*abort; ++tile) {
            for (int sb = 0; sb < nsb; ++sb, ++sb_it) {
                const uint32_t rs = sb_it % kRawStages, rph = (sb_it / kRawStages) & 1u;
                if (!mbar_wait_warp(&sm->raw_full[rs], rph, abort)) goto done;
                typename Dec::Block blk;
                Dec::open(raw_stage + rs * Plan::kRawStageBytes + slot, (x_row + (uint32_t)sb * Dec::kBlockBytes) & 15u, blk);
                if (h == 0) {
                    bool bad;
                    const float2 dd = Dec::scales(blk, bad);
                    if constexpr (kHasMin) dscale[(sb_it % kScaleRing) * kTileM + row] = dd;
                    else dscale[(sb_it % kScaleRing) * kTileM + row] = dd.x;
                    if (bad) raise(p.status, YVEX_B200_STATUS_NUMERIC);
                }
                // a chunk's words and table entries are read, and its first half converted, before the wait for its stage
                // (2 % against converting all of it behind the wait; converting all of it before is no better)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    typename Dec::Half half;
                    Dec::fetch(blk, c, h, tab, lane4, half);
                    uint32_t v[8];
                    Dec::convert(half, 0, v);
                    if (!mbar_wait_warp(&sm->a_empty[a.s], a.ph ^ 1u, abort)) goto done;
                    tc_fence_after();
                    tmem_st8(a_at + a.s * (kChunkK / 2), v);
                    Dec::convert(half, 1, v);
                    tmem_st8(a_at + a.s * (kChunkK / 2) + 8u, v);
                    tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sm->a_full[a.s]);
                    a.next<kAStages>();
                }
                if (kHasMin) {
                    const uint32_t buf = sb_it & 1u, bph = (sb_it >> 1) & 1u;
                    if (!mbar_wait_warp(&sm->min_empty[buf], bph ^ 1u, abort)) goto done;
                    Dec::mins(blk, h, min_a + buf * kMinTileBytes, row);
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sm->min_full[buf]);
                }
                __syncwarp();                                   // every lane is done reading the stage
                if (lane == 0) mbar_arrive(&sm->raw_empty[rs]);
            }
        }
    } else {
        // ---------------- epilogue ----------------
        set_registers<Plan::kEpiRegs, kLaunched>();
        constexpr int kCols = Plan::kColsPerWarp;
        const int ew = warp - (4 + kProducerWarps), quarter = warp & 3, colhalf = ew >> 2;     // TMEM lanes 32*quarter.., columns kCols*colhalf..
        const int row = 32 * quarter + lane;
        const uint32_t lane_addr = (uint32_t)(32 * quarter) << 16;
        uint32_t sb_it = 0;
        for (uint32_t tn = 0; tn < my_tiles && !*abort; ++tn) {
            Tile cb;
            {
                const uint32_t i = tn % kTileRing;
                if (!mbar_wait_warp(&sm->tile_full[i], (tn / kTileRing) & 1u, abort)) goto done;
                const int4 v = sm->tile[i];
                cb.row0 = v.x; cb.ncols = v.y; cb.mt = v.w;
                __syncwarp();
                if (lane == 0) mbar_arrive(&sm->tile_empty[i]);
            }
            const int mt = cb.mt;
            float acc[kCols];
#pragma unroll
            for (int i = 0; i < kCols; ++i) acc[i] = 0.0f;
            const int ncols_here = cb.ncols - kCols * colhalf;    // columns this warp owns that are real
            // fused form: the route weights of this warp's columns, lane l holding those of columns l and
            // 32 + l; loaded here so that their latency is long gone when the tile ends
            float w_lo = 0.0f, w_hi = 0.0f;
            if constexpr (kFused) {
                const float *wcol = p.col_weight + cb.row0 + kCols * colhalf;
                if (lane < ncols_here) w_lo = __ldg(wcol + lane);
                if (kCols > 32 && 32 + lane < ncols_here) w_hi = __ldg(wcol + 32 + lane);
            }
            for (int sb = 0; sb < nsb; ++sb, ++sb_it) {
                const uint32_t buf = sb_it & 1u, bph = (sb_it >> 1) & 1u;
                if (!mbar_wait_warp(&sm->acc_full[buf], bph, abort)) goto done;
                tc_fence_after();
                // written by the row's producer before its last chunk of this superblock was published
                float d, dmin = 0.0f;
                if constexpr (kHasMin) { const float2 dd = dscale[(sb_it % kScaleRing) * kTileM + row]; d = dd.x; dmin = dd.y; }
                else d = dscale[(sb_it % kScaleRing) * kTileM + row];
                {
                    // (16-column groups without a real column are skipped: their sums stay zero, and the
                    // columns of a ragged group hold sums over neighbouring real rows, so every sum is
                    // finite unless real data is not)
#pragma unroll
                    for (int q = 0; q < kCols / 16; ++q) {
                        if (16 * q >= ncols_here) break;
                        uint32_t v[16];
                        tmem_ld16(tmem + lane_addr + buf * kTileN + kCols * colhalf + 16 * q, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; i += 2) fma2(acc[16 * q + i], acc[16 * q + i + 1], d, v[i], v[i + 1]);
                        if (kHasMin) {
                            tmem_ld16(tmem + lane_addr + Plan::kMinCol + kCols * colhalf + 16 * q, v);
                            tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < 16; i += 2) fma2(acc[16 * q + i], acc[16 * q + i + 1], -dmin, v[i], v[i + 1]);
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sm->acc_empty[buf]);
            }
            if (ncols_here <= 0) continue;                      // no real column: nothing to store
            // non-finite sums are refused: x * 0 is zero for finite x and NaN otherwise
            float poison = 0.0f, poison2 = 0.0f;
#pragma unroll
            for (int i = 0; i < kCols; i += 2) fma2(poison, poison2, 0.0f, __float_as_uint(acc[i]), __float_as_uint(acc[i + 1]));
            if (poison != poison || poison2 != poison2) raise(p.status, YVEX_B200_STATUS_NUMERIC);
            if constexpr (kFused) {
                // Even lanes hold the gate row of intermediate i = row / 2, odd lanes its up row. A pair of
                // lanes swaps every other column, so the even lane ends up with gate and up of the even
                // columns, the odd lane of the odd ones, and each evaluates half of the pair's SwiGLUs.
                // Then the four lanes of equal parity in every aligned group of eight transpose 4 x 4
                // blocks (intermediates x columns) with shuffles: lane (a, r, parity) ends up with
                // intermediates 4a..4a+3 of column 8b + 2r + parity, multiplies by that column's route
                // weight and stores them as one 8-byte vector.
                // A shuffle takes tens of cycles to come back (its pipe also serves the producers' reads), and
                // nothing of a tile end hides behind the two accumulators. It is therefore written in ROUNDS of
                // independent shuffles (all swaps; all first transpose steps; all second steps) rather than block
                // by block with three dependent shuffles each.
                const bool odd = lane & 1, o2 = lane & 2, o4 = lane & 4;
                const int rr = (lane >> 1) & 3;
                const uint64_t m0 = (uint64_t)mt * kRowsPerMat + 16 * quarter + 4 * (lane >> 3);
                bool bad = false;
                // (32 columns, sixteen swaps, at a time: steps without a real column are left out)
#pragma unroll
                for (int c0 = 0; c0 < kCols; c0 += 32) {
                    if (c0 >= ncols_here) break;
                    float *g = acc + c0;
#pragma unroll
                    for (int m = 0; m < 16; ++m) {                      // g[2m] = gate, g[2m + 1] = up of column c0 + 2m + parity
                        const float keep = odd ? g[2 * m + 1] : g[2 * m];
                        const float got = __shfl_xor_sync(0xffffffffu, odd ? g[2 * m] : g[2 * m + 1], 1);
                        g[2 * m] = odd ? got : keep;
                        g[2 * m + 1] = odd ? keep : got;
                    }
                    const float wl = c0 ? w_hi : w_lo;
                    float wv[4];                                        // route weight of column c0 + 8b + 2rr + parity
#pragma unroll
                    for (int b = 0; b < 4; ++b) wv[b] = __shfl_sync(0xffffffffu, wl, 8 * b + 2 * rr + (odd ? 1 : 0));
#pragma unroll
                    for (int m = 0; m < 16; ++m)                        // g[m] = silu(gate) * up
                        g[m] = swiglu_product(g[2 * m], g[2 * m + 1], 1.0f, p.limit);
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        float *r = g + 4 * b;
                        const float s0 = __shfl_xor_sync(0xffffffffu, o2 ? r[0] : r[1], 2), s1 = __shfl_xor_sync(0xffffffffu, o2 ? r[2] : r[3], 2);
                        if (o2) { r[0] = s0; r[2] = s1; } else { r[1] = s0; r[3] = s1; }
                    }
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        float *r = g + 4 * b;
                        const float s0 = __shfl_xor_sync(0xffffffffu, o4 ? r[0] : r[2], 4), s1 = __shfl_xor_sync(0xffffffffu, o4 ? r[1] : r[3], 4);
                        if (o4) { r[0] = s0; r[1] = s1; } else { r[2] = s0; r[3] = s1; }
                    }
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        const int col = c0 + 8 * b + 2 * rr + (odd ? 1 : 0);
                        if (col < ncols_here) {
                            const uint64_t srow = (uint64_t)cb.row0 + kCols * colhalf + col;
                            const float r0 = g[4 * b] * wv[b], r1 = g[4 * b + 1] * wv[b], r2 = g[4 * b + 2] * wv[b], r3 = g[4 * b + 3] * wv[b];
                            bad |= !isfinite(r0) || !isfinite(r1) || !isfinite(r2) || !isfinite(r3);
                            // f32 -> bf16 (round to nearest even; the product is finite or the launch is refused) -> the same values as fp16
                            const __nv_bfloat162 b01 = __floats2bfloat162_rn(r0, r1), b23 = __floats2bfloat162_rn(r2, r3);
                            const __half2 h01 = __float22half2_rn(__bfloat1622float2(b01)), h23 = __float22half2_rn(__bfloat1622float2(b23));
                            *reinterpret_cast<uint2 *>(p.mid + srow * p.M + m0) =
                                make_uint2(*reinterpret_cast<const uint32_t *>(&h01), *reinterpret_cast<const uint32_t *>(&h23));
                        }
                    }
                }
                if (bad) raise(p.status, YVEX_B200_STATUS_NUMERIC);
            } else {
                // store: out[(row0 + n)][mt*128 + row]. A thread holds 64 (affine qtypes: 32) token columns of ONE weight row, so a
                // direct store is one instruction per column and 2 bytes per lane. Instead every aligned
                // group of four lanes transposes 4 x 4 blocks with shuffles: lane 4a+j ends up with weight
                // rows 4a..4a+3 of token column 4b+j and stores them as one 8-byte vector (a quarter of
                // the store instructions). Two rounds of independent shuffles, as above.
                const bool odd = lane & 1, hi = lane & 2;
                const int j4 = lane & 3;
                const uint64_t m0 = (uint64_t)mt * kTileM + 32 * quarter + (lane & ~3);
#pragma unroll
                for (int b0 = 0; b0 < kCols / 4; b0 += 4) {           // four blocks (eight shuffles) per round
#pragma unroll
                    for (int b = b0; b < b0 + 4; ++b) {
                        float *r = acc + 4 * b;
                        const float s0 = __shfl_xor_sync(0xffffffffu, odd ? r[0] : r[1], 1), s1 = __shfl_xor_sync(0xffffffffu, odd ? r[2] : r[3], 1);
                        if (odd) { r[0] = s0; r[2] = s1; } else { r[1] = s0; r[3] = s1; }
                    }
#pragma unroll
                    for (int b = b0; b < b0 + 4; ++b) {
                        float *r = acc + 4 * b;
                        const float s0 = __shfl_xor_sync(0xffffffffu, hi ? r[0] : r[2], 2), s1 = __shfl_xor_sync(0xffffffffu, hi ? r[1] : r[3], 2);
                        if (hi) { r[0] = s0; r[1] = s1; } else { r[2] = s0; r[3] = s1; }
                    }
                }
#pragma unroll
                for (int b = 0; b < kCols / 4; ++b) {
                    const int col = 4 * b + j4;
                    if (col < ncols_here) {
                        const uint64_t srow = (uint64_t)cb.row0 + kCols * colhalf + col;
                        uint16_t *dst;
                        if (p.out_addr) dst = reinterpret_cast<uint16_t *>(__ldg(p.out_addr + srow));
                        else dst = p.out_bf16 + (p.out_rows ? (uint64_t)__ldg(p.out_rows + srow) : srow) * p.M;
                        // streaming stores: the results are not read again by this kernel and must not push the
                        // activation tiles and weight rows that other CTAs are about to reuse out of L2
                        // (round to nearest even; a launch with a non-finite sum is refused)
                        const __nv_bfloat162 lo = __floats2bfloat162_rn(acc[4 * b], acc[4 * b + 1]), hi2 = __floats2bfloat162_rn(acc[4 * b + 2], acc[4 * b + 3]);
                        if (dst) __stcs(reinterpret_cast<uint2 *>(dst + m0),
                                        make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi2)));
                    }
                }
            }
        }
    }
done:
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && sm->abort) raise(p.status, YVEX_B200_STATUS_TIMEOUT);
    if (warp == 0) tmem_dealloc(tmem, kTmemCols);
}

}  // namespace yb
