// A8W8 FP8 (E4M3) NT GEMM for sm_100a: C[M,N] = A[M,K] . B[N,K]^T with fp32 accumulation.
//
// Replaces the device kernels of the reference (gemm_a8w8_kernel, opus_gemm/gemm_a8w8_8wave.cc:261-563;
// gemm_a8w8_blockscale_kernel + scale_c_tile, block_scale_gemm/gemm_a8w8_blockscale_kernel_template.hpp:24-39,
// 203-591; flatmm_kernel for M above the skinny range, opus_fmm/flatmm_a8w8_gfx950.cc:243-548).
//
// One persistent CTA per SM, 12 warps:
//   warp 0      TMA producer   (one elected lane)  global -> shared ring, mbarrier complete_tx
//   warp 1      UMMA issuer    (one elected lane)  tcgen05.mma kind::f8f6f4 / kind::mxf8f6f4, TMEM alloc
//   warp 2      block scales: brings the scales into shared memory beside the operands (up to 192 columns), or reads them into L1 ahead of
//               their use (256 columns, ScaleToucher)
//   warp 3      block scales in a grid of one round: asks for the first ring of B ahead of the wait for the predecessor; idle otherwise, as warp 2 is
//               without block scales (register re-allocation works on whole warpgroups)
//   warps 4-11  epilogue: TMEM -> registers -> scale -> global
// TMEM holds two accumulator buffers of BN columns (three or four with block scales and fewer than 192).  Per-tensor / unscaled / MX modes accumulate a
// whole tile in one buffer while the epilogue drains the other.  Block-scale mode gives every
// 128-wide K group a FRESH buffer (the reference does the same with a fresh MFMA accumulator,
// kernel_template.hpp:317,334) and the epilogue warps fold it into register accumulators with
// acc += partial * (sfa[g][row] * sfb[nblk][g]) -- the analogue of scale_c_tile.
// Tiles are 128 rows by 128 or 256 columns, or in a grid of one round by as few as bring all SMs to work (32 to 224, MX 64 or 192, one_round_columns()
// of the launcher), or without block scales in several rounds by 160 or 192 (MX 192) where those waste less of the last one.  Few tiles with a long K: the CTAs of a cluster take a part of a 128 x 128 tile's K each (SPLIT) and sum their results in
// distributed shared memory; tile_splits() of the launcher says when.
#pragma once

#include <type_traits>

#include "sm100_ptx.cuh"

namespace b200 {

// MODE_ACC16: the accumulate-mode pipeline on bf16 operands (every K quantity counted in bytes by the launcher)
enum : int { MODE_ACC = 0, MODE_BLOCK = 1, MODE_MX = 2, MODE_ACC16 = 3 };
enum : int { BL_NK = 0, BL_FLAT = 1 };
enum : int { OUT_F32 = 0, OUT_BF16 = 1 };

struct GemmParams {
    CUtensorMap tmap_a;          // u8 [batch][M][K], box 128 bytes x a_rows, 128-byte swizzle
    CUtensorMap tmap_b;          // u8 [batch][N][K] (same box) or the flat 4-D view
    CUtensorMap tmap_sfa;        // pair kernels, MX: scale atoms as u8 [atoms*2][256], box 256 x 2
    CUtensorMap tmap_sfb;        // pair kernels, MX: box 256 x 2*atoms
    CUtensorMap tmap_c;          // pair kernels, block-scale, bf16 out: C [batch][M][N], box 64 x 32, 128-byte swizzle
    void* c;
    const float* sfa;            // block: fp32 [K/128][M];   MX: E8M0 atoms (uint8, see sf_relayout)
    const float* sfb;            // block: fp32 [N/128][K/128]; MX: E8M0 atoms
    const float* scale_a;        // per-tensor device scalars (may be null -> 1)
    const float* scale_b;
    long long ldc, c_batch;
    long long sfa_stride, sfb_stride, sfa_batch, sfb_batch;
    int m, n, k, batch;
    int tiles_m, tiles_n, tiles_total, kblocks;
    int a_rows;                  // rows of A's box (single-CTA kernels): 128, or M where that is little
    int out_dtype;
    int c_tma;                   // block-scale pair kernels: finished tiles leave through TMA bulk stores
    int inputs_ready;            // pair kernels: operands do not depend on the previous kernel (see b200_gemm_flags)
    int b_shared;                // pair kernels: every batch multiplies by the same B (B is read at batch coordinate 0)
    int batch_epoch;             // pair kernels: value a batch's ready word must have reached (with batch_ready)
    const int* batch_ready;      // pair kernels: one ready word per batch, or null
    // pair kernels, 256 x 256 tiles, 8-bit operands, not MX: the tiles from tail_first on (the last, partly filled
    // round of the persistent schedule) are each computed as tail_split (2 or 4) column parts of 256 / tail_split
    // columns by as many CTA pairs -- narrower MMAs over the full K, so every output element is summed exactly as in a
    // whole tile.  tmap_b_tail is B with a box of 128 / tail_split rows.  tail_split == 0: whole tiles only.
    CUtensorMap tmap_b_tail;
    int tail_first, tail_split;
    // single-CTA 128 x 128 tiles: the CTAs of a cluster take kb_per_split K blocks each of one tile (splits == 1: whole tiles)
    int splits, kb_per_split;
    int b_ahead;                 // single-CTA kernels, block scales, one round: the first K blocks of B are asked for ahead
    int* status;
};

// Work unit u of a pair kernel -> its tile and column part (part < 0: the whole tile).
__device__ __forceinline__ void unit_coords(const GemmParams& p, int u, int& t, int& part) {
    if (p.tail_split == 0 || u < p.tail_first) {
        t = u;
        part = -1;
    } else {
        const int r = u - p.tail_first;
        t = p.tail_first + r / p.tail_split;
        part = r - (t - p.tail_first) * p.tail_split;
    }
}

// store staging of one epilogue warp (see store_chunk_coalesced)
static constexpr int kOutStagePitch = 80;
static constexpr int kOutStageBytesPerWarp = 32 * kOutStagePitch;

template <int BN_, int MODE_, int BLAYOUT_, bool SPLIT_ = false>
struct GemmCfg {
    static constexpr bool SPLIT = SPLIT_;                           // a tile's K is split over a cluster
    static constexpr bool TOUCH = MODE_ == MODE_BLOCK && BN_ == 256;   // a warp reads the scales ahead of their use
    static constexpr bool FEED = MODE_ == MODE_BLOCK && BN_ != 256;    // a warp brings the scales into shared memory beside the operands
    static constexpr bool AB16 = MODE_ == MODE_ACC16;               // bf16 operands: same bytes, kind::f16 MMAs
    static constexpr int BM = 128, BN = BN_, BK = 128, MODE = AB16 ? MODE_ACC : MODE_, BLAYOUT = BLAYOUT_;
    static constexpr int A_BYTES = BM * BK;
    static constexpr int B_BYTES = BN * BK;
    static constexpr int SFA_BYTES = (MODE == MODE_MX) ? 512 : 0;
    static constexpr int SFB_ATOMS = (BN + 127) / 128;
    static constexpr int SFB_BYTES = (MODE == MODE_MX) ? SFB_ATOMS * 512 : 0;
    static constexpr int STAGE_BYTES = ((A_BYTES + B_BYTES + SFA_BYTES + SFB_BYTES + 1023) / 1024) * 1024;
    static constexpr int OUT_STAGE_BYTES = 8 * kOutStageBytesPerWarp;        // store staging of the eight epilogue warps
    // FEED: scales of so many K blocks, each the tile's rows of A and its one or two blocks of B.  Eight warps that load the scales themselves wait for them
    // however early they ask: a load queues behind all the operand tiles in flight, 200 KB a CTA.  Six register sets, requested six groups
    // ahead / a ring that fills with the operands (and so with a stage less of those), us: 333 x 5120 x 2048 9.0 / 7.9, 128 x 8192 x 8192 23.9 / 20.1 (no
    // loads at all 19.7), 512 x 4096 x 4096 13.9 / 12.0, 1024 x 1024 x 512 4.26 / 4.11, 2500 x 5120 x 3072 53.8 / 48.7.  Also tried on 128 x 8192 x 8192: the
    // reading-ahead warp of the 256 columns 22.8, register sets of 8 and 16 groups loaded together 23.7, 22.0.  On 256 columns the epilogue's
    // registers do not take it (spills, 333 x 7168 x 2048 12.0 / 15.2).
    static constexpr int SF_SLOTS = FEED ? 16 : 0, SF_SLOT_BYTES = (BM + 4) * 4;
    static constexpr int ROOM = 227 * 1024 - 1024 /*barriers*/ - 1024 /*alignment slack*/ - SF_SLOTS * SF_SLOT_BYTES;
    static constexpr int STAGES = (ROOM - OUT_STAGE_BYTES) / STAGE_BYTES < 8 ? (ROOM - OUT_STAGE_BYTES) / STAGE_BYTES : 8;   // ring with the staging behind it
    // Ring of a CTA with one tile, whose staging lies in the ring: 128 columns without block or MX scales seven stages instead of six.  Behind six
    // of them a long K waits for its operands, us, six / seven: 8-bit 128 x 8192 x 8192 19.8 / 18.4, 512 x 4096 x 4096 11.6 / 11.0, bf16
    // 128 x 8192 x 8192 35.1 / 33.0.  CTAs with several tiles keep the staging of its own: the next tile's loads are under way while
    // a result leaves, and stores from registers instead cost more than the stage gives (2500 x 5120 x 3072 45.0 / 41.5).
    static constexpr int STAGES_ONE = ROOM / STAGE_BYTES < 8 ? ROOM / STAGE_BYTES : 8;
    static constexpr int STAGING_END = STAGES * STAGE_BYTES + OUT_STAGE_BYTES;
    static constexpr int RING_BYTES = STAGES_ONE * STAGE_BYTES > STAGING_END ? STAGES_ONE * STAGE_BYTES : STAGING_END;
    static constexpr int SMEM_BYTES = RING_BYTES + 1024 /*barriers*/ + SF_SLOTS * SF_SLOT_BYTES + 1024 /*alignment slack*/;
    // accumulator buffers; block scales, a hand-off per K block: up to four, as many as tensor memory holds
    static constexpr int BUFS = !FEED ? 2 : BN <= 128 ? 4 : 512 / BN;
    static constexpr int ACC_COLS = BUFS * BN;
    static constexpr int SF_COLS = (MODE == MODE_MX) ? 4 + 4 * SFB_ATOMS : 0;
    static constexpr int TMEM_COLS = (ACC_COLS + SF_COLS) <= 32 ? 32 : (ACC_COLS + SF_COLS) <= 64 ? 64
                                   : (ACC_COLS + SF_COLS) <= 128 ? 128 : (ACC_COLS + SF_COLS) <= 256 ? 256 : 512;
    static constexpr int NCH = BN / 2;              // columns owned by one epilogue thread
    static constexpr bool STRADDLE = BN % 128 != 0 && 128 % BN != 0;    // a tile lies in two of the 128-column scale blocks
    static constexpr int THREADS = 384;
    static_assert(ACC_COLS + SF_COLS <= 512, "TMEM overflow");
    static_assert(BN % 32 == 0 && BN <= 256, "BN must be a multiple of 32, at most 256");
    static_assert(MODE != MODE_MX || BN % 64 == 0, "MX scales: a tile begins at the first or third column word of an atom of 128 columns");
    static_assert(STAGES >= 3 && STAGES_ONE <= 8, "ring depth");
    // a stage that is free says that the group STAGES + BUFS before its next one has been drained
    static_assert(!FEED || STAGES_ONE + BUFS <= SF_SLOTS, "scales stay until their group has been drained");
    static_assert(OUT_STAGE_BYTES <= STAGES * STAGE_BYTES, "the staging fits the ring");
    static_assert(!SPLIT || (BN == 128 && BM * BN * 4 <= RING_BYTES), "the partial sums fit the ring");
};

// Block scales: a warp that reads from every line of a tile's scales once, a few K groups before the TMA producer asks for the operands, so that the
// epilogue finds it in L1.  An epilogue warp that runs behind has some 300 clocks between asking for a group's scales and using
// them; a load that L1 misses takes 350 of a quiet L2 and 700 behind the operand tiles in flight, an L1 hit 110.  A hint: nothing waits
// for it.  (prefetch.global.L1 comes as far as L2, a later load takes 280 clocks: a third of the gain.)
struct ScaleToucher {
    static constexpr int kBatch = 4, kAhead = 3;             // groups per request; groups ahead of the producer
    float x[kBatch + 1] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f}, sum = 0.0f;
    int q = 0;                                               // K groups behind this one
    // One tile: A's rows [row0, row0 + 128), B's columns from col0 on.  *requested: the K block the producer is at.  False: give up.
    __device__ __forceinline__ bool tile(const GemmParams& p, int b, int row0, int col0, int bn, int groups, int lane, volatile int* requested,
                                         volatile int* abort_flag) {
        // A: the lanes' rows are at most five apart and the first and the last of the 128 are among them, so that every 32-byte sector has
        // one, wherever a group's scales begin.  B: two lanes for each 128-column block of the tile, the first and the last of the groups.
        // (A lane per 16 bytes of A and per block of B missed a sector where a row of scales is not a whole number of them, us, best of 15:
        // 16381 x 7168 x 8192 923.4 / 918.4; 16384 rows the same.)
        const int row = row0 + lane * 127 / 31, blk = (col0 >> 7) + (lane >> 1);
        const float* pa = p.sfa + b * p.sfa_batch + (row < p.m ? row : p.m - 1);
        const bool col_ok = blk <= (col0 + bn - 1) >> 7 && (blk << 7) < p.n;
        const float* pb = p.sfb + b * p.sfb_batch + (col_ok ? static_cast<long long>(blk) * p.sfb_stride : 0);
        bool go = true;
        for (int g = 0; g < groups && go; g += kBatch) {
            const int cnt = groups - g < kBatch ? groups - g : kBatch;
            int polls = 0;
            while (q > *requested + kAhead && go) {
                go = !*abort_flag && ++polls < (1 << 20);
                __nanosleep(200);
            }
            go = __all_sync(0xFFFFFFFFu, go);
            // (added up only here, so that the loads of the batch before have had its time to arrive)
#pragma unroll
            for (int i = 0; i <= kBatch; ++i) sum += x[i];
#pragma unroll
            for (int i = 0; i < kBatch; ++i)
                if (i < cnt) x[i] = ld_nc_f32(pa + static_cast<long long>(g + i) * p.sfa_stride);
            if (col_ok) x[kBatch] = ld_nc_f32(pb + g + (lane & 1 ? cnt - 1 : 0));
            q += cnt;
        }
        return go;
    }
    // keeps the loads (no sum has these bits)
    __device__ __forceinline__ void finish(volatile int* requested) {
#pragma unroll
        for (int i = 0; i <= kBatch; ++i) sum += x[i];
        if (__float_as_uint(sum) == 0xFFFFFFFFu) *requested = -1;
    }
};

// tile index -> (batch, m tile, n tile): groups of 8 M tiles walk N, so that the tiles resident at
// one time share few A row panels and few B column panels in L2.
__device__ __forceinline__ void tile_coords(const GemmParams& p, int t, int& b, int& mi, int& ni) {
    const int per_batch = p.tiles_m * p.tiles_n;
    b = t / per_batch;
    int r = t - b * per_batch;
    constexpr int GM = 8;
    const int group_sz = GM * p.tiles_n;
    const int grp = r / group_sz;
    const int first_m = grp * GM;
    const int rows = (p.tiles_m - first_m) < GM ? (p.tiles_m - first_m) : GM;
    const int in_grp = r - grp * group_sz;
    mi = first_m + in_grp % rows;
    ni = in_grp / rows;
}

// Store CNT consecutive output columns of one row, 16 bytes at a time where the address allows (vec_ok) and the columns are there.  bf16, element by
// element wherever one of the CNT columns is missing / by whole pieces, us: 4000 x 4088 x 512 18.7 / 13.7, 100 x 2040 x 1024 9.2 / 7.0, MX 2000 x
// 2040 x 1024 11.0 / 8.6, bf16 operands 2000 x 4040 x 512 11.6 / 11.15.  fp32 gains nothing by pieces (4000 x 4072 x 512 20.1), and a chunk that is all there
// has its own branch: both cost few rows their code (3 x 3592 x 256, fp32, 3.0 / 3.25).  A chunk that lies behind the last column is left out as a whole: its
// pieces, all looked at one by one, cost a last tile of few rows 0.6 (bf16 18 x 8512 x 64, four batches, 128 x 256 tiles 4.91 / 4.29; 40 rows 5.06 / 4.63).
template <int CNT>
__device__ __forceinline__ void store_row_chunk(const GemmParams& p, void* crow, int col0, const float* v,
                                                bool vec_ok) {
    const bool whole = vec_ok && col0 + CNT <= p.n;
    if (p.out_dtype == OUT_BF16) {
        __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(crow) + col0;
        auto piece = [&](const int j) {
            uint4 w;
            w.x = pack_bf16x2(v[j + 0], v[j + 1]);
            w.y = pack_bf16x2(v[j + 2], v[j + 3]);
            w.z = pack_bf16x2(v[j + 4], v[j + 5]);
            w.w = pack_bf16x2(v[j + 6], v[j + 7]);
            *reinterpret_cast<uint4*>(dst + j) = w;
        };
        if (whole) {
#pragma unroll
            for (int j = 0; j < CNT; j += 8) piece(j);
        } else if (!vec_ok || col0 < p.n) {
#pragma unroll
            for (int j = 0; j < CNT; j += 8) {
                if (vec_ok && col0 + j + 8 <= p.n) {
                    piece(j);
                } else {
#pragma unroll
                    for (int i = j; i < j + 8; ++i)
                        if (col0 + i < p.n) dst[i] = __float2bfloat16_rn(v[i]);
                }
            }
        }
    } else {
        float* dst = reinterpret_cast<float*>(crow) + col0;
        if (whole) {
#pragma unroll
            for (int j = 0; j < CNT; j += 4)
                *reinterpret_cast<float4*>(dst + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        } else {
#pragma unroll
            for (int j = 0; j < CNT; ++j)
                if (col0 + j < p.n) dst[j] = v[j];
        }
    }
}

// Coalesced store of one warp's 32-row x CNT-column chunk.  Every lane holds CNT consecutive columns of ITS row
// (the TMEM load layout), so a direct store would touch 32 different rows per instruction.  The chunk is written
// to a warp-private shared-memory buffer (row pitch 80 B: 16-byte accesses stay conflict-free) and read back
// transposed, so that one store instruction covers whole 32- or 64-byte row segments.
// `row0` is the output row of lane 0; `stage` is this warp's 2560-byte buffer.
// The way out of the last tile is in nobody's shadow.  With the pieces per row known at compile time and every read issued
// ahead of the stores (a loop with run-time divisions, one read and one store at a time, before), us: four batches of 700 x 2064 x 1152,
// fp32, 256 x 192 tiles 13.7 -> 12.7, 256 x 256 tiles 14.9 -> 13.2; 256 x 512 x 1024, bf16, 256 x 256 tiles 8.0 -> 7.3.
// store_chunk_staged: all columns in range, 16-byte stores allowed.  bf16: 16 or 32 columns; fp32: 16, a row of the buffer.
template <int CNT, bool BF16>
__device__ __forceinline__ void store_chunk_staged(const GemmParams& p, uint8_t* cbatch, uint8_t* stage, int row0, int col0, const float* v, int lane) {
    static_assert(CNT * (BF16 ? 2 : 4) <= 64, "a row of the staging buffer holds 64 bytes");
    constexpr int ESZ = BF16 ? 2 : 4, PIECES = CNT * ESZ / 16, ROWS = 32 / PIECES;       // 16-byte pieces per row, rows per instruction
    uint8_t* mine = stage + lane * kOutStagePitch;
    if constexpr (BF16) {
#pragma unroll
        for (int j = 0; j < CNT; j += 8) {
            uint4 w;
            w.x = pack_bf16x2(v[j + 0], v[j + 1]);
            w.y = pack_bf16x2(v[j + 2], v[j + 3]);
            w.z = pack_bf16x2(v[j + 4], v[j + 5]);
            w.w = pack_bf16x2(v[j + 6], v[j + 7]);
            *reinterpret_cast<uint4*>(mine + j * 2) = w;
        }
    } else {
#pragma unroll
        for (int j = 0; j < CNT; j += 4) *reinterpret_cast<float4*>(mine + j * 4) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
    }
    __syncwarp();
    const int c = lane % PIECES, r = lane / PIECES;
    const size_t pitch_c = static_cast<size_t>(p.ldc) * ESZ;
    const uint8_t* src = stage + r * kOutStagePitch + c * 16;
    uint8_t* dst = cbatch + (row0 + r) * pitch_c + static_cast<size_t>(col0) * ESZ + c * 16;
    // with all rows in range the reads go out together, then the stores
    if (row0 + 32 <= p.m) {
        uint4 w[PIECES];
#pragma unroll
        for (int i = 0; i < PIECES; ++i) w[i] = *reinterpret_cast<const uint4*>(src + i * ROWS * kOutStagePitch);
#pragma unroll
        for (int i = 0; i < PIECES; ++i) *reinterpret_cast<uint4*>(dst + i * ROWS * pitch_c) = w[i];
    } else {
#pragma unroll
        for (int i = 0; i < PIECES; ++i)
            if (row0 + r + i * ROWS < p.m)
                *reinterpret_cast<uint4*>(dst + i * ROWS * pitch_c) = *reinterpret_cast<const uint4*>(src + i * ROWS * kOutStagePitch);
    }
    __syncwarp();
}
// A chunk of 16 columns, or of 32 when the output is bf16 (any other goes out lane by lane, as the ragged and unaligned ones do).  kRagged: a chunk
// may lie across the last column; where none does, the code for it costs the block-scale pair kernel's loop (4096 x 7168 x 2048 66.4 / 67.3 us).
template <int CNT, bool kRagged = true>
__device__ __forceinline__ void store_chunk_coalesced(const GemmParams& p, uint8_t* cbatch, uint8_t* stage, int row0,
                                                      int col0, const float* v, int lane, bool vec_ok) {
    const bool bf16 = p.out_dtype == OUT_BF16;
    const int esz = bf16 ? 2 : 4;
    if (!(vec_ok && col0 + CNT <= p.n) || CNT * esz > 64) {
        const int row = row0 + lane;
        if (row < p.m) store_row_chunk<CNT>(p, cbatch + static_cast<size_t>(row) * p.ldc * esz, col0, v, kRagged && vec_ok);
        return;
    }
    if (bf16) store_chunk_staged<CNT, true>(p, cbatch, stage, row0, col0, v, lane);
    else if constexpr (CNT <= 16) store_chunk_staged<CNT, false>(p, cbatch, stage, row0, col0, v, lane);
}

// One epilogue warp's part of a split tile: rows split + ew * S, ... in steps of 8 S, each summed over the S CTAs of the cluster in
// the order of K, a lane four columns.  All the loads of a step are issued before the first is waited for (one row at a time, a
// remote load's latency per row, the sum of a 2-CTA cluster was most of what a split tile took longer).
template <int S>
__device__ __forceinline__ void sum_splits(const GemmParams& p, uint32_t smem_base, int t, int split, int ew, int lane, float scale, bool vec_ok) {
    constexpr int ROWS = (16 + S - 1) / S;                          // rows per step: a whole tile's in one
    int b, mi, ni;
    tile_coords(p, t, b, mi, ni);
    const int rows = p.m - mi * 128 < 128 ? p.m - mi * 128 : 128, col = ni * 128 + lane * 4;
    const size_t esz = (p.out_dtype == OUT_BF16) ? 2 : 4;
    float4 v[ROWS][S];
    const int r0 = split + ew * S;
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        const int r = r0 + i * 8 * S;
        const uint32_t at = smem_base + r * 512 + ((lane ^ (r & 7)) << 4);
        if (r < rows) {
#pragma unroll
            for (int q = 0; q < S; ++q) v[i][q] = ld_shared_cluster_f32x4(mapa_shared(at, q));
        }
    }
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        const int r = r0 + i * 8 * S;
        if (r >= rows) break;
        float4 sum = v[i][0];
#pragma unroll
        for (int q = 1; q < S; ++q) {
            sum.x += v[i][q].x;
            sum.y += v[i][q].y;
            sum.z += v[i][q].z;
            sum.w += v[i][q].w;
        }
        const float o[4] = {sum.x * scale, sum.y * scale, sum.z * scale, sum.w * scale};
        uint8_t* dst = reinterpret_cast<uint8_t*>(p.c) + (static_cast<size_t>(b) * p.c_batch + static_cast<size_t>(mi * 128 + r) * p.ldc + col) * esz;
        if (vec_ok && col + 4 <= p.n) {
            if (p.out_dtype == OUT_BF16) *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]));
            else *reinterpret_cast<float4*>(dst) = make_float4(o[0], o[1], o[2], o[3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (col + j >= p.n) continue;
                if (p.out_dtype == OUT_BF16) reinterpret_cast<__nv_bfloat16*>(dst)[j] = __float2bfloat16_rn(o[j]);
                else reinterpret_cast<float*>(dst)[j] = o[j];
            }
        }
    }
}

template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, 1) gemm_a8w8_sm100_kernel(const __grid_constant__ GemmParams p) {
    constexpr int BM = Cfg::BM, BN = Cfg::BN, BK = Cfg::BK, MODE = Cfg::MODE;
    constexpr int NCH = Cfg::NCH;

    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    // A CTA that computes one tile stages its result in the ring: every load and MMA has completed when the last accumulator has.
    const bool one_tile = Cfg::SPLIT || p.tiles_total <= static_cast<int>(gridDim.x);
    const uint32_t stages = one_tile ? Cfg::STAGES_ONE : Cfg::STAGES;
    // barrier block sits after the ring
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem_gen + Cfg::RING_BYTES);
    const uint32_t bar_full0 = smem_base + Cfg::RING_BYTES;
    const uint32_t bar_empty0 = bar_full0 + Cfg::STAGES_ONE * 8;
    const uint32_t bar_accf0 = bar_empty0 + Cfg::STAGES_ONE * 8;
    constexpr int BUFS = Cfg::BUFS;
    const uint32_t bar_acce0 = bar_accf0 + BUFS * 8;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * Cfg::STAGES_ONE + 2 * BUFS);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* requested = reinterpret_cast<volatile int*>(tmem_slot + 2);    // TOUCH: the K block the TMA producer is at
    const uint32_t sf0 = smem_base + Cfg::RING_BYTES + 1024;                     // FEED: the scales

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    // Launched with programmatic serialization: barriers, tensor memory and descriptors are set up while the predecessor
    // drains; nothing of its output is read, and nothing written, before pdl_wait().  In plain order / so, us
    // back to back: 8-bit 122 x 256 x 5120 12.3 / 11.4, quantiser and block-scale 100 x 7168 x 2048 12.1 / 11.0, MX 40 x 2048 x 2048
    // 10.0 / 8.8, bf16 1 x 4096 x 4096 16.6 / 16.0.
    pdl_launch_dependents();
    // With block scales a quantiser runs in front, as a rule, which leaves HBM idle.  Where B is a microsecond of it and more and several CTAs share a
    // tile of it, those of the first row of tiles ask for their first ring of B into L2 before the wait.  Quantiser and GEMM, weights
    // from HBM, not / so, us: 333 x 7168 x 2048 12.7 / 12.3, 500 x 8192 x 1024 11.25 / 10.6, 250 x 6144 x 1024 8.5 / 8.1, 180 x 9600 x 3072 15.0 / 14.5, 1000 x
    // 4096 x 2048 16.2 / 15.8; one row of tiles 120 x 4096 x 2048 9.0 / 9.1; MX 200 x 6144 x 4096 15.9 / 16.1.  Not without scales: behind another GEMM
    // it takes from that one's tail, twice where rows are not whole lines apart (802 x 4232 x 1776 13.4 / 13.8).
    if constexpr (MODE == MODE_BLOCK && !Cfg::SPLIT) {
        if (threadIdx.x == 3 * 32 && p.b_ahead) {
            int b, mi, ni;
            tile_coords(p, blockIdx.x, b, mi, ni);
            const int most = mi > 0 ? 0 : (p.kblocks < static_cast<int>(stages) ? p.kblocks : static_cast<int>(stages));
            for (int kb = 0; kb < most; ++kb) {
                if constexpr (Cfg::BLAYOUT == BL_NK) tma_prefetch_3d(&p.tmap_b, kb * BK, ni * BN, b);
                else tma_prefetch_4d(&p.tmap_b, 0, ni * (BN / 16), kb * (BK / 16), b);
            }
        }
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < Cfg::STAGES_ONE; ++s) {
            mbar_init(bar_full0 + s * 8, Cfg::FEED ? 33 : 1);    // FEED: and every lane of the feeding warp
            mbar_init(bar_empty0 + s * 8, 1);
        }
        for (int s = 0; s < BUFS; ++s) {
            mbar_init(bar_accf0 + s * 8, 1);
            mbar_init(bar_acce0 + s * 8, 8);     // one arrival per epilogue warp
        }
        *abort_flag = 0;
        *requested = 0;
        fence_barrier_init();
        fence_proxy_async_smem();
    }
    if (warp == 1) {
        tmem_alloc<1>(smem_u32(tmem_slot), Cfg::TMEM_COLS);
        tmem_relinquish<1>();
    }
    if (warp == 0 && lane == 0) {
        prefetch_tmap(&p.tmap_a);
        prefetch_tmap(&p.tmap_b);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();

    // A CTA of a split tile has that tile only, and K blocks [kb0, kb0 + kblocks) of it.  (Whole tiles walk blockIdx.x and gridDim.x
    // themselves: through variables of their own, MX 436 x 2432 x 2432 8.9 -> 9.6 us, bf16 1216 x 1416 x 7040 26.8 -> 28.1.)
    const int split = Cfg::SPLIT ? static_cast<int>(cluster_ctarank()) : 0;
    const int split_tile = Cfg::SPLIT ? static_cast<int>(blockIdx.x) / p.splits : 0;
    const int kb0 = split * p.kb_per_split;
    const int kblocks = Cfg::SPLIT ? (p.kb_per_split < p.kblocks - kb0 ? p.kb_per_split : p.kblocks - kb0) : p.kblocks;
    const int groups = (MODE == MODE_BLOCK) ? kblocks : 1;            // accumulator phases per tile
    const int kb_per_group = (MODE == MODE_BLOCK) ? 1 : kblocks;

    auto next_stage = [stages](uint32_t& s, uint32_t& ph) {           // ring stage and its phase
        if (++s == stages) {
            s = 0;
            ph ^= 1;
        }
    };

    if (warp < 4) {
        setmaxnreg_dec<40>();
        if (warp == 0 && lane == 0) {
            // ------------------------------ TMA producer ------------------------------
            uint32_t s = 0, ph = 0;
            bool ok = true;
            int asked = 0;
            for (int t = Cfg::SPLIT ? split_tile : static_cast<int>(blockIdx.x); t < p.tiles_total && ok; t += Cfg::SPLIT ? p.tiles_total : static_cast<int>(gridDim.x)) {
                int b, mi, ni;
                tile_coords(p, t, b, mi, ni);
                // MX: the atoms of 128 columns that the tile lies in, as far as there are
                const int atom_b = ni * BN / 128;
                const uint32_t sfb_bytes = MODE != MODE_MX ? 0u : BN <= 128 || atom_b + 1 < p.sfb_stride ? Cfg::SFB_BYTES : 512u;
                const uint32_t bytes = p.a_rows * BK + Cfg::B_BYTES + Cfg::SFA_BYTES + sfb_bytes;
                for (int kb = kb0; kb < kb0 + kblocks; ++kb, next_stage(s, ph)) {
                    if (!mbar_wait(bar_empty0 + s * 8, ph ^ 1, abort_flag, p.status, KSTAT_TIMEOUT_EMPTY)) {
                        ok = false;
                        break;
                    }
                    const uint32_t sa = smem_base + s * Cfg::STAGE_BYTES;
                    const uint32_t sb = sa + Cfg::A_BYTES;
                    const uint32_t full = bar_full0 + s * 8;
                    if constexpr (Cfg::TOUCH) *requested = asked++;
                    mbar_arrive_expect_tx(full, bytes);
                    tma_load_3d(sa, &p.tmap_a, full, kb * BK, mi * BM, b);
                    if constexpr (Cfg::BLAYOUT == BL_NK)
                        tma_load_3d(sb, &p.tmap_b, full, kb * BK, ni * BN, b);
                    else
                        tma_load_4d(sb, &p.tmap_b, full, 0, ni * (BN / 16), kb * (BK / 16), b);
                    if constexpr (MODE == MODE_MX) {
                        // scale-factor atoms: [batch][K/128][rows/128][512 B]
                        const uint8_t* sfa = reinterpret_cast<const uint8_t*>(p.sfa) + b * p.sfa_batch +
                                             (static_cast<long long>(kb) * p.sfa_stride + mi) * 512;
                        const uint8_t* sfb = reinterpret_cast<const uint8_t*>(p.sfb) + b * p.sfb_batch +
                                             (static_cast<long long>(kb) * p.sfb_stride + atom_b) * 512;
                        bulk_load(sb + Cfg::B_BYTES, sfa, 512, full);
                        bulk_load(sb + Cfg::B_BYTES + 512, sfb, sfb_bytes, full);
                    }
                }
            }
        } else if (warp == 1) {
            // ------------------------------ UMMA issuer (the warp; an elected lane issues) ------------
            const bool elected = elect_one() != 0;
            uint32_t s = 0, ph = 0, phase = 0;
            // Block scales, two waits a K block: both barriers of the next one are looked at ahead of this one's MMAs, so that a wait that is over costs
            // nothing then.  Without / with, us: 333 x 5120 x 2048 9.0 / 8.6, 512 x 4096 x 4096 14.0 / 13.5, 256 x 2048 x 8192 12.1 / 11.6; unscaled 10.3 / 10.5,
            // the pair kernel 21.3 / 26.5 (256 x 512 x 8192): there the next operands or buffer are seldom ready yet.
            bool ok = true, full_seen = false, free_seen = false;
            constexpr uint32_t idesc = make_idesc_f8(BM, BN);
            for (int t = Cfg::SPLIT ? split_tile : static_cast<int>(blockIdx.x); t < p.tiles_total && ok; t += Cfg::SPLIT ? p.tiles_total : static_cast<int>(gridDim.x)) {
                uint32_t sf_col = 0;                             // MX: the tile's first scale word in its first atom
                if constexpr (MODE == MODE_MX && BN % 128 != 0) {
                    int b, mi, ni;
                    tile_coords(p, t, b, mi, ni);
                    sf_col = (ni * BN & 127) / 32;
                }
                for (int g = 0; g < groups && ok; ++g, ++phase) {
                    const uint32_t as = phase % BUFS;
                    const uint32_t aph = (phase / BUFS) & 1;
                    if (!role_all<true>(free_seen) && !role_all<true>(mbar_wait(bar_acce0 + as * 8, aph ^ 1, abort_flag, p.status, KSTAT_TIMEOUT_ACC_E))) {
                        ok = false;
                        break;
                    }
                    const uint32_t tacc = tmem_base + as * BN;
                    for (int kb = 0; kb < kb_per_group; ++kb, next_stage(s, ph)) {
                        // The descriptors are formed before the wait, so that the MMAs follow it at once.  Behind it / before it, us, 128 x 128
                        // tiles: 8-bit 512 x 4096 x 4096 11.4 / 10.9, 128 x 8192 x 4096 15.4 / 14.7, block scales 512 x 4096 x 4096 13.85 / 13.05, bf16
                        // 333 x 5120 x 1024 7.3 / 7.0.
                        const uint32_t sa = smem_base + s * Cfg::STAGE_BYTES;
                        const uint32_t sb = sa + Cfg::A_BYTES;
                        constexpr uint32_t LBO = (BN / 16) * 256;
                        uint64_t da0 = make_smem_desc(sa, 16, 1024, kSwizzle128B);
                        uint64_t db0 = Cfg::BLAYOUT == BL_NK ? make_smem_desc(sb, 16, 1024, kSwizzle128B) : make_smem_desc(sb, LBO, 128, kSwizzleNone);
                        uint64_t dsf0 = make_smem_desc(sb + Cfg::B_BYTES, 0, 128, kSwizzleNone);                 // MX
                        asm volatile("" : "+l"(da0), "+l"(db0), "+l"(dsf0));
                        if (!role_all<true>(full_seen) && !role_all<true>(mbar_wait(bar_full0 + s * 8, ph, abort_flag, p.status, KSTAT_TIMEOUT_FULL))) {
                            ok = false;
                            break;
                        }
                        if constexpr (Cfg::FEED) {
                            uint32_t s1 = s, ph1 = ph;
                            next_stage(s1, ph1);
                            full_seen = mbar_probe(bar_full0 + s1 * 8, ph1);
                            free_seen = mbar_probe(bar_acce0 + (phase + 1) % BUFS * 8, (((phase + 1) / BUFS) & 1) ^ 1);
                        }
                        tc_fence_after();
                        if (!elected) continue;
                        if constexpr (MODE == MODE_MX) {
                            const uint32_t tsf = tmem_base + Cfg::ACC_COLS;
                            tmem_cp_sf<1>(tsf, dsf0);
#pragma unroll
                            for (int a = 0; a < Cfg::SFB_ATOMS; ++a) tmem_cp_sf<1>(tsf + 4 + 4 * a, dsf0 + 32 + 32 * a);
                        }
#pragma unroll
                        for (int k = 0; k < BK / 32; ++k) {
                            const uint64_t da = da0 + k * 2, db = db0 + (Cfg::BLAYOUT == BL_NK ? k * 2u : (k * 2 * LBO) >> 4);
                            const uint32_t accum = (kb > 0 || k > 0) ? 1u : 0u;
                            if constexpr (MODE == MODE_MX) {
                                const uint32_t tsf = tmem_base + Cfg::ACC_COLS;
                                umma_mxf8<1>(tacc, da, db, make_idesc_mxf8(BM, BN, k, k), accum, tsf, tsf + 4 + sf_col);
                            } else {
                                if constexpr (Cfg::AB16) umma_f16<1>(tacc, da, db, make_idesc_bf16(BM, BN), accum);
                                else umma_f8<1>(tacc, da, db, idesc, accum);
                            }
                        }
                        umma_commit<1>(bar_empty0 + s * 8);      // stage free once these MMAs retire
                    }
                    if (ok && elected) umma_commit<1>(bar_accf0 + as * 8);  // accumulator phase complete
                }
            }
        }
        if constexpr (Cfg::TOUCH) {
            // (Not for one tile of few K groups, all of which the epilogue asks for as early as this warp could.  With / without, one-round
            // grids, fp32 result, us: 3670 x 1280 x 128 6.33 / 6.24, 578 x 6272 x 256 6.84 / 6.74, 4734 x 1024 x 384 7.22 / 7.11; bf16 the same.)
            if (warp == 2 && !(one_tile && groups <= ScaleToucher::kAhead)) {
                ScaleToucher touch;
                bool go = true;
                for (int t = blockIdx.x; t < p.tiles_total && go; t += gridDim.x) {
                    int b, mi, ni;
                    tile_coords(p, t, b, mi, ni);
                    go = touch.tile(p, b, mi * BM, ni * BN, BN, groups, lane, requested, abort_flag);
                }
                touch.finish(requested);
            }
        }
        if constexpr (Cfg::FEED) {
            if (warp == 2) {
                // ------------------------------ scales into shared memory (the warp) ------------------------------
                // Four-byte copies, since a row of scales begins anywhere; they count towards the stage's full barrier, and whoever then sees the
                // group's accumulator sees its scales.
                uint32_t s = 0, ph = 0, it = 0;
                bool ok = true;
                for (int t = Cfg::SPLIT ? split_tile : static_cast<int>(blockIdx.x); t < p.tiles_total && ok; t += Cfg::SPLIT ? p.tiles_total : static_cast<int>(gridDim.x)) {
                    int b, mi, ni;
                    tile_coords(p, t, b, mi, ni);
                    const float* pa = p.sfa + b * p.sfa_batch + static_cast<long long>(kb0) * p.sfa_stride;
                    int row[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) row[j] = mi * BM + j * 32 + lane < p.m ? mi * BM + j * 32 + lane : p.m - 1;
                    // (a tile of a width between lies in two 128-column blocks of B; the second may be beyond the last)
                    const int blk = ni * BN / 128 + lane;
                    const float* pb = p.sfb + b * p.sfb_batch + static_cast<long long>(blk * 128 < p.n ? blk : p.n / 128 - 1) * p.sfb_stride + kb0;
                    for (int kb = 0; kb < kblocks; ++kb, ++it, next_stage(s, ph)) {
                        if (!role_all<true>(mbar_wait(bar_empty0 + s * 8, ph ^ 1, abort_flag, p.status, KSTAT_TIMEOUT_EMPTY))) {
                            ok = false;
                            break;
                        }
                        const uint32_t slot = sf0 + it % Cfg::SF_SLOTS * Cfg::SF_SLOT_BYTES;
#pragma unroll
                        for (int j = 0; j < 4; ++j) cp_async_4(slot + (j * 32 + lane) * 4, pa + row[j]);
                        if (lane <= (Cfg::STRADDLE ? 1 : 0)) cp_async_4(slot + (BM + lane) * 4, pb + kb);
                        cp_async_arrive(bar_full0 + s * 8);
                        pa += p.sfa_stride;
                    }
                }
                cp_async_wait_all();
            }
        }
        if constexpr (Cfg::SPLIT) {
            __syncwarp();
            cluster_arrive();
            cluster_wait();
        }
    } else {
        // ---------------------------------- epilogue ----------------------------------
        setmaxnreg_inc<232>();
        const int ew = warp - 4;
        const int quad = warp & 3;                 // TMEM lane quadrant this warp may touch
        const int half = ew >> 2;                  // which BN/2 column range
        const int row_in_tile = quad * 32 + lane;
        const uint32_t tmem_lane = static_cast<uint32_t>(quad * 32) << 16;
        const size_t esz = (p.out_dtype == OUT_BF16) ? 2 : 4;
        const bool vec_ok = ((reinterpret_cast<uintptr_t>(p.c) & 15) == 0) && ((p.ldc * esz) % 16 == 0) &&
                            ((p.c_batch * esz) % 16 == 0);
        float tscale = 1.0f;
        if constexpr (MODE == MODE_ACC) {
            if (p.scale_a) tscale *= __ldg(p.scale_a);
            if (p.scale_b) tscale *= __ldg(p.scale_b);
        }
        uint8_t* out_stage = smem_gen + (one_tile ? 0 : Cfg::STAGES * Cfg::STAGE_BYTES) + ew * kOutStageBytesPerWarp;
        uint32_t phase = 0;
        bool ok = true;
        for (int t = Cfg::SPLIT ? split_tile : static_cast<int>(blockIdx.x); t < p.tiles_total && ok; t += Cfg::SPLIT ? p.tiles_total : static_cast<int>(gridDim.x)) {
            int b, mi, ni;
            tile_coords(p, t, b, mi, ni);
            const int row = mi * BM + row_in_tile;
            const int col_base = ni * BN + half * NCH;
            uint8_t* cbatch = reinterpret_cast<uint8_t*>(p.c) + static_cast<size_t>(b) * p.c_batch * esz;
            // A warp whose 32 rows are not all there, and every warp of a tile of at most 32 rows, stores from its registers: with few
            // rows an instruction touches few lines, and there is nothing to wait for.  From registers / staged, us, 8-bit 128 x 128 tiles,
            // fp32 result: 1, 16, 32 x 2048 x 1024 4.77 / 5.26, 4.78 / 5.24, 4.99 / 5.25; bf16 result 1 x 2048 x 1024 4.77 / 4.87.  From 33
            // rows on staged, which wins where many CTAs store: 48, 64 x 12288 x 512 5.73 / 5.21, 6.19 / 5.25 (on few CTAs
            // 48 x 2048 x 1024 5.28 / 5.32).  (Block scales have no such tiles but the last of many rows.)
            const int rows = p.m - mi * BM;
            const bool direct = MODE != MODE_BLOCK && (rows <= 32 || rows - quad * 32 < 32);
            // this warp's 32 rows x CW columns of its part, from column `c` of it on
            auto put = [&](auto width, const int c, const float* o) {
                constexpr int CW = decltype(width)::value;
                if constexpr (Cfg::SPLIT) {
                    // partial sums, row by row; the 16-byte pieces of eight neighbouring rows lie in different banks
                    uint8_t* mine = smem_gen + row_in_tile * (BN * 4);
#pragma unroll
                    for (int j = 0; j < CW / 4; ++j)
                        *reinterpret_cast<float4*>(mine + (((half * (NCH / 4) + c / 4 + j) ^ (lane & 7)) << 4)) =
                            make_float4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
                    return;
                }
                const int row0 = mi * BM + quad * 32, col0 = col_base + c;
                if (direct || !vec_ok || col0 + CW > p.n) {
                    // (block scales: N is a multiple of 128, so that a chunk is all there or not at all, and these are the stores of an unaligned C)
                    if (row < p.m) store_row_chunk<CW>(p, cbatch + static_cast<size_t>(row) * p.ldc * esz, col0, o, MODE != MODE_BLOCK && vec_ok);
                } else if (p.out_dtype == OUT_BF16) {
                    store_chunk_staged<CW, true>(p, cbatch, out_stage, row0, col0, o, lane);
                } else {
#pragma unroll
                    for (int j = 0; j < CW; j += 16) store_chunk_staged<16, false>(p, cbatch, out_stage, row0, col0 + j, o + j, lane);
                }
            };
            using W32 = std::integral_constant<int, 32>;
            using W16 = std::integral_constant<int, 16>;

            if constexpr (Cfg::FEED) {
                // 64 columns per thread leave room to have both loads of a group in flight, and the buffer goes back before the FMAs;
                // four buffers keep the tensor core busy meanwhile.  Two buffers, handed back after the FMAs, scalar FMAs and stores
                // from registers / this loop and staged stores, us: 100 x 7168 x 2048 10.6 / 9.2, 200 x 7168 x 2048 11.3 / 9.6, 512 x 4096 x
                // 4096 16.8 / 15.0, 2500 x 5120 x 3072 77 / 59.
                constexpr int C32 = NCH / 32, TAIL = NCH % 32;       // loads of a group: 32 columns each, and one of 16
                static_assert(TAIL == 0 || TAIL == 16, "a thread's columns are a multiple of 16");
                unsigned long long acc2[NCH / 2];
#pragma unroll
                for (int j = 0; j < NCH / 2; ++j) acc2[j] = 0ull;
                // Columns up to the next scale block, and which of the tile's two blocks they begin in.  A loop for each place where the
                // blocks meet within a thread's columns (one loop that chooses: 512 x 4096 x 4096 on 160 columns 16.2 -> 15.7 us).
                const int left = 128 - (col_base & 127);
                const int blk = Cfg::STRADDLE ? (col_base >> 7) - (ni * BN >> 7) : 0;
                const uint32_t sf_row = sf0 + row_in_tile * 4, sf_col = sf0 + (BM + blk) * 4;
                auto k_loop = [&](auto left_tag) {
                    constexpr int LEFT = decltype(left_tag)::value;
                    for (int g = 0; g < groups; ++g, ++phase) {
                        const uint32_t as = phase % BUFS;
                        const uint32_t aph = (phase / BUFS) & 1;
                        if (!mbar_wait(bar_accf0 + as * 8, aph, abort_flag, p.status, KSTAT_TIMEOUT_ACC_F)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t taddr = tmem_base + tmem_lane + as * BN + half * NCH;
                        float v[NCH];
#pragma unroll
                        for (int c = 0; c < C32; ++c) tmem_ld32(taddr + c * 32, v + c * 32);
                        if constexpr (TAIL) tmem_ld16(taddr + C32 * 32, v + C32 * 32);
                        const uint32_t slot = phase % Cfg::SF_SLOTS * Cfg::SF_SLOT_BYTES;
                        const float sa = ld_shared_f32(sf_row + slot);
                        const float sc = sa * ld_shared_f32(sf_col + slot);
                        const unsigned long long sc2 = pack_f32x2(sc, sc);
                        unsigned long long sd2 = sc2;
                        if constexpr (LEFT < NCH) {
                            const float sd = sa * ld_shared_f32(sf_col + 4 + slot);
                            sd2 = pack_f32x2(sd, sd);
                        }
                        tmem_ld_wait();
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_acce0 + as * 8);
#pragma unroll
                        for (int j = 0; j < NCH / 2; ++j) acc2[j] = ffma2(pack_f32x2(v[2 * j], v[2 * j + 1]), 2 * j < LEFT ? sc2 : sd2, acc2[j]);
                    }
                };
                if constexpr (!Cfg::STRADDLE) {
                    k_loop(std::integral_constant<int, NCH>{});
                } else {
                    if (left >= NCH) k_loop(std::integral_constant<int, NCH>{});
                    else if (NCH > 64 && left == 64) k_loop(std::integral_constant<int, 64>{});
                    else if (TAIL && NCH > 48 && left == 48) k_loop(std::integral_constant<int, 48>{});
                    else if (left == 32) k_loop(std::integral_constant<int, 32>{});
                    else if constexpr (TAIL) k_loop(std::integral_constant<int, 16>{});
                }
                if (ok) {
                    float o[32];
#pragma unroll
                    for (int c = 0; c < C32; ++c) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) unpack_f32x2(acc2[c * 16 + j], o[2 * j], o[2 * j + 1]);
                        // (N is a multiple of 128: 16 columns are all there or none of them)
                        if (!TAIL || col_base + c * 32 + 32 <= p.n) {
                            put(W32{}, c * 32, o);
                        } else if (col_base + c * 32 + 16 <= p.n) {
                            put(W16{}, c * 32, o);
                        }
                    }
                    if constexpr (TAIL) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) unpack_f32x2(acc2[C32 * 16 + j], o[2 * j], o[2 * j + 1]);
                        if (col_base + C32 * 32 + 16 <= p.n) put(W16{}, C32 * 32, o);
                    }
                }
            } else if constexpr (MODE == MODE_BLOCK) {
                // 128 columns per thread: two 32-column loads in flight beside the accumulators, the buffer handed back when the last of
                // four has landed, scales of the next group (in L1, see ScaleToucher) asked for after that.  One load at a time, scalar FMAs,
                // the buffer handed back last and scales from L2 / so, us: 333 x 7168 x 2048 12.6 / 11.8, 4096 x 7168 x 2048 80.7 / 70.5, 8192^3
                // 661 / 585, 700 x 2048 x 7168 44.8 / 39.5.
                unsigned long long acc2[NCH / 2];
#pragma unroll
                for (int j = 0; j < NCH / 2; ++j) acc2[j] = 0ull;
                const float* sfa_p = p.sfa + b * p.sfa_batch + (row < p.m ? row : 0);
                const float* sfb_p = p.sfb + b * p.sfb_batch + static_cast<long long>(col_base / 128) * p.sfb_stride;
                const bool col_ok = col_base < p.n;
                float sa_cur = __ldg(sfa_p);
                float sb_cur = col_ok ? __ldg(sfb_p) : 0.0f;
                for (int g = 0; g < groups; ++g, ++phase) {
                    const uint32_t as = phase & 1;
                    const uint32_t aph = (phase >> 1) & 1;
                    if (!mbar_wait(bar_accf0 + as * 8, aph, abort_flag, p.status, KSTAT_TIMEOUT_ACC_F)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t taddr = tmem_base + tmem_lane + as * BN + half * NCH;
                    float v[2][32];
                    tmem_ld32(taddr, v[0]);
                    tmem_ld32(taddr + 32, v[1]);
                    const float sc = sa_cur * sb_cur;
                    const unsigned long long sc2 = pack_f32x2(sc, sc);
#pragma unroll
                    for (int c = 0; c < NCH / 32; ++c) {
                        if (c % 2 == 0) tmem_ld_wait();
                        if (c == NCH / 32 - 2) {
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(bar_acce0 + as * 8);
                            if (g + 1 < groups) {
                                sfa_p += p.sfa_stride;
                                ++sfb_p;
                                sa_cur = __ldg(sfa_p);
                                sb_cur = col_ok ? __ldg(sfb_p) : 0.0f;
                            }
                        }
#pragma unroll
                        for (int j = 0; j < 16; ++j) acc2[c * 16 + j] = ffma2(pack_f32x2(v[c & 1][2 * j], v[c & 1][2 * j + 1]), sc2, acc2[c * 16 + j]);
                        if (c + 2 < NCH / 32) tmem_ld32(taddr + (c + 2) * 32, v[c & 1]);
                    }
                }
                if (ok) {
#pragma unroll
                    for (int c = 0; c < NCH / 32; ++c) {
                        float o[32];
#pragma unroll
                        for (int j = 0; j < 16; ++j) unpack_f32x2(acc2[c * 16 + j], o[2 * j], o[2 * j + 1]);
                        put(W32{}, c * 32, o);
                    }
                }
            } else {
                const uint32_t as = phase & 1;
                const uint32_t aph = (phase >> 1) & 1;
                if (!mbar_wait(bar_accf0 + as * 8, aph, abort_flag, p.status, KSTAT_TIMEOUT_ACC_F)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t taddr = tmem_base + tmem_lane + as * BN + half * NCH;
                constexpr int CW = NCH % 32 == 0 ? 32 : 16, NC = NCH / CW;
                float v[2][CW];
                tmem_ld<CW>(taddr, v[0]);
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    tmem_ld_wait();
                    if (c + 1 < NC) tmem_ld<CW>(taddr + (c + 1) * CW, v[(c + 1) & 1]);
                    if (c + 1 == NC) {
                        // every column of this warp is in registers: hand the buffer back early
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_acce0 + as * 8);
                    }
                    if (MODE == MODE_ACC && !Cfg::SPLIT) {
#pragma unroll
                        for (int j = 0; j < CW; ++j) v[c & 1][j] *= tscale;
                    }
                    put(std::integral_constant<int, CW>{}, c * CW, v[c & 1]);
                }
                ++phase;
            }
        }
        if constexpr (Cfg::SPLIT) {
            // CTA r of the cluster sums rows r, r + splits, ... over all of them, in the order of K, a lane four columns
            __syncwarp();
            cluster_arrive();
            cluster_wait();
            // A split that gave up (an expired wait) has no sums to add: the tile is left unwritten then.
            const uint32_t gave_up = lane < p.splits ? ld_shared_cluster_u32(mapa_shared(smem_u32(tmem_slot + 1), lane)) : 0u;
            if (!__any_sync(0xFFFFFFFFu, gave_up != 0u)) {
                switch (p.splits) {
                    case 2: sum_splits<2>(p, smem_base, split_tile, split, ew, lane, tscale, vec_ok); break;
                    case 3: sum_splits<3>(p, smem_base, split_tile, split, ew, lane, tscale, vec_ok); break;
                    case 4: sum_splits<4>(p, smem_base, split_tile, split, ew, lane, tscale, vec_ok); break;
                    case 5: sum_splits<5>(p, smem_base, split_tile, split, ew, lane, tscale, vec_ok); break;
                    case 6: sum_splits<6>(p, smem_base, split_tile, split, ew, lane, tscale, vec_ok); break;
                    case 7: sum_splits<7>(p, smem_base, split_tile, split, ew, lane, tscale, vec_ok); break;
                    default: sum_splits<8>(p, smem_base, split_tile, split, ew, lane, tscale, vec_ok); break;
                }
            }
        }
    }
    if constexpr (Cfg::SPLIT) {
        // no CTA leaves while another one reads its partial sums
        __syncwarp();
        cluster_arrive();
        cluster_wait();
    }
    // ---------------------------------- teardown ----------------------------------
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc<1>(tmem_base, Cfg::TMEM_COLS);
    }
}

}  // namespace b200
