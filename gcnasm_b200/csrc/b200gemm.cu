// Host side of libb200gemm.so: argument validation, tile-config selection, TMA tensor-map
// construction and kernel launches behind the C ABI declared in include/b200gemm.h.
//
// Tile-config selection replaces the reference's compile-time traits structs
// (opus_gemm/gemm_a8w8_8wave.cc:36-96, block_scale_gemm/gemm_a8w8_blockscale_common.h:28-84,
// opus_fmm/flatmm_a8w8_gfx950.cc:36-104) with a run-time choice from a small static table.
#include "../../include/b200gemm.h"

#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "aux_kernels.cuh"
#include "decode_sm100.cuh"
#include "gemm_pair_sm100.cuh"
#include "gemm_sm100.cuh"
#include "host_staging.h"
#include "recent_table.h"
#include "weight_file.h"

namespace {

using namespace b200;

std::atomic<uint64_t> g_launches{0};
thread_local int g_last_cuda = 0;

__device__ int g_status_word;

#define CU_TRY(expr)                                   \
    do {                                               \
        cudaError_t e_ = (expr);                       \
        if (e_ != cudaSuccess) {                       \
            g_last_cuda = static_cast<int>(e_);        \
            return B200_ERR_CUDA;                      \
        }                                              \
    } while (0)

// ---- per-device state ------------------------------------------------------------------------
constexpr int kMaxDevices = 64;
struct DeviceState {
    bool init = false;
    int sm_count = 0;
    int cc_major = 0;
    int* status_ptr = nullptr;
    // cached buffers of b200_gemm_a8w8_host
    void* buf[8] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    size_t cap[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    // b200_gemm_a8w8_host: second stream for the copy-back of finished row slabs, one event per slab
    cudaStream_t copy_stream = nullptr;
    cudaEvent_t slab_done[16] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                                 nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    cudaEvent_t copies_done = nullptr;
    cudaStream_t peek_stream = nullptr;   // b200_peek_status: reads the status word without waiting for other streams
    Staging staging;                      // b200_gemm_a8w8_host: pinned ring for pageable operands (host_entry_mu)
    int* status_host = nullptr;           // ... and the pinned word its final look at the status goes to
    std::mutex host_entry_mu;             // b200_gemm_a8w8_host: one caller at a time per device (shared staging buffers)
};
DeviceState g_dev[kMaxDevices];
std::mutex g_mu;

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn g_encode = nullptr;
typedef CUresult (*StreamWriteValue32Fn)(CUstream, CUdeviceptr, cuuint32_t, unsigned int);
StreamWriteValue32Fn g_write_value32 = nullptr;     // null when the driver does not offer stream memory operations
StreamWriteValue32Fn g_wait_value32 = nullptr;      // cuStreamWaitValue32 has the same signature


int device_state(DeviceState** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        g_last_cuda = static_cast<int>(e);
        return B200_ERR_NO_DEVICE;
    }
    if (dev < 0 || dev >= kMaxDevices) return B200_ERR_NO_DEVICE;
    std::lock_guard<std::mutex> lk(g_mu);
    DeviceState& s = g_dev[dev];
    if (!s.init) {
        cudaDeviceProp prop;
        CU_TRY(cudaGetDeviceProperties(&prop, dev));
        s.sm_count = prop.multiProcessorCount;
        // B200GEMM_MAX_SMS caps the SMs the persistent GEMM grids occupy, so that a collective running on another
        // stream (the activation broadcast of the N-sharded mode) finds free SMs and overlaps with the GEMM
        if (const char* cap = std::getenv("B200GEMM_MAX_SMS")) {
            const int v = std::atoi(cap);
            if (v >= 2 && v < s.sm_count) s.sm_count = v;
        }
        s.cc_major = prop.major;
        if (prop.major != 10) return B200_ERR_NO_DEVICE;
        void* sym = nullptr;
        CU_TRY(cudaGetSymbolAddress(&sym, g_status_word));
        s.status_ptr = static_cast<int*>(sym);
        CU_TRY(cudaMemset(s.status_ptr, 0, sizeof(int)));
        if (!g_encode) {
            void* fn = nullptr;
            cudaDriverEntryPointQueryResult q;
            CU_TRY(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q));
            if (q != cudaDriverEntryPointSuccess || !fn) return B200_ERR_NO_DEVICE;
            g_encode = reinterpret_cast<EncodeTiledFn>(fn);
            void* wv = nullptr;
            if (cudaGetDriverEntryPoint("cuStreamWriteValue32", &wv, cudaEnableDefault, &q) == cudaSuccess &&
                q == cudaDriverEntryPointSuccess && wv)
                g_write_value32 = reinterpret_cast<StreamWriteValue32Fn>(wv);
            else
                cudaGetLastError();
            wv = nullptr;
            if (cudaGetDriverEntryPoint("cuStreamWaitValue32", &wv, cudaEnableDefault, &q) == cudaSuccess &&
                q == cudaDriverEntryPointSuccess && wv)
                g_wait_value32 = reinterpret_cast<StreamWriteValue32Fn>(wv);
            else
                cudaGetLastError();
        }
        s.init = true;
    }
    *out = &s;
    return B200_OK;
}

// SMs of the current device, whatever B200GEMM_MAX_SMS says (148 where it cannot be asked; asked once per device)
int physical_sms() {
    static std::atomic<int> known[kMaxDevices];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 148;
    int n = known[dev].load(std::memory_order_relaxed);
    if (n == 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
        known[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

// u8 tensor map of rank `rank`; dims/strides innermost first, strides[i] = byte stride of dim i+1
// Encoding a tensor map costs a driver call; serving loops present the same few buffers over and over, so
// the most recent encodings are kept (keyed by every encode parameter; a map holds no device-specific state
// beyond the address it was encoded for).
struct TmapKey {
    const void* base;
    uint64_t dims[5], strides[4];
    uint32_t box[5];
    int rank, swz, dtype;
};
// 512: weights, activations and results of some sixty layers.  Host time of a launch in a loop over 24, 64 and 156 maps, us: a list of 64 that is searched
// 3.29, 3.38, 3.66; 64 sets of two by hash, which lose some of a loop from 24 maps on, 3.25, 3.29, 3.34; this 3.24, 3.23, 3.23.
RecentTable<TmapKey, CUtensorMap, 512> g_tmaps;

int make_tmap(CUtensorMap* tm, const void* base, int rank, const uint64_t* dims, const uint64_t* strides,
              const uint32_t* box, CUtensorMapSwizzle swz, CUtensorMapDataType dtype = CU_TENSOR_MAP_DATA_TYPE_UINT8) {
    TmapKey key;
    std::memset(&key, 0, sizeof(key));
    key.base = base;
    key.rank = rank;
    key.swz = static_cast<int>(swz);
    key.dtype = static_cast<int>(dtype);
    for (int i = 0; i < rank; ++i) {
        key.dims[i] = dims[i];
        key.box[i] = box[i];
    }
    for (int i = 0; i + 1 < rank; ++i) key.strides[i] = strides[i];
    if (g_tmaps.find(key, tm)) return B200_OK;
    cuuint64_t gd[5], gs[4];
    cuuint32_t bx[5], es[5];
    for (int i = 0; i < rank; ++i) {
        gd[i] = dims[i];
        bx[i] = box[i];
        es[i] = 1;
    }
    for (int i = 0; i + 1 < rank; ++i) gs[i] = strides[i];
    CUresult r = g_encode(tm, dtype, static_cast<cuuint32_t>(rank), const_cast<void*>(base), gd,
                          gs, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        g_last_cuda = 100000 + static_cast<int>(r);
        return B200_ERR_CUDA;
    }
    g_tmaps.add(key, *tm);
    return B200_OK;
}

// row-major u8 [batch][rows][K] with a 128-byte-swizzled box of 128 (K) x box_rows
int make_rowmajor_tmap(CUtensorMap* tm, const void* base, int64_t rows, int64_t k, int64_t ld, int64_t batch,
                       int64_t batch_stride, uint32_t box_rows) {
    const uint64_t dims[3] = {static_cast<uint64_t>(k), static_cast<uint64_t>(rows), static_cast<uint64_t>(batch)};
    const uint64_t strides[2] = {static_cast<uint64_t>(ld),
                                 static_cast<uint64_t>(batch > 1 ? batch_stride : ld * rows)};
    const uint32_t box[3] = {128, box_rows, 1};
    return make_tmap(tm, base, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

// flat image [N/16][K/16][256 B] viewed as (256 B, slab, k-chunk, batch): a box {256, rows/16, 8, 1}
// lands in shared memory as [k-chunk][slab][256 B]
int make_flat_tmap(CUtensorMap* tm, const void* base, int64_t n, int64_t k, int64_t batch, int64_t batch_stride,
                   uint32_t box_rows) {
    const uint64_t dims[4] = {256, static_cast<uint64_t>(n / 16), static_cast<uint64_t>(k / 16),
                              static_cast<uint64_t>(batch)};
    const uint64_t strides[3] = {static_cast<uint64_t>(k * 16), 256,
                                 static_cast<uint64_t>(batch > 1 ? batch_stride : n * k)};
    const uint32_t box[4] = {256, box_rows / 16, 8, 1};
    return make_tmap(tm, base, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE);
}

// ---- validation and config selection -----------------------------------------------------------
struct Plan {
    int tile;        // b200_tile_hint value actually used
    int mt;          // decode token block
    int splits;      // decode K splits; otherwise, above 1: 128 x 128 tiles, each shared by so many CTAs, whatever `tile` says
    int columns;     // above 0: one CTA's tiles of 128 rows and so many columns, whatever `tile` says
};

// MX with few tokens: the K blocks from which the skinny-M kernel beats the 128 x 128 tiles, which have the shorter fixed part.  Its own
// is the sum over the splits of a panel: tokens / splits rows of remote loads, on every warp of the panel's CTAs; what the splits save
// grows with K.  So one split (more panels than half the SMs) and few tokens cross over early, 64 tokens in two splits late.  Time with
// the skinny kernel over time with the tiles, at 768, 1024, 1536, 2048, 2560 (N = 128 panels):
//   panels 75, 144 (one split)   m = 1  0.65 0.66 0.73 0.72 0.69   64  0.81 0.83 0.95 0.98 0.94     144:  1  0.77 .. 0.67  64  0.93 .. 0.97
//   panels 16                    m = 16 0.89 0.80 0.76 0.68 0.59   64  1.20 1.05 0.95 0.84 0.79
//   panels 64 (two splits)       m = 16 0.97 0.94 0.90 0.86 0.84   32  1.08 1.04 0.98 0.93 0.91   48  1.14 1.09 1.03 0.98 0.91
//                                m = 64 1.26 1.19 1.12 1.05 0.97
//   panels 74                    m = 32 1.04 1.01 1.00 0.98 0.92   48  1.15 1.13 1.10 1.07 0.97   64  1.28 1.22 1.18 1.14 1.03
// For instance, us, skinny kernel / tiles: 64 x 8192 x 1536 7.6 / 6.8, 64 x 9472 x 1664 8.5 / 7.2, 16 x 8192 x 1024 5.1 / 5.4, 64 x 9600 x 1024
// 4.7 / 5.7, 1 x 12288 x 1024 4.6 / 7.3.  Below six K blocks only four were measured (64 x 512 x 512 5.0 / 3.8).
constexpr int kMxSkinnyLeast = 6;
int64_t mx_skinny_kblocks(int64_t m, int64_t panels, int sm_count) {
    if (m <= 16 || panels * 2 > sm_count) return kMxSkinnyLeast;
    if (m <= 32 || panels * 4 <= sm_count) return 12;
    const int64_t line = (m + 2 * panels * 148 / sm_count - 88 + 5) / 6;       // a plane through the crossings of 33-64 tokens, 38-74 panels
    return line > 12 ? line : 12;
}

// CTAs that share a 128 x 128 tile, each with a part of K: as many as bring the K blocks of a CTA down furthest, if the clusters are all
// resident and what is saved is worth more than the exchange of the partial sums.  In K blocks, that takes 9 (block and MX scales, 0.25 and
// 0.31 us a block) or 13 (0.2 us; 15 on tiles of few rows, whose blocks are shorter) on few tiles, more on many, and a cluster of more than
// four two more.  Whole 128 x 128 tiles / split, us, weights from HBM, K = 2048, 4096, 8192 (narrow whole tiles where that is in brackets):
//   8-bit         100 x 512 (4 tiles)    6.2 (5.6)    9.2 / 6.6   15.1 / 7.5     256 x 4608 (72)   6.9 (6.3)    9.9 (9.4)    16.4 / 14.2
//                 256 x 2048 (32)        6.5 (5.8)    9.6 / 8.7   15.6 / 10.8
//   block scales  100 x 512              6.9 (6.1)   10.6 / 6.9   18.8 / 7.8     256 x 4608        7.4 (6.9)   11.9 / 10.8   20.1 / 15.0
//                 256 x 2048             7.2 (6.3)   11.4 / 9.0   19.5 / 11.3
//   MX            100 x 512              7.4 / 6.4   11.8 / 6.8   20.8 / 8.1     256 x 4608        8.1 / 8.1   12.7 / 11.5   21.8 / 16.8
// (At 1024 8-bit operands lose 1 us, block scales 0.5; MX 1705 x 256 x 1536 6.4 / 6.9, 8-bit 12 x 4232 x 3328 8.1 / 8.7.)
constexpr int kMaxTileSplits = 8;
constexpr int kSplitClusters[kMaxTileSplits + 1] = {0, 148, 74, 45, 33, 26, 22, 15, 15};     // resident at once on 148 SMs
// Tiles of up to 24 rows, the grid just too large for three CTAs a tile (46 to 50 tiles): two are slower than one where rows of A and B are
// not whole 128-byte lines apart, and up to 47 K blocks where B comes out of L2; with more tiles a whole tile is the slow one.  Whole /
// split, us, without scales: 4 x 6024 x 5872 15.6 / 19.7, x 8176 23.0 / 29.7, x 5376 with B from HBM 15.9 / 14.5, out of L2 12.0 / 13.9.  Mean
// of split / whole over 3000 sizes: other pitches 0.98 (0.7 to 1.4), whole lines and 48 K blocks or more 0.84, with B out of L2 0.87.
// (What had made them slower were the rows of A's box that are not there, see kBoxRows.  Since that box is of the rows that there are, these calls run on whole tiles of 64
// columns, and two CTAs a tile would be the faster ones at these sizes too: 4 x 6024 x 5872 11.7 / 10.7, out of L2 11.0 / 9.0, bf16 24 x 6256 x 4088 16.1 / 14.4, 14.6 / 12.9; 146
// random sizes 0.86 to 0.94, 0.78 to 0.87.  The line is older and test_split_of_few_rows holds it.)
// *equal: the K blocks that a CTA would take as long for; lines: rows of A and B whole 128-byte lines apart
int tile_splits(int64_t m, int64_t tiles, int64_t kblocks, bool slow, bool lines, int sm_count, int64_t* equal = nullptr) {
    const int64_t exchange = slow ? 9 + tiles / 32 : (m <= 32 ? 15 : 13) + tiles / 12;
    if (equal) *equal = kblocks;
    if (kblocks <= exchange) return 1;
    int best = 1;
    int64_t best_cost = kblocks;
    for (int s = 2; s <= kMaxTileSplits; ++s) {
        const int64_t per = (kblocks + s - 1) / s, cost = per + exchange + (s > 4 ? 2 : 0);
        if (per * (s - 1) >= kblocks || tiles > static_cast<int64_t>(kSplitClusters[s]) * sm_count / 148 || cost >= best_cost) continue;
        if (s == 2 && m <= 24 && tiles <= 50 && !(lines && kblocks >= 48)) continue;
        best = s;
        best_cost = cost;
    }
    if (equal) *equal = best_cost;
    return best;
}

// How the rows of an operand lie in memory, best first: each begins at a whole 128-byte line; at whole 32-byte sectors, some at a line; all of them within a line; every other
// one within a sector; all of them within a sector (a view that begins at an odd multiple of 16 bytes).  A row of a box then is in two lines, with the last two also in five
// sectors instead of four.
enum : int { kLines = 0, kSectors = 1, kOffLines = 2, kHalfSectors = 3, kNoSectors = 4 };
int row_starts(const void* base, int64_t pitch, int64_t batch_stride) {
    if (pitch % 32 != 0) return kHalfSectors;
    const uintptr_t at = reinterpret_cast<uintptr_t>(base) | static_cast<uintptr_t>(batch_stride);
    return (at & 31) != 0 ? kNoSectors : pitch % 128 != 0 ? kSectors : (at & 127) != 0 ? kOffLines : kLines;
}

// A grid of one round on `w` columns against a pair's tiles: the K blocks from which the pair is kept.  It takes less out of L2 for a K block, and of what the rows make
// dear; one CTA has the shorter way in and out.  One CTA / pair, mean over K blocks (100,000 random sizes; * with two rows of tiles):
//   whole lines    8-bit  192*  0.96 from 16 on, 1.00 at 24 to 31, 1.04 above (245 x 11920 x 6272 21.9 / 20.1), more rows 0.85 to 0.98; 224* 1.00 to 31, 1.02 above, four rows 1.01 from 40
//   whole sectors  8-bit  160   0.95 at 20;  192 0.92 at 9;  bf16 224 1.00 from 24 on, 160 and 192 0.75 to 0.96
//   off lines      8-bit  160   0.95 to 24, 1.03 above, 1.09 from 40;  192 1.00 at 12, 1.03 at 20, 1.17 above 40, * 0.96 at 15, 1.05 at 20;  224 1.08 to 1.16 (1794 x 1888 x 7168 28.3 / 22.4)
//                  bf16   192   0.99 at 35, 1.05 above 40;  224 0.98 at 20, 1.04 at 27, 1.12 above 30;  MX 192 0.97 at 27, 1.02 at 35, 1.06 above 40
//   half sectors   8-bit  160   0.97 from 12 to 14, 1.01 to 17, then 1.03;  192 0.98 at 9
//                  bf16   160   0.99 from 33 to 38, then 1.01 to 1.03, * 0.97 at 24, 1.02 at 27;  192 0.96 from 15, 1.00 from 18, 1.03 from 24, then to 1.13, * 1.00 at 15, 1.07 at
//                               18 (142 x 13792 x 3480 37.2 / 30.9);  224 0.98 from 9, 1.00 from 12, 1.04 from 15 to 1.10, * 1.03 from 9
//   no sectors     8-bit  160   0.97 from 9 to 14, then 1.04 to 1.19;  192 0.99 at 9, 1.10 from 12 on to 1.36;  224 1.25 to 1.46;  bf16 about as half sectors;  MX 192 0.96 from
//                               12, 1.00 from 15, 1.04 from 21 to 1.20
int64_t pair_from(int w, int64_t tm, int rows, bool block, bool mx, bool ab16) {
    constexpr int64_t never = int64_t{1} << 62;
    if (w < 160 || (block && rows == kOffLines)) return never;
    if (rows == kLines) return ab16 || mx || block ? never : w == 192 && tm <= 2 ? 28 : w == 224 && tm <= 4 ? (tm <= 2 ? 32 : 40) : never;
    if (ab16) {
        if (rows <= kOffLines) return w == 224 ? 24 : w == 192 && rows == kOffLines ? 40 : never;
        return w == 160 ? (tm <= 2 ? 25 : 36) : w == 192 ? (tm <= 2 ? 15 : 18) : (tm <= 2 ? 10 : 13);
    }
    if (mx) return rows == kNoSectors ? 16 : rows == kOffLines ? 34 : 10;
    if (w == 160) return rows == kSectors ? 20 : rows == kOffLines ? 25 : 15;
    return rows == kOffLines ? (tm <= 2 ? 16 : 13) : 10;
}

// ... and in several rounds against a pair's 256 columns.  By K blocks, 192 columns: half sectors 8-bit 0.97 at 6, 0.99 at 7, 1.05 at 8, bf16 0.99 at 8, 1.00 at 9, MX 0.99 at 9;
// no sectors 8-bit 0.97 at 5, 1.03 at 6, bf16 0.98 at 6, 1.00 at 7, MX 0.98 at 7, 1.00 at 8; off lines 8-bit 1.00 at 11, 1.04 at 14, bf16 0.97 at 14, 1.00 at 17.  160 columns: off
// lines 1.00 at 35, 1.02 above; no sectors 8-bit 1.04 at 9, bf16 0.95 at 11.
int64_t pair_from_rounds(int w, int rows, bool mx, bool ab16) {
    if (mx) return rows == kNoSectors ? 8 : 10;
    switch (rows) {
        case kLines: return int64_t{1} << 62;
        case kOffLines: return w == 160 ? 40 : ab16 ? 17 : 12;
        case kHalfSectors: return w == 160 ? 10 : ab16 ? 9 : 7;
        case kNoSectors: return w == 160 ? (ab16 ? 14 : 9) : ab16 ? 7 : 6;
        default: return 10;
    }
}

// One CTA's tiles in a grid of one round: the fewest columns that make one.  A K block takes what its operand tiles take out of L2, 128 rows of
// A and the tile's of B at some 70 bytes a clock, and the way in and out of a tile is the shorter the narrower it is, so as long as SMs are
// idle a narrower tile on more of them wins; and 160 to 224 columns make one round of what would be two of 128, or 256 with SMs idle.  us, kind of tile as
// before / narrowest, mean over 1300 to 1500 sizes each (up to 3000 rows, 18432 columns, K 8192): unscaled 0.884, block scales 0.896, bf16 0.874.
//   8-bit         256 x 512 x 1024    128 columns 4.5 / 32 3.6       333 x 7168 x 2048   256 columns 10.7 / 160 8.5    700 x 2048 x 7168  128 15.6 / 96 14.9
//   block scales  129 x 1024 x 1024   128         5.0 / 32 4.1       333 x 7168 x 2048   256         11.9 / 160 9.7    100 x 7168 x 2048  128  7.8 / 64  7.1
//   bf16          64 x 8192 x 2048    128        10.4 / 64 9.7       333 x 7168 x 1024   256 (pair)  10.9 / 160 8.5
//   MX            256 x 1024 x 1024   128         5.1 / 64 4.6       333 x 7168 x 2048   256 (pair)  11.3 / 192 9.3    1000 x 3456 x 2048  256  11.1 / 192 9.2
// MX: 64, 128 and 192, which begin at the first or the third scale word of an atom of 128 columns (mean of 1850 sizes 0.944).
// Not 96 or 224 columns for a short K (96 for 128: 175 x 6272 x 384 3.72 / 3.86; 224 for 256: 269 x 10240 x 256 4.96 / 5.67), not 224 with block scales,
// whose 256 columns take no longer, and nothing in the place of 256 (two rows of tiles and a long K are the pair's: 430 x 8448 x 7552 26.8 / 29.8).
// pair: the tile would be a pair's, rows: how they lie in memory (see row_starts).
int one_round_columns(int64_t tm, int64_t n, int64_t batch, int64_t kblocks, bool block, bool mx, bool pair, int rows, bool ab16, int sm_count) {
    for (int w : {32, 64, 96, 128, 160, 192, 224}) {
        if (tm * ((n + w - 1) / w) * batch > sm_count || (mx && w % 64 != 0)) continue;
        if ((w == 96 || w == 224) && kblocks < 6) continue;
        // Every other row begins within a sector and 128 columns give each tile two SMs, which share their way to L2: 128 / 96, mean of 28 sizes of 17 to 32
        // K blocks 1.04, 28 longer ones 0.99, 35 shorter 0.97 (100 x 9568 x 2064 9.2 / 10.5, bf16 119 x 9792 x 1096 10.1 / 11.7)
        if (w == 96 && tm == 1 && rows == kHalfSectors && kblocks > 16 && ((n + 127) / 128) * batch <= 76) continue;
        if (pair && kblocks >= pair_from(w, tm, rows, block, mx, ab16)) return 0;
        return w == 224 && block ? 0 : w;
    }
    return 0;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// ab16: `a` is the byte view of a bf16 problem (K and the A/B strides counted in bytes)
int validate(const b200_gemm_args* a, int sm_count, Plan* plan, bool ab16 = false) {
    if (!a || !a->ptr_a || !a->ptr_b || !a->ptr_c) return B200_ERR_BAD_ARG;
    if (a->m <= 0 || a->n <= 0 || a->k <= 0 || a->batch <= 0) return B200_ERR_BAD_ARG;
    if (a->scale_mode < 0 || a->scale_mode > 3 || a->b_layout < 0 || a->b_layout > 1 || a->out_dtype < 0 ||
        a->out_dtype > 1 || a->tile_hint < 0 || a->tile_hint > 8)
        return B200_ERR_BAD_ARG;
    if (ab16 && (a->scale_mode == B200_SCALE_BLOCK || a->scale_mode == B200_SCALE_MX)) return B200_ERR_UNSUPPORTED;
    if (a->m > 0x7FFFFFFF || a->n > 0x7FFFFFFF || a->k > 0x7FFFFFFF || a->batch > 65535) return B200_ERR_TOO_LARGE;
    if (a->stride_a < a->k || a->stride_c < a->n) return B200_ERR_BAD_ARG;
    // TMA: 16-byte aligned bases and row pitches
    if (!aligned16(a->ptr_a) || !aligned16(a->ptr_b)) return B200_ERR_UNSUPPORTED;
    if (a->stride_a % 16 != 0 || a->k % 16 != 0) return B200_ERR_UNSUPPORTED;
    if (a->batch > 1 && (a->stride_a_batch % 16 != 0 || a->stride_b_batch % 16 != 0)) return B200_ERR_UNSUPPORTED;
    if (a->b_layout == B200_B_NK_ROWMAJOR) {
        if (a->stride_b < a->k) return B200_ERR_BAD_ARG;
        if (a->stride_b % 16 != 0) return B200_ERR_UNSUPPORTED;
    } else {
        if (a->n % 16 != 0 || a->k % 128 != 0) return B200_ERR_UNSUPPORTED;   // flat needs whole 16x16 blocks
    }
    if (a->scale_mode == B200_SCALE_BLOCK) {
        if (!a->ptr_sfa || !a->ptr_sfb) return B200_ERR_BAD_ARG;
        // GROUP_M/N/K = 1/128/128 check of gemm_a8w8_blockscale_host.cc:183
        if (a->n % 128 != 0 || a->k % 128 != 0) return B200_ERR_UNSUPPORTED;
        if (a->stride_sfa < a->m || a->stride_sfb < a->k / 128) return B200_ERR_BAD_ARG;
    }
    if (a->scale_mode == B200_SCALE_MX) {
        if (!a->ptr_sfa || !a->ptr_sfb) return B200_ERR_BAD_ARG;
        if (a->k % 128 != 0) return B200_ERR_UNSUPPORTED;
        if (!aligned16(a->ptr_sfa) || !aligned16(a->ptr_sfb)) return B200_ERR_UNSUPPORTED;
        if (a->batch > 1 && (a->stride_sfa_batch % 16 != 0 || a->stride_sfb_batch % 16 != 0)) return B200_ERR_UNSUPPORTED;
    }

    // slabs that are still arriving, and one B for every batch: the 2-CTA tile kernels only
    const bool batch_ready = (a->flags & B200_GEMM_BATCH_READY) != 0;
    const bool b_shared = a->batch > 1 && a->stride_b_batch == 0;
    const bool pair_only = batch_ready || b_shared;
    if (batch_ready && !a->ptr_batch_ready) return B200_ERR_BAD_ARG;
    if (batch_ready && (ab16 || a->scale_mode == B200_SCALE_MX)) return B200_ERR_UNSUPPORTED;
    if (b_shared && a->scale_mode == B200_SCALE_BLOCK && a->stride_sfb_batch != 0) return B200_ERR_BAD_ARG;
    if (pair_only && a->m <= 128) return B200_ERR_UNSUPPORTED;

    Plan pl{B200_TILE_128x128, 0, 1, 0};
    const int64_t kblocks = (a->k + 127) / 128;
    const bool decode_ok = !pair_only && !ab16 && a->m <= 64 && (a->n % 16 == 0);
    int hint = a->tile_hint;
    if (hint == B200_TILE_DECODE && (!decode_ok || (a->scale_mode == B200_SCALE_MX && kblocks < kMxSkinnyLeast))) return B200_ERR_UNSUPPORTED;
    if (hint == B200_TILE_128x64) return B200_ERR_UNSUPPORTED;
    const bool mx = a->scale_mode == B200_SCALE_MX, slow = mx || a->scale_mode == B200_SCALE_BLOCK;
    // MX pair kernels address the scale atoms through a tensor map: batch strides in whole atoms
    const bool mx_pair_ok = !mx || a->batch == 1 || (a->stride_sfa_batch % 512 == 0 && a->stride_sfb_batch % 512 == 0);
    if (hint == B200_TILE_AUTO) {
        if (decode_ok && (!mx || kblocks >= mx_skinny_kblocks(a->m, (a->n + 127) / 128 * a->batch, sm_count))) {
            hint = B200_TILE_DECODE;
        } else {
            // cost of a persistent schedule: rounds (in tenths) x time per tile, proportional to the tile's N; with block
            // scales the tail of 256 x 256 pair tiles counts with the share of a round that its column parts take (plan_tail).
            // Not without: counted there too, 24 of 152 sizes (256...8192 in each dimension) go to 256 x 256 tiles, 10 of them up to
            // 10 % faster (4486 x 1232 x 1104 16.1 -> 14.5 us) and 14 up to 15 % slower (705 x 6160 x 416 9.15 -> 10.5); 1 % slower
            // in the mean.
            const int pairs = sm_count / 2;
            const int64_t tm2 = (a->m + 255) / 256, tm1 = (a->m + 127) / 128;
            int64_t best = -1;
            auto consider = [&](int tile, int bn, bool pair) {
                const int64_t tiles = (pair ? tm2 : tm1) * ((a->n + bn - 1) / bn) * a->batch;
                const int64_t units = pair ? pairs : sm_count;
                const bool block = a->scale_mode == B200_SCALE_BLOCK;
                int64_t tenths = (tiles + units - 1) / units * 10;
                const int64_t rem = tiles % units;
                if (pair && bn == 256 && block && tiles > units && rem > 0 && kblocks >= 4 && rem * 2 <= units)
                    tenths += (rem * 4 <= units ? 4 : 6) - 10;
                // w = time per output column, measured on 4096 x 7168 x 2048 (us a round and 1000 columns, 8-bit / block scales:
                // pair 256 27 / 40, 224 30 / 54, 192 30 / 56, 128 39 / 53; one CTA 256 33 / 49, 128 42 / 59; block scales, their scales
                // read ahead into L1, 37, 48, 49, 55; 41, 57): narrow and single-CTA tiles re-read more of A and B per flop, tiles that straddle the 128-column scale blocks
                // pay for the second scale, and the 224-column epilogue works in half-width pieces, which a short K shows.
                // Against the weights before (us): 4096^3 52.6 -> 47.9, 3794 x 3712 x 512 20.3 -> 16.7, 2750 x 7040 x 384 23.6 ->
                // 18.5; with block scales 3794 x 3712 x 512 20.3 -> 16.7.
                int64_t w;
                // A grid of one round is another matter: nothing hides a tile's way in and out, and both are shorter without a
                // partner CTA.  Against that stands what a K block takes, so for some kinds K decides; pair / one CTA, us back to back at
                // K = 512, 2048, 4096, 8192:
                //   8-bit, 128 columns       256 x 512 (8 tiles)   4.5 / 3.9   7.1 / 6.2   10.6 / 9.3    17.7 / 15.5
                //                            256 x 8192 (128)      5.3 / 4.0   8.3 / 7.0   12.2 / 10.5   21.5 / 20.0     one CTA
                //   block scales, 128        256 x 512 (8)         5.1 / 4.5   8.6 / 8.1   13.2 / 13.1   22.5 / 23.0
                //                            700 x 2048 (96)       5.6 / 4.5   9.4 / 9.0   14.7 / 14.7   24.6 / 25.6
                //                            2048 x 1024 (128)     6.0 / 4.5   9.8 / 9.0   15.1 / 14.9   35.0 / 25.9
                // With block scales a pair hands its accumulator over once for twice the rows, which wins from K = 4096 on until the
                // single tiles, one per SM, have more SMs than the pairs can use.  8-bit, 256 columns against the pair's best:
                // 769 x 4608 x 512 6.9 / 5.4, 1110 x 3968 x 3072 16.2 / 12.1, 1398 x 2688 x 4096 14.9 / 14.5, but 1096 x 2816 x 7168 21.5 /
                // 23.4 and, two rows of tiles and B streaming from HBM, 190 x 16640 x 4096 18.7 / 20.0: a single tile fetches 48 KB per K
                // block through four stages, a CTA of a pair 32 through six.
                // (Calls whose inputs are ready keep the pair's tiles: those start under the predecessor's last tiles, a single CTA waits.)
                // Block scales on 256 columns: as fast per column as the pair in one round, as long as K is not long (pair / one CTA 333 x 7168 x
                // 2048 12.2 / 11.8, 769 x 4608 x 512 7.6 / 6.4, 1024 x 4608 x 2048 13.4 / 12.3, 512 x 9472 x 8192 37.8 / 39.0); in several rounds
                // 1.02-1.18 times the pair's (the weights are the best of a sweep over 5783 sizes, all tiles timed; with fewer than four
                // K blocks the ones before it stand: 1332 x 7296 x 256, four batches, 27.0 / 29.5 on this tile).
                const bool ready = (a->flags & B200_GEMM_INPUTS_READY) != 0;
                const bool one_round = !pair && tiles <= units && !ab16 && !ready;
                if (one_round && block && bn >= 256) w = kblocks <= 40 ? 93 : 102;
                else if (block && !pair && bn >= 256 && !ready && kblocks >= 4) w = 110;
                else if (one_round && block && (kblocks <= 32 || tiles * 2 > units)) w = 125;
                else if (one_round && !block && (bn < 256 || kblocks <= (tm1 > 2 ? 32 : 24))) w = bn >= 256 ? 95 : 130;
                else if (!pair) w = bn >= 256 ? 125 : 155;
                else if (bn == 256) w = 100;
                else if (bn == 128) w = block && kblocks < 4 ? 130 : 140;
                else w = block ? 140 : (bn == 224 && kblocks < 8 ? 120 : 110);
                const int64_t cost = tenths * bn * w;
                if (best < 0 || cost < best) {
                    best = cost;
                    hint = tile;
                }
            };
            if (mx) {
                if (mx_pair_ok && a->m > 128) consider(B200_TILE_PAIR_256x256, 256, true);
                if (!pair_only) consider(B200_TILE_128x128, 128, false);
            } else {
                if (a->m > 128) {
                    consider(B200_TILE_PAIR_256x256, 256, true);
                }
                if (a->m > 128 && !ab16) {
                    consider(B200_TILE_PAIR_256x224, 224, true);
                    consider(B200_TILE_PAIR_256x192, 192, true);
                    consider(B200_TILE_PAIR_256x128, 128, true);
                }
                if (!pair_only) {
                    consider(B200_TILE_128x256, 256, false);
                    consider(B200_TILE_128x128, 128, false);
                }
            }
            // Few tiles with a long K: 128 x 128 tiles whose K is split may be the better ones (w as for a grid of one round).  A hint is
            // another matter: who names a tile gets it whole, with the bits that every kind of whole tile gives.  Where inputs are ready a
            // pair tile is kept, since it starts under its predecessor and a split one waits (in a chain, pair / split, us: 8-bit 256 x 512 x
            // 8192 2.9 / 8.3, 256 x 4608 x 8192 10.6 / 14.1, block scales 3.0 / 9.1, 12.3 / 16.0); a whole single-CTA tile waits as well (whole /
            // split: 8-bit 100 x 512 x 8192 15.1 / 7.4, MX 256 x 4608 x 8192 21.6 / 16.7, bf16 256 x 2048 x 4096 15.4 / 10.6).
            const bool starts_early = (a->flags & B200_GEMM_INPUTS_READY) && hint != B200_TILE_128x128 && hint != B200_TILE_128x256;
            if (!pair_only && !starts_early) {
                int64_t equal;
                const int rows_a = row_starts(a->ptr_a, a->stride_a, a->batch > 1 ? a->stride_a_batch : 0);
                const int rows_b = a->b_layout == B200_B_FLAT_16x16 ? kLines : row_starts(a->ptr_b, a->stride_b, a->batch > 1 ? a->stride_b_batch : 0);
                const int rows = rows_a > rows_b ? rows_a : rows_b;
                const bool lines = rows == kLines || rows == kOffLines;
                const int s = tile_splits(a->m, tm1 * ((a->n + 127) / 128) * a->batch, kblocks, slow, lines, sm_count, &equal);
                if (s > 1 && 10 * 128 * (ab16 ? 155 : a->scale_mode == B200_SCALE_BLOCK ? 125 : 130) * equal < best * kblocks) pl.splits = s;
                const bool block = a->scale_mode == B200_SCALE_BLOCK, single = hint == B200_TILE_128x128 || hint == B200_TILE_128x256;
                const int columns = one_round_columns(tm1, a->n, a->batch, kblocks, block, mx, !single, rows, ab16, sm_count);
                // A split takes as long as `equal` K blocks on 128 columns; narrow tiles are worth two more (block scales three), 32 columns one more.
                // Narrow over split by kblocks - equal, mean of 430 / 990 sizes: 8-bit 32 columns 0.92 at 1, 0.94 at 2, 0.96 at 3, from five parts on with up to 112 rows 1.06 at 3
                // (92 x 448 x 2688 6.2 / 5.8), 64 columns of several rows of tiles for two parts 1.02 at 1 and 2 (2106 x 312 x 4608 11.4 / 9.8); block scales 0.86, 0.89, 0.92, 0.95 at 4.
                // Rows that begin within sectors: 8-bit 32 columns 0.99 at 1, 1.02 at 2, otherwise to 1.14; block scales 64 columns 0.97, 1.01, 1.01, 32 as above.
                // Not for few rows, whose sums are quick (2 x 392 x 2816 4.4 / 6.1, block scales 68 x 384 x 2304, two batches, 6.1 / 6.6).
                int64_t worth = (block ? 4 : 3) + (columns == 32 && !(!block && s > 4 && a->m <= 112));
                if (ab16 || mx || a->m <= 80) worth = 0;
                else if (!lines) worth = rows != kNoSectors ? 1 : columns != 32 ? (block ? 2 : 1) : block ? worth : 2;
                else if (!block && columns == 64 && tm1 > 1 && s == 2) worth = 1;
                if (columns && kblocks - equal < worth) pl.splits = 1;
                if (pl.splits == 1) pl.columns = columns;
                // Several rounds without scales: 160 and 192 columns on one CTA, where they waste less of the last round (weights as above; bf16 has no pair tiles
                // of other widths to choose from).  Tile as before / so, mean of random sizes: bf16 0.865 (a third of 1690 sizes change), 8-bit 0.88 (one of 16);
                // 2000 x 3000 x 1024 bf16 15.5 / 14.7, 1000 x 6000 x 512 10.7 / 9.5.  A pair stays where rows are not whole lines apart, from ten K blocks on (bf16 1.0
                // at 16 to 24, 1.07 above 40), and with block scales, whose 160 and 192 columns take as long as 256 (700 x 8192 x 1024 12.6 / 13.4).  MX: 192 columns
                // for the pair's 256, up to ten K blocks (0.81 up to three, 0.88 to nine, then 0.97 and above twenty 1.02).
                // Not for a pair's 224 or 192 where rows begin within sectors (1.00 to 1.06; 2546 x 1304 x 912 10.0 / 9.3, 1352 x 2480 x 1040, two batches, 17.2 / 15.1),
                // nor for 224 of whole sectors (1.00) or of whole lines in three rounds (1.00).
                if (pl.splits == 1 && !columns && !block) {
                    constexpr int kWide[2][2] = {{160, 135}, {192, 125}};
                    const bool pair224 = hint == B200_TILE_PAIR_256x224, narrow_pair = pair224 || hint == B200_TILE_PAIR_256x192;
                    for (const auto& c : kWide) {
                        const int64_t rounds = (tm1 * ((a->n + c[0] - 1) / c[0]) * a->batch + sm_count - 1) / sm_count, cost = rounds * 10 * c[0] * c[1];
                        if ((mx && (single || c[0] != 192)) || (!single && kblocks >= pair_from_rounds(c[0], rows, mx, ab16))) continue;
                        if (c[0] == 192 && ((narrow_pair && rows >= kHalfSectors) || (pair224 && (rows == kSectors || (rounds > 2 && kblocks >= 10))))) continue;
                        if (rounds > 1 && cost < best) {
                            best = cost;
                            pl.columns = c[0];
                        }
                    }
                }
            }
        }
    }
    if (pair_only && !(hint == B200_TILE_PAIR_256x256 || hint == B200_TILE_PAIR_256x224 || hint == B200_TILE_PAIR_256x192 ||
                       hint == B200_TILE_PAIR_256x128))
        return B200_ERR_UNSUPPORTED;
    if (mx && !(hint == B200_TILE_128x128 || hint == B200_TILE_DECODE || (hint == B200_TILE_PAIR_256x256 && mx_pair_ok))) return B200_ERR_UNSUPPORTED;
    // bf16 operands: pair 256x256 and the two single-CTA tiles are built
    if (ab16 && !(hint == B200_TILE_128x128 || hint == B200_TILE_128x256 || hint == B200_TILE_PAIR_256x256)) return B200_ERR_UNSUPPORTED;
    pl.tile = hint;
    if (hint == B200_TILE_DECODE) {
        pl.mt = a->m <= 16 ? 16 : (a->m <= 32 ? 32 : 64);
        // K splits: fill the machine when there are fewer weight panels than SMs, and keep the
        // per-CTA scale staging within its shared-memory budget
        const int64_t tiles = ((a->n + 127) / 128) * a->batch;
        int splits = 1;
        while (tiles * splits * 2 <= sm_count && splits * 2 <= kblocks && splits < 16) splits *= 2;
        if (a->scale_mode == B200_SCALE_BLOCK) {
            const int64_t cap = decode_sf_bytes(pl.mt) / 4;
            while (((kblocks + splits - 1) / splits) * (pl.mt + 1) > cap) {
                splits *= 2;
                if (splits > kblocks) return B200_ERR_TOO_LARGE;
            }
        }
        pl.splits = splits;
    }
    if (plan) *plan = pl;
    return B200_OK;
}

// (one call per kernel and device: the attribute sticks, and a launch should cost no more host time than it has to)
template <auto kKernel>
int set_smem(int bytes) {
    static std::atomic<bool> done[kMaxDevices];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return B200_ERR_NO_DEVICE;
    if (done[dev].load(std::memory_order_acquire)) return B200_OK;
    CU_TRY(cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    done[dev].store(true, std::memory_order_release);
    return B200_OK;
}

// Launch with programmatic serialization: the kernel may be scheduled while its predecessor drains, and itself waits
// (griddepcontrol.wait) before it touches anything the predecessor may still be writing or reading.
template <class... P, class... A>
int launch_pdl_cluster(int cluster, void (*kernel)(P...), unsigned grid, unsigned threads, size_t smem, cudaStream_t st, const A&... args) {
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    std::memset(attr, 0, sizeof(attr));
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = static_cast<unsigned>(cluster);
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    CU_TRY(cudaLaunchKernelEx(&cfg, kernel, args...));
    g_launches.fetch_add(1);
    return B200_OK;
}
template <class... P, class... A>
int launch_pdl(void (*kernel)(P...), unsigned grid, unsigned threads, size_t smem, cudaStream_t st, const A&... args) {
    return launch_pdl_cluster(1, kernel, grid, threads, smem, st, args...);
}

// Clusters of `size` CTAs of a kernel that are resident at once (0: it cannot be told)
template <class Kernel>
int resident_clusters(Kernel kernel, int size, int threads, int smem) {
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(static_cast<unsigned>(size), 1, 1);
    cfg.blockDim = dim3(static_cast<unsigned>(threads), 1, 1);
    cfg.dynamicSmemBytes = static_cast<size_t>(smem);
    cudaLaunchAttribute attr;
    std::memset(&attr, 0, sizeof(attr));
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = static_cast<unsigned>(size);
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    return n;
}

template <int BN, int MODE, int BL>
int launch_gemm(const GemmParams& p, int grid, cudaStream_t st) {
    using Cfg = GemmCfg<BN, MODE, BL>;
    constexpr auto kernel = gemm_a8w8_sm100_kernel<Cfg>;
    int rc = set_smem<kernel>(Cfg::SMEM_BYTES);
    if (rc) return rc;
    return launch_pdl(kernel, static_cast<unsigned>(grid), Cfg::THREADS, Cfg::SMEM_BYTES, st, p);
}

template <int MODE, int BL>
int split_clusters(int size, int sm_count) {
    using Cfg = GemmCfg<128, MODE, BL, true>;
    constexpr auto kernel = gemm_a8w8_sm100_kernel<Cfg>;
    static std::atomic<int> known[kMaxDevices][kMaxTileSplits + 1];        // clusters resident at once + 1; 0: not asked yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
    int n = known[dev][size].load() - 1;
    if (n < 0) {
        if (set_smem<kernel>(Cfg::SMEM_BYTES)) return 0;
        n = resident_clusters(kernel, size, Cfg::THREADS, Cfg::SMEM_BYTES);
        if (n > 0) known[dev][size].store(n + 1);                           // (a question that failed is asked again)
    }
    return n < sm_count / size ? n : sm_count / size;
}
template <int BL>
int split_clusters(const b200_gemm_args* a, bool ab16, int size, int sm_count) {
    if (ab16) return split_clusters<MODE_ACC16, BL>(size, sm_count);
    switch (a->scale_mode) {
        case B200_SCALE_BLOCK: return split_clusters<MODE_BLOCK, BL>(size, sm_count);
        case B200_SCALE_MX: return split_clusters<MODE_MX, BL>(size, sm_count);
        default: return split_clusters<MODE_ACC, BL>(size, sm_count);
    }
}

thread_local int t_last_k_split = 0, t_last_columns = 0;           // the calling thread's last tile-kernel launch (b200_last_k_split, b200_last_columns)
// 128 x 128 tiles on one CTA each or, with p.splits > 1, on a cluster each
template <int MODE, int BL>
int launch_gemm128(const GemmParams& p, int grid, cudaStream_t st) {
    if (p.splits <= 1) return launch_gemm<128, MODE, BL>(p, grid, st);
    using Cfg = GemmCfg<128, MODE, BL, true>;
    constexpr auto kernel = gemm_a8w8_sm100_kernel<Cfg>;
    int rc = set_smem<kernel>(Cfg::SMEM_BYTES);
    if (rc) return rc;
    t_last_k_split = p.splits;
    return launch_pdl_cluster(p.splits, kernel, static_cast<unsigned>(p.tiles_total * p.splits), Cfg::THREADS, Cfg::SMEM_BYTES, st, p);
}

// ... and of any width that is built
template <int MODE, int BL>
int launch_columns(int columns, const GemmParams& p, int grid, cudaStream_t st) {
    if constexpr (MODE == MODE_MX) {
        switch (columns) {
            case 64: return launch_gemm<64, MODE, BL>(p, grid, st);
            case 128: return launch_gemm128<MODE, BL>(p, grid, st);
            case 192: return launch_gemm<192, MODE, BL>(p, grid, st);
            default: return B200_ERR_UNSUPPORTED;
        }
    } else
    switch (columns) {
        case 32: return launch_gemm<32, MODE, BL>(p, grid, st);
        case 64: return launch_gemm<64, MODE, BL>(p, grid, st);
        case 96: return launch_gemm<96, MODE, BL>(p, grid, st);
        case 128: return launch_gemm128<MODE, BL>(p, grid, st);
        case 160: return launch_gemm<160, MODE, BL>(p, grid, st);
        case 192: return launch_gemm<192, MODE, BL>(p, grid, st);
        case 224:
            if constexpr (MODE != MODE_BLOCK) return launch_gemm<224, MODE, BL>(p, grid, st);
            else return B200_ERR_UNSUPPORTED;
        default: return launch_gemm<256, MODE, BL>(p, grid, st);
    }
}

// K splits of the decode kernel that work as one cluster (above 8 the size is not portable and asked for explicitly)
constexpr int kMaxDecodeCluster = 16;

template <int MT, int MODE, int BL>
int decode_attrs() {
    using Cfg = DecodeCfg<MT, MODE, BL>;
    auto kernel = decode_a8w8_sm100_kernel<Cfg>;
    static std::atomic<bool> done[kMaxDevices];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return B200_ERR_NO_DEVICE;
    if (done[dev].load()) return B200_OK;
    CU_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
    CU_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    done[dev].store(true);
    return B200_OK;
}

// Clusters of `size` CTAs of this kernel that are resident at once (one CTA per SM; the SMs of a cluster belong to one
// GPC, so 16 clusters of 9 do not fit where 9 of 16 do).  Asked once per device and size.
template <int MT, int MODE, int BL>
int decode_clusters(int size, int sm_count) {
    using Cfg = DecodeCfg<MT, MODE, BL>;
    static std::atomic<int> known[kMaxDevices][kMaxDecodeCluster + 1];     // capacity + 1; 0: not asked yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
    int n = known[dev][size].load() - 1;
    if (n < 0) {
        if (decode_attrs<MT, MODE, BL>()) return 0;
        n = resident_clusters(decode_a8w8_sm100_kernel<Cfg>, size, Cfg::THREADS, Cfg::SMEM_BYTES);
        if (n > 0) known[dev][size].store(n + 1);
    }
    return n < sm_count / size ? n : sm_count / size;
}

// splits == 1: plain launch; > 1 without a workspace: the splits of a panel form a cluster
template <int MT, int MODE, int BL>
int launch_decode(const DecodeParams& p, int grid, cudaStream_t st) {
    using Cfg = DecodeCfg<MT, MODE, BL>;
    int rc = decode_attrs<MT, MODE, BL>();
    if (rc) return rc;
    const int cluster = p.splits > 1 && !p.partial ? p.splits : 1;
    return launch_pdl_cluster(cluster, decode_a8w8_sm100_kernel<Cfg>, static_cast<unsigned>(grid), Cfg::THREADS, Cfg::SMEM_BYTES, st, p);
}

// number of CTA pairs that can be resident at once (GPCs with an odd SM count strand one SM)
template <class Kernel>
int max_pairs(Kernel kernel, int threads, int smem, int sm_count) {
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(static_cast<unsigned>(sm_count & ~1), 1, 1);
    cfg.blockDim = dim3(static_cast<unsigned>(threads), 1, 1);
    cfg.dynamicSmemBytes = static_cast<size_t>(smem);
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) {
        cudaGetLastError();
        n = sm_count / 2;
    }
    return n < sm_count / 2 ? n : sm_count / 2;
}

// CTA pairs of this kernel that are resident at once on the current device (0 on failure)
template <int BN, int MODE, int BL>
int pair_capacity(int sm_count) {
    using Cfg = PairCfg<BN, MODE, BL>;
    constexpr auto kernel = gemm_a8w8_pair_sm100_kernel<Cfg>;
    if (set_smem<kernel>(Cfg::SMEM_BYTES)) return 0;
    static int pairs_cached[kMaxDevices] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= kMaxDevices) return 0;
    if (pairs_cached[dev] == 0) pairs_cached[dev] = max_pairs(kernel, Cfg::THREADS, Cfg::SMEM_BYTES, sm_count);
    return pairs_cached[dev];
}

// The last round of a persistent schedule is rarely full: 448 tiles on 74 CTA pairs leave 4 tiles for a seventh round, and 70
// pairs idle while those are computed.  GEMMs of 8-bit operands on 256 x 256 tiles (MX apart) therefore compute the
// tiles of a partial last round as 4 (or 2) column parts each, one part per pair, when there are pairs enough: the
// same K loop with 64- (128-) column MMAs, so every element is summed in exactly the order of a whole tile and
// nothing meets in memory.  4096 x 7168 x 2048, block scales, pre-shuffled B, without and with: 67.7 / 64.2 us; bf16 4096^3
// gains nothing (105.6 / 104.6, in a loop 119.9 both).  Sets p.tail_first / p.tail_split; B200GEMM_TAIL_SPLIT=0 in the
// environment (read once) switches it off.
thread_local int t_last_tail[2] = {0, 0};      // the calling thread's last pair launch (b200_last_tail_split)
void plan_tail(GemmParams& p, int capacity) {
    static const bool off = [] {
        const char* e = std::getenv("B200GEMM_TAIL_SPLIT");
        return e && *e == '0';
    }();
    p.tail_first = p.tiles_total;
    p.tail_split = 0;
    if (off || capacity <= 0 || p.kblocks < 4) return;
    const int full = (p.tiles_total / capacity) * capacity;
    const int rem = p.tiles_total - full;
    // (a problem of less than one round is left alone: measured, four times as many pairs on quarter tiles gain nothing there)
    if (rem == 0 || full == 0) return;
    const int split = rem * 4 <= capacity ? 4 : (rem * 2 <= capacity ? 2 : 0);
    if (!split) return;
    p.tail_first = full;
    p.tail_split = split;
    t_last_tail[0] = full;
    t_last_tail[1] = split;
}

template <int BN, int MODE, int BL>
int launch_pair(const GemmParams& p, int sm_count, cudaStream_t st) {
    using Cfg = PairCfg<BN, MODE, BL>;
    auto kernel = gemm_a8w8_pair_sm100_kernel<Cfg>;
    if (!p.tail_split) t_last_tail[0] = t_last_tail[1] = 0;
    const int capacity = pair_capacity<BN, MODE, BL>(sm_count);
    if (capacity <= 0) return B200_ERR_CUDA;
    int pairs = p.tiles_total < capacity ? p.tiles_total : capacity;
    if (p.tail_split) pairs = capacity;              // (plan_tail: whole rounds, then one round of parts)
    // programmatic serialization: this launch may begin while its predecessor drains; the kernel decides what it
    // does before the predecessor is complete (b200_gemm_flags)
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(static_cast<unsigned>(2 * pairs), 1, 1);
    cfg.blockDim = dim3(Cfg::THREADS, 1, 1);
    cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    std::memset(&attr, 0, sizeof(attr));
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    // A launch that waits for ready words starts in plain stream order, after its predecessor has COMPLETED.  With
    // programmatic serialization its first CTAs would be placed on whatever SMs the predecessor leaves free -- the very
    // SMs a capped grid (B200GEMM_MAX_SMS) sets aside for the collective that delivers the slabs -- and spin there on
    // words that collective can then never write.
    cfg.numAttrs = p.batch_ready ? 0 : 1;
    CU_TRY(cudaLaunchKernelEx(&cfg, kernel, p));
    g_launches.fetch_add(1);
    return B200_OK;
}

template <int BN>
int launch_pair_modes(const b200_gemm_args* a, const GemmParams& p, int sm_count, cudaStream_t st) {
    const bool flat = a->b_layout == B200_B_FLAT_16x16;
    switch (a->scale_mode) {
        case B200_SCALE_BLOCK:
            return flat ? launch_pair<BN, MODE_BLOCK, BL_FLAT>(p, sm_count, st) : launch_pair<BN, MODE_BLOCK, BL_NK>(p, sm_count, st);
        case B200_SCALE_MX:
            if constexpr (BN == 256)
                return flat ? launch_pair<BN, MODE_MX, BL_FLAT>(p, sm_count, st) : launch_pair<BN, MODE_MX, BL_NK>(p, sm_count, st);
            else
                return B200_ERR_UNSUPPORTED;
        default:
            return flat ? launch_pair<BN, MODE_ACC, BL_FLAT>(p, sm_count, st) : launch_pair<BN, MODE_ACC, BL_NK>(p, sm_count, st);
    }
}

template <int MODE, int BL>
int launch_decode_mt(int mt, const DecodeParams& p, int grid, cudaStream_t st) {
    switch (mt) {
        case 16: return launch_decode<16, MODE, BL>(p, grid, st);
        case 32: return launch_decode<32, MODE, BL>(p, grid, st);
        default: return launch_decode<64, MODE, BL>(p, grid, st);
    }
}
template <int MODE, int BL>
int decode_clusters_mt(int mt, int size, int sm_count) {
    switch (mt) {
        case 16: return decode_clusters<16, MODE, BL>(size, sm_count);
        case 32: return decode_clusters<32, MODE, BL>(size, sm_count);
        default: return decode_clusters<64, MODE, BL>(size, sm_count);
    }
}
int decode_clusters_any(int scale_mode, bool flat, int mt, int size, int sm_count) {
    if (scale_mode == B200_SCALE_MX) return flat ? decode_clusters_mt<MODE_MX, BL_FLAT>(mt, size, sm_count) : decode_clusters_mt<MODE_MX, BL_NK>(mt, size, sm_count);
    if (scale_mode == B200_SCALE_BLOCK) return flat ? decode_clusters_mt<MODE_BLOCK, BL_FLAT>(mt, size, sm_count) : decode_clusters_mt<MODE_BLOCK, BL_NK>(mt, size, sm_count);
    return flat ? decode_clusters_mt<MODE_ACC, BL_FLAT>(mt, size, sm_count) : decode_clusters_mt<MODE_ACC, BL_NK>(mt, size, sm_count);
}

// K splits of a decode launch that reduces in its clusters: of the counts whose clusters are all resident at once, the
// smallest one with the fewest K blocks per CTA, at least kMinSplitBlocks (1024 x 1024: 1 split 5.8 us, 2 5.3, 4 5.0, 8
// 5.3; a count whose clusters are not all resident costs a second wave: 7168 x 2048 2 splits 8.6 us, 3 12.9).  Block scales
// bound a CTA's K blocks by its staging area; when that takes more splits than fit a cluster the answer is 0 and the partials
// go through a workspace.
int cluster_splits(int64_t tiles, int64_t kblocks, int scale_mode, bool flat, int mt, int sm_count) {
    const bool block = scale_mode == B200_SCALE_BLOCK;
    constexpr int kMinSplitBlocks = 2;
    const int64_t most = block ? decode_sf_bytes(mt) / 4 / (mt + 1) : kblocks;      // K blocks one CTA can take
    const int64_t need = (kblocks + most - 1) / most;
    if (need > kMaxDecodeCluster || (need > 1 && decode_clusters_any(scale_mode, flat, mt, static_cast<int>(need), sm_count) < 1)) return 0;
    int best = static_cast<int>(need);
    for (int s = best + 1; s <= kMaxDecodeCluster && (kblocks + s - 1) / s >= kMinSplitBlocks; ++s)
        if (tiles * s <= sm_count && (kblocks + s - 1) / s < (kblocks + best - 1) / best && decode_clusters_any(scale_mode, flat, mt, s, sm_count) >= tiles) best = s;
    return best;
}

// Split-K workspaces of the skinny-M path.  One per (device, stream): launches on different streams never share
// partials.  A workspace that has been handed to a launch is never freed or moved before b200_release() -- a
// launch still in flight, or a CUDA graph that captured one, keeps using the pointer it was given -- so a stream
// that needs more gets an additional, larger one and the old one merely stops being handed out.
struct Scratch {
    int dev;
    cudaStream_t stream;
    float* ptr;
    size_t cap;          // bytes
    bool current;        // the one handed out for (dev, stream); older, smaller ones stay allocated until release
};
constexpr int kMaxScratch = 256;
Scratch g_scratch[kMaxScratch];
int g_scratch_count = 0;

int scratch_for(int dev, cudaStream_t st, size_t need, float** out) {
    std::lock_guard<std::mutex> lk(g_mu);
    Scratch* cur = nullptr;
    for (int i = 0; i < g_scratch_count; ++i)
        if (g_scratch[i].current && g_scratch[i].dev == dev && g_scratch[i].stream == st) cur = &g_scratch[i];
    if (cur && cur->cap >= need) {
        *out = cur->ptr;
        return B200_OK;
    }
    if (g_scratch_count == kMaxScratch) return B200_ERR_TOO_LARGE;      // too many (stream, size) generations
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) == cudaSuccess && cap != cudaStreamCaptureStatusNone)
        return B200_ERR_UNSUPPORTED;                                      // no allocation inside a capture
    float* ptr = nullptr;
    CU_TRY(cudaMalloc(&ptr, need));
    if (cur) cur->current = false;
    g_scratch[g_scratch_count++] = Scratch{dev, st, ptr, need, true};
    *out = ptr;
    return B200_OK;
}

// ---- allocation-free decode variant -------------------------------------------------------------------
// Split-K scratch that lives in the library image instead of in cudaMalloc'd memory: every GPU that loads the
// library holds these bytes until the process exits.  In host code the NAME of the array is only a host-side
// handle, not a device address; the address each device uses comes from cudaGetSymbolAddress, asked once
// per device with that device current.
constexpr size_t kStaticScratchFloats = 256 * 1024;                   // 1 MiB
static __device__ __align__(256) float g_static_scratch[kStaticScratchFloats];
float* g_static_scratch_ptr[kMaxDevices] = {nullptr};

int static_scratch(size_t need_floats, float** out) {
    int dev = 0;
    CU_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return B200_ERR_NO_DEVICE;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (!g_static_scratch_ptr[dev]) {
            void* sym = nullptr;
            CU_TRY(cudaGetSymbolAddress(&sym, g_static_scratch));     // this device's copy of the array
            g_static_scratch_ptr[dev] = static_cast<float*>(sym);
        }
        *out = g_static_scratch_ptr[dev];
    }
    return need_floats > kStaticScratchFloats ? B200_ERR_TOO_LARGE : B200_OK;
}

// use_static: the split-K partials go to the fixed array above (b200_gemm_a8w8_decode_static) instead of a
// cudaMalloc'd per-stream workspace.  Every element of the partials that the reduction reads is written by the
// launch first, so neither kind of workspace is ever cleared.
int run_decode(const b200_gemm_args* a, const Plan& pl, DeviceState* ds, cudaStream_t st, bool use_static = false) {
    DecodeParams p;
    std::memset(&p, 0, sizeof(p));
    const bool block = a->scale_mode == B200_SCALE_BLOCK, flat = a->b_layout == B200_B_FLAT_16x16;
    // (the limit of b200_gemm_a8w8_decode_static counts the splits a launch without clusters would make)
    const size_t need_floats = pl.splits > 1 ? static_cast<size_t>(pl.splits) * a->batch * a->m * a->n : 0;
    float* scratch = nullptr;
    if (use_static) {
        int rc0 = static_scratch(need_floats, &scratch);
        if (rc0) return rc0;
    }
    int splits = cluster_splits((a->n + 127) / 128 * a->batch, (a->k + 127) / 128, a->scale_mode, flat, pl.mt, ds->sm_count);
    if (splits == 0) {
        splits = pl.splits;
        if (use_static) {
            p.partial = scratch;
        } else if (splits > 1) {
            int dev = 0;
            CU_TRY(cudaGetDevice(&dev));
            int rc0 = scratch_for(dev, st, need_floats * sizeof(float), &p.partial);
            if (rc0) return rc0;
        }
    }
    int rc;
    if (a->b_layout == B200_B_NK_ROWMAJOR)
        rc = make_rowmajor_tmap(&p.tmap_w, a->ptr_b, a->n, a->k, a->stride_b, a->batch, a->stride_b_batch, 128);
    else
        rc = make_flat_tmap(&p.tmap_w, a->ptr_b, a->n, a->k, a->batch, a->stride_b_batch, 128);
    if (rc) return rc;
    rc = make_rowmajor_tmap(&p.tmap_x, a->ptr_a, a->m, a->k, a->stride_a, a->batch, a->stride_a_batch, static_cast<uint32_t>(a->m));
    if (rc) return rc;
    p.c = a->ptr_c;
    p.sfa = static_cast<const float*>(a->ptr_sfa);
    p.sfb = static_cast<const float*>(a->ptr_sfb);
    p.scale_a = a->scale_mode == B200_SCALE_TENSOR ? a->ptr_scale_a : nullptr;
    p.scale_b = a->scale_mode == B200_SCALE_TENSOR ? a->ptr_scale_b : nullptr;
    p.ldc = a->stride_c;
    p.c_batch = a->stride_c_batch;
    const bool mx = a->scale_mode == B200_SCALE_MX;
    p.sfa_stride = mx ? (a->m + 127) / 128 : a->stride_sfa;       // MX: atoms per K block
    p.sfb_stride = mx ? (a->n + 127) / 128 : a->stride_sfb;
    p.sfa_batch = a->stride_sfa_batch;
    p.sfb_batch = a->stride_sfb_batch;
    p.m = static_cast<int>(a->m);
    p.n = static_cast<int>(a->n);
    p.k = static_cast<int>(a->k);
    p.batch = static_cast<int>(a->batch);
    p.tiles_n = static_cast<int>((a->n + 127) / 128);
    p.kblocks = static_cast<int>((a->k + 127) / 128);
    p.splits = splits;
    p.kb_per_split = (p.kblocks + splits - 1) / splits;
    p.out_dtype = a->out_dtype;
    p.inputs_ready = (a->flags & B200_GEMM_INPUTS_READY) ? 1 : 0;
    p.status = ds->status_ptr;
    const int grid = p.tiles_n * p.batch * splits;
    if (flat)
        rc = mx ? launch_decode_mt<MODE_MX, BL_FLAT>(pl.mt, p, grid, st)
                : (block ? launch_decode_mt<MODE_BLOCK, BL_FLAT>(pl.mt, p, grid, st) : launch_decode_mt<MODE_ACC, BL_FLAT>(pl.mt, p, grid, st));
    else
        rc = mx ? launch_decode_mt<MODE_MX, BL_NK>(pl.mt, p, grid, st)
                : (block ? launch_decode_mt<MODE_BLOCK, BL_NK>(pl.mt, p, grid, st) : launch_decode_mt<MODE_ACC, BL_NK>(pl.mt, p, grid, st));
    if (rc) return rc;
    if (splits > 1 && p.partial) {
        const long long per_split = static_cast<long long>(a->batch) * a->m * a->n;
        const int threads = 256;
        const unsigned blocks = static_cast<unsigned>((per_split + threads - 1) / threads);
        decode_splitk_reduce_kernel<<<blocks, threads, 0, st>>>(p.partial, a->ptr_c, splits, per_split, p.m, p.n,
                                                               p.ldc, p.c_batch, p.out_dtype);
        CU_TRY(cudaGetLastError());
        g_launches.fetch_add(1);
    }
    return B200_OK;
}

// Up to so many rows, A's box is of the rows that there are (what lies behind them in a stage is anything, and so are the rows of the
// accumulator that nobody stores).  A box that reaches beyond the matrix is filled with zeros, but each row that is not there still
// costs a request, all of them in few places of L2: boxes of 128 rows in a ring of six on 144 CTAs take 918 clocks each with one row there,
// 806 with 24, 522 with 32 and more; boxes of 16 rows with one there 522.  128 rows / the rows there are, us: bf16 1 x 5440 x 1792 11.7 / 8.8, 16 x 5440 x
// 2048 10.6 / 8.2, 4 x 8192 x 4096 18.9 / 14.5, 8-bit 5 x 5448 x 4096 10.5 / 7.9; 40 x 5440 x 2048 and 1 x 1024 x 1024 (8 tiles) the same.  The few rows
// of a last tile below others are not worth a second box: its CTAs are half of a grid at most (8-bit 140 x 8192 x 2048 6.4 / 6.45).
constexpr int kBoxRows = 127;

int run_gemm(const b200_gemm_args* a, const Plan& pl, DeviceState* ds, cudaStream_t st, bool ab16 = false) {
    int BN = 128;
    bool pair = false;
    // The plan took the clusters that are resident at once from a table; where this device holds fewer, the tile that b200_gemm_check reports is launched whole.
    // (On 148 SMs, and on any part of them, as many are resident as the table says.)
    int splits = pl.splits;
    if (splits > 1) {
        const int64_t tiles = (a->m + 127) / 128 * ((a->n + 127) / 128) * a->batch;
        const int room = a->b_layout == B200_B_FLAT_16x16 ? split_clusters<BL_FLAT>(a, ab16, splits, ds->sm_count)
                                                          : split_clusters<BL_NK>(a, ab16, splits, ds->sm_count);
        if (room < tiles) splits = 1;
    }
    switch (splits > 1 || pl.columns ? B200_TILE_128x128 : pl.tile) {
        case B200_TILE_128x256: BN = 256; break;
        case B200_TILE_PAIR_256x256: BN = 256; pair = true; break;
        case B200_TILE_PAIR_256x224: BN = 224; pair = true; break;
        case B200_TILE_PAIR_256x192: BN = 192; pair = true; break;
        case B200_TILE_PAIR_256x128: BN = 128; pair = true; break;
        default: BN = pl.columns ? pl.columns : 128; break;
    }
    const int BMT = pair ? 256 : 128;                 // output rows per tile
    const int BROWS = pair ? BN / 2 : BN;             // B rows one CTA loads
    GemmParams p;
    std::memset(&p, 0, sizeof(p));
    p.a_rows = !pair && a->m <= kBoxRows ? static_cast<int>(a->m) : 128;
    int rc = make_rowmajor_tmap(&p.tmap_a, a->ptr_a, a->m, a->k, a->stride_a, a->batch, a->stride_a_batch, static_cast<uint32_t>(p.a_rows));
    if (rc) return rc;
    const bool b_shared = a->batch > 1 && a->stride_b_batch == 0;      // one B for every batch (validate(): pair tiles)
    const int64_t b_batches = b_shared ? 1 : a->batch;
    if (a->b_layout == B200_B_NK_ROWMAJOR)
        rc = make_rowmajor_tmap(&p.tmap_b, a->ptr_b, a->n, a->k, a->stride_b, b_batches, a->stride_b_batch, BROWS);
    else
        rc = make_flat_tmap(&p.tmap_b, a->ptr_b, a->n, a->k, b_batches, a->stride_b_batch, BROWS);
    if (rc) return rc;
    if (pair && a->scale_mode == B200_SCALE_MX) {
        // scale atoms as rows of 256 bytes; one atom = 2 rows
        const uint64_t bytes_a = a->batch > 1 ? static_cast<uint64_t>(a->stride_sfa_batch) * a->batch : b200_mx_sf_bytes(a->m, a->k);
        const uint64_t bytes_b = a->batch > 1 ? static_cast<uint64_t>(a->stride_sfb_batch) * a->batch : b200_mx_sf_bytes(a->n, a->k);
        const uint64_t da[2] = {256, bytes_a / 256}, db[2] = {256, bytes_b / 256};
        const uint64_t str[1] = {256};
        const uint32_t box_a[2] = {256, 2}, box_b[2] = {256, static_cast<uint32_t>(2 * ((BN + 127) / 128))};
        if ((rc = make_tmap(&p.tmap_sfa, a->ptr_sfa, 2, da, str, box_a, CU_TENSOR_MAP_SWIZZLE_NONE))) return rc;
        if ((rc = make_tmap(&p.tmap_sfb, a->ptr_sfb, 2, db, str, box_b, CU_TENSOR_MAP_SWIZZLE_NONE))) return rc;
    }
    if (pair && a->scale_mode == B200_SCALE_BLOCK && a->out_dtype == B200_OUT_BF16 && aligned16(a->ptr_c) &&
        a->stride_c % 8 == 0 && (a->batch == 1 || a->stride_c_batch % 8 == 0)) {
        // bf16 C [batch][M][N] for the epilogue's bulk stores: 64-column x 32-row boxes, clipped at the edges
        const uint64_t d[3] = {static_cast<uint64_t>(a->n), static_cast<uint64_t>(a->m), static_cast<uint64_t>(a->batch)};
        const uint64_t st[2] = {static_cast<uint64_t>(a->stride_c) * 2,
                                static_cast<uint64_t>(a->batch > 1 ? a->stride_c_batch : a->stride_c * a->m) * 2};
        const uint32_t bx[3] = {64, 32, 1};
        if ((rc = make_tmap(&p.tmap_c, a->ptr_c, 3, d, st, bx, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16))) return rc;
        p.c_tma = 1;
    }
    p.c = a->ptr_c;
    p.sfa = static_cast<const float*>(a->ptr_sfa);
    p.sfb = static_cast<const float*>(a->ptr_sfb);
    p.scale_a = a->scale_mode == B200_SCALE_TENSOR ? a->ptr_scale_a : nullptr;
    p.scale_b = a->scale_mode == B200_SCALE_TENSOR ? a->ptr_scale_b : nullptr;
    p.ldc = a->stride_c;
    p.c_batch = a->stride_c_batch;
    p.m = static_cast<int>(a->m);
    p.n = static_cast<int>(a->n);
    p.k = static_cast<int>(a->k);
    p.batch = static_cast<int>(a->batch);
    p.tiles_m = static_cast<int>((a->m + BMT - 1) / BMT);
    p.tiles_n = static_cast<int>((a->n + BN - 1) / BN);
    const long long total = static_cast<long long>(p.tiles_m) * p.tiles_n * p.batch;
    if (total > 0x7FFFFFFF) return B200_ERR_TOO_LARGE;
    p.tiles_total = static_cast<int>(total);
    p.kblocks = static_cast<int>((a->k + 127) / 128);
    p.kb_per_split = (p.kblocks + splits - 1) / splits;
    p.splits = splits;
    p.b_ahead = !pair && p.tiles_m > 1 && p.tiles_total <= ds->sm_count && a->n * a->k >= (int64_t{6} << 20) ? 1 : 0;
    p.out_dtype = a->out_dtype;
    p.inputs_ready = (a->flags & (B200_GEMM_INPUTS_READY | B200_GEMM_BATCH_READY)) ? 1 : 0;
    p.b_shared = b_shared ? 1 : 0;
    if (a->flags & B200_GEMM_BATCH_READY) {
        p.batch_ready = reinterpret_cast<const int*>(a->ptr_batch_ready);
        p.batch_epoch = a->batch_epoch;
    }
    p.status = ds->status_ptr;
    if (a->scale_mode == B200_SCALE_MX) {
        // atoms [K/128][rows/128][512 B]: strides in atoms, batch strides in bytes
        p.sfa_stride = (a->m + 127) / 128;
        p.sfb_stride = (a->n + 127) / 128;
        p.sfa_batch = a->stride_sfa_batch;
        p.sfb_batch = a->stride_sfb_batch;
    } else {
        p.sfa_stride = a->stride_sfa;
        p.sfb_stride = a->stride_sfb;
        p.sfa_batch = a->stride_sfa_batch;
        p.sfb_batch = a->stride_sfb_batch;
    }
    t_last_k_split = 0;
    t_last_columns = BN;
    const bool flat = a->b_layout == B200_B_FLAT_16x16;
    if (pair && BN == 256 && !ab16 && a->scale_mode != B200_SCALE_MX) {
        const int sms = ds->sm_count;
        plan_tail(p, a->scale_mode == B200_SCALE_BLOCK
                         ? (flat ? pair_capacity<256, MODE_BLOCK, BL_FLAT>(sms) : pair_capacity<256, MODE_BLOCK, BL_NK>(sms))
                         : (flat ? pair_capacity<256, MODE_ACC, BL_FLAT>(sms) : pair_capacity<256, MODE_ACC, BL_NK>(sms)));
        if (p.tail_split) {
            const uint32_t rows = static_cast<uint32_t>(BROWS / p.tail_split);
            rc = flat ? make_flat_tmap(&p.tmap_b_tail, a->ptr_b, a->n, a->k, b_batches, a->stride_b_batch, rows)
                      : make_rowmajor_tmap(&p.tmap_b_tail, a->ptr_b, a->n, a->k, a->stride_b, b_batches, a->stride_b_batch, rows);
            if (rc) return rc;
        }
    }
    if (ab16) {
        if (pair) return flat ? launch_pair<256, MODE_ACC16, BL_FLAT>(p, ds->sm_count, st) : launch_pair<256, MODE_ACC16, BL_NK>(p, ds->sm_count, st);
        const int grid16 = p.tiles_total < ds->sm_count ? p.tiles_total : ds->sm_count;
        return flat ? launch_columns<MODE_ACC16, BL_FLAT>(BN, p, grid16, st) : launch_columns<MODE_ACC16, BL_NK>(BN, p, grid16, st);
    }
    if (pair) {
        switch (BN) {
            case 256: return launch_pair_modes<256>(a, p, ds->sm_count, st);
            case 224: return launch_pair_modes<224>(a, p, ds->sm_count, st);
            case 192: return launch_pair_modes<192>(a, p, ds->sm_count, st);
            default: return launch_pair_modes<128>(a, p, ds->sm_count, st);
        }
    }
    const int grid = p.tiles_total < ds->sm_count ? p.tiles_total : ds->sm_count;
    switch (a->scale_mode) {
        case B200_SCALE_BLOCK:
            return flat ? launch_columns<MODE_BLOCK, BL_FLAT>(BN, p, grid, st) : launch_columns<MODE_BLOCK, BL_NK>(BN, p, grid, st);
        case B200_SCALE_MX:
            return flat ? launch_columns<MODE_MX, BL_FLAT>(BN, p, grid, st) : launch_columns<MODE_MX, BL_NK>(BN, p, grid, st);
        default:
            return flat ? launch_columns<MODE_ACC, BL_FLAT>(BN, p, grid, st) : launch_columns<MODE_ACC, BL_NK>(BN, p, grid, st);
    }
}

// ---- host generators ----------------------------------------------------------------------------
inline uint64_t mix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
inline uint64_t stream_key(uint64_t seed, uint32_t tensor_id) {
    return mix64(seed ^ (static_cast<uint64_t>(tensor_id) << 32) ^ 0xA8F8A8F8ull);
}
inline uint64_t draw64(uint64_t key, uint64_t idx) { return mix64(key + idx * 0xD1342543DE82EF95ull); }

int ensure(DeviceState* ds, int slot, size_t bytes) {
    if (ds->cap[slot] >= bytes) return B200_OK;
    if (ds->buf[slot]) CU_TRY(cudaFree(ds->buf[slot]));
    ds->buf[slot] = nullptr;
    ds->cap[slot] = 0;
    const size_t want = bytes + (bytes >> 3) + 256;
    CU_TRY(cudaMalloc(&ds->buf[slot], want));
    ds->cap[slot] = want;
    return B200_OK;
}

}  // namespace

// =================================================================================================
extern "C" {

int b200_gemm_check(const b200_gemm_args* args, int32_t* chosen_tile) {
    Plan pl;
    int sms = 148;
    int rc = validate(args, sms, &pl);
    if (rc == B200_OK && chosen_tile) *chosen_tile = pl.tile;
    return rc;
}
int b200_gemm_check_split(const b200_gemm_args* args, int32_t* parts) {
    Plan pl;
    int rc = validate(args, 148, &pl);
    if (rc == B200_OK && parts) *parts = pl.tile == B200_TILE_DECODE ? 1 : pl.splits;
    return rc;
}

static int byte_view16(const b200_gemm_args* a, b200_gemm_args* v);
int b200_gemm_check_columns(const b200_gemm_args* args, int32_t bf16_operands, int32_t* columns) {
    b200_gemm_args v;
    int rc = bf16_operands ? byte_view16(args, &v) : B200_OK;
    if (rc) return rc;
    Plan pl;
    rc = validate(bf16_operands ? &v : args, 148, &pl, bf16_operands != 0);
    if (rc == B200_OK && columns) *columns = pl.columns;
    return rc;
}

int b200_gemm_a8w8(const b200_gemm_args* args, void* cuda_stream) {
    Plan pl;
    int rc = validate(args, 148, &pl);
    if (rc) return rc;
    DeviceState* ds = nullptr;
    rc = device_state(&ds);
    if (rc) return rc;
    if (ds->sm_count != 148) rc = validate(args, ds->sm_count, &pl);
    if (rc) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
    if (pl.tile == B200_TILE_DECODE) return run_decode(args, pl, ds, st);
    return run_gemm(args, pl, ds, st);
}

// bf16 operands: the same pipeline on the byte view of the problem (a bf16 row of K elements is a row of 2K bytes;
// tile bytes, swizzle and descriptor steps are those of the 8-bit path), with kind::f16 MMAs
static int byte_view16(const b200_gemm_args* a, b200_gemm_args* v) {
    if (!a) return B200_ERR_BAD_ARG;
    if (a->k > 0x3FFFFFFF) return B200_ERR_TOO_LARGE;
    *v = *a;
    v->k = a->k * 2;
    v->stride_a = a->stride_a * 2;
    v->stride_b = a->stride_b * 2;
    v->stride_a_batch = a->stride_a_batch * 2;
    v->stride_b_batch = a->stride_b_batch * 2;
    return B200_OK;
}
int b200_gemm_a16w16_check(const b200_gemm_args* args, int32_t* chosen_tile) {
    b200_gemm_args v;
    int rc = byte_view16(args, &v);
    if (rc) return rc;
    Plan pl;
    rc = validate(&v, 148, &pl, true);
    if (rc == B200_OK && chosen_tile) *chosen_tile = pl.tile;
    return rc;
}
int b200_gemm_a16w16_check_split(const b200_gemm_args* args, int32_t* parts) {
    b200_gemm_args v;
    int rc = byte_view16(args, &v);
    if (rc) return rc;
    Plan pl;
    rc = validate(&v, 148, &pl, true);
    if (rc == B200_OK && parts) *parts = pl.splits;
    return rc;
}
int b200_gemm_a16w16(const b200_gemm_args* args, void* cuda_stream) {
    b200_gemm_args v;
    int rc = byte_view16(args, &v);
    if (rc) return rc;
    Plan pl;
    rc = validate(&v, 148, &pl, true);
    if (rc) return rc;
    DeviceState* ds = nullptr;
    rc = device_state(&ds);
    if (rc) return rc;
    rc = validate(&v, ds->sm_count, &pl, true);
    if (rc) return rc;
    return run_gemm(&v, pl, ds, static_cast<cudaStream_t>(cuda_stream), true);
}

int b200_gemm_a8w8_decode_static(const b200_gemm_args* args, void* cuda_stream) {
    Plan pl;
    int rc = validate(args, 148, &pl);
    if (rc) return rc;
    DeviceState* ds = nullptr;
    rc = device_state(&ds);
    if (rc) return rc;
    rc = validate(args, ds->sm_count, &pl);
    if (rc) return rc;
    // only the skinny-M kernel has this variant, and not with MX scales
    if (pl.tile != B200_TILE_DECODE || args->scale_mode == B200_SCALE_MX) return B200_ERR_UNSUPPORTED;
    return run_decode(args, pl, ds, static_cast<cudaStream_t>(cuda_stream), true);
}

int b200_gemm_a8w8_simple(const b200_gemm_args* a, void* cuda_stream) {
    if (!a || !a->ptr_a || !a->ptr_b || !a->ptr_c) return B200_ERR_BAD_ARG;
    if (a->m <= 0 || a->n <= 0 || a->k <= 0 || a->batch <= 0 || a->m > 65535 * 1LL * 65535 || a->batch > 65535) return B200_ERR_BAD_ARG;
    if (a->m > 65535) return B200_ERR_TOO_LARGE;
    if ((a->scale_mode == B200_SCALE_BLOCK || a->scale_mode == B200_SCALE_MX) && (!a->ptr_sfa || !a->ptr_sfb)) return B200_ERR_BAD_ARG;
    SimpleParams p;
    p.a = static_cast<const uint8_t*>(a->ptr_a);
    p.b = static_cast<const uint8_t*>(a->ptr_b);
    p.c = a->ptr_c;
    p.sfa = a->ptr_sfa;
    p.sfb = a->ptr_sfb;
    p.scale_a = a->ptr_scale_a;
    p.scale_b = a->ptr_scale_b;
    p.m = a->m; p.n = a->n; p.k = a->k; p.batch = a->batch;
    p.lda = a->stride_a; p.ldb = a->stride_b; p.ldc = a->stride_c;
    p.a_batch = a->stride_a_batch; p.b_batch = a->stride_b_batch; p.c_batch = a->stride_c_batch;
    if (a->scale_mode == B200_SCALE_MX) {
        p.sfa_stride = (a->m + 127) / 128;
        p.sfb_stride = (a->n + 127) / 128;
    } else {
        p.sfa_stride = a->stride_sfa;
        p.sfb_stride = a->stride_sfb;
    }
    p.sfa_batch = a->stride_sfa_batch; p.sfb_batch = a->stride_sfb_batch;
    p.scale_mode = a->scale_mode; p.b_layout = a->b_layout; p.out_dtype = a->out_dtype;
    dim3 grid(static_cast<unsigned>((a->n + 127) / 128), static_cast<unsigned>(a->m), static_cast<unsigned>(a->batch));
    gemm_simple_kernel<<<grid, 128, 0, static_cast<cudaStream_t>(cuda_stream)>>>(p);
    CU_TRY(cudaGetLastError());
    g_launches.fetch_add(1);
    return B200_OK;
}

// End of the synchronous host-buffer entry: wait for the stream, then look at the status word, so that a launch
// that gave up (an expired wait, a pair whose CTAs disagreed on their tensor-memory address) is an error HERE and
// not a silently wrong C.  The word is left for b200_last_status() to report and clear.
static int host_entry_finish(DeviceState* ds, HostCall& call, cudaStream_t st) {
    int unpinned = 0;                                    // (no pinned word to be had: the copy then waits for the stream)
    int* v = ds->status_host ? ds->status_host : &unpinned;
    CU_TRY(cudaMemcpyAsync(v, ds->status_ptr, sizeof(int), cudaMemcpyDeviceToHost, st));
    CU_TRY(call.finish());
    return *v == 0 ? B200_OK : B200_ERR_DEVICE_TIMEOUT;
}

// a * b for non-negative operands, or -1 when the product does not fit in 2^46 bytes (64 TiB: far above any device)
static int64_t mul_checked(int64_t a, int64_t b) {
    if (a < 0 || b < 0) return -1;
    if (a == 0 || b == 0) return 0;
    if (a > (int64_t(1) << 46) / b) return -1;
    return a * b;
}

int b200_gemm_a8w8_host(const b200_gemm_args* h, void* cuda_stream) {
    Plan pl;
    if (!h || !h->ptr_a || !h->ptr_b || !h->ptr_c) return B200_ERR_BAD_ARG;
    if (h->flags & B200_GEMM_BATCH_READY) return B200_ERR_UNSUPPORTED;       // ready words are device memory
    DeviceState* ds = nullptr;
    int rc = device_state(&ds);
    if (rc) return rc;
    // validate before anything is allocated, copied or queued: the same checks as the device entry, run on a copy
    // whose operand pointers are stand-ins with the alignment the library's own buffers will have
    {
        b200_gemm_args probe = *h;
        probe.ptr_a = probe.ptr_b = probe.ptr_c = reinterpret_cast<void*>(uintptr_t(256));
        if (h->scale_mode == B200_SCALE_BLOCK || h->scale_mode == B200_SCALE_MX) {
            if (!h->ptr_sfa || !h->ptr_sfb) return B200_ERR_BAD_ARG;
            probe.ptr_sfa = probe.ptr_sfb = reinterpret_cast<void*>(uintptr_t(256));
        }
        if ((rc = validate(&probe, ds->sm_count, &pl))) return rc;
        if (h->b_layout == B200_B_NK_ROWMAJOR && h->stride_b < h->k) return B200_ERR_BAD_ARG;
    }
    cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
    // A call that returns finished results cannot be captured.  Refused before the ring's events are recorded: an event that
    // was last recorded inside a capture fails every later wait for it.
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    CU_TRY(cudaStreamIsCapturing(st, &capturing));
    if (capturing != cudaStreamCaptureStatusNone) CU_TRY(cudaErrorStreamCaptureUnsupported);
    const int64_t esz = h->out_dtype == B200_OUT_BF16 ? 2 : 4;
    const int64_t a_sz = h->batch > 1 ? mul_checked(h->stride_a_batch, h->batch) : mul_checked(h->stride_a, h->m);
    const int64_t b_sz = h->batch > 1 ? mul_checked(h->stride_b_batch, h->batch)
                                      : (h->b_layout == B200_B_FLAT_16x16 ? mul_checked(h->n, h->k) : mul_checked(h->stride_b, h->n));
    const int64_t c_sz = mul_checked(h->batch > 1 ? mul_checked(h->stride_c_batch, h->batch) : mul_checked(h->stride_c, h->m), esz);
    int64_t sfa_sz = 0, sfb_sz = 0;
    if (h->scale_mode == B200_SCALE_BLOCK) {
        sfa_sz = mul_checked(h->batch > 1 ? mul_checked(h->stride_sfa_batch, h->batch) : mul_checked(h->stride_sfa, h->k / 128), 4);
        sfb_sz = mul_checked(h->batch > 1 ? mul_checked(h->stride_sfb_batch, h->batch) : mul_checked(h->stride_sfb, h->n / 128), 4);
    } else if (h->scale_mode == B200_SCALE_MX) {
        sfa_sz = h->batch > 1 ? mul_checked(h->stride_sfa_batch, h->batch) : static_cast<int64_t>(b200_mx_sf_bytes(h->m, h->k));
        sfb_sz = h->batch > 1 ? mul_checked(h->stride_sfb_batch, h->batch) : static_cast<int64_t>(b200_mx_sf_bytes(h->n, h->k));
    }
    if (a_sz <= 0 || b_sz <= 0 || c_sz <= 0 || sfa_sz < 0 || sfb_sz < 0) return B200_ERR_BAD_ARG;   // zero, negative or overflowing
    const size_t a_bytes = static_cast<size_t>(a_sz), b_bytes = static_cast<size_t>(b_sz), c_bytes = static_cast<size_t>(c_sz);
    const size_t sfa_bytes = static_cast<size_t>(sfa_sz), sfb_bytes = static_cast<size_t>(sfb_sz);
    // the staging buffers, the copy stream and its events are per device: one caller at a time
    std::lock_guard<std::mutex> entry(ds->host_entry_mu);
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if ((rc = ensure(ds, 0, a_bytes)) || (rc = ensure(ds, 1, b_bytes)) || (rc = ensure(ds, 2, c_bytes)) ||
            (rc = ensure(ds, 3, sfa_bytes + 16)) || (rc = ensure(ds, 4, sfb_bytes + 16)) || (rc = ensure(ds, 5, 64)))
            return rc;
    }
    b200_gemm_args d = *h;
    d.ptr_a = ds->buf[0];
    d.ptr_b = ds->buf[1];
    d.ptr_c = ds->buf[2];
    rc = validate(&d, ds->sm_count, &pl);
    if (rc) return rc;
    // Large single-batch problems run as row slabs: the copy-back of slab i (the largest transfer of the call)
    // proceeds on a second stream while slab i+1 is uploaded and computed, so the two PCIe directions overlap.
    // (MX scale atoms are indexed by the full M, so MX problems take the single-shot path.)
    const int64_t slab_rows = ((h->m + 7) / 8 + 255) / 256 * 256;
    const bool slabs = h->batch == 1 && h->m >= 2048 && h->scale_mode != B200_SCALE_MX && (h->m + slab_rows - 1) / slab_rows <= 16;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (slabs && !ds->copy_stream) {
            CU_TRY(cudaStreamCreateWithFlags(&ds->copy_stream, cudaStreamNonBlocking));
            for (auto& e : ds->slab_done) CU_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
            CU_TRY(cudaEventCreateWithFlags(&ds->copies_done, cudaEventDisableTiming));
        }
        if (!ds->status_host && cudaHostAlloc(&ds->status_host, sizeof(int), cudaHostAllocDefault) != cudaSuccess) {
            cudaGetLastError();
            ds->status_host = nullptr;
        }
    }
    Staging& io = ds->staging;
    HostCall call(io, st, ds->copy_stream);              // from here on every way out waits for what has been queued
    CU_TRY(io.upload(ds->buf[1], h->ptr_b, b_bytes, st));
    if (sfa_bytes) {
        CU_TRY(io.upload(ds->buf[3], h->ptr_sfa, sfa_bytes, st));
        CU_TRY(io.upload(ds->buf[4], h->ptr_sfb, sfb_bytes, st));
        d.ptr_sfa = ds->buf[3];
        d.ptr_sfb = ds->buf[4];
    }
    if (h->scale_mode == B200_SCALE_TENSOR) {
        float* sc = static_cast<float*>(ds->buf[5]);
        if (h->ptr_scale_a) {
            CU_TRY(cudaMemcpyAsync(sc, h->ptr_scale_a, 4, cudaMemcpyHostToDevice, st));
            d.ptr_scale_a = sc;
        }
        if (h->ptr_scale_b) {
            CU_TRY(cudaMemcpyAsync(sc + 1, h->ptr_scale_b, 4, cudaMemcpyHostToDevice, st));
            d.ptr_scale_b = sc + 1;
        }
    }
    if (!slabs) {
        CU_TRY(io.upload(ds->buf[0], h->ptr_a, a_bytes, st));
        rc = b200_gemm_a8w8(&d, st);
        if (rc) return rc;
        CU_TRY(io.download(h->ptr_c, ds->buf[2], c_bytes, st));
        return host_entry_finish(ds, call, st);
    }
    int slab = 0;
    for (int64_t r0 = 0; r0 < h->m; r0 += slab_rows, ++slab) {
        const int64_t rows = (h->m - r0) < slab_rows ? (h->m - r0) : slab_rows;
        b200_gemm_args s = d;
        s.m = rows;
        s.ptr_a = static_cast<const uint8_t*>(d.ptr_a) + r0 * h->stride_a;
        s.ptr_c = static_cast<uint8_t*>(d.ptr_c) + static_cast<size_t>(r0) * h->stride_c * esz;
        if (h->scale_mode == B200_SCALE_BLOCK) s.ptr_sfa = static_cast<const float*>(d.ptr_sfa) + r0;   // [K/128][M]: same pitch
        CU_TRY(io.upload(const_cast<void*>(s.ptr_a), static_cast<const uint8_t*>(h->ptr_a) + r0 * h->stride_a,
                         static_cast<size_t>(rows * h->stride_a), st));
        rc = b200_gemm_a8w8(&s, st);
        if (rc) return rc;
        CU_TRY(cudaEventRecord(ds->slab_done[slab], st));
        CU_TRY(cudaStreamWaitEvent(ds->copy_stream, ds->slab_done[slab], 0));
        CU_TRY(io.download(static_cast<uint8_t*>(h->ptr_c) + static_cast<size_t>(r0) * h->stride_c * esz, s.ptr_c,
                           static_cast<size_t>(rows * h->stride_c) * esz, ds->copy_stream));
    }
    CU_TRY(cudaEventRecord(ds->copies_done, ds->copy_stream));
    CU_TRY(cudaStreamWaitEvent(st, ds->copies_done, 0));
    return host_entry_finish(ds, call, st);
}

// ---- layout ----------------------------------------------------------------------------------------
static int shuffle_common(const void* src, void* dst, int64_t n, int64_t k, int32_t kn, bool to_flat, void* stream) {
    if (!src || !dst || n <= 0 || k <= 0) return B200_ERR_BAD_ARG;
    if (n % 16 != 0 || k % 16 != 0) return B200_ERR_UNSUPPORTED;
    if (!aligned16(src) || !aligned16(dst)) return B200_ERR_UNSUPPORTED;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (kn) {
        dim3 grid(static_cast<unsigned>((n + 255) / 256), static_cast<unsigned>((k + 63) / 64));
        if (grid.y > 65535) return B200_ERR_TOO_LARGE;
        if (to_flat) shuffle_kn_kernel<true><<<grid, 256, 0, st>>>(static_cast<const uint8_t*>(src), static_cast<uint8_t*>(dst), n, k);
        else shuffle_kn_kernel<false><<<grid, 256, 0, st>>>(static_cast<const uint8_t*>(src), static_cast<uint8_t*>(dst), n, k);
    } else {
        dim3 grid(static_cast<unsigned>((k / 16 + 63) / 64), static_cast<unsigned>(n / 16));
        if (grid.y > 65535) return B200_ERR_TOO_LARGE;
        if (to_flat) shuffle_nk_kernel<true><<<grid, 256, 0, st>>>(static_cast<const uint4*>(src), static_cast<uint4*>(dst), n, k);
        else shuffle_nk_kernel<false><<<grid, 256, 0, st>>>(static_cast<const uint4*>(src), static_cast<uint4*>(dst), n, k);
    }
    CU_TRY(cudaGetLastError());
    g_launches.fetch_add(1);
    return B200_OK;
}
int b200_shuffle_b(const void* src, void* dst, int64_t n, int64_t k, int32_t src_is_kn, void* stream) {
    return shuffle_common(src, dst, n, k, src_is_kn, true, stream);
}
int b200_unshuffle_b(const void* flat, void* dst, int64_t n, int64_t k, int32_t dst_is_kn, void* stream) {
    return shuffle_common(flat, dst, n, k, dst_is_kn, false, stream);
}

static int shuffle16_common(const void* src, void* dst, int64_t n, int64_t k, int32_t kn, bool to_flat, void* stream) {
    if (!src || !dst || n <= 0 || k <= 0) return B200_ERR_BAD_ARG;
    if (n % 16 != 0 || k % 8 != 0) return B200_ERR_UNSUPPORTED;
    if (!kn) return shuffle_common(src, dst, n, 2 * k, 0, to_flat, stream);      // [N][K] bf16 = [N][2K] bytes
    if (!aligned16(src) || !aligned16(dst)) return B200_ERR_UNSUPPORTED;
    dim3 grid(static_cast<unsigned>((n + 63) / 64), static_cast<unsigned>((k + 63) / 64));
    if (grid.y > 65535) return B200_ERR_TOO_LARGE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (to_flat) shuffle_kn16_kernel<true><<<grid, 256, 0, st>>>(static_cast<const uint16_t*>(src), static_cast<uint16_t*>(dst), n, k);
    else shuffle_kn16_kernel<false><<<grid, 256, 0, st>>>(static_cast<const uint16_t*>(src), static_cast<uint16_t*>(dst), n, k);
    CU_TRY(cudaGetLastError());
    g_launches.fetch_add(1);
    return B200_OK;
}
int b200_shuffle_b_bf16(const void* src, void* dst, int64_t n, int64_t k, int32_t src_is_kn, void* stream) {
    return shuffle16_common(src, dst, n, k, src_is_kn, true, stream);
}
int b200_unshuffle_b_bf16(const void* flat, void* dst, int64_t n, int64_t k, int32_t dst_is_kn, void* stream) {
    return shuffle16_common(flat, dst, n, k, dst_is_kn, false, stream);
}

// ---- quantisers ------------------------------------------------------------------------------------
static unsigned grid_for(int64_t work_items, int threads) {
    int64_t blocks = (work_items + threads - 1) / threads;
    if (blocks > 148 * 16) blocks = 148 * 16;
    if (blocks < 1) blocks = 1;
    return static_cast<unsigned>(blocks);
}
int b200_cast_e4m3(const float* x, void* q, int64_t count, void* stream) {
    if (!x || !q || count <= 0) return B200_ERR_BAD_ARG;
    if (!aligned16(x) || (reinterpret_cast<uintptr_t>(q) & 3)) return B200_ERR_UNSUPPORTED;
    cast_e4m3_kernel<<<grid_for(count / 4 + 1, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(x, static_cast<uint8_t*>(q), count);
    CU_TRY(cudaGetLastError());
    g_launches.fetch_add(1);
    return B200_OK;
}
size_t b200_quantize_tensor_workspace(void) { return 256; }
int b200_quantize_tensor(const float* x, void* q, float* scale, int64_t count, void* workspace, void* stream) {
    if (!x || !q || !scale || !workspace || count <= 0) return B200_ERR_BAD_ARG;
    if (!aligned16(x) || (reinterpret_cast<uintptr_t>(q) & 3) || (reinterpret_cast<uintptr_t>(workspace) & 3)) return B200_ERR_UNSUPPORTED;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    unsigned int* amax = static_cast<unsigned int*>(workspace);
    CU_TRY(cudaMemsetAsync(amax, 0, sizeof(unsigned int), st));
    amax_kernel<<<grid_for(count / 4 + 1, 256), 256, 0, st>>>(x, count, amax);
    CU_TRY(cudaGetLastError());
    quant_tensor_kernel<<<grid_for(count / 4 + 1, 256), 256, 0, st>>>(x, static_cast<uint8_t*>(q), scale, count, amax);
    CU_TRY(cudaGetLastError());
    g_launches.fetch_add(2);
    return B200_OK;
}
int b200_quantize_1x128(const float* x, void* q, float* sfa, int64_t m, int64_t k, void* stream) {
    if (!x || !q || !sfa || m <= 0 || k <= 0) return B200_ERR_BAD_ARG;
    if (k % 128 != 0 || !aligned16(x) || (reinterpret_cast<uintptr_t>(q) & 3)) return B200_ERR_UNSUPPORTED;
    const int64_t warps = m * (k / 128);
    const int64_t blocks = (warps + 7) / 8;
    if (blocks > 0x7FFFFFFF) return B200_ERR_TOO_LARGE;
    quant_1x128_kernel<<<static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(x, static_cast<uint8_t*>(q), sfa, m, k);
    CU_TRY(cudaGetLastError());
    g_launches.fetch_add(1);
    return B200_OK;
}
// persistent grid of the probe kernels: two 1024-thread blocks per SM, fewer for small buffers
static unsigned membw_grid(int sm_count, unsigned long long n16) {
    const unsigned long long want = (n16 + 1023) / 1024;
    const unsigned long long cap = static_cast<unsigned long long>(sm_count) * 2;
    return static_cast<unsigned>(want < cap ? (want ? want : 1) : cap);
}
int b200_membw_read(const void* src, size_t bytes, uint32_t* word_sum, void* stream) {
    if (!src || !word_sum || bytes == 0) return B200_ERR_BAD_ARG;
    if (bytes % 16 != 0 || !aligned16(src)) return B200_ERR_UNSUPPORTED;
    DeviceState* ds = nullptr;
    int rc = device_state(&ds);
    if (rc) return rc;
    const unsigned long long n16 = bytes / 16;
    membw_read_kernel<<<membw_grid(ds->sm_count, n16), 1024, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint4*>(src), n16, word_sum);
    CU_TRY(cudaGetLastError());
    g_launches.fetch_add(1);
    return B200_OK;
}
int b200_membw_copy(const void* src, void* dst, size_t bytes, void* stream) {
    if (!src || !dst || bytes == 0) return B200_ERR_BAD_ARG;
    if (bytes % 16 != 0 || !aligned16(src) || !aligned16(dst)) return B200_ERR_UNSUPPORTED;
    DeviceState* ds = nullptr;
    int rc = device_state(&ds);
    if (rc) return rc;
    const unsigned long long n16 = bytes / 16;
    membw_copy_kernel<<<membw_grid(ds->sm_count, n16), 1024, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint4*>(src), static_cast<uint4*>(dst), n16);
    CU_TRY(cudaGetLastError());
    g_launches.fetch_add(1);
    return B200_OK;
}
int b200_quantize_act_bf16_1x128(const void* x_bf16, int64_t ldx, void* q, int64_t ldq, float* sfa, int64_t stride_sfa,
                                 int64_t m, int64_t k, void* stream) {
    if (!x_bf16 || !q || !sfa || m <= 0 || k <= 0) return B200_ERR_BAD_ARG;
    if (ldx < k || ldq < k || stride_sfa < m) return B200_ERR_BAD_ARG;
    // 16-byte loads of eight bf16 and 8-byte stores of eight e4m3: pitches and bases must keep that alignment
    if (k % 128 != 0 || ldx % 8 != 0 || ldq % 8 != 0 || (reinterpret_cast<uintptr_t>(x_bf16) & 15) ||
        (reinterpret_cast<uintptr_t>(q) & 7))
        return B200_ERR_UNSUPPORTED;
    // four rows per warp (see the kernel) unless that leaves an SM with fewer than eight warps
    const int64_t pairs = (k / 128 + 1) / 2;
    const bool wide = (m + 3) / 4 * pairs >= physical_sms() * 8;
    const int64_t blocks = ((wide ? (m + 3) / 4 : m) * pairs + 7) / 8;
    if (k > 0x7FFFFFFF || blocks > (1 << 28)) return B200_ERR_TOO_LARGE;
    return launch_pdl(wide ? act_quant_bf16_1x128_kernel<4> : act_quant_bf16_1x128_kernel<1>, static_cast<unsigned>(blocks), 256, 0,
                      static_cast<cudaStream_t>(stream), static_cast<const uint16_t*>(x_bf16), static_cast<long long>(ldx),
                      static_cast<uint8_t*>(q), static_cast<long long>(ldq), sfa, static_cast<long long>(stride_sfa),
                      static_cast<long long>(m), static_cast<int>(k / 128));
}
int b200_quantize_act_bf16_mx32(const void* x_bf16, int64_t ldx, void* q, int64_t ldq, void* sf_atoms, int64_t rows, int64_t k,
                                void* stream) {
    if (!x_bf16 || !q || !sf_atoms || rows <= 0 || k <= 0) return B200_ERR_BAD_ARG;
    if (ldx < k || ldq < k) return B200_ERR_BAD_ARG;
    if (k % 128 != 0 || ldx % 4 != 0 || ldq % 4 != 0 || (reinterpret_cast<uintptr_t>(x_bf16) & 7) ||
        (reinterpret_cast<uintptr_t>(q) & 3) || (reinterpret_cast<uintptr_t>(sf_atoms) & 3))
        return B200_ERR_UNSUPPORTED;
    const int64_t blocks = ((rows + 127) / 128 * 32 * ((k / 128 + 1) / 2) + 7) / 8;
    if (k > 0x7FFFFFFF || blocks > (1 << 28)) return B200_ERR_TOO_LARGE;
    const bool aligned = ldx % 8 == 0 && ldq % 8 == 0 && aligned16(x_bf16) && (reinterpret_cast<uintptr_t>(q) & 7) == 0;
    return launch_pdl(aligned ? act_quant_bf16_mx32_kernel<true> : act_quant_bf16_mx32_kernel<false>,
                      static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream),
                      static_cast<const uint16_t*>(x_bf16), static_cast<long long>(ldx), static_cast<uint8_t*>(q),
                      static_cast<long long>(ldq), static_cast<uint32_t*>(sf_atoms), static_cast<long long>(rows),
                      static_cast<int>(k / 128));
}
int b200_quantize_128x128(const float* x, void* q, float* sfb, int64_t n, int64_t k, void* stream) {
    if (!x || !q || !sfb || n <= 0 || k <= 0) return B200_ERR_BAD_ARG;
    if (n % 128 != 0 || k % 128 != 0 || !aligned16(x) || (reinterpret_cast<uintptr_t>(q) & 3)) return B200_ERR_UNSUPPORTED;
    dim3 grid(static_cast<unsigned>(k / 128), static_cast<unsigned>(n / 128));
    if (grid.y > 65535) return B200_ERR_TOO_LARGE;
    quant_128x128_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(x, static_cast<uint8_t*>(q), sfb, n, k);
    CU_TRY(cudaGetLastError());
    g_launches.fetch_add(1);
    return B200_OK;
}
int b200_quantize_mx32(const float* x, void* q, void* sf, int64_t rows, int64_t k, void* stream) {
    if (!x || !q || !sf || rows <= 0 || k <= 0) return B200_ERR_BAD_ARG;
    if (k % 32 != 0 || !aligned16(x) || (reinterpret_cast<uintptr_t>(q) & 3)) return B200_ERR_UNSUPPORTED;
    const int64_t threads = rows * (k / 32) * 8;
    const int64_t blocks = (threads + 255) / 256;
    if (blocks > 0x7FFFFFFF) return B200_ERR_TOO_LARGE;
    quant_mx32_kernel<<<static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(x, static_cast<uint8_t*>(q), static_cast<uint8_t*>(sf), rows, k);
    CU_TRY(cudaGetLastError());
    g_launches.fetch_add(1);
    return B200_OK;
}
size_t b200_mx_sf_bytes(int64_t rows, int64_t k) {
    if (rows <= 0 || k <= 0) return 0;
    return static_cast<size_t>((k + 127) / 128) * static_cast<size_t>((rows + 127) / 128) * 512;
}
int b200_mx_sf_relayout(const void* sf_logical, void* sf_atoms, int64_t rows, int64_t k, void* stream) {
    if (!sf_logical || !sf_atoms || rows <= 0 || k <= 0) return B200_ERR_BAD_ARG;
    if (k % 128 != 0 || (reinterpret_cast<uintptr_t>(sf_logical) & 3) || !aligned16(sf_atoms)) return B200_ERR_UNSUPPORTED;
    const int64_t words = (k / 128) * ((rows + 127) / 128) * 128;
    const int64_t blocks = (words + 255) / 256;
    if (blocks > 0x7FFFFFFF) return B200_ERR_TOO_LARGE;
    mx_sf_relayout_kernel<<<static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint8_t*>(sf_logical), static_cast<uint32_t*>(sf_atoms), rows, k);
    CU_TRY(cudaGetLastError());
    g_launches.fetch_add(1);
    return B200_OK;
}

// ---- seeded inputs ---------------------------------------------------------------------------------
void b200_fill_uniform(float* out, size_t count, uint64_t seed, uint32_t tensor_id, float lo, float hi) {
    const uint64_t key = stream_key(seed, tensor_id);
    const float span = hi - lo;
#pragma omp parallel for schedule(static)
    for (long long i = 0; i < static_cast<long long>(count); ++i) {
        const uint32_t r = static_cast<uint32_t>(draw64(key, static_cast<uint64_t>(i)) >> 40);
        const float u = static_cast<float>(r) * (1.0f / 16777216.0f);
        volatile float prod = span * u;      // keep the multiply and the add separately rounded
        out[i] = lo + prod;
    }
}
void b200_fill_normal(float* out, size_t count, uint64_t seed, uint32_t tensor_id) {
    const uint64_t key = stream_key(seed, tensor_id);
#pragma omp parallel for schedule(static)
    for (long long i = 0; i < static_cast<long long>(count); ++i) {
        const uint64_t d = draw64(key, static_cast<uint64_t>(i));
        const uint32_t r1 = static_cast<uint32_t>(d >> 40);
        const uint32_t r2 = static_cast<uint32_t>(d >> 8) & 0xFFFFFFu;
        const double u1 = (static_cast<double>(r1) + 1.0) * (1.0 / 16777216.0);
        const double u2 = static_cast<double>(r2) * (1.0 / 16777216.0);
        out[i] = static_cast<float>(std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2));
    }
}

// ---- status ------------------------------------------------------------------------------------------
int b200_last_status(void) {
    DeviceState* ds = nullptr;
    int rc = device_state(&ds);
    if (rc) return rc;
    CU_TRY(cudaDeviceSynchronize());
    int v = 0;
    CU_TRY(cudaMemcpy(&v, ds->status_ptr, sizeof(int), cudaMemcpyDeviceToHost));
    if (v != 0) CU_TRY(cudaMemset(ds->status_ptr, 0, sizeof(int)));
    return v;
}
int b200_peek_status(void) {
    DeviceState* ds = nullptr;
    int rc = device_state(&ds);
    if (rc) return rc;
    {
        // (created on first use, not with the per-device state: the allocation-free entry point must not create anything)
        std::lock_guard<std::mutex> lk(g_mu);
        if (!ds->peek_stream) CU_TRY(cudaStreamCreateWithFlags(&ds->peek_stream, cudaStreamNonBlocking));
    }
    int v = 0;
    CU_TRY(cudaMemcpyAsync(&v, ds->status_ptr, sizeof(int), cudaMemcpyDeviceToHost, ds->peek_stream));
    CU_TRY(cudaStreamSynchronize(ds->peek_stream));
    return v;
}
int b200_flag_write(int32_t* flag, int32_t value, void* cuda_stream) {
    if (!flag || (reinterpret_cast<uintptr_t>(flag) & 3)) return B200_ERR_BAD_ARG;
    DeviceState* ds = nullptr;
    int rc = device_state(&ds);
    if (rc) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
    if (g_write_value32) {
        const CUresult r = g_write_value32(reinterpret_cast<CUstream>(st), reinterpret_cast<CUdeviceptr>(flag),
                                           static_cast<cuuint32_t>(value), 0 /* CU_STREAM_WRITE_VALUE_DEFAULT */);
        if (r == CUDA_SUCCESS) return B200_OK;
        g_last_cuda = 100000 + static_cast<int>(r);
        return B200_ERR_CUDA;
    }
    // A driver without stream memory operations: a one-thread kernel could do the write, but it would need an SM,
    // and the consumer of these words is a persistent GEMM that may hold every SM while it waits for them.
    return B200_ERR_UNSUPPORTED;
}
int b200_flag_wait(const int32_t* flag, int32_t value, void* cuda_stream) {
    if (!flag || (reinterpret_cast<uintptr_t>(flag) & 3)) return B200_ERR_BAD_ARG;
    DeviceState* ds = nullptr;
    int rc = device_state(&ds);
    if (rc) return rc;
    if (!g_wait_value32) return B200_ERR_UNSUPPORTED;
    const CUresult r = g_wait_value32(reinterpret_cast<CUstream>(cuda_stream), reinterpret_cast<CUdeviceptr>(flag),
                                      static_cast<cuuint32_t>(value), 0x0 /* CU_STREAM_WAIT_VALUE_GEQ */);
    if (r == CUDA_SUCCESS) return B200_OK;
    g_last_cuda = 100000 + static_cast<int>(r);
    return B200_ERR_CUDA;
}
int b200_stream_copy(void* dst, const void* src, size_t bytes, void* cuda_stream) {
    if (!dst || !src || bytes == 0) return B200_ERR_BAD_ARG;
    CU_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, static_cast<cudaStream_t>(cuda_stream)));
    return B200_OK;
}
int b200_ipc_alloc(size_t bytes, void** dev_ptr, void* handle64) {
    static_assert(sizeof(cudaIpcMemHandle_t) == 64, "the handle travels as 64 bytes");
    if (!dev_ptr || !handle64 || bytes == 0) return B200_ERR_BAD_ARG;
    DeviceState* ds = nullptr;
    int rc = device_state(&ds);
    if (rc) return rc;
    void* p = nullptr;
    CU_TRY(cudaMalloc(&p, bytes));
    cudaIpcMemHandle_t h;
    const cudaError_t e = cudaIpcGetMemHandle(&h, p);
    if (e != cudaSuccess) {
        g_last_cuda = static_cast<int>(e);
        cudaFree(p);
        return B200_ERR_CUDA;
    }
    std::memcpy(handle64, &h, sizeof(h));
    *dev_ptr = p;
    return B200_OK;
}
int b200_ipc_open(const void* handle64, void** dev_ptr) {
    if (!handle64 || !dev_ptr) return B200_ERR_BAD_ARG;
    DeviceState* ds = nullptr;
    int rc = device_state(&ds);
    if (rc) return rc;
    cudaIpcMemHandle_t h;
    std::memcpy(&h, handle64, sizeof(h));
    void* p = nullptr;
    CU_TRY(cudaIpcOpenMemHandle(&p, h, cudaIpcMemLazyEnablePeerAccess));
    *dev_ptr = p;
    return B200_OK;
}
int b200_ipc_close(void* dev_ptr) {
    if (!dev_ptr) return B200_ERR_BAD_ARG;
    CU_TRY(cudaIpcCloseMemHandle(dev_ptr));
    return B200_OK;
}
int b200_ipc_free(void* dev_ptr) {
    if (!dev_ptr) return B200_ERR_BAD_ARG;
    CU_TRY(cudaFree(dev_ptr));
    return B200_OK;
}
size_t b200_slab_bytes(int64_t slab_rows, int64_t k) {
    if (slab_rows <= 0 || k <= 0 || k % 128 != 0 || slab_rows % 4 != 0) return 0;
    return static_cast<size_t>(slab_rows) * static_cast<size_t>(k) + 4 * static_cast<size_t>(k / 128) * static_cast<size_t>(slab_rows);
}
int b200_slab_upload(const void* host_a, const float* host_sfa, void* dev_slabs, int64_t m, int64_t k, int64_t slab_rows,
                     int64_t slab, void* cuda_stream) {
    if (!host_a || !host_sfa || !dev_slabs || m <= 0 || slab < 0) return B200_ERR_BAD_ARG;
    const size_t bytes = b200_slab_bytes(slab_rows, k);
    if (bytes == 0) return B200_ERR_UNSUPPORTED;
    if (m % slab_rows != 0 || (slab + 1) * slab_rows > m) return B200_ERR_BAD_ARG;
    cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
    uint8_t* dst = static_cast<uint8_t*>(dev_slabs) + static_cast<size_t>(slab) * bytes;
    const size_t a_bytes = static_cast<size_t>(slab_rows) * static_cast<size_t>(k);
    CU_TRY(cudaMemcpyAsync(dst, static_cast<const uint8_t*>(host_a) + static_cast<size_t>(slab) * a_bytes, a_bytes,
                           cudaMemcpyHostToDevice, st));
    // the slab's columns of every K group: K/128 rows of slab_rows floats, source pitch M floats
    CU_TRY(cudaMemcpy2DAsync(dst + a_bytes, static_cast<size_t>(slab_rows) * 4, host_sfa + slab * slab_rows,
                             static_cast<size_t>(m) * 4, static_cast<size_t>(slab_rows) * 4, static_cast<size_t>(k / 128),
                             cudaMemcpyHostToDevice, st));
    return B200_OK;
}
int b200_selftest_bounded_wait(int64_t budget_us, int32_t polling, void* cuda_stream) {
    if (budget_us < 100 || budget_us > 100000) return B200_ERR_BAD_ARG;          // 0.1 ms .. 100 ms
    DeviceState* ds = nullptr;
    int rc = device_state(&ds);
    if (rc) return rc;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if ((rc = ensure(ds, 6, 64))) return rc;
    }
    cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
    int* returned = static_cast<int*>(ds->buf[6]);
    CU_TRY(cudaMemsetAsync(returned, 0, sizeof(int), st));
    selftest_bounded_wait_kernel<<<1, 64, 0, st>>>(ds->status_ptr, static_cast<unsigned long long>(budget_us) * 1000ull,
                                                   polling, returned);
    CU_TRY(cudaGetLastError());
    CU_TRY(cudaStreamSynchronize(st));
    int n = 0;
    CU_TRY(cudaMemcpy(&n, returned, sizeof(int), cudaMemcpyDeviceToHost));
    return n == 2 ? B200_OK : B200_ERR_DEVICE_TIMEOUT;       // both waits must have returned "gave up"
}
int b200_last_cuda_error(void) { return g_last_cuda; }
int b200_weight_file_write(const char* path, int32_t b_layout, int32_t scale_mode, int64_t n, int64_t k, const void* data,
                           const void* scales) {
    return b200::weight_file_write(path, b_layout, scale_mode, n, k, data, scales);
}
int b200_weight_file_stat(const char* path, b200_weight_desc* out) { return b200::weight_file_stat(path, out); }
int b200_weight_file_read(const char* path, void* data, size_t data_capacity, void* scales, size_t scale_capacity) {
    return b200::weight_file_read(path, data, data_capacity, scales, scale_capacity);
}
const char* b200_strerror(int code) {
    switch (code) {
        case B200_OK: return "ok";
        case B200_ERR_BAD_ARG: return "bad argument";
        case B200_ERR_UNSUPPORTED: return "unsupported shape, stride or alignment";
        case B200_ERR_CUDA: return "CUDA call failed";
        case B200_ERR_DEVICE_TIMEOUT: return "bounded device wait expired";
        case B200_ERR_NO_DEVICE: return "no sm_100 device";
        case B200_ERR_TOO_LARGE: return "request exceeds an internal capacity";
        case B200_ERR_IO: return "weight file i/o failed";
        case B200_ERR_CORRUPT: return "weight file checksum mismatch";
        default: return "unknown";
    }
}
int b200_sm_count(void) {
    DeviceState* ds = nullptr;
    int rc = device_state(&ds);
    return rc ? rc : ds->sm_count;
}
int b200_release(void) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return B200_ERR_NO_DEVICE;
    std::lock_guard<std::mutex> lk(g_mu);
    DeviceState& s = g_dev[dev];
    for (int i = 0; i < 8; ++i) {
        if (s.buf[i]) cudaFree(s.buf[i]);
        s.buf[i] = nullptr;
        s.cap[i] = 0;
    }
    {
        int kept = 0;
        for (int i = 0; i < g_scratch_count; ++i) {
            if (g_scratch[i].dev == dev) cudaFree(g_scratch[i].ptr);
            else g_scratch[kept++] = g_scratch[i];
        }
        g_scratch_count = kept;
    }
    s.staging.release();
    if (s.status_host) cudaFreeHost(s.status_host);
    s.status_host = nullptr;
    CopyPool::get().release();
    if (s.copy_stream) {
        cudaStreamDestroy(s.copy_stream);
        s.copy_stream = nullptr;
        for (auto& e : s.slab_done) {
            cudaEventDestroy(e);
            e = nullptr;
        }
        cudaEventDestroy(s.copies_done);
        s.copies_done = nullptr;
    }
    return B200_OK;
}
const char* b200_version(void) { return "b200gemm 0.1 (sm_100a)"; }
#ifdef B200_TRACE
int b200_trace_read(long long* host, int count) {
    CU_TRY(cudaDeviceSynchronize());
    CU_TRY(cudaMemcpyFromSymbol(host, b200::g_trace, sizeof(long long) * count));
    return 0;
}
#endif
uint64_t b200_launch_count(void) { return g_launches.load(); }
int b200_last_tail_split(int32_t* first_tile, int32_t* parts) {
    if (first_tile) *first_tile = t_last_tail[0];
    if (parts) *parts = t_last_tail[1];
    return t_last_tail[1] > 0 ? 1 : 0;
}
int b200_last_k_split(void) { return t_last_k_split; }
int b200_last_columns(void) { return t_last_columns; }

}  // extern "C"
