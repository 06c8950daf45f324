// hpmc_column_core.cuh -- column classification on sm_100a (shadergen.cpp:86-171
// fused with the first five reductions): the parts shared by the TMA column
// classifiers (kernels_build.cu) and the direct column classifier below, which
// include/hpmc_functor.cuh also instantiates for a caller's functor types.
//
// A column = one 32x32 cell footprint of the slice tiles x column_slices
// slices, taken in boxes of 8 sample layers.  Per layer, every warp turns rows
// of samples into bits (f < iso) with one ballot per row.  Per slice, ONE warp
// classifies the whole 32x32 block, bit-sliced: lane y holds the 32 cells of
// row y as eight 32-bit words, word k = bit k (dx + 2dy + 4dz) of the 32 codes.
// AND/OR over the eight words marks the cells that are neither all-inside nor
// all-outside (the only ones with vertices); only those go through the count
// table.  The warp sum is the block's level-5 entry.
#pragma once
#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>
#include <type_traits>

#include "hpmc_classify_core.cuh"
#include "hpmc_device.cuh"
#include "hpmc_fetch.cuh"

namespace hpmc {

namespace {

// Sample below the iso-value; uint8 samples against the threshold byte.
template <typename T>
__device__ __forceinline__ bool below(T v, float iso, int u8_thr) {
    if constexpr (std::is_same<T, float>::value)
        return v < iso;  // strict; NaN -> false (shadergen.cpp:137-142)
    else
        return (int)v < u8_thr;
}

// 8x8 bit-matrix transpose: byte r bit c -> byte c bit r.
__device__ __forceinline__ uint64_t transpose8(uint64_t x) {
    uint64_t t;
    t = (x ^ (x >> 7)) & 0x00AA00AA00AA00AAull;
    x = x ^ t ^ (t << 7);
    t = (x ^ (x >> 14)) & 0x0000CCCC0000CCCCull;
    x = x ^ t ^ (t << 14);
    t = (x ^ (x >> 28)) & 0x00000000F0F0F0F0ull;
    x = x ^ t ^ (t << 28);
    return x;
}

// Bit-sliced codes of one 32-cell row -> 32 byte codes (w[i] = cells 4i..4i+3).
__device__ __forceinline__ void slices_to_codes(const uint32_t c[8], uint32_t w[8]) {
#pragma unroll
    for (int g = 0; g < 4; g++) {
        const uint32_t sel = (uint32_t)g | ((uint32_t)(g + 4) << 4);
        const uint32_t lo = __byte_perm(__byte_perm(c[0], c[1], sel), __byte_perm(c[2], c[3], sel), 0x5410);
        const uint32_t hi = __byte_perm(__byte_perm(c[4], c[5], sel), __byte_perm(c[6], c[7], sel), 0x5410);
        const uint64_t x = transpose8((uint64_t)lo | ((uint64_t)hi << 32));
        w[2 * g] = (uint32_t)x;
        w[2 * g + 1] = (uint32_t)(x >> 32);
    }
}

// One warp: classify slice z of footprint (fx, fy) from sample-bit rows of the
// lower layer (rows_b/col_b) and the upper layer (rows_t/col_t).  Every block
// gets its level-5 count; blocks with vertices store their sample bits and
// their tiles' vertices in their slot.  full: every cell of the footprint lies inside the
// grid (vmask is all ones in every lane).  b: the block's level-5 index,
// column_block_index(V, z, fx, fy).
__device__ __forceinline__ void classify_slice_warp(const Volume& V, int z, int fx, int fy, uint32_t b, int lane,
                                                    uint32_t vmask, bool full, const uint32_t* rows_b,
                                                    uint64_t col_b, const uint32_t* rows_t, uint64_t col_t,
                                                    const uint8_t* s_cnt) {
    // rows y and y+1 of both layers; bit 32 of a row (column x0+32) comes
    // from the column word: (row >> 1) | colbit << 31 is the row shifted by one cell
    const uint32_t cbl = (uint32_t)col_b, cbh = (uint32_t)(col_b >> 32);
    const uint32_t ctl = (uint32_t)col_t, cth = (uint32_t)(col_t >> 32);
    const uint32_t a0 = rows_b[lane], a1 = rows_b[lane + 1];
    const uint32_t b0 = rows_t[lane], b1 = rows_t[lane + 1];
    if (full && !V.codes_out) {
        // A full block has no vertices iff its 33x33x2 samples all lie on one
        // side of the iso-value (two samples that differ have some edge
        // between them that differs, and every edge belongs to a cell of the
        // block): one AND and one OR of the lane's two rows in both layers
        // and of its two column bits, two votes.
        const uint32_t cb = __funnelshift_r(cbl, cbh, lane) & 3u, ct = __funnelshift_r(ctl, cth, lane) & 3u;
        const bool below_all = ((a0 & a1 & b0 & b1) == 0xffffffffu) && ((cb & ct) == 3u);
        const bool above_all = ((a0 | a1 | b0 | b1) == 0u) && ((cb | ct) == 0u);
        if (__all_sync(0xffffffffu, below_all) || __all_sync(0xffffffffu, above_all)) {
            if (lane == 0) V.levels[V.level_off[kBlockLevel] + b] = 0u;
            return;
        }
    }
    uint32_t c[8];
    c[0] = a0;                                                   // (x,   y,   z)
    c[1] = (a0 >> 1) | (((cbl >> lane) & 1u) << 31);             // (x+1, y,   z)
    c[2] = a1;                                                   // (x,   y+1, z)
    c[3] = (a1 >> 1) | ((__funnelshift_rc(cbl, cbh, lane + 1) & 1u) << 31);
    c[4] = b0;                                                   // (x,   y,   z+1)
    c[5] = (b0 >> 1) | (((ctl >> lane) & 1u) << 31);
    c[6] = b1;
    c[7] = (b1 >> 1) | ((__funnelshift_rc(ctl, cth, lane + 1) & 1u) << 31);
    uint32_t all = c[0], any = c[0];
#pragma unroll
    for (int k = 1; k < 8; k++) {
        all &= c[k];
        any |= c[k];
    }
    // cells that are neither all-inside nor all-outside: the only ones with
    // vertices (every other MC case has at least one triangle)
    const uint32_t active = (all ^ any) & vmask;
    const bool has_vertices = __any_sync(0xffffffffu, active != 0u);
    if (!has_vertices) {
        if (lane == 0) V.levels[V.level_off[kBlockLevel] + b] = 0u;
        if (!V.codes_out) return;
    }
    // codes of this row (cells outside the grid are masked to 0)
#pragma unroll
    for (int k = 0; k < 8; k++) c[k] &= vmask;
    uint32_t w[8];
    slices_to_codes(c, w);
    if (has_vertices) {
        // the block's vertices: 32 independent count lookups per lane (byte j
        // of seg = the row's cells 8j .. 8j+7, at most 96), one warp
        // reduction (inactive cells have codes 0 or 255, count 0)
        uint32_t seg = 0;
#pragma unroll
        for (int i = 0; i < 32; i++) seg += (uint32_t)s_cnt[(w[i >> 2] >> (8 * (i & 3))) & 0xffu] << (8 * (i >> 3));
        const uint32_t vs = (seg & 0xffu) + ((seg >> 8) & 0xffu) + ((seg >> 16) & 0xffu) + (seg >> 24);
        const uint32_t total = __reduce_add_sync(0xffffffffu, vs);
        if (lane == 0) V.levels[V.level_off[kBlockLevel] + b] = total;
        // the block's sample bits (see kRowSlotWords)
        uint32_t* dst = V.arena + (((long long)z * V.nfy + fy) * V.nfx + fx) * kRowSlotWords;
        dst[lane] = a0;
        dst[32 + lane] = b0;
        if (lane == 0) *reinterpret_cast<uint4*>(dst + 64) = make_uint4(rows_b[32], rows_t[32], cbl, ctl);
        if (lane == 1) dst[68] = (cbh & 1u) | ((cth & 1u) << 1);
        // Morton tile `lane` is the 8x4 cells at rows ty .. ty+3, columns tx ..
        // tx+7: its vertices from the rows' segment counts
        const uint32_t q = (uint32_t)lane;
        const int ty = morton_tile_y(q);
        const uint32_t tx = morton_tile_x(q);
        uint32_t tcnt = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) tcnt += (__shfl_sync(0xffffffffu, seg, ty + i) >> tx) & 0xffu;
        reinterpret_cast<uint16_t*>(dst + kRowSlotCounts)[lane] = (uint16_t)tcnt;
    }
    if (V.codes_out) {
        const int y = fy * 32 + lane;
        if (y < V.cells[1]) {
            uint8_t* row = V.codes_out + ((long long)z * V.cells[1] + y) * V.cells[0] + fx * 32;
            const int nx = min(32, V.cells[0] - fx * 32);
#pragma unroll
            for (int i = 0; i < 32; i++)
                if (i < nx) row[i] = (uint8_t)(w[i >> 2] >> (8 * (i & 3)));
        }
    }
}

// Bit rows and tables of a column classifier CTA.  Bit rows are kept for the last
// kRowBuffers sample layers (indexed by a running layer counter mod
// kRowBuffers): while a slow warp still classifies the slices of box p
// (layers 8p-1 .. 8p+7) other warps already convert box p+1 (layers 8p+8 ..
// 8p+15), so the buffers of the two boxes must not alias.
constexpr int kRowBuffers = 32;
constexpr int kSliceTable = 1024;

struct ColumnBits {
    // 16-byte aligned: warps store 4 rows at a time (uint4), whatever the
    // number of ring stages before it
    alignas(16) uint32_t rows[kRowBuffers][36];  // bit x = sample (x0 + x, y0 + r) below iso; [32] = row 32
    uint64_t col[kRowBuffers];                   // bit r = sample (x0 + 32, y0 + r) below iso; bit 32 = corner
    uint8_t cnt[256];
    // level-5 index of block (0, 0) of slice zfirst + i, i < kSliceTable: a
    // footprint's block is that OR its own Morton part (the footprint's bits
    // lie below the tile's), so a slice costs one load instead of two bit spreads
    uint32_t zbase[kSliceTable];
    int zfirst;
};
static_assert(offsetof(ColumnBits, rows) % 16 == 0 && (36 * 4) % 16 == 0, "uint4 row stores need 16-byte alignment");

static_assert(kWarps == 8 && kLayersPerBox <= kWarps, "a box's layers and slices map onto the 8 warps mod 8");
static_assert(kRowBuffers % kLayersPerBox == 0, "a box's bit-row buffers never wrap");

// The samples one lane turns into bits in a box: rows 4 warp .. 4 warp + 3 of
// every layer at column `lane`, and of one layer row 32, column 32 and the corner.
template <typename T>
struct BoxSamples {
    T v[kLayersPerBox][4];
    T row, col, corner;
};

// The layer of a box (first layer at running index gl0) whose row 32 and
// column 32 this warp takes.
__device__ __forceinline__ int edge_layer(uint32_t gl0, int warp) { return (int)(((uint32_t)warp - gl0 - 3u) & 7u); }

// Bit rows of the nl layers of one box, layer l stored at running index
// gl0 + l.  Warp w converts rows 4w .. 4w+3 of every layer; row 32 and column
// x0+32 of layer g go to warp (g + 3) mod 8.
template <typename T>
__device__ __forceinline__ void box_bits(const BoxSamples<T>& s, int nl, uint32_t gl0, float iso, int u8_thr, int warp,
                                         int lane, ColumnBits& C) {
    // gl0 is a multiple of kLayersPerBox and kRowBuffers of that, so a box's
    // buffers are g0 .. g0 + kLayersPerBox - 1 without wrapping
    const uint32_t g0 = gl0 & (kRowBuffers - 1);
    uint4* const rows_w = reinterpret_cast<uint4*>(&C.rows[g0][4 * warp]);
#pragma unroll
    for (int l = 0; l < kLayersPerBox; l++) {
        uint32_t b[4];
#pragma unroll
        for (int i = 0; i < 4; i++) b[i] = __ballot_sync(0xffffffffu, below(s.v[l][i], iso, u8_thr));
        if (l < nl && lane == 0) rows_w[l * (36 / 4)] = make_uint4(b[0], b[1], b[2], b[3]);
    }
    const uint32_t r32 = __ballot_sync(0xffffffffu, below(s.row, iso, u8_thr));
    const uint32_t col = __ballot_sync(0xffffffffu, below(s.col, iso, u8_thr));
    const bool corner = below(s.corner, iso, u8_thr);
    const int le = edge_layer(gl0, warp);
    if (le < nl && lane == 0) {
        const uint32_t buf = g0 + (uint32_t)le;
        C.rows[buf][32] = r32;
        C.col[buf] = (uint64_t)col | ((uint64_t)corner << 32);
    }
}

// Morton part of footprint (fx, fy) in a block index.
__device__ __forceinline__ uint32_t footprint_morton(int fx, int fy) {
    return morton_spread16((uint32_t)fx) | (morton_spread16((uint32_t)fy) << 1);
}

// Tables of the CTA (all threads; a barrier follows): case counts and the
// slice table from slice z0 on, up to slice z1.
__device__ __forceinline__ void fill_column_tables(const Volume& V, ColumnBits& C, int z0, int z1) {
    if (threadIdx.x == 0) C.zfirst = z0;
    C.cnt[threadIdx.x] = c_vertex_count[threadIdx.x];
    const int n = min(z1 - z0, kSliceTable);
    for (int i = threadIdx.x; i < n; i += blockDim.x) C.zbase[i] = (uint32_t)column_block_index(V, z0 + i, 0, 0);
}

__device__ __forceinline__ uint32_t slice_block(const Volume& V, const ColumnBits& C, int z, uint32_t fm) {
    const int i = z - C.zfirst;
    return (i < kSliceTable ? C.zbase[i] : (uint32_t)column_block_index(V, z, 0, 0)) | fm;
}

// After the box barrier: the slices whose upper layer arrived in this box
// (column-relative slices lb-1 .. lb+nl-2), warp (glu + slice) mod 8 each, so
// the work rotates over the warps from box to box.  glu = running index of
// the column's layer 0.
__device__ __forceinline__ void classify_box_slices(const Volume& V, int z0, int fx, int fy, uint32_t fm, int lb,
                                                    int nl, uint32_t glu, int warp, int lane, uint32_t vmask,
                                                    bool full, ColumnBits& C) {
    // the slice of this warp, if any.  glu + lb is the running index of the
    // box's first layer, a multiple of kLayersPerBox: with 8-layer boxes the
    // warp's offset in the box is the same in every box
    const uint32_t w1 = kLayersPerBox == 8 ? (uint32_t)(warp + 1) & 7u
                                           : ((uint32_t)warp - (glu + (uint32_t)lb - 1u)) & 7u;
    const int sl = lb - 1 + (int)w1;
    if (sl >= 0 && sl <= lb + nl - 2) {
        const uint32_t g = glu + (uint32_t)sl;
        const uint32_t bb = g & (kRowBuffers - 1), bt = (g + 1u) & (kRowBuffers - 1);
        const int z = z0 + sl;
        classify_slice_warp(V, z, fx, fy, slice_block(V, C, z, fm), lane, vmask, full, C.rows[bb], C.col[bb],
                            C.rows[bt], C.col[bt], C.cnt);
    }
}

// Cells of row `lane` of footprint (x0, y0) inside the grid (masked codes are
// 0, shadergen.cpp:112-125).
__device__ __forceinline__ uint32_t row_mask(const Volume& V, int x0, int y0, int lane) {
    const int xv = V.cells[0] - x0;
    const uint32_t xmask = xv >= 32 ? 0xffffffffu : ((1u << xv) - 1u);
    return (y0 + lane < V.cells[1]) ? xmask : 0u;
}

// Element type a field's samples are compared in.
template <int FT>
using SampleT = typename std::conditional<FT == kFieldU8 || FT == kFieldUNorm8, uint8_t, float>::type;

// Resident direct-classifier CTAs per SM the registers are held to: 3 against
// 2, 4, 5 measured on whole calls: f32 301x257x129 45.7 us (48.8, 45.4, 48.2),
// cubic functor 128^3 56.1 (56.2, 60.7, 59.6).
constexpr int kDirectCtas = 3;

// One sample of an array field, (x, y, z) inside the lattice.
template <int FT>
__device__ __forceinline__ SampleT<FT> direct_sample(const Volume& V, int x, int y, int z) {
    const long long at = (long long)z * V.slice_pitch + (long long)y * V.row_pitch + x;
    if constexpr (FT == kFieldU8 || FT == kFieldUNorm8)
        return __ldg(static_cast<const uint8_t*>(V.field) + at);
    else
        return fetch_raw<FT>(V, at);
}

// Bit rows of a box of an array field whose first layer is lattice layer z,
// straight from global memory, four layers of loads at a time; indices past the
// lattice are clamped (their cells are outside the grid and masked).
template <int FT>
__device__ __forceinline__ void direct_box_bits(const Volume& V, int x0, int y0, int z, int nl, uint32_t gl0, float iso,
                                                int warp, int lane, ColumnBits& C) {
    constexpr int kHalf = kLayersPerBox / 2;
    const int mx = V.lattice[0] - 1, my = V.lattice[1] - 1, mz = V.lattice[2] - 1;
    const int x = min(x0 + lane, mx), x32 = min(x0 + 32, mx), y32 = min(y0 + 32, my);
    const uint32_t g0 = gl0 & (kRowBuffers - 1);
    const int le = edge_layer(gl0, warp), ze = min(z + le, mz);
    const SampleT<FT> row = direct_sample<FT>(V, x, y32, ze), col = direct_sample<FT>(V, x32, min(y0 + lane, my), ze),
                      corner = direct_sample<FT>(V, x32, y32, ze);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        if (h * kHalf >= nl) break;
        SampleT<FT> v[kHalf][4];
#pragma unroll
        for (int l = 0; l < kHalf; l++)
#pragma unroll
            for (int i = 0; i < 4; i++)
                v[l][i] = direct_sample<FT>(V, x, min(y0 + 4 * warp + i, my), min(z + h * kHalf + l, mz));
#pragma unroll
        for (int l = 0; l < kHalf; l++) {
            uint32_t b[4];
#pragma unroll
            for (int i = 0; i < 4; i++) b[i] = __ballot_sync(0xffffffffu, below(v[l][i], iso, V.u8_thr));
            if (h * kHalf + l < nl && lane == 0)
                *reinterpret_cast<uint4*>(&C.rows[g0 + h * kHalf + l][4 * warp]) = make_uint4(b[0], b[1], b[2], b[3]);
        }
    }
    const uint32_t r32 = __ballot_sync(0xffffffffu, below(row, iso, V.u8_thr));
    const uint32_t c32 = __ballot_sync(0xffffffffu, below(col, iso, V.u8_thr));
    if (le < nl && lane == 0) {
        C.rows[g0 + (uint32_t)le][32] = r32;
        C.col[g0 + (uint32_t)le] = (uint64_t)c32 | ((uint64_t)below(corner, iso, V.u8_thr) << 32);
    }
}

// Bit rows of a box of a functor field: box_bits with every sample evaluated
// where it is compared.  A layer's four rows are evaluated together (their
// chains of dependent operations overlap) and the loops around them stay
// rolled: 35 inlined copies of a functor do not fit the instruction cache
// (the cubic at 128^3: 47.4 us unrolled, 16.4 us with one copy in the form of that
// measurement; 12.9 us now).
template <int FT, class UF>
__device__ __forceinline__ void functor_box_bits(const Volume& V, int x0, int y0, int z, int nl, uint32_t gl0, float iso,
                                                 int warp, int lane, ColumnBits& C) {
    const int mx = V.lattice[0] - 1, my = V.lattice[1] - 1;
    const uint32_t g0 = gl0 & (kRowBuffers - 1);
    const int x = min(x0 + lane, mx);
#pragma unroll 1
    for (int l = 0; l < nl; l++) {
        uint32_t b[4];
#pragma unroll
        for (int i = 0; i < 4; i++)
            b[i] = __ballot_sync(0xffffffffu, fetch<FT, UF>(V, x, min(y0 + 4 * warp + i, my), z + l) < iso);
        if (lane == 0) *reinterpret_cast<uint4*>(&C.rows[g0 + l][4 * warp]) = make_uint4(b[0], b[1], b[2], b[3]);
    }
    const int le = edge_layer(gl0, warp);
    if (le >= nl) return;
    uint64_t col = 0;
#pragma unroll 1
    for (int i = 0; i < 3; i++) {  // row 32, column 32, the corner
        const uint32_t b = __ballot_sync(
            0xffffffffu, fetch<FT, UF>(V, i == 0 ? x : min(x0 + 32, mx), min(y0 + (i == 1 ? lane : 32), my), z + le) < iso);
        if (i == 0 && lane == 0) C.rows[g0 + le][32] = b;
        if (i > 0) col |= i == 1 ? (uint64_t)b : (uint64_t)(b & 1u) << 32;
    }
    if (lane == 0) C.col[g0 + le] = col;
}

}  // namespace

// ---------------------------------------------------------------------------
// Direct column classifier: column layouts whose field no tensor map covers --
// rows that are no multiple of 16 bytes, float4 fields, functors.  One CTA per
// column.  Array samples come straight into registers (one coalesced row per
// load, 16 in flight per lane: keeping a whole next box in registers as well
// leaves room for 2 CTAs per SM only); functors are evaluated once per sample.  The block
// classifier it takes over from loads or evaluates 18 samples per 4 cells and
// visits the padding blocks of the layout.  Kernel times, block classifier ->
// this one: f32 301x257x129 51.9 -> 17.9 us, UNORM8 253x231x197 62.6 -> 24.0,
// float4 128^3 18.1 -> 9.7, the cubic functor at 128^3 44.7 -> 12.9.  Issue-
// bound on array fields (ballots and slice classification), not by memory.
//
// CTA body: column `u` (footprint-fastest) of V.  WAIT: also wait for the
// previous grid before the field and the pyramid are touched.
template <int FT, class UF, bool WAIT>
__device__ __forceinline__ void classify_column_direct(const Volume& V, int u, ColumnBits& C) {
    constexpr bool kArray = FT != kFieldFunctor && FT != kFieldUser;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per_slab = V.nfx * V.nfy;
    const int zc = u / per_slab, r = u - zc * per_slab;
    const int fy = r / V.nfx, fx = r - fy * V.nfx;
    const int x0 = fx * 32, y0 = fy * 32, z0 = zc * V.column_slices;
    const int z1 = min(V.cells[2], z0 + V.column_slices);
    const int nlayers = z1 - z0 + 1;
    const float iso = V.binary ? 0.5f : V.iso;
    fill_column_tables(V, C, z0, z1);
    const uint32_t fm = footprint_morton(fx, fy);
    const uint32_t vmask = row_mask(V, x0, y0, lane);
    const bool full = __all_sync(0xffffffffu, vmask == 0xffffffffu);
    if (WAIT) wait_prior_grid();
    for (int lb = 0; lb < nlayers; lb += kLayersPerBox) {
        const int nl = min(kLayersPerBox, nlayers - lb);
        if constexpr (kArray) direct_box_bits<FT>(V, x0, y0, z0 + lb, nl, (uint32_t)lb, iso, warp, lane, C);
        else functor_box_bits<FT, UF>(V, x0, y0, z0 + lb, nl, (uint32_t)lb, iso, warp, lane, C);
        __syncthreads();  // bit rows of this box ready, and every slice of the box before the last classified
        classify_box_slices(V, z0, fx, fy, fm, lb, nl, 0u, warp, lane, vmask, full, C);
    }
}

template <int FT, class UF = NoUserField>
__global__ void __launch_bounds__(kThreads, kDirectCtas) classify_columns_direct(const __grid_constant__ Volume V) {
    __shared__ __align__(16) ColumnBits C;
    classify_column_direct<FT, UF, true>(V, blockIdx.x, C);
}

// Columns of a volume (the direct classifier's grid).
inline int column_count(const Volume& V) {
    return V.nfx * V.nfy * ((V.cells[2] + V.column_slices - 1) / V.column_slices);
}

}  // namespace hpmc
