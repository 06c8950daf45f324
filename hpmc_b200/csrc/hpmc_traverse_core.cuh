// hpmc_traverse_core.cuh -- the per-vertex HistoPyramid traversal on sm_100a:
// shared-memory layout, case tables, the descent, the windows of active cells
// with their distinct edges, and the extraction kernel template.
//
// Reference: the traversal vertex shader extractVertex (shadergen.cpp:436-565,
// GL3+ path) driven by HPMCextractVertices (triface.cpp:332-457), one
// invocation per output vertex in batches of 3000 (constants.cpp:198).
//
// Included by kernels_traverse.cu (the library's field types) and by
// include/hpmc_functor.cuh (a caller's functor types, instantiated in the
// caller's own translation unit).  Every translation unit gets its own copy
// of the tables in its own device module.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "hpmc_device.cuh"
#include "hpmc_fetch.cuh"
#include "hpmc_geometry.cuh"
#include "hpmc_kernels.h"
#include "_gen/hpmc_case_tables.h"

namespace hpmc {

// Case tables of this translation unit's device module (HPMC's, generated at
// build time from its tables.cpp; see gen_tables.py).
static __constant__ uint8_t c_vertex_count_t[256] = HPMC_GEN_VERTEX_COUNT;
static __constant__ uint64_t c_edge_nibbles[256] = HPMC_GEN_EDGE_NIBBLES;
static __device__ const float g_binary_normals[256 * 16 * 3] = HPMC_GEN_BINARY_NORMALS;
constexpr uint64_t kEdgeGeometry = HPMC_GEN_EDGE_GEOMETRY;

enum { kModeForward = kGeomForward, kModeCentral = kGeomCentral, kModeBinary = kGeomBinary };

namespace {

// Edges of a cell by axis and the offset (sx, sy, sz) of their lower end.
__host__ __device__ constexpr uint32_t edge_geometry(int e) { return (uint32_t)(kEdgeGeometry >> (5 * e)) & 31u; }
__host__ __device__ constexpr int edge_id(int axis, int sx, int sy, int sz) {
    for (int e = 0; e < 12; e++)
        if (edge_geometry(e) == (uint32_t)(sx | (sy << 1) | (sz << 2) | (axis << 3))) return e;
    return 12;
}
// Edges with lower end at offset sx = 1 (sy = 1), and below edge e.
__host__ __device__ constexpr uint32_t edges_at(int bit) {
    uint32_t m = 0;
    for (int e = 0; e < 12; e++) m |= ((edge_geometry(e) >> bit) & 1u) << e;
    return m;
}
constexpr uint32_t kRightEdges = edges_at(0), kUpperEdges = edges_at(1);
__host__ __device__ constexpr uint32_t below_edge(int e) { return (1u << e) - 1u; }

constexpr int kWindowCells = 32;   // active cells a warp works on at a time (one per lane)
constexpr int kWindowEdges = 96;   // distinct edges of a window (8 cells never have more)

// One warp's working memory.
struct WarpArea {
    // what the window's edges hold (extraction: position x y, position z and
    // normal x, normal y z of the edge's vertex; three float2 cost fewer
    // shared-memory wavefronts to gather than two float4).  Before that, `data`
    // maps cells of the window to lanes.
    float2 data[3][kWindowEdges];
    uint4 row[33];                       // sample rows of the block: lower layer bits 0..31, bit 32, upper layer
    int4 strides[12];                    // edge_strides of the 12 edges
    uint2 cell[2 * kWindowCells];        // cells waiting for a window (see pack_cell)
    uint8_t slot[16 * kWindowCells];     // per vertex of the window: the slot of its edge
    uint16_t edge[kWindowEdges];         // edge | geometry << 4 | lane of its cell << 9
    uint16_t list[2 * kWindowCells];     // the block's next cells: x | y << 5
};
static_assert(kWindowEdges >= 96 && kWindowEdges <= 128 && kWindowCells == 32, "slots are bytes below 128");

// A waiting cell: x, y, z (below 2^14: lattices have at most 16384 samples per
// axis), its case, and the number (mod 64) of its block among those the warp
// has visited.
__device__ __forceinline__ uint2 pack_cell(int x, int y, int z, uint32_t code, uint32_t visit) {
    return make_uint2((uint32_t)x | ((uint32_t)y << 14), (uint32_t)z | (code << 14) | (visit << 22));
}

struct TraverseSmem {
    WarpArea warp[kWarps];
    uint64_t edge[256];
    alignas(16) uint32_t top[kTopCacheEntries];
    uint16_t cross[256];         // edges with a vertex, per case
    uint8_t cnt[256];
};

constexpr size_t kTraverseSmem = sizeof(TraverseSmem);
// Batched: a volume descriptor per warp follows.
static_assert(sizeof(TraverseSmem) % 16 == 0 && kVolumeHead % 8 == 0, "descriptors are copied in 8-byte words");
constexpr size_t kBatchSmem = sizeof(TraverseSmem) + kWarps * kVolumeHead;
// Dynamic shared memory without an opt-in per kernel, device and context; the
// adjoint has 6 KB of its own.
static_assert(kBatchSmem <= 48 * 1024 && kTraverseSmem + 6 * 1024 <= 48 * 1024, "at most 48 KB");

// The block a warp is working in: its vertices base .. base + count - 1, its
// key-space origin and, for the column layout, the lattice cell of its first
// key (every cell of such a block lies in the same slice tile).  Lane t holds
// the active cells of Morton tile t and the tile's first vertex and count.
struct WarpBlock {
    uint32_t b, base, count;
    uint32_t X0, Y0;
    int ox, oy, oz;
    uint32_t active, tstart, tcount;
    const uint32_t* slot;  // its arena slot
};

__device__ __forceinline__ uint32_t compact32(uint32_t v) {
    v &= 0x55555555u;
    v = (v | (v >> 1)) & 0x33333333u;
    v = (v | (v >> 2)) & 0x0f0f0f0fu;
    v = (v | (v >> 4)) & 0x00ff00ffu;
    v = (v | (v >> 8)) & 0x0000ffffu;
    return v;
}

// 16 bits -> Morton positions of an 8x2 cell tile: bit x of the low byte goes
// to bit (x0 | x1 << 2 | x2 << 4), bit x of the high byte to that + 8.
__device__ __forceinline__ uint32_t spread16(uint32_t t) {
    t = (t | (t << 12)) & 0x0F0F0F0Fu;
    return (t | (t << 2)) & 0x33333333u;
}

// prmt: byte i of the result is the byte of (hi, lo) that nibble i of sel
// numbers, or, where the nibble's top bit is set, that byte's sign in every bit
// (__byte_perm ignores the top bit).
__device__ __forceinline__ uint32_t select_bytes(uint32_t lo, uint32_t hi, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(lo), "r"(hi), "r"(sel));
    return r;
}

template <typename T>
__device__ __forceinline__ T warp_inclusive_scan(T v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Where block B.b lies: key-space origin, lattice cell of its first key (column
// layout) and arena slot, clamped to the arena (no clamping happens for
// consistent data).
__device__ __forceinline__ void locate_block(const Volume& V, WarpBlock& B) {
    B.X0 = compact32(B.b) << 5;
    B.Y0 = compact32(B.b >> 1) << 5;
    B.ox = (int)(B.X0 & ((1u << V.wx_l2) - 1u));
    B.oy = (int)(B.Y0 & ((1u << V.wy_l2) - 1u));
    B.oz = (int)(((B.Y0 >> V.wy_l2) << V.lx_l2) | (B.X0 >> V.wx_l2));
    uint32_t slot = V.column_layout ? ((uint32_t)B.oz * (uint32_t)V.nfy + ((uint32_t)B.oy >> 5)) * (uint32_t)V.nfx +
                                          ((uint32_t)B.ox >> 5)
                                    : B.b;
    if ((long long)slot >= V.arena_slots) slot = (uint32_t)(V.arena_slots - 1);
    B.slot = V.arena + (size_t)slot * (size_t)V.slot_words;
}

// One warp: the active cells of the (located) block from its arena slot.  Column layout:
// lane y takes sample rows y and y + 1 of both layers (bits below the
// iso-value), AND/OR over a cell's eight corners gives the active cells of
// row y, and four rows make a Morton tile's mask; the rows stay in shared
// memory for the cells' codes.
__device__ __forceinline__ void load_block(const Volume& V, WarpArea& W, int lane, WarpBlock& B) {
    const uint32_t* sw = B.slot;
    if (V.column_layout) {
        const uint32_t a0 = __ldg(sw + lane), b0 = __ldg(sw + 32 + lane);
        const uint4 ex = __ldg(reinterpret_cast<const uint4*>(sw + 64));
        const uint32_t corner = __ldg(sw + 68);
        B.tcount = __ldg(reinterpret_cast<const uint16_t*>(sw + kRowSlotCounts) + lane);
        const uint32_t ca = (ex.z >> lane) & 1u, cb = (ex.w >> lane) & 1u;
        W.row[lane] = make_uint4(a0, ca, b0, cb);
        if (lane == 0) W.row[32] = make_uint4(ex.x, corner & 1u, ex.y, corner >> 1);
        uint32_t a1 = __shfl_down_sync(0xffffffffu, a0, 1), b1 = __shfl_down_sync(0xffffffffu, b0, 1);
        a1 = lane == 31 ? ex.x : a1;
        b1 = lane == 31 ? ex.y : b1;
        const uint32_t ca1 = __funnelshift_rc(ex.z, corner, lane + 1) & 1u;
        const uint32_t cb1 = __funnelshift_rc(ex.w, corner >> 1, lane + 1) & 1u;
        const uint32_t a0x = (a0 >> 1) | (ca << 31), b0x = (b0 >> 1) | (cb << 31);
        const uint32_t a1x = (a1 >> 1) | (ca1 << 31), b1x = (b1 >> 1) | (cb1 << 31);
        const uint32_t all = a0 & a0x & a1 & a1x & b0 & b0x & b1 & b1x;
        const uint32_t any = a0 | a0x | a1 | a1x | b0 | b0x | b1 | b1x;
        const int xv = V.cells[0] - B.ox;
        const uint32_t xmask = xv >= 32 ? 0xffffffffu : ((1u << xv) - 1u);
        const uint32_t active = lane < V.cells[1] - B.oy ? (any & ~all) & xmask : 0u;
        const int ty = morton_tile_y((uint32_t)lane);
        const uint32_t tx = morton_tile_x((uint32_t)lane);
        uint32_t r[4];
#pragma unroll
        for (int i = 0; i < 4; i++) r[i] = (__shfl_sync(0xffffffffu, active, ty + i) >> tx) & 0xffu;
        // rows 0/2 on Morton bit 3 = 0/1 with bit 1 = 0; rows 1/3 shifted by 2 (bit 1 = 1)
        B.active = spread16(r[0] | (r[2] << 8)) | (spread16(r[1] | (r[3] << 8)) << 2);
    } else {
        B.active = __ldg(sw + kCodeSlotMasks + lane);
        B.tcount = __ldg(reinterpret_cast<const uint16_t*>(sw + kCodeSlotCounts) + lane);
    }
    B.tstart = warp_inclusive_scan(B.tcount, lane) - B.tcount;
}

// Case tables (no barrier).
__device__ __forceinline__ void load_base_tables(TraverseSmem& S) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {
        const uint32_t n = c_vertex_count_t[i];
        const uint64_t w = c_edge_nibbles[i];
        uint32_t m = 0;
        for (uint32_t k = 0; k < n; k++) m |= 1u << ((uint32_t)(w >> (4 * k)) & 15u);
        S.cnt[i] = (uint8_t)n;
        S.edge[i] = w;
        S.cross[i] = (uint16_t)m;
    }
}

__device__ __forceinline__ void load_tables(const Volume& V, TraverseSmem& S) {
    load_base_tables(S);
    // the pyramid and the control block only after the previous grid (the
    // build)
    wait_prior_grid();
    for (int i = threadIdx.x; i < V.top_cached; i += blockDim.x) S.top[i] = V.levels[i];
    __syncthreads();
}

// Descent through the dense levels (jtop-1 .. 5) for vertex key `key`
// (warp-uniform: every lane passes the same key).
__device__ __forceinline__ void descend(const Volume& V, const TraverseSmem& S, uint32_t key, uint32_t& block,
                                        uint32_t& base, uint32_t& count) {
    uint32_t node = 0;
    base = 0;
    count = V.top_cached ? S.top[0] : V.levels[V.level_off[V.jtop]];
    for (int j = V.jtop - 1; j >= kBlockLevel; j--) {
        const uint32_t idx = (uint32_t)V.level_off[j] + 4u * node;
        const uint4 s = (idx + 4u <= (uint32_t)V.top_cached)
                            ? *reinterpret_cast<const uint4*>(&S.top[idx])
                            : __ldg(reinterpret_cast<const uint4*>(V.levels + idx));
        const uint32_t s0 = s.x, s1 = s0 + s.y, s2 = s1 + s.z;
        const uint32_t c = (uint32_t)(key >= s0) + (uint32_t)(key >= s1) + (uint32_t)(key >= s2);
        const uint32_t skip = c == 0 ? 0u : c == 1 ? s0 : c == 2 ? s1 : s2;
        count = c == 0 ? s.x : c == 1 ? s.y : c == 2 ? s.z : s.w;
        key -= skip;
        base += skip;
        node = 4u * node + c;
    }
    block = node;
}

// Vertices of block b + 1 + lane (level 5): a warp walking forward out of block
// b takes the next block with vertices from them if there is one (one coalesced
// load instead of a descent through dependent loads).  Entries of padding
// blocks are zero: every level buffer is cleared when it is allocated and only
// the generic classifier writes those entries (with zero).
__device__ __forceinline__ uint32_t sibling_counts(const Volume& V, int lane, uint32_t b) {
    const unsigned long long e = (unsigned long long)b + 1ull + (unsigned long long)lane;
    return e < (unsigned long long)V.nblocks ? __ldg(V.levels + V.level_off[kBlockLevel] + e) : 0u;
}

__device__ __forceinline__ void prefetch_l1(const void* p) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// A group of cells of one window, ready for its edges and vertices: their
// distinct edges are numbered 0 .. nedges-1 (slots), and vertices
// first .. last-1 have their records.
struct CellGroup {
    const Volume& V;
    const TraverseSmem& S;
    WarpArea& W;
    int lane;
    uint32_t xy, z, code;    // this lane's cell: x | y << 14, z, MC case
    uint32_t at;             // element index of its first sample, bit 31: not an interior cell
    unsigned int lanes;      // the group's cells (a run of lanes)
    uint32_t start;          // this lane's first vertex
    uint32_t nedges, first, last;

    // f(slot, edge) for every distinct edge, 32 at a time.
    template <class F>
    __device__ __forceinline__ void edges(F&& f) const {
#pragma unroll 1
        for (uint32_t i0 = 0; i0 < nedges; i0 += 32) {
            const uint32_t i = i0 + (uint32_t)lane;
            const uint32_t id = W.edge[i < nedges ? i : nedges - 1u];
            const int l = (int)(id >> 9);
            const uint32_t cxy = __shfl_sync(0xffffffffu, xy, l), cz = __shfl_sync(0xffffffffu, z, l),
                           cat = __shfl_sync(0xffffffffu, at, l);
            if (i < nedges) {
                const int4 o = W.strides[id & 15u];
                EdgeAt E;
                E.a[0] = (int)((cxy & 0x3fffu) + ((id >> 4) & 1u));
                E.a[1] = (int)((cxy >> 14) + ((id >> 5) & 1u));
                E.a[2] = (int)(cz + ((id >> 6) & 1u));
                E.axis = (int)((id >> 7) & 3u);
                E.interior = (cat >> 31) == 0u;
                E.at = cat + (uint32_t)o.x;
                E.ou = o.y;
                E.ov = o.z;
                E.ow = o.w;
                f(i, E);
            }
        }
        __syncwarp();
    }

    // For the outputs that need a vertex's cell: one bit per cell that starts
    // among the 32 vertices from first + i0 on.
    __device__ __forceinline__ uint32_t starts(uint32_t i0) const {
        const uint32_t d = start - first - i0;
        return __reduce_or_sync(0xffffffffu, ((lanes >> lane) & 1u) && d < 32u ? 1u << d : 0u);
    }
};

// One window: the warp's first n waiting cells, one per lane, in vertex order;
// `pos` is the first one's first vertex, advanced past the last one's.  Cells
// whose first vertex lies in [v0, v1) are worked on, group by group: a group
// has at most kWindowEdges distinct edges; nearly always the whole window is
// one.  Vertices from N on are not written.
//
// An edge shared by several cells of the group belongs to the one with the
// largest (x, y) of the same block: a cell owns its crossed edges except those
// its right and upper neighbours in the group have too.  Slots number the owned
// edges in lane order, so a cell finds the slot of a neighbour's edge from that
// neighbour's owned mask and first slot.
template <class P>
__device__ __forceinline__ void process_window(const Volume& V, const TraverseSmem& S, WarpArea& W, int lane, uint32_t n,
                                               uint32_t& pos, uint32_t v0, uint32_t v1, uint32_t N, P& p) {
    const bool has = (uint32_t)lane < n;
    const uint2 c = W.cell[lane];
    const uint32_t xy = c.x, z = c.y & 0x3fffu, code = has ? (c.y >> 14) & 0xffu : 0u;
    const uint32_t cnt = S.cnt[code], cross = S.cross[code];  // none for code 0
    uint32_t start = warp_inclusive_scan(cnt, lane);
    const uint32_t total = __shfl_sync(0xffffffffu, start, 31);
    start += pos - cnt;
    pos += total;
    unsigned int chosen = __ballot_sync(0xffffffffu, has && start >= v0 && start < v1);
    if (!chosen) return;
    uint32_t at = 0x80000000u;
    if (V.idx32 && has && interior_cell(V, (int)(xy & 0x3fffu), (int)(xy >> 14), (int)z))
        at = z * (uint32_t)V.slice_pitch + (xy >> 14) * (uint32_t)V.row_pitch + (xy & 0x3fffu);
    // position in the block with room between its rows, so that key + 1, + 63,
    // + 64, + 65 are the right, upper left, upper and upper right neighbours or
    // no cell at all, and the block's number above; where lattice neighbours
    // need not be neighbours in the block (narrow tiles) no two are related
    const uint32_t key = V.column_layout ? (xy & 31u) | (((xy >> 14) & 31u) << 6) | ((c.y >> 22) << 12)
                                         : 70u * (uint32_t)lane;
    static_assert(31 + 31 * 64 + 65 < (int)sizeof(W.data) && 31 * 70 + 65 < (int)sizeof(W.data), "the map fits the edges' area");
    uint8_t* const lane_of = reinterpret_cast<uint8_t*>(W.data) + (key & 0xfffu);
    while (chosen) {
        unsigned int lanes = chosen;
        uint32_t own, ent, scan, nedges;
        uint32_t entR, entU, entL, entC;  // right, upper, upper left, upper right neighbour's entry
        bool hasR, hasU, hasL, hasC;
        if ((chosen >> lane) & 1u) *lane_of = (uint8_t)lane;
        __syncwarp();
        const int r = lane_of[1] & 31, ul = lane_of[63] & 31, u = lane_of[64] & 31, ur = lane_of[65] & 31;
        for (;;) {
            const bool mine = (lanes >> lane) & 1u;
            // a neighbour's lane is checked against that lane's own key (the
            // map is not cleared between windows)
            const uint32_t k = mine ? key : 0xffffffffu;
            hasR = __shfl_sync(0xffffffffu, k, r) == key + 1u;
            hasL = __shfl_sync(0xffffffffu, k, ul) == key + 63u;
            hasU = __shfl_sync(0xffffffffu, k, u) == key + 64u;
            hasC = __shfl_sync(0xffffffffu, k, ur) == key + 65u;
            own = mine ? cross : 0u;
            if (hasR) own &= ~kRightEdges;
            if (hasU) own &= ~kUpperEdges;
            if (hasL) own &= ~(1u << edge_id(2, 0, 1, 0));
            if (hasC) own &= ~(1u << edge_id(2, 1, 1, 0));
            const uint32_t m = (uint32_t)__popc(own);
            scan = warp_inclusive_scan(m, lane);
            nedges = __shfl_sync(0xffffffffu, scan, 31);
            scan -= m;
            ent = own | (scan << 16);
            entR = __shfl_sync(0xffffffffu, ent, r);
            entU = __shfl_sync(0xffffffffu, ent, u);
            entL = __shfl_sync(0xffffffffu, ent, ul);
            entC = __shfl_sync(0xffffffffu, ent, ur);
            if (nedges <= (uint32_t)kWindowEdges) break;
            // too many: the first half of the cells (8 cells always fit)
            lanes &= (2u << (__ffs((int)lanes) - 1 + (__popc(lanes) >> 1) - 1)) - 1u;
        }
        __syncwarp();  // every lane has read the map
        auto slot = [](uint32_t entry, uint32_t below) { return (entry >> 16) + (uint32_t)__popc(entry & below); };
        uint32_t w[3] = {0u, 0u, 0u};
        auto put = [&](int e, uint32_t s) {
            w[e >> 2] |= s << (8 * (e & 3));
            if ((own >> e) & 1u) W.edge[s] = (uint16_t)((uint32_t)e | (edge_geometry(e) << 4) | ((uint32_t)lane << 9));
        };
#pragma unroll
        for (int sz = 0; sz < 2; sz++) {
            constexpr uint32_t (*b)(int) = below_edge;
            put(edge_id(0, 0, 0, sz), slot(ent, b(edge_id(0, 0, 0, sz))));
            put(edge_id(1, 0, 0, sz), slot(ent, b(edge_id(1, 0, 0, sz))));
            put(edge_id(0, 0, 1, sz), slot(hasU ? entU : ent, hasU ? b(edge_id(0, 0, 0, sz)) : b(edge_id(0, 0, 1, sz))));
            put(edge_id(1, 1, 0, sz), slot(hasR ? entR : ent, hasR ? b(edge_id(1, 0, 0, sz)) : b(edge_id(1, 1, 0, sz))));
        }
        constexpr int z00 = edge_id(2, 0, 0, 0), z10 = edge_id(2, 1, 0, 0), z01 = edge_id(2, 0, 1, 0),
                      z11 = edge_id(2, 1, 1, 0);
        constexpr uint32_t b00 = below_edge(z00), b10 = below_edge(z10), b01 = below_edge(z01), b11 = below_edge(z11);
        put(z00, slot(ent, b00));
        put(z10, slot(hasR ? entR : ent, hasR ? b00 : b10));
        put(z01, slot(hasU ? entU : hasL ? entL : ent, hasU ? b00 : hasL ? b10 : b01));
        put(z11, slot(hasC ? entC : hasU ? entU : hasR ? entR : ent, hasC ? b00 : hasU ? b10 : hasR ? b01 : b11));
        const int l0 = __ffs((int)lanes) - 1, l1 = 31 - __clz((int)lanes);
        const uint32_t first = __shfl_sync(0xffffffffu, start, l0);
        const uint32_t last = __shfl_sync(0xffffffffu, start + cnt, l1);
#pragma unroll
        for (int i = 0; i < 3; i++) w[i] &= 0x7f7f7f7fu;  // (edges without a vertex may have larger numbers)
        // the vertices' slots: vertex k lies on the edge in nibble k of the
        // case's word, and the nibbles are byte selectors as they stand -- of
        // w[0], w[1] for edges 0..7, with the top bit flipped of w[2] for 8..11
        // (a selector with the top bit set gives the sign of a byte below 128: 0)
        const uint32_t nv = (lanes >> lane) & 1u ? cnt : 0u;
        const uint32_t most = __reduce_max_sync(0xffffffffu, nv);
        uint8_t* const to = W.slot + (start - first);
        const uint64_t nibbles = S.edge[code];
#pragma unroll
        for (uint32_t k = 0; k < 15; k += 4) {
            if (k >= most) break;
            const uint32_t sel = (uint32_t)(k < 8 ? nibbles : nibbles >> 32) >> (4 * (k & 7));
            const uint32_t four = select_bytes(w[0], w[1], sel) | select_bytes(w[2], 0u, sel ^ 0x8888u);
#pragma unroll
            for (uint32_t j = 0; j < 4 && k + j < 15; j++)
                if (k + j < nv) to[k + j] = (uint8_t)(four >> (8 * j));
        }
        __syncwarp();  // edges and slots ready
        p.run(CellGroup{V, S, W, lane, xy, z, code, at, lanes, start, nedges, first, min(last, N)});
        chosen &= ~lanes;
    }
}

// The cells whose first vertex lies in [v0, v1); vertices from N on are not
// written.  One descent, then block by block (the next block's slot is on its
// way to L1 while a block is worked on).  A block's active cells are listed in
// Morton (= vertex) order, tile by tile with one lane per cell, their cases
// read from the block's sample rows, and queued; windows of 32 cells are taken
// from the queue, whatever blocks they come from.  Tiles outside the range are
// skipped by their counts.
template <class P>
__device__ __forceinline__ void walk_range(const Volume& V, const TraverseSmem& S, WarpArea& W, int lane, uint32_t v0,
                                           uint32_t v1, uint32_t N, P& p) {
    WarpBlock B;
    uint32_t queued = 0, pos = 0, visit = 0, next = v0;
    bool found = false;  // B is the block of vertex `next`, and located
    // this lane's cell in a tile and the first cell of tile `lane`, x | y << 5
    const uint32_t in_tile = morton_tile_cell((uint32_t)lane);
    const uint32_t tile_at = morton_tile_x((uint32_t)lane) | ((uint32_t)morton_tile_y((uint32_t)lane) << 5);
    for (;;) {
        if (!found) {
            descend(V, S, next, B.b, B.base, B.count);
            locate_block(V, B);
        }
        next = B.base + B.count;
        const bool more = next < v1 && B.count != 0u;
        const uint32_t sib = more ? sibling_counts(V, lane, B.b) : 0u;
        load_block(V, W, lane, B);
        const uint32_t sm = __ballot_sync(0xffffffffu, sib != 0u);
        found = sm != 0u;
        WarpBlock N1 = B;
        if (found) {
            const uint32_t ahead = (uint32_t)__ffs((int)sm);  // the next block is b + ahead
            N1.b += ahead;
            N1.base = next;
            N1.count = __shfl_sync(0xffffffffu, sib, (int)ahead - 1);
            locate_block(V, N1);
            if (lane < 3) prefetch_l1(N1.slot + 32 * lane);  // a row slot; part of a code slot
        }
        const uint32_t k0 = v0 > B.base ? v0 - B.base : 0u, k1 = v1 - B.base;
        uint32_t tiles = __ballot_sync(0xffffffffu, B.active != 0u && B.tstart < k1 && B.tstart + B.tcount > k0);
        // (nothing is queued before the first block)
        if (!queued && tiles) pos = B.base + __shfl_sync(0xffffffffu, B.tstart, __ffs((int)tiles) - 1);
        uint32_t listed = 0;
        // the last block also empties the queue
        while (tiles || listed || (!more && queued)) {
            while (listed < kWindowCells && tiles) {
                const int t = __ffs((int)tiles) - 1;
                tiles &= tiles - 1u;
                const uint32_t m = __shfl_sync(0xffffffffu, B.active, t);
                const uint32_t at = __shfl_sync(0xffffffffu, tile_at, t);
                if ((m >> lane) & 1u)
                    W.list[listed + (uint32_t)__popc(m & ((1u << lane) - 1u))] = (uint16_t)(at + in_tile);
                listed += (uint32_t)__popc(m);
            }
            __syncwarp();  // the list (and the block's rows) are visible
            const uint32_t n = min(listed, (uint32_t)kWindowCells);
            const uint32_t later = W.list[kWindowCells + lane];
            if ((uint32_t)lane < n) {
                const uint32_t xy = W.list[lane], x = xy & 31u, y = (xy >> 5) & 31u;
                int cx = B.ox + (int)x, cy = B.oy + (int)y, cz = B.oz;
                uint32_t code;
                if (V.column_layout) {
                    const uint4 q0 = W.row[y], q1 = W.row[y + 1];
                    code = (__funnelshift_r(q0.x, q0.y, x) & 3u) | ((__funnelshift_r(q1.x, q1.y, x) & 3u) << 2) |
                           ((__funnelshift_r(q0.z, q0.w, x) & 3u) << 4) | ((__funnelshift_r(q1.z, q1.w, x) & 3u) << 6);
                } else {
                    code = __ldg(reinterpret_cast<const uint8_t*>(B.slot) + (morton_spread16(x) | (morton_spread16(y) << 1)));
                    virtual_to_cell(V, B.X0 + x, B.Y0 + y, cx, cy, cz);
                }
                W.cell[queued + (uint32_t)lane] = pack_cell(cx, cy, cz, code, visit);
            }
            __syncwarp();
            W.list[lane] = (uint16_t)later;  // the cells past these 32 move up
            listed -= n;
            queued += n;
            if (queued >= kWindowCells || (!more && !tiles && !listed)) {
                const uint2 rest = W.cell[kWindowCells + lane];
                const uint32_t m = min(queued, (uint32_t)kWindowCells);
                process_window(V, S, W, lane, m, pos, v0, v1, N, p);
                __syncwarp();
                W.cell[lane] = rest;
                queued -= m;
            }
            __syncwarp();
        }
        if (!more) break;
        if (found) B = N1;
        visit = (visit + 1u) & 63u;
    }
    __syncwarp();
}

// The strides of the volume's 12 edges (a warp).
__device__ __forceinline__ void set_volume(const Volume& V, WarpArea& W, int lane) {
    if (lane < 12) W.strides[lane] = edge_strides(V, (uint32_t)(kEdgeGeometry >> (5 * lane)) & 31u);
    __syncwarp();
}

// Rounds of 32 vertices per work item: one item per warp of the (resident,
// persistent) grid, i.e. a contiguous vertex range per warp.  Every item
// starts with a descent through dependent loads of the upper levels; after
// that the warp walks from block to block, so fewer, longer items are faster
// (measured: one item per warp beats two or four per warp), and per-vertex
// work is uniform enough that the ranges stay balanced.  At least
// kMinRounds, so that a window's set-up serves more than a few cells.
__device__ __forceinline__ uint32_t item_rounds(uint32_t N, uint32_t ctas) {
    const uint32_t warps = ctas * (uint32_t)kWarps;
    const uint32_t r = (uint32_t)(((unsigned long long)N + 32u * warps - 1u) / (32u * warps));
    return r < (uint32_t)kMinRounds ? (uint32_t)kMinRounds : r;
}

// Dynamic work queue over vertex chunks (balances the persistent grid):
// lane 0 takes the next chunk for its warp.
__device__ __forceinline__ uint32_t next_chunk(const Volume& V, int lane) {
    uint32_t c = 0;
    if (lane == 0) c = atomicAdd(&V.ctrl->work_next, 1u);
    return __shfl_sync(0xffffffffu, c, 0);
}

// The last CTA to finish resets the queue for the next launch on the stream
// (and, after an extraction, clears the pyramid's extraction flag).
__device__ __forceinline__ void finish_queue(const Volume& V, bool extraction = false) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&V.ctrl->work_done, 1u) == gridDim.x - 1) {
            V.ctrl->work_next = 0;
            V.ctrl->work_done = 0;
            if (extraction) V.ctrl->extracting = 0;
            __threadfence();
        }
    }
}

__device__ __forceinline__ uint32_t next_chunk_batch(const BatchDev& Bt, int lane) {
    uint32_t c = 0;
    if (lane == 0) c = atomicAdd(&Bt.ctrl->work_next, 1u);
    return __shfl_sync(0xffffffffu, c, 0);
}

__device__ __forceinline__ void finish_queue_batch(const BatchDev& Bt) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&Bt.ctrl->work_done, 1u) == gridDim.x - 1) {
            Bt.ctrl->work_next = 0;
            Bt.ctrl->work_done = 0;
            __threadfence();
        }
    }
}

}  // namespace

// ---------------------------------------------------------------------------
// The extraction: every vertex of the last build (up to the outputs'
// capacity), in the reference's vertex order.
//
// What bounds it: the L1 data pipe where the surface is dense (a gather of 32
// edges touches about 12 lines), else the instructions and latencies of the
// block walk.  A warp used to take 32 vertices a round and compute each one's
// geometry (489 warp instructions a round, 14 gathers a vertex); an edge's
// vertex is emitted by 6 triangles, so computing each distinct edge of a window
// once removes more than half of the gathers.  Windows span blocks because a
// sparse surface leaves only about 50 active cells in a block.  kTraverseCtas:
// 3 CTAs of 39 KB leave L1 room for the gathers; 4 (64 registers) measured 1 to
// 5 % slower, 5 (spills) 5 to 25 %, and a 222 KB footprint of the shared memory
// 15 % slower on the 512^3 cubic.  kWindowEdges: 96 against 128, the same
// except the batch, 12 % faster.  The batched form spills 52 to 100 bytes at its 80
// registers, the others nothing.  Kernel times before -> now: 512^3 cubic 84.5
// -> 72.8 us, 512x512x33 slab 46.9 -> 33.2, uint8 noise 256^3 360 -> 305,
// UNORM8 noise 253x231x197 225 -> 161, float4 128^3 28.6 -> 18.8, 64 volumes
// batched 364 -> 247, metaballs 64^3 24.3 -> 14.6.  UF: a caller's functor type
// when FT == kFieldUser (include/hpmc_functor.cuh).  EXTRA: the interleaved
// feedback and inspection outputs may be set (false: positions and normals
// only, without their per-vertex tests).
template <int FT, int MODE, class UF, bool EXTRA>
struct ExtractVertices {
    static constexpr bool kInfo = EXTRA || MODE == kModeBinary;
    const TraverseOut& O;
    unsigned long long out;  // output index of the volume's first vertex

    __device__ __forceinline__ void run(const CellGroup& G) {
        const Volume& V = G.V;
        WarpArea& W = G.W;
        G.edges([&](uint32_t slot, const EdgeAt& E) {
            float q[3], n[3], t;
            edge_vertex<FT, MODE, UF>(V, E, q, n, t);
            W.data[0][slot] = make_float2(q[0], q[1]);
            W.data[1][slot] = make_float2(q[2], n[0]);
            W.data[2][slot] = make_float2(n[1], n[2]);
        });
        const uint32_t n = G.last - G.first;
        const unsigned long long o0 = out + G.first;
        if (!kInfo) {
            float4* pos = O.pos + o0 + G.lane;
            float4* nrm = O.nrm + o0 + G.lane;
            const bool p = O.pos != nullptr, q = O.nrm != nullptr;
#pragma unroll 1
            for (uint32_t i = (uint32_t)G.lane; i < n; i += 32, pos += 32, nrm += 32) {
                const float2* d = &W.data[0][W.slot[i]];
                const float2 d0 = d[0], d1 = d[kWindowEdges], d2 = d[2 * kWindowEdges];
                if (p) __stcs(pos, make_float4(d0.x, d0.y, d1.x, 1.0f));
                if (q) __stcs(nrm, make_float4(d1.y, d2.x, d2.y, 0.0f));
            }
            __syncwarp();
            return;
        }
        uint32_t c0 = (uint32_t)__ffs((int)G.lanes) - 2u;  // + cells that start at or before the vertex
#pragma unroll 1
        for (uint32_t i0 = 0; i0 < n; i0 += 32) {
            // a lane's cell follows from the cells that start in this round
            const uint32_t i = i0 + (uint32_t)G.lane, starts = G.starts(i0);
            const int c = (int)((c0 + (uint32_t)__popc(starts & (0xffffffffu >> (31 - G.lane)))) & 31u);
            c0 += (uint32_t)__popc(starts);
            const uint32_t code = __shfl_sync(0xffffffffu, G.code, c);
            const uint32_t k = (G.first + i - __shfl_sync(0xffffffffu, G.start, c)) & 15u;
            const uint32_t xy = EXTRA ? __shfl_sync(0xffffffffu, G.xy, c) : 0u;
            const uint32_t z = EXTRA ? __shfl_sync(0xffffffffu, G.z, c) : 0u;
            if (i >= n) continue;
            const unsigned long long o = o0 + i;
            const float2* d = &W.data[0][W.slot[i]];
            const float2 d0 = d[0], d1 = d[kWindowEdges], d2 = d[2 * kWindowEdges];
            float m[3] = {d1.y, d2.x, d2.y};
            if (MODE == kModeBinary) {
                // the reference's table normal of the case's vertex (constants.cpp:217-273)
                const float* b = g_binary_normals + 3u * (16u * code + k);
#pragma unroll
                for (int j = 0; j < 3; j++) m[j] = b[j] * V.scale[j];
            }
            if (O.pos) __stcs(O.pos + o, make_float4(d0.x, d0.y, d1.x, 1.0f));
            if (O.nrm) __stcs(O.nrm + o, make_float4(m[0], m[1], m[2], 0.0f));
            if (EXTRA && O.feedback) {
                float2* fb = reinterpret_cast<float2*>(O.feedback + 6ull * o);
                __stcs(fb + 0, make_float2(m[0], m[1]));
                __stcs(fb + 1, make_float2(m[2], d0.x));
                __stcs(fb + 2, make_float2(d0.y, d1.x));
            }
            if (EXTRA && (O.dbg_cell || O.dbg_t)) {
                const int x = (int)(xy & 0x3fffu), y = (int)(xy >> 14);
                const uint32_t e = (uint32_t)(G.S.edge[code] >> (4u * k)) & 15u;
                if (O.dbg_cell) O.dbg_cell[o] = make_int4(x, y, (int)z, (int)(code | (k << 8) | (e << 16)));
                if (O.dbg_t) {  // the crossing parameter again, from the vertex's own edge
                    float q[3], u[3], t;
                    edge_vertex<FT, MODE, UF>(V, edge_at(V, x, y, (int)z, (uint32_t)(kEdgeGeometry >> (5u * e)) & 31u), q,
                                              u, t);
                    O.dbg_t[o] = t;
                }
            }
        }
        __syncwarp();
    }
};

template <int FT, int MODE, class UF = NoUserField, bool EXTRA = true>
__global__ void __launch_bounds__(kThreads, kTraverseCtas) traverse_kernel(const __grid_constant__ Volume V,
                                                                           const __grid_constant__ TraverseOut O) {
    extern __shared__ __align__(16) uint8_t s_traverse[];
    TraverseSmem& S = *reinterpret_cast<TraverseSmem*>(s_traverse);
    load_tables(V, S);
    // The next grid (normally the next build) may launch now.  The flag,
    // written before any CTA of this one lets it launch, tells that build's
    // column classifier that the previous grid is this extraction, which
    // neither writes the field nor reads the set of levels and arena that the
    // build writes next; the last CTA clears it.
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        V.ctrl->extracting = 1u;
        __threadfence();
    }
    __syncthreads();
    allow_next_grid();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned long long total = V.ctrl->total;
    const uint32_t N = (uint32_t)(total < O.capacity ? total : O.capacity);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (total > O.capacity) atomicOr(&V.ctrl->status, kStatusCapacity);
        V.ctrl->written = N;
    }
    const uint32_t VW = 32u * item_rounds(N, gridDim.x);
    const uint32_t nchunks = (N + VW - 1) / VW;
    set_volume(V, S.warp[warp], lane);
    ExtractVertices<FT, MODE, UF, EXTRA> p{O, V.vertex_base};
    for (uint32_t chunk = next_chunk(V, lane); chunk < nchunks; chunk = next_chunk(V, lane))
        walk_range(V, S, S.warp[warp], lane, chunk * VW, min(N, (chunk + 1u) * VW), N, p);
    finish_queue(V, true);
}

// Launch of one instantiation of the extraction.
template <int FT, int MODE, class UF, bool EXTRA>
inline cudaError_t launch_traverse_kernel(const Volume& V, const TraverseOut& O, int grid, cudaStream_t st) {
    return launch_dependent(traverse_kernel<FT, MODE, UF, EXTRA>, grid, kThreads, kTraverseSmem, st, V, O);
}

}  // namespace hpmc
