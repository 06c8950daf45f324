// kernels_traverse.cu -- per-vertex HistoPyramid traversal, geometry and the
// adjoint, on sm_100a.
//
// Reference: the traversal vertex shader extractVertex (shadergen.cpp:436-565,
// GL3+ path) driven by HPMCextractVertices (triface.cpp:332-457), one
// invocation per output vertex in batches of 3000 (constants.cpp:198).
//
// Here one persistent grid walks the vertex range, a contiguous range per warp:
//   1. descent (warp-cooperative): the warp descends the dense levels for its
//      first vertex, from the top (cached in shared memory) to the 1024-key
//      block, taking the first child whose running sum exceeds the key exactly
//      as shadergen.cpp:448-467 does; a warp that walks out of its block takes
//      the next non-empty one from the following 32 level-5 entries (one
//      coalesced load) when it lies there.
//   2. cells (warp-cooperative; replaces the base-level steps of
//      shadergen.cpp:469-495): the classifier left every non-empty block's
//      sample bits in the block's arena slot; the warp derives the active
//      cells in Morton (= vertex) order and takes them 32 at a time, one per
//      lane: code, vertex count, and one scan for the first vertices.
//   3. edges: the distinct crossed edges of the 32 cells are numbered, and
//      each one's vertex -- crossing parameter, position, normal
//      (shadergen.cpp:497-563) -- is computed once, into shared memory; FP32
//      arithmetic with a float-float fallback for ill-conditioned normals.
//   4. vertices: a lane finds its vertex's cell with one OR-reduction and a
//      popcount, the edge from the case table, and copies the edge's vertex to
//      the outputs with coalesced streaming float4 stores.
#include <cuda_runtime.h>
#include <cstdint>

#include "hpmc_batch.cuh"
#include "hpmc_device.cuh"
#include "hpmc_fetch.cuh"
#include "hpmc_geometry.cuh"
#include "hpmc_kernels.h"
#include "hpmc_traverse_core.cuh"

namespace hpmc {

// ---------------------------------------------------------------------------
// Adjoint: recompute the traversal of each vertex and scatter
// dL/dp . dp/df + dL/dn . dn/df onto the field samples the vertex read.
//   t = (f_a - iso)/(f_a - f_b):  dt/df_a = (iso - f_b)/(f_a - f_b)^2,
//                                 dt/df_b = (f_a - iso)/(f_a - f_b)^2
//   p_axis = (a_axis + t) s_axis
//   forward: n_i = ((1-t)(iso - f(a+e_i)) + t(iso - f(b+e_i))) s_i
//   central: n_i = -1/2((1-t)(f(a+e_i) - f(a-e_i)) + t(f(b+e_i) - f(b-e_i))) s_i
// Clamped samples scatter to the sample that was read.
namespace {
__device__ __forceinline__ void scatter(const Volume& V, float* dfield, const int* a, int dx, int dy, int dz,
                                        float g) {
    const int x = min(max(a[0] + dx, 0), V.lattice[0] - 1);
    const int y = min(max(a[1] + dy, 0), V.lattice[1] - 1);
    const int z = min(max(a[2] + dz, 0), V.lattice[2] - 1);
    atomicAdd(dfield + (long long)z * V.slice_pitch + (long long)y * V.row_pitch + x, g);
}
}  // namespace

// The last group may be cut inside a cell: an edge that only vertices past the
// cut lie on has no cotangent, and 0 times an overflowing derivative is not 0.
// The first vertex's edge takes its place, once more with no cotangent.  (Where
// nothing is cut every edge is seen.)  n: the group's vertices; seen: a word per edge.
static __device__ __noinline__ void drop_unseen_edges(WarpArea& W, uint32_t* seen, uint32_t nedges, uint32_t n, int lane) {
    static_assert(kWindowEdges <= 32 * 6, "the staging area has a word per edge");
    for (uint32_t i = (uint32_t)lane; i < nedges; i += 32) seen[i] = 0u;
    __syncwarp();
    for (uint32_t i = (uint32_t)lane; i < n; i += 32) seen[W.slot[i]] = 1u;
    __syncwarp();
    for (uint32_t i = (uint32_t)lane; i < nedges; i += 32)
        if (!seen[i]) W.edge[i] = W.edge[W.slot[0]];
    __syncwarp();
}

// Every distinct edge of a group of cells is differentiated once: the vertices
// on it -- the same crossing emitted by neighbouring triangles -- have the same
// Jacobian, so their cotangents are summed into the edge's slot first.  (Summing
// only within rounds of 32 vertices, with a third of the lanes then gathering
// and scattering, took 50 us on the 128^3 spheres; this takes 27.)
template <int FT, int MODE>
struct AdjointVertices {
    const AdjointIO& A;
    float (*agg)[6];    // the warp's staging area, one row per lane
    unsigned long long out;
    uint32_t end;       // vertices differentiated

    __device__ __forceinline__ void run(const CellGroup& G) {
        const Volume& V = G.V;
        WarpArea& W = G.W;
        for (uint32_t i = (uint32_t)G.lane; i < G.nedges; i += 32)
            W.data[0][i] = W.data[1][i] = W.data[2][i] = make_float2(0.f, 0.f);
        __syncwarp();
        const uint32_t n = G.last - G.first;
#pragma unroll 1
        for (uint32_t i0 = 0; i0 < n; i0 += 32) {
            const uint32_t i = i0 + (uint32_t)G.lane;
            const bool act = i < n;
            const uint32_t slot = act ? W.slot[i] : 0x10000u | (uint32_t)G.lane;
            float4 dp = make_float4(0.f, 0.f, 0.f, 0.f), dn = dp;
            if (act) {
                const unsigned long long o = out + G.first + i;
                if (A.dpos) dp = __ldg(A.dpos + o);
                if (A.dnrm) dn = __ldg(A.dnrm + o);
            }
            // lanes on the same edge: the lowest one adds up their cotangents
            const unsigned int peers = __match_any_sync(0xffffffffu, slot);
            float* mine = agg[G.lane];
            mine[0] = dp.x; mine[1] = dp.y; mine[2] = dp.z;
            mine[3] = dn.x; mine[4] = dn.y; mine[5] = dn.z;
            __syncwarp();
            if (act && __ffs((int)peers) - 1 == G.lane) {
                for (unsigned int rest = peers & (peers - 1u); rest; rest &= rest - 1u) {
                    const float* q = agg[__ffs((int)rest) - 1];
                    dp.x += q[0]; dp.y += q[1]; dp.z += q[2];
                    dn.x += q[3]; dn.y += q[4]; dn.z += q[5];
                }
                float2 &s0 = W.data[0][slot], &s1 = W.data[1][slot], &s2 = W.data[2][slot];
                s0.x += dp.x; s0.y += dp.y; s1.x += dp.z;
                s1.y += dn.x; s2.x += dn.y; s2.y += dn.z;
            }
            __syncwarp();
        }
        if (G.last == end) drop_unseen_edges(W, reinterpret_cast<uint32_t*>(agg), G.nedges, n, G.lane);
        G.edges([&](uint32_t slot, const EdgeAt& E) {
            const int ax = E.axis;
            const float iso = V.iso;
            const float2 s0 = W.data[0][slot], s1 = W.data[1][slot], s2 = W.data[2][slot];
            EdgeField F{};
            gather_edge<FT, MODE == kModeCentral>(V, E, F);
            // along (u, v, w): the edge's axis and the two after it
            const float sc[3] = {V.scale[0], V.scale[1], V.scale[2]};
            const float dp[3] = {s0.x * sc[0], s0.y * sc[1], s1.x * sc[2]};
            const float dn[3] = {s1.y * sc[0], s2.x * sc[1], s2.y * sc[2]};
            const float du = ax == 0 ? dn[0] : ax == 1 ? dn[1] : dn[2];
            const float dvw[2] = {ax == 0 ? dn[1] : ax == 1 ? dn[2] : dn[0], ax == 0 ? dn[2] : ax == 1 ? dn[0] : dn[1]};
            const int u[3] = {ax == 0, ax == 1, ax == 2};
            auto add = [&](int nu, int nv, int nw, float g) {
                if (E.interior) {
                    atomicAdd(A.dfield + (E.at + (uint32_t)(nu * E.ou + nv * E.ov + nw * E.ow)), g);
                    return;
                }
                scatter(V, A.dfield, E.a, nu * u[0] + nv * u[2] + nw * u[1], nu * u[1] + nv * u[0] + nw * u[2],
                        nu * u[2] + nv * u[1] + nw * u[0], g);
            };
            const float den = F.va - F.vb;
            const FF tf = ff_ratio_of_diffs(F.va, iso, F.va, F.vb);
            const float t = tf.hi + tf.lo;
            const float omt = 1.0f - t;
            float dLdt = ax == 0 ? dp[0] : ax == 1 ? dp[1] : dp[2];
            float ga = 0.0f, gb = 0.0f;  // direct contributions to samples a and b
            if (MODE == kModeForward) {
                dLdt += du * (F.vb - F.bp);
                gb -= omt * du;
                add(2, 0, 0, -t * du);
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    dLdt += dvw[i] * (F.ap[i] - F.bpv[i]);
                    add(0, i == 0, i == 1, -omt * dvw[i]);
                    add(1, i == 0, i == 1, -t * dvw[i]);
                }
            } else {
                dLdt -= 0.5f * du * ((F.bp - F.va) - (F.vb - F.am));
                const float wa = -0.5f * omt * du, wb = -0.5f * t * du;
                gb += wa;
                ga -= wb;
                add(-1, 0, 0, -wa);
                add(2, 0, 0, wb);
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    dLdt -= 0.5f * dvw[i] * ((F.bpv[i] - F.bmv[i]) - (F.ap[i] - F.amv[i]));
                    const float va = -0.5f * omt * dvw[i], vb = -0.5f * t * dvw[i];
                    add(0, i == 0, i == 1, va);
                    add(0, -(i == 0), -(i == 1), -va);
                    add(1, i == 0, i == 1, vb);
                    add(1, -(i == 0), -(i == 1), -vb);
                }
            }
            const float inv = 1.0f / (den * den);
            ga += dLdt * (iso - F.vb) * inv;
            gb += dLdt * (F.va - iso) * inv;
            add(0, 0, 0, ga);
            add(1, 0, 0, gb);
        });
    }
};

template <int FT, int MODE>
__global__ void __launch_bounds__(kThreads, kTraverseCtas) adjoint_kernel(const __grid_constant__ Volume V,
                                                                          const __grid_constant__ AdjointIO A) {
    extern __shared__ __align__(16) uint8_t s_traverse[];
    TraverseSmem& S = *reinterpret_cast<TraverseSmem*>(s_traverse);
    __shared__ float S_agg[kWarps][32][6];  // cotangents of lanes sharing an edge
    load_tables(V, S);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned long long total = V.ctrl->total;
    const uint32_t N = (uint32_t)(total < A.count ? total : A.count);
    const uint32_t VW = 32u * item_rounds(N, gridDim.x);
    const uint32_t nchunks = (N + VW - 1) / VW;
    set_volume(V, S.warp[warp], lane);
    AdjointVertices<FT, MODE> p{A, S_agg[warp], V.vertex_base, N};
    for (uint32_t chunk = next_chunk(V, lane); chunk < nchunks; chunk = next_chunk(V, lane))
        walk_range(V, S, S.warp[warp], lane, chunk * VW, min(N, (chunk + 1u) * VW), N, p);
    finish_queue(V);
}

// ---------------------------------------------------------------------------
// Batched traversal: one persistent grid over the work items of every volume
// (chunk_start, written by the batched reduction).  A warp that takes an item
// of another volume copies that volume's descriptor into its own shared slot;
// the descriptors have top_cached = 0, so the descent reads the dense levels
// through L1 instead of a per-CTA cache.
template <int FT, int MODE>
__global__ void __launch_bounds__(kThreads, kTraverseCtas) traverse_batch(const __grid_constant__ BatchDev Bt,
                                                                          const __grid_constant__ TraverseOut O) {
    // dynamic: TraverseSmem, then one volume descriptor per warp
    extern __shared__ __align__(16) uint8_t s_traverse[];
    TraverseSmem& S = *reinterpret_cast<TraverseSmem*>(s_traverse);
    load_base_tables(S);
    __syncthreads();
    if (Bt.host && blockIdx.x == 0) {
        // offsets and whether any status bit is set, for the host: from here the
        // writes across PCIe overlap the traversal (from the reduction they
        // would hold up its end by 2 us)
        uint32_t status = threadIdx.x == 0 ? __ldcg(&Bt.ctrl->status) : 0u;
        for (int v = (int)threadIdx.x; v <= Bt.nvol; v += kThreads) {
            Bt.host[2 + v] = __ldcg(Bt.vbase + v);
            if (v < Bt.nvol) status |= __ldcg(&Bt.vols[v].ctrl->status);
        }
        status = (uint32_t)__syncthreads_or((int)status);
        if (threadIdx.x == 0) Bt.host[0] = status;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t VW = 32u * (uint32_t)Bt.rounds;
    const uint32_t nitems = __ldcg(Bt.chunk_start + Bt.nvol);
    Volume* const s_vol = reinterpret_cast<Volume*>(s_traverse + sizeof(TraverseSmem) + warp * kVolumeHead);
    const Volume& V = *s_vol;
    int cur = -1;
    uint32_t c0 = 0, c1 = 0, N = 0;
    ExtractVertices<FT, MODE, NoUserField, false> p{O, 0ull};
    for (uint32_t item = next_chunk_batch(Bt, lane); item < nitems; item = next_chunk_batch(Bt, lane)) {
        if (cur < 0 || item < c0 || item >= c1) {
            const int v = find_segment(Bt.chunk_start, Bt.nvol, item);
            __syncwarp();
            copy_volume(s_vol, Bt.vols + v, lane, 32);
            __syncwarp();
            set_volume(V, S.warp[warp], lane);
            cur = v;
            c0 = __ldcg(Bt.chunk_start + v);
            c1 = __ldcg(Bt.chunk_start + v + 1);
            p.out = __ldcg(Bt.vbase + v);
            const unsigned long long total = __ldcg(&V.ctrl->total);
            const unsigned long long room = Bt.capacity > p.out ? Bt.capacity - p.out : 0ull;
            N = (uint32_t)(total < room ? total : room);
        }
        const uint32_t first = (item - c0) * VW;
        walk_range(V, S, S.warp[warp], lane, first, min(N, first + VW), N, p);
    }
    finish_queue_batch(Bt);
}

// ---------------------------------------------------------------------------
// Indexed (welded) output.  No counterpart in the reference, which emits
// triangle soup only.  Every soup vertex lies on a lattice edge (a, axis);
// welding keeps one vertex per edge, numbered in order of first occurrence
// in the soup, and an index per soup vertex (three per triangle, the soup's
// triangle order).
//   mesh_edges    traversal without geometry: lists every group's distinct
//                 edges with their first soup vertex in the group, and per soup
//                 vertex its edge; clears the table;
//   mesh_insert   open-addressing table key -> smallest soup index (atomicCAS
//                 on the key, atomicMin on the index), an edge's slot kept;
//   mesh_mark     one bit per soup vertex that is the first on its edge;
//   mesh_scan     exclusive scan of the bits = unique vertex numbers;
//   mesh_vertices per edge its number, and for the first one the geometry
//                 (bit-identical to the soup vertex's);
//   mesh_indices  per soup vertex its edge's number.
// The table sees a group's distinct edges, 0.4 per soup vertex, and is probed
// once for each (every soup vertex inserted and looked up: 99 us of kernels at
// 192^3 with 0.9 M soup vertices).  Bound by launches and atomics in L2.
__device__ __forceinline__ unsigned long long mesh_key(const int a[3], int axis) {
    return (unsigned long long)a[0] | ((unsigned long long)a[1] << 14) | ((unsigned long long)a[2] << 28) |
           ((unsigned long long)axis << 42);
}

constexpr unsigned long long kEmptyKey = ~0ull;

struct MeshEdges {
    const MeshIO& M;
    unsigned int* count;
    bool meta;

    __device__ __forceinline__ void run(const CellGroup& G) {
        unsigned long long* key = reinterpret_cast<unsigned long long*>(G.W.data[0]);
        uint32_t* first = reinterpret_cast<uint32_t*>(G.W.data[1]);
        uint32_t j0 = 0;
        if (G.lane == 0) j0 = atomicAdd(count, G.nedges);
        j0 = __shfl_sync(0xffffffffu, j0, 0);
        G.edges([&](uint32_t slot, const EdgeAt& E) {
            key[slot] = mesh_key(E.a, E.axis);
            first[slot] = 0xffffffffu;
        });
        const uint32_t n = G.last - G.first;
        for (uint32_t i = (uint32_t)G.lane; i < n; i += 32) {
            const uint32_t slot = G.W.slot[i];
            atomicMin(&first[slot], G.first + i);
            M.vertex[G.first + i] = j0 + slot;
        }
        if (meta) {
            uint32_t c0 = (uint32_t)__ffs((int)G.lanes) - 2u;
#pragma unroll 1
            for (uint32_t i0 = 0; i0 < n; i0 += 32) {
                const uint32_t i = i0 + (uint32_t)G.lane, starts = G.starts(i0);
                const int c = (int)((c0 + (uint32_t)__popc(starts & (0xffffffffu >> (31 - G.lane)))) & 31u);
                c0 += (uint32_t)__popc(starts);
                const uint32_t code = __shfl_sync(0xffffffffu, G.code, c);
                const uint32_t k = (G.first + i - __shfl_sync(0xffffffffu, G.start, c)) & 15u;
                if (i < n) M.meta[G.first + i] = (uint16_t)(code | (k << 8));
            }
        }
        __syncwarp();
        for (uint32_t i = (uint32_t)G.lane; i < G.nedges; i += 32) {
            if (j0 + i >= M.edges) break;
            M.keys[j0 + i] = key[i];
            M.first[j0 + i] = first[i];
        }
        __syncwarp();
    }
};

// The listed edges.
__device__ __forceinline__ uint32_t listed_edges(const MeshIO& M, const Ctrl* ctrl) {
    const uint32_t n = __ldcg(&ctrl->mesh_edges);
    return n < M.edges ? n : M.edges;
}

__global__ void __launch_bounds__(kThreads, kTraverseCtas) mesh_edges(const __grid_constant__ Volume V,
                                                                      const __grid_constant__ MeshIO M) {
    extern __shared__ __align__(16) uint8_t s_traverse[];
    TraverseSmem& S = *reinterpret_cast<TraverseSmem*>(s_traverse);
    load_tables(V, S);
    allow_next_grid();
    const uint32_t t0 = blockIdx.x * kThreads + threadIdx.x, nt = gridDim.x * kThreads;
    uint4* table = reinterpret_cast<uint4*>(M.table_keys);  // keys and, behind them, vals: a multiple of 16 bytes
    const size_t quads = 3 * ((size_t)M.table_mask + 1) / 4;
    for (size_t i = t0; i < quads; i += nt) table[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
    for (uint32_t i = t0; i < (M.count + 31u) / 32u; i += nt) M.bits[i] = 0u;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned long long total = V.ctrl->total;
    const uint32_t N = (uint32_t)(total < M.count ? total : M.count);
    const uint32_t VW = 32u * item_rounds(N, gridDim.x);
    const uint32_t nchunks = (N + VW - 1) / VW;
    set_volume(V, S.warp[warp], lane);
    MeshEdges p{M, &V.ctrl->mesh_edges, V.binary != 0};
    // one item per warp at most, by its number: the queue's two atomics per warp
    // on one address cost 4 us here (the extraction, whose CTAs start at
    // different times beside the reduction, is 2 % faster with its queue)
    for (uint32_t chunk = warp * gridDim.x + blockIdx.x; chunk < nchunks; chunk += kWarps * gridDim.x)
        walk_range(V, S, S.warp[warp], lane, chunk * VW, min(N, (chunk + 1u) * VW), N, p);
}

__device__ __forceinline__ uint32_t key_hash(unsigned long long k) {
    k ^= k >> 33;
    k *= 0xff51afd7ed558ccdull;
    k ^= k >> 33;
    return (uint32_t)k;
}

__global__ void __launch_bounds__(kThreads) mesh_insert(const __grid_constant__ MeshIO M, Ctrl* ctrl) {
    wait_prior_grid();
    allow_next_grid();
    const uint32_t n = listed_edges(M, ctrl);
    for (uint32_t j = blockIdx.x * kThreads + threadIdx.x; j < n; j += gridDim.x * kThreads) {
        if (M.first[j] >= M.count) {  // only vertices past the count lie on it
            M.place[j] = 0xffffffffu;
            continue;
        }
        const unsigned long long key = M.keys[j];
        uint32_t h = key_hash(key) & M.table_mask, place = 0xffffffffu;
        for (uint32_t probe = 0; probe <= M.table_mask; probe++) {  // the table has more slots than keys
            const unsigned long long prev = atomicCAS(&M.table_keys[h], kEmptyKey, key);
            if (prev == kEmptyKey || prev == key) {
                atomicMin(&M.table_vals[h], M.first[j]);
                place = h;
                break;
            }
            h = (h + 1u) & M.table_mask;
        }
        M.place[j] = place;
        if (place == 0xffffffffu) atomicOr(&ctrl->status, kStatusCapacity);
    }
}

__global__ void __launch_bounds__(kThreads) mesh_mark(const __grid_constant__ MeshIO M, Ctrl* ctrl) {
    wait_prior_grid();
    allow_next_grid();
    const uint32_t n = listed_edges(M, ctrl);
    for (uint32_t j = blockIdx.x * kThreads + threadIdx.x; j < n; j += gridDim.x * kThreads) {
        const uint32_t h = M.place[j], f = M.first[j];
        if (f < M.count && h <= M.table_mask && M.table_vals[h] == f) atomicOr(&M.bits[f >> 5], 1u << (f & 31u));
    }
}

constexpr int kScanItems = 8;                          // words of bits per thread
constexpr uint32_t kScanTile = kThreads * kScanItems;  // per CTA

// scan[w] = bits set before word w in its tile; the last CTA turns the tiles'
// sums into their exclusive scan and writes the number of unique vertices.
__global__ void __launch_bounds__(kThreads) mesh_scan(const __grid_constant__ MeshIO M, Ctrl* ctrl) {
    __shared__ uint32_t s_warp[kWarps];
    __shared__ int s_last;
    wait_prior_grid();
    allow_next_grid();
    const uint32_t words = (M.count + 31u) / 32u;
    const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto block_scan = [&](uint32_t x, uint32_t& total) {  // exclusive
        const uint32_t inc = warp_inclusive_scan(x, lane);
        if (lane == 31) s_warp[warp] = inc;
        __syncthreads();
        uint32_t off = 0;
        total = 0;
#pragma unroll
        for (int w = 0; w < kWarps; w++) {
            if (w < warp) off += s_warp[w];
            total += s_warp[w];
        }
        __syncthreads();
        return off + inc - x;
    };
    uint32_t f[kScanItems], sum = 0, total;
#pragma unroll
    for (int j = 0; j < kScanItems; j++) {
        f[j] = base + j < words ? (uint32_t)__popc(__ldcg(&M.bits[base + j])) : 0u;
        sum += f[j];
    }
    uint32_t run = block_scan(sum, total);
#pragma unroll
    for (int j = 0; j < kScanItems; j++) {
        if (base + j < words) M.scan[base + j] = run;
        run += f[j];
    }
    if (threadIdx.x == 0) {
        M.tile_sums[blockIdx.x] = total;
        __threadfence();
        s_last = atomicAdd(&ctrl->mesh_done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    uint32_t carry = 0;
    for (uint32_t b = 0; b < gridDim.x; b += kThreads) {
        const uint32_t i = b + threadIdx.x;
        const uint32_t off = block_scan(i < gridDim.x ? __ldcg(&M.tile_sums[i]) : 0u, total);
        if (i < gridDim.x) M.tile_sums[i] = carry + off;
        carry += total;
    }
    if (threadIdx.x == 0) {
        *M.unique = carry;
        ctrl->mesh_done = 0;
    }
}

template <int FT, int MODE>
__global__ void __launch_bounds__(kThreads) mesh_vertices(const __grid_constant__ Volume V,
                                                          const __grid_constant__ MeshIO M) {
    wait_prior_grid();
    allow_next_grid();
    const uint32_t n = listed_edges(M, V.ctrl);
    for (uint32_t j = blockIdx.x * kThreads + threadIdx.x; j < n; j += gridDim.x * kThreads) {
        const uint32_t h = M.place[j];
        if (h > M.table_mask) continue;  // not inserted
        const uint32_t f = M.table_vals[h], word = f >> 5;
        if (f >= M.count) continue;
        const uint32_t u = M.tile_sums[word / kScanTile] + M.scan[word] +
                           (uint32_t)__popc(M.bits[word] & ((1u << (f & 31u)) - 1u));
        M.place[j] = u;
        if (M.first[j] != f || u >= M.vcap) continue;
        const unsigned long long key = M.keys[j];
        float p[3], nn[3], t;
        edge_vertex<FT, MODE>(V, edge_at(V, (int)(key & 0x3fffu), (int)((key >> 14) & 0x3fffu), (int)((key >> 28) & 0x3fffu),
                                         (uint32_t)(key >> 42) << 3), p, nn, t);
        if (MODE == kModeBinary) {
            const uint16_t m = M.meta[f];
#pragma unroll
            for (int c = 0; c < 3; c++) nn[c] = g_binary_normals[3 * (16 * (m & 0xff) + ((m >> 8) & 15)) + c] * V.scale[c];
        }
        if (M.pos) M.pos[u] = make_float4(p[0], p[1], p[2], 1.0f);
        if (M.nrm) M.nrm[u] = make_float4(nn[0], nn[1], nn[2], 0.0f);
    }
}

__global__ void __launch_bounds__(kThreads) mesh_indices(const __grid_constant__ MeshIO M, Ctrl* ctrl) {
    wait_prior_grid();
    if (blockIdx.x == 0 && threadIdx.x == 0) ctrl->mesh_edges = 0;
    if (!M.indices) return;
    // (vertices past the total were not listed)
    const unsigned long long total = ctrl->total < M.count ? ctrl->total : M.count;
    const uint32_t n = (uint32_t)(M.icap < total ? M.icap : total);
    for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
        const uint32_t j = M.vertex[i];
        M.indices[i] = j < M.edges ? M.place[j] : 0xffffffffu;
    }
}

template <int FT>
static cudaError_t launch_mesh_vertices(const Volume& V, const MeshIO& M, int mode, int grid, cudaStream_t st) {
    return mode == kModeBinary    ? launch_dependent(mesh_vertices<FT, kModeBinary>, grid, kThreads, 0, st, V, M)
           : mode == kModeCentral ? launch_dependent(mesh_vertices<FT, kModeCentral>, grid, kThreads, 0, st, V, M)
                                  : launch_dependent(mesh_vertices<FT, kModeForward>, grid, kThreads, 0, st, V, M);
}

cudaError_t launch_mesh(const Volume& V, const MeshIO& M, int normal_mode, int traverse_grid, int grid,
                        cudaStream_t st) {
    if (M.count == 0) return cudaSuccess;
    const int mode = V.binary ? kModeBinary : (normal_mode == kNormalsCentral ? kModeCentral : kModeForward);
    const unsigned int tiles = ((M.count + 31u) / 32u + kScanTile - 1) / kScanTile;
    cudaError_t e = launch_dependent(mesh_edges, traverse_grid, kThreads, kTraverseSmem, st, V, M);
    if (e == cudaSuccess) e = launch_dependent(mesh_insert, grid, kThreads, 0, st, M, V.ctrl);
    if (e == cudaSuccess) e = launch_dependent(mesh_mark, grid, kThreads, 0, st, M, V.ctrl);
    if (e == cudaSuccess) e = launch_dependent(mesh_scan, tiles, kThreads, 0, st, M, V.ctrl);
    if (e == cudaSuccess) {
        switch (V.ftype) {
            case kFieldF32: e = launch_mesh_vertices<kFieldF32>(V, M, mode, grid, st); break;
            case kFieldU8: e = launch_mesh_vertices<kFieldU8>(V, M, mode, grid, st); break;
            case kFieldUNorm8: e = launch_mesh_vertices<kFieldUNorm8>(V, M, mode, grid, st); break;
            case kFieldFunctor: e = launch_mesh_vertices<kFieldFunctor>(V, M, mode, grid, st); break;
            case kFieldF32X4: e = launch_mesh_vertices<kFieldF32X4>(V, M, mode, grid, st); break;
            default: return cudaErrorInvalidValue;
        }
    }
    if (e == cudaSuccess) e = launch_dependent(mesh_indices, grid, kThreads, 0, st, M, V.ctrl);
    return e;
}

// ---------------------------------------------------------------------------
cudaError_t launch_traverse(const Volume& V, const TraverseOut& O, int normal_mode, int grid,
                            cudaStream_t st) {
    const int mode = V.binary ? kModeBinary : (normal_mode == kNormalsCentral ? kModeCentral : kModeForward);
    const bool extra = O.feedback || O.dbg_cell || O.dbg_t;
#define HPMC_TRAVERSE_LAUNCH(FT_, MODE_)                                                 \
    return extra ? launch_traverse_kernel<FT_, MODE_, NoUserField, true>(V, O, grid, st) \
                 : launch_traverse_kernel<FT_, MODE_, NoUserField, false>(V, O, grid, st);
#define HPMC_TRAVERSE_CASE(FT_)                                             \
    case FT_:                                                               \
        if (mode == kModeBinary) HPMC_TRAVERSE_LAUNCH(FT_, kModeBinary)     \
        if (mode == kModeCentral) HPMC_TRAVERSE_LAUNCH(FT_, kModeCentral)   \
        HPMC_TRAVERSE_LAUNCH(FT_, kModeForward)
    switch (V.ftype) {
        HPMC_TRAVERSE_CASE(kFieldF32)
        HPMC_TRAVERSE_CASE(kFieldU8)
        HPMC_TRAVERSE_CASE(kFieldUNorm8)
        HPMC_TRAVERSE_CASE(kFieldFunctor)
        HPMC_TRAVERSE_CASE(kFieldF32X4)
        default: return cudaErrorInvalidValue;
    }
#undef HPMC_TRAVERSE_CASE
#undef HPMC_TRAVERSE_LAUNCH
}

template <int FT, int MODE>
static cudaError_t launch_adjoint_kernel(const Volume& V, const AdjointIO& A, int grid, cudaStream_t st) {
    adjoint_kernel<FT, MODE><<<grid, kThreads, kTraverseSmem, st>>>(V, A);
    return cudaGetLastError();
}

cudaError_t launch_adjoint(const Volume& V, const AdjointIO& A, int normal_mode, int grid, cudaStream_t st) {
    const bool central = normal_mode == kNormalsCentral;
    switch (V.ftype) {
        case kFieldF32:
            return central ? launch_adjoint_kernel<kFieldF32, kModeCentral>(V, A, grid, st)
                           : launch_adjoint_kernel<kFieldF32, kModeForward>(V, A, grid, st);
        case kFieldU8:
            return central ? launch_adjoint_kernel<kFieldU8, kModeCentral>(V, A, grid, st)
                           : launch_adjoint_kernel<kFieldU8, kModeForward>(V, A, grid, st);
        case kFieldUNorm8:
            return central ? launch_adjoint_kernel<kFieldUNorm8, kModeCentral>(V, A, grid, st)
                           : launch_adjoint_kernel<kFieldUNorm8, kModeForward>(V, A, grid, st);
        default:
            return cudaErrorInvalidValue;
    }
}

template <int FT, int MODE>
static cudaError_t launch_batch_kernel(const BatchDev& B, const TraverseOut& O, int grid, cudaStream_t st) {
    traverse_batch<FT, MODE><<<grid, kThreads, kBatchSmem, st>>>(B, O);
    return cudaGetLastError();
}

cudaError_t launch_traverse_batch(const BatchDev& B, const TraverseOut& O, int ftype, int normal_mode, int grid,
                                  cudaStream_t st) {
    const bool central = normal_mode == kNormalsCentral;
    switch (ftype) {
        case kFieldF32:
            return central ? launch_batch_kernel<kFieldF32, kModeCentral>(B, O, grid, st)
                           : launch_batch_kernel<kFieldF32, kModeForward>(B, O, grid, st);
        case kFieldU8:
            return central ? launch_batch_kernel<kFieldU8, kModeCentral>(B, O, grid, st)
                           : launch_batch_kernel<kFieldU8, kModeForward>(B, O, grid, st);
        case kFieldUNorm8:
            return central ? launch_batch_kernel<kFieldUNorm8, kModeCentral>(B, O, grid, st)
                           : launch_batch_kernel<kFieldUNorm8, kModeForward>(B, O, grid, st);
        default:
            return cudaErrorInvalidValue;
    }
}

// Resident CTAs per SM of one kernel with `bytes` of dynamic shared memory.
template <class K>
static int resident_ctas(K* kernel, size_t bytes) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kThreads, bytes) != cudaSuccess || n < 1)
        n = 1;
    return n;
}

int traverse_batch_blocks_per_sm() { return resident_ctas(traverse_batch<kFieldF32, kModeCentral>, kBatchSmem); }

int traverse_blocks_per_sm() {
    return resident_ctas(traverse_kernel<kFieldF32, kModeCentral, NoUserField, false>, kTraverseSmem);
}

}  // namespace hpmc
