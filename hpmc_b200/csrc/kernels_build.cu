// kernels_build.cu -- HistoPyramid build on sm_100a: classification fused
// with the first five reductions, then the upper reductions.
//
// Reference passes replaced (hpmc/src/buildpass.cpp:42-178):
//   base level  (shadergen.cpp:86-171)  -> classify_columns / classify_blocks
//   first reduction + 4 upper levels    -> fused into classification (a 32x32
//                                          cell block = 4^5 keys is summed in
//                                          registers and warp reductions)
//   remaining upper reductions          -> reduce_levels (one launch,
//                                          last-block-done chaining)
//   top readback (buildpass.cpp:161-168)-> Ctrl::total in device memory
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>

#include "hpmc_batch.cuh"
#include "hpmc_device.cuh"
#include "hpmc_fetch.cuh"
#include "hpmc_kernels.h"
#include "hpmc_tma.cuh"
#include "hpmc_column_core.cuh"

namespace hpmc {

// ---------------------------------------------------------------------------
// TMA column classification (hpmc_column_core.cuh has the classification of a
// box): a column's boxes stream through a TMA ring (each sample leaves HBM
// once; halo rows/columns are shared with neighbouring columns through L2).
// The single-volume kernel is persistent (columns from a device queue); the
// batched one takes one column brick per CTA.
template <int FT>
struct ColumnGeom {
    using T = typename std::conditional<FT == kFieldF32, float, uint8_t>::type;
    static constexpr int BXE = (FT == kFieldF32) ? 36 : 48;  // box width (16-byte multiple)
    static constexpr int LAYER = BXE * 33;                    // elements of one sample layer
    static constexpr int STAGE_BYTES = LAYER * kLayersPerBox * (int)sizeof(T);
    static constexpr int STAGE_STRIDE = (STAGE_BYTES + 127) & ~127;
};

struct ColumnSmem {
    ColumnBits bits;
    uint64_t bar[kRingStages];
};

// Bit rows of the nl layers of one box (ring stage st).
template <int FT>
__device__ __forceinline__ void convert_box(const typename ColumnGeom<FT>::T* st, int nl, uint32_t gl0, float iso,
                                            int u8_thr, int warp, int lane, ColumnBits& C) {
    using G = ColumnGeom<FT>;
    // Every sample first, then the ballots and stores: the compiler cannot
    // tell the bit-row stores from the ring stage, so loads issued after a
    // store would wait for it.  A stage always holds kLayersPerBox layers
    // (copies past the volume read zeros), so all of them are read; layers
    // past nl are not stored.
    BoxSamples<typename G::T> s;
    const typename G::T* row = st + 4 * warp * G::BXE + lane;
#pragma unroll
    for (int l = 0; l < kLayersPerBox; l++)
#pragma unroll
        for (int i = 0; i < 4; i++) s.v[l][i] = row[l * G::LAYER + i * G::BXE];
    const int le = edge_layer(gl0, warp);
    const typename G::T* layer = st + (le < kLayersPerBox ? le : 0) * G::LAYER;  // inside the stage for any box depth
    s.row = layer[32 * G::BXE + lane];
    s.col = layer[lane * G::BXE + 32];
    s.corner = layer[32 * G::BXE + 32];
    box_bits(s, nl, gl0, iso, u8_thr, warp, lane, C);
}

template <int FT>
__device__ __forceinline__ uint8_t* ring_base() {
    extern __shared__ __align__(128) uint8_t s_dyn[];
    // TMA destinations must be 128-byte aligned: align the ring explicitly
    // (the launch reserves 128 spare bytes)
    return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(s_dyn) + 127) & ~uintptr_t(127));
}

// Issues box k of the column at (x0, y0, z0) into its ring stage (one thread).
template <int FT>
__device__ __forceinline__ void issue_box(uint8_t* ring, uint64_t* bar, const CUtensorMap* tmap, int x0, int y0, int z0,
                                          int k, uint64_t pol) {
    using G = ColumnGeom<FT>;
    const int s = k % kRingStages;
    mbar_arrive_expect_tx(&bar[s], G::STAGE_BYTES);
    tma_load_3d(ring + s * G::STAGE_STRIDE, tmap, x0, y0, z0 + k * kLayersPerBox, &bar[s], pol);
}

// Column CTA body (one column per CTA): footprint (fx, fy) of the slice tiles,
// `slices` slices from z0 on, field boxes from `tmap`; the first kRingStages
// boxes are on their way, the tables filled.  stall: the box that never arrives
// (-1: none).
template <int FT>
__device__ __forceinline__ void classify_column_body(const CUtensorMap* tmap, const Volume& V, int fx, int fy, int z0,
                                                     int slices, int stall, uint64_t pol, uint8_t* s_ring,
                                                     ColumnSmem& C) {
    using G = ColumnGeom<FT>;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int x0 = fx * 32, y0 = fy * 32;
    const int nlayers = slices + 1;
    const int nbox = (nlayers + kLayersPerBox - 1) / kLayersPerBox;
    const float iso = V.binary ? 0.5f : V.iso;
    const int u8_thr = V.u8_thr;
    const uint32_t fm = footprint_morton(fx, fy);
    const uint32_t vmask = row_mask(V, x0, y0, lane);
    const bool full = __all_sync(0xffffffffu, vmask == 0xffffffffu);

    bool timed_out = false;
    int k = 0;
    for (; k < nbox; k++) {
        const int s = k % kRingStages;
        const uint32_t parity = (uint32_t)(k / kRingStages) & 1u;
        const int lb = k * kLayersPerBox;
        const int nl = min(kLayersPerBox, nlayers - lb);
        // every warp waits on the box's mbarrier (suspended in hardware, not spinning)
        if (!mbar_wait_bounded(&C.bar[s], parity, V.wait_limit_ns, &V.ctrl->status, kStatusTimeout)) timed_out = true;
        if (!timed_out)
            convert_box<FT>(reinterpret_cast<const typename G::T*>(s_ring + s * G::STAGE_STRIDE), nl, (uint32_t)lb,
                            iso, u8_thr, warp, lane, C.bits);
        // the only CTA barrier of a box: stage s consumed, bit rows of layers
        // lb .. lb+nl-1 ready, and a uniform decision on a timed-out wait
        if (__syncthreads_or(timed_out)) break;
        if (tid == 0 && k + kRingStages < nbox && k + kRingStages != stall)
            issue_box<FT>(s_ring, C.bar, tmap, x0, y0, z0, k + kRingStages, pol);
        classify_box_slices(V, z0, fx, fy, fm, lb, nl, 0u, warp, lane, vmask, full, C.bits);
    }
    if (timed_out) {
        // drain the boxes still in flight (bounded) before the CTA exits
        if (tid == 0) {
            for (int l = k; l < nbox && l < k + kRingStages; l++)
                mbar_wait_bounded(&C.bar[l % kRingStages], (uint32_t)(l / kRingStages) & 1u, V.wait_limit_ns,
                                  nullptr, 0u);
            atomicOr(&V.ctrl->status, kStatusTimeout);
        }
    }
}

// Persistent column classifier (column = footprint (fx, fy) x one run of
// column_slices slices, numbered footprint-fastest so that neighbouring
// columns share halo samples in L2).  Thread 0 claims columns from a device
// queue (one atomic per column: a CTA whose columns end early takes more) and
// streams their boxes back to back through the ring, tagging every stage with
// its column and box, so the copy engine never idles between columns; after
// the last column it arrives on the next stage without a copy, tagged -1.
// The last CTA to finish resets the queue for the next launch.
template <int FT>
__global__ void __launch_bounds__(kThreads) classify_columns(const __grid_constant__ CUtensorMap tmap,
                                                             const __grid_constant__ Volume V, int ncolumns) {
    using G = ColumnGeom<FT>;
    uint8_t* const s_ring = ring_base<FT>();
    __shared__ __align__(16) ColumnSmem C;
    // per ring stage: box k | layers << 16 of its column (-1: end), footprint
    // fx | fy << 16, first slice and the footprint's Morton part -- decoded
    // once by the producer, so that the consumers start converting without
    // integer divisions after each wait
    __shared__ int4 s_tag[kRingStages];
    // per ring stage: the column's x mask and valid rows (bit 31: every row
    // valid and the mask full), so a lane's row mask is one compare
    __shared__ uint2 s_rowmask[kRingStages];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int per_slab = V.nfx * V.nfy;
    const float iso = V.binary ? 0.5f : V.iso;
    const int u8_thr = V.u8_thr;
    // column u -> footprint, first slice, layers (slices + 1)
    auto column = [&](int u, int& fx, int& fy, int& z0, int& nlayers) {
        const int zc = u / per_slab;
        const int r = u - zc * per_slab;
        fy = r / V.nfx;
        fx = r - fy * V.nfx;
        z0 = zc * V.column_slices;
        nlayers = min(V.cells[2], z0 + V.column_slices) - z0 + 1;
    };

    __shared__ int s_early;
    fill_column_tables(V, C.bits, 0, V.cells[2]);
    if (tid == 0) {
        for (int s = 0; s < kRingStages; s++) mbar_init(&C.bar[s], 1);
        mbar_fence_init();
        // The previous grid may still be this pyramid's extraction (its
        // flag is set before it lets this launch begin and cleared by its
        // last CTA): then this CTA streams at once and waits at its end.  A
        // CTA that sees the flag clear takes the ordinary path; a stale clear
        // flag only costs the overlap.
        s_early = V.overlap && *reinterpret_cast<volatile unsigned int*>(&V.ctrl->extracting) != 0u;
    }
    __syncthreads();
    const bool early = s_early != 0;
    // Otherwise global memory (field, pyramid, control block) only after the
    // previous grid.  No early trigger: the reduce launches as these CTAs
    // exit (reduce CTAs resident and waiting through the whole build measured
    // ~2% slower).
    if (!early) wait_prior_grid();
    // producer state (thread 0): next box to issue = box pk of column pu; the
    // following column is claimed one column ahead (pnext), so the atomic's
    // round trip overlaps the current column
    int pu = -1, pk = 0, pnl = 0, pz0 = 0, pfx = 0, pfy = 0, pnext = -1;
    const uint64_t pol = l2_evict_first_policy();  // the field is read once
    bool pdone = false;
    uint32_t issued = 0;
    if (tid == 0) pnext = (int)atomicAdd(&V.ctrl->col_next, 1u);
    auto issue_next = [&]() {
        if (pdone) return;
        const int s = (int)(issued % kRingStages);
        if (pu < 0 || pk * kLayersPerBox >= pnl) {
            pu = pnext;
            if (pu < ncolumns) pnext = (int)atomicAdd(&V.ctrl->col_next, 1u);
            pk = 0;
            if (pu >= ncolumns) {
                s_tag[s] = make_int4(-1, 0, 0, 0);
                mbar_arrive(&C.bar[s]);  // completes the phase: the consumers see the end tag
                issued++;
                pdone = true;
                return;
            }
            column(pu, pfx, pfy, pz0, pnl);
        }
        s_tag[s] = make_int4(pk | (pnl << 16), pfx | (pfy << 16), pz0, (int)footprint_morton(pfx, pfy));
        {
            const int xv = V.cells[0] - pfx * 32, yv = V.cells[1] - pfy * 32;
            const uint32_t xm = xv >= 32 ? 0xffffffffu : ((1u << xv) - 1u);
            const uint32_t rows = (uint32_t)min(yv, 32);
            s_rowmask[s] = make_uint2(xm, rows | ((xm == 0xffffffffu && rows == 32u) ? 0x80000000u : 0u));
        }
        // test hook: a CTA never issues its box stall_box (its waits run out)
        if ((int)issued != V.stall_box) {
            mbar_arrive_expect_tx(&C.bar[s], G::STAGE_BYTES);
            tma_load_3d(s_ring + s * G::STAGE_STRIDE, &tmap, pfx * 32, pfy * 32, pz0 + pk * kLayersPerBox, &C.bar[s],
                        pol);
        }
        issued++;
        pk++;
    };
    if (tid == 0)
        for (int i = 0; i < kRingStages; i++) issue_next();

    bool timed_out = false;
    uint32_t pos = 0;  // running box position (ring slot, phase, row-buffer index)
    for (;; pos++) {
        const int s = (int)(pos % kRingStages);
        const uint32_t parity = (pos / kRingStages) & 1u;
        const bool ok = mbar_wait_bounded(&C.bar[s], parity, V.wait_limit_ns, &V.ctrl->status, kStatusTimeout);
        // the stage's tag was written before the producer's arrival (release) on its barrier
        const int4 tag = ok ? s_tag[s] : make_int4(-1, 0, 0, 0);
        const uint2 rm = ok ? s_rowmask[s] : make_uint2(0u, 0u);  // read before the producer refills stage s
        const int fx = tag.y & 0xffff, fy = tag.y >> 16, z0 = tag.z;
        const uint32_t fm = (uint32_t)tag.w;
        const int k = tag.x & 0xffff, nlayers = tag.x >> 16;
        const int lb = k * kLayersPerBox;
        const int nl = min(kLayersPerBox, nlayers - lb);
        if (ok && tag.x >= 0)
            convert_box<FT>(reinterpret_cast<const typename G::T*>(s_ring + s * G::STAGE_STRIDE), nl,
                            pos * kLayersPerBox, iso, u8_thr, warp, lane, C.bits);
        // the only CTA barrier of a box (uniform decision on a timed-out wait);
        // the producer rewrites the stage and its tag only after it
        if (__syncthreads_or(!ok)) {
            timed_out = true;
            break;
        }
        if (tag.x < 0) break;        // the end tag (the same for every thread)
        if (tid == 0) issue_next();  // refill stage s
        const uint32_t vmask = (uint32_t)lane < (rm.y & 0xffu) ? rm.x : 0u;  // == row_mask(V, 32 fx, 32 fy, lane)
        const bool full = (rm.y >> 31) != 0u;
        classify_box_slices(V, z0, fx, fy, fm, lb, nl, (pos - (uint32_t)k) * kLayersPerBox, warp, lane, vmask, full,
                            C.bits);
    }
    if (timed_out && tid == 0) {
        // drain the boxes still in flight (bounded) before the CTA exits
        for (uint32_t p = pos; p < issued; p++)
            mbar_wait_bounded(&C.bar[p % kRingStages], (p / kRingStages) & 1u, V.wait_limit_ns, nullptr, 0u);
        atomicOr(&V.ctrl->status, kStatusTimeout);
    }
    // an early CTA ends only after the extraction it overlapped, so the
    // reduce (and all later work) still follows every earlier grid
    if (early) wait_prior_grid();
    // the last CTA to finish resets the column queue for the next launch
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(&V.ctrl->col_done, 1u) == gridDim.x - 1) {
            V.ctrl->col_next = 0;
            V.ctrl->col_done = 0;
            __threadfence();
        }
    }
}


// ---------------------------------------------------------------------------
// Upper reductions (shadergen.cpp:174-225 without the floor filter): level
// j+1 entry e = sum of level j entries 4e..4e+3.  CTA c reduces 1024 entries
// of level j_in (5 levels: registers, shuffles and one shared-memory
// exchange); the last CTA to finish carries on from those partial tops to
// level j_stop.  The top entry is the vertex count (hpiface.cpp:323-327).
// Level-5 entries of padding blocks (footprints past the grid) are zero: the
// levels are cleared when they are set up and only the generic classifier
// writes those entries, with zero.
constexpr int kReduceChunk = 1024;  // level entries per CTA (5 levels)
constexpr int kReduceTop = 4096;    // entries the last CTA can finish (6 levels)


__device__ void reduce_tree(const Volume& V, uint32_t* buf0, uint32_t* buf1, int& j, int j_stop, long long n,
                            long long out_base, bool& overflow) {
    // buf0 holds n entries of level j (n a power of 4); out_base = index of the
    // first entry of level j in this chunk.  Leaves the last level in buf0.
    uint32_t* src = buf0;
    uint32_t* dst = buf1;
    while (j < j_stop && n >= 4) {
        n >>= 2;
        out_base >>= 2;
        j++;
        for (long long i = threadIdx.x; i < n; i += blockDim.x) {
            const unsigned long long s =
                (unsigned long long)src[4 * i] + src[4 * i + 1] + src[4 * i + 2] + src[4 * i + 3];
            if (s > 0xffffffffull) overflow = true;
            dst[i] = (uint32_t)s;
            V.levels[V.level_off[j] + out_base + i] = (uint32_t)s;
        }
        __syncthreads();
        uint32_t* t = src;
        src = dst;
        dst = t;
    }
    if (src != buf0) {
        for (long long i = threadIdx.x; i < n; i += blockDim.x) buf0[i] = src[i];
        __syncthreads();
    }
}

// The vertex count (one thread), after every status bit of the build.
__device__ __forceinline__ void write_total(const Volume& V, uint32_t total) {
    V.ctrl->total = total;
    if (V.host) {
        V.host->total = total;
        V.host->status = __ldcg(&V.ctrl->status);
    }
}

// One chunk of kReduceChunk level-j_in entries (chunk `chunk` of `nchunks`).
// Returns true in the CTA that wrote the vertex count (level jtop reached).
__device__ __forceinline__ bool reduce_chunk(const Volume& V, int j_in, int j_stop, long long chunk, unsigned int nchunks, uint32_t* buf0, uint32_t* buf1,
                                             int* s_last) {
    bool overflow = false;
    const long long n_in = level_entries(V.size_l2, j_in);
    const long long base = chunk * kReduceChunk;
    const long long n = min((long long)kReduceChunk, n_in - base);  // a power of 4 (>= 4), or 1 at the top
    const int t = threadIdx.x;
    int j = j_in;
    if (n == kReduceChunk && j_stop - j_in >= 5) {
        // a full chunk, five levels without shared-memory round trips: thread
        // t's four entries make level j+1 entry t, groups of 4 and 16 lanes
        // (shuffles) levels j+2 and j+3, pairs of warps and then all eight
        // (one exchange) levels j+4 and j+5.  A chunk's sums stay below 2^32
        // (1024 entries of at most 15 * 1024 vertices each).
        const uint4 v = *reinterpret_cast<const uint4*>(V.levels + V.level_off[j_in] + base + 4 * t);
        uint32_t a = v.x + v.y + v.z + v.w;
        V.levels[V.level_off[j_in + 1] + (base >> 2) + t] = a;
        a += __shfl_xor_sync(0xffffffffu, a, 1);
        a += __shfl_xor_sync(0xffffffffu, a, 2);
        if ((t & 3) == 0) V.levels[V.level_off[j_in + 2] + (base >> 4) + (t >> 2)] = a;
        a += __shfl_xor_sync(0xffffffffu, a, 4);
        a += __shfl_xor_sync(0xffffffffu, a, 8);
        if ((t & 15) == 0) V.levels[V.level_off[j_in + 3] + (base >> 6) + (t >> 4)] = a;
        a += __shfl_xor_sync(0xffffffffu, a, 16);
        if ((t & 31) == 0) buf1[t >> 5] = a;  // the warps' sums
        __syncthreads();
        if (t < kWarps / 2) {
            const uint32_t p = buf1[2 * t] + buf1[2 * t + 1];
            V.levels[V.level_off[j_in + 4] + (base >> 8) + t] = p;
            buf1[kWarps + t] = p;
        }
        __syncthreads();
        if (t == 0) {
            const uint32_t c = buf1[kWarps] + buf1[kWarps + 1] + buf1[kWarps + 2] + buf1[kWarps + 3];
            V.levels[V.level_off[j_in + 5] + (base >> 10)] = c;
            buf0[0] = c;
        }
        __syncthreads();
        j = j_in + 5;
    } else {
        if (4 * t < n)
            *reinterpret_cast<uint4*>(&buf0[4 * t]) =
                *reinterpret_cast<const uint4*>(V.levels + V.level_off[j_in] + base + 4 * t);
        __syncthreads();
        reduce_tree(V, buf0, buf1, j, j_stop, n, base, overflow);
    }
    if (j < j_stop) {
        // levels remain above this chunk's top: the last CTA to finish continues
        if (overflow) atomicOr(&V.ctrl->status, kStatusOverflow);
        __threadfence();
        if (threadIdx.x == 0) *s_last = (atomicAdd(&V.ctrl->reduce_done, 1u) == nchunks - 1);
        __syncthreads();
        if (!*s_last) return false;
        __threadfence();
        const long long m = level_entries(V.size_l2, j);  // == nchunks entries, <= kReduceTop
        for (long long i = threadIdx.x; i < m; i += blockDim.x) buf0[i] = __ldcg(&V.levels[V.level_off[j] + i]);
        __syncthreads();
        reduce_tree(V, buf0, buf1, j, j_stop, m, 0, overflow);
        if (threadIdx.x == 0) V.ctrl->reduce_done = 0;
    }
    if (overflow) atomicOr(&V.ctrl->status, kStatusOverflow);
    if (j == V.jtop) {
        __syncthreads();
        if (threadIdx.x == 0) write_total(V, buf0[0]);
    }
    return j == V.jtop;
}

__global__ void __launch_bounds__(kThreads) reduce_levels(const __grid_constant__ Volume V, int j_in, int j_stop) {
    __shared__ __align__(16) uint32_t buf0[kReduceTop];
    __shared__ uint32_t buf1[kReduceTop / 4];
    __shared__ int s_last;
    wait_prior_grid();
    allow_next_grid();
    reduce_chunk(V, j_in, j_stop, blockIdx.x, gridDim.x, buf0, buf1, &s_last);
}

// Top entry when the whole pyramid is one block (no reduction launch needed).
__global__ void copy_total(const __grid_constant__ Volume V) {
    wait_prior_grid();
    allow_next_grid();
    if (threadIdx.x == 0) write_total(V, V.levels[V.level_off[V.jtop]]);
}

// ---------------------------------------------------------------------------
// Batched build.  One classify launch covers the column bricks of every volume
// with a tensor map (CTA = one brick), one the bricks of the others; one
// reduce launch covers the reduction chunks of every volume (each volume's
// pyramid finished by its own last CTA), and the CTA that completes the last
// volume scans the per-volume counts into output offsets and traversal work
// items.  Volume descriptors are copied into shared memory per CTA.
//
// A brick's descriptor says all that its first boxes need, so they are on their
// way before the CTA fetches the volume's descriptor and fills its tables.
// Finding the volume by bisection and the brick's place by divisions came first
// once: kernel for 64 volumes of 335 MB 125 -> 115 us, for the 36 aligned bricks
// of a ragged batch 7.4 -> 5.3.  Issue-bound (the slices with vertices).
template <int FT>
__global__ void __launch_bounds__(kThreads) classify_batch_tma(const __grid_constant__ BatchDev B) {
    uint8_t* const s_ring = ring_base<FT>();
    __shared__ __align__(16) Volume sV;
    __shared__ __align__(16) ColumnSmem C;
    const uint2 brick = __ldg(B.bricks + blockIdx.x);
    const int v = (int)(brick.x & 0xfffffu), slices = (int)(brick.x >> 20);
    const int fx = (int)(brick.y & 511u), fy = (int)((brick.y >> 9) & 511u), zc = (int)(brick.y >> 18);
    const int z0 = zc * B.column_slices;
    // test hook: the first column of a volume never receives box stall_box
    const int stall = (v == B.stall_volume && fx == 0 && fy == 0 && zc == 0) ? B.stall_box : -1;
    const uint64_t pol = l2_evict_first_policy();  // the field is read once
    if (threadIdx.x == 0) {
        for (int s = 0; s < kRingStages; s++) mbar_init(&C.bar[s], 1);
        mbar_fence_init();
        for (int k = 0; k < kRingStages && k * kLayersPerBox <= slices; k++)
            if (k != stall) issue_box<FT>(s_ring, C.bar, B.tmaps + v, fx * 32, fy * 32, z0, k, pol);
    }
    copy_volume(&sV, B.vols + v, threadIdx.x, blockDim.x);
    __syncthreads();
    fill_column_tables(sV, C.bits, z0, z0 + slices);
    __syncthreads();
    classify_column_body<FT>(B.tmaps + v, sV, fx, fy, z0, slices, stall, pol, s_ring, C);
}

// The bricks of the volumes without a tensor map, one per CTA: columns (direct
// classifier) or, for narrow tiles, 32x32 blocks.  One launch for all of them:
// a launch per volume leaves the GPU nearly empty for about 5 us each (24 byte
// volumes of edge 20..120: 23 launches, 128 us in all; this one 15 us).
template <int FT>
__global__ void __launch_bounds__(kThreads, kDirectCtas) classify_batch_direct(const __grid_constant__ BatchDev B) {
    __shared__ __align__(16) Volume sV;
    __shared__ __align__(16) ColumnBits C;
    __shared__ uint32_t s_warp[kWarps];
    const uint2 brick = __ldg(B.direct_bricks + blockIdx.x);  // volume, its column or block
    copy_volume(&sV, B.vols + brick.x, threadIdx.x, blockDim.x);
    C.cnt[threadIdx.x] = c_vertex_count[threadIdx.x];
    __syncthreads();
    const uint32_t u = brick.y;
    if (sV.column_layout) classify_column_direct<FT, NoUserField, false>(sV, (int)u, C);
    else classify_block_body<FT>(sV, u, C.cnt, s_warp);
}

namespace {

// Block-wide exclusive scan (kThreads threads); `total` receives the sum.
template <typename T>
__device__ __forceinline__ T block_exclusive_scan(T x, T* s_warp, T& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T inc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    T off = 0, tot = 0;
#pragma unroll
    for (int w = 0; w < kWarps; w++) {
        const T s = s_warp[w];
        if (w < warp) off += s;
        tot += s;
    }
    __syncthreads();
    total = tot;
    return off + inc - x;
}

// Output offsets (exclusive scan of the vertex counts) and traversal work
// items (vertices that fit the output, in items of 32 * rounds).
__device__ void batch_scan(const BatchDev& B) {
    __shared__ unsigned long long s_w64[kWarps];
    __shared__ uint32_t s_w32[kWarps];
    const uint32_t VW = 32u * (uint32_t)B.rounds;
    unsigned long long carry = 0;
    uint32_t ccarry = 0;
    for (int base = 0; base < B.nvol; base += kThreads) {
        const int v = base + (int)threadIdx.x;
        unsigned long long tot = 0;
        if (v < B.nvol) {
            const Ctrl* c = B.vols[v].ctrl;
            tot = __ldcg(&c->total);
        }
        unsigned long long sum64;
        const unsigned long long vb = carry + block_exclusive_scan<unsigned long long>(tot, s_w64, sum64);
        const unsigned long long room = B.capacity > vb ? B.capacity - vb : 0ull;
        const unsigned long long nw = tot < room ? tot : room;
        const uint32_t items = (uint32_t)((nw + VW - 1) / VW);
        uint32_t sum32;
        const uint32_t cs = ccarry + block_exclusive_scan<uint32_t>(items, s_w32, sum32);
        if (v < B.nvol) {
            B.vbase[v] = vb;
            B.chunk_start[v] = cs;
        }
        carry += sum64;
        ccarry += sum32;
    }
    if (threadIdx.x == 0) {
        B.vbase[B.nvol] = carry;
        B.chunk_start[B.nvol] = ccarry;
        B.ctrl->total = carry;
        if (carry > B.capacity) atomicOr(&B.ctrl->status, kStatusCapacity);
        B.ctrl->reduce_done = 0;
        __threadfence();
    }
}

}  // namespace

__global__ void __launch_bounds__(kThreads) reduce_batch(const __grid_constant__ BatchDev B) {
    __shared__ __align__(16) uint32_t buf0[kReduceTop];
    __shared__ uint32_t buf1[kReduceTop / 4];
    __shared__ __align__(16) Volume sV;
    __shared__ int s_last, s_all;
    const int v = find_segment(B.reduce_start, B.nvol, blockIdx.x);
    copy_volume(&sV, B.vols + v, threadIdx.x, blockDim.x);
    __syncthreads();
    const uint32_t c0 = __ldg(B.reduce_start + v);
    const uint32_t nchunks = __ldg(B.reduce_start + v + 1) - c0;
    // every batch volume reaches its top in this launch (jtop - 5 <= 11)
    const bool finished =
        reduce_chunk(sV, kBlockLevel, sV.jtop, (long long)(blockIdx.x - c0), nchunks, buf0, buf1, &s_last);
    if (!finished) return;  // uniform across the CTA
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();  // this volume's total before the batch counter
        s_all = (atomicAdd(&B.ctrl->reduce_done, 1u) == (unsigned)B.nvol - 1u);
    }
    __syncthreads();
    if (s_all) {
        __threadfence();
        batch_scan(B);
    }
}

// ---------------------------------------------------------------------------
// Host launchers
constexpr int kRingBytesF32 = kRingStages * ((36 * 33 * 4 * kLayersPerBox + 127) & ~127) + 128;
constexpr int kRingBytesU8 = kRingStages * ((48 * 33 * kLayersPerBox + 127) & ~127) + 128;

// Resident column-classifier CTAs per SM (shared-memory bound).
static int column_ctas_per_sm() {
    static int n = 0;
    if (n == 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, classify_columns<kFieldF32>, kThreads,
                                                          kRingBytesF32) !=
                cudaSuccess ||
            n < 1)
            n = 1;
    }
    return n;
}

cudaError_t launch_classify(const Volume& V, const CUtensorMap* tmap, int max_ctas, cudaStream_t st) {
    if (V.column_layout && tmap) {
        const int ncolumns = column_count(V);
        // persistent: every resident CTA slot (max_ctas = 16 per SM)
        const int slots = (max_ctas / 16) * column_ctas_per_sm();
        const int grid = ncolumns < slots ? ncolumns : slots;
        if (V.ftype == kFieldF32)
            return launch_dependent(classify_columns<kFieldF32>, grid, kThreads, kRingBytesF32, st, *tmap, V, ncolumns);
        else if (V.ftype == kFieldU8)
            return launch_dependent(classify_columns<kFieldU8>, grid, kThreads, kRingBytesU8, st, *tmap, V, ncolumns);
        else
            return launch_dependent(classify_columns<kFieldUNorm8>, grid, kThreads, kRingBytesU8, st, *tmap, V,
                                    ncolumns);
    } else if (V.column_layout) {
        const int grid = column_count(V);
        switch (V.ftype) {
            case kFieldF32: return launch_dependent(classify_columns_direct<kFieldF32>, grid, kThreads, 0, st, V);
            case kFieldU8: return launch_dependent(classify_columns_direct<kFieldU8>, grid, kThreads, 0, st, V);
            case kFieldUNorm8: return launch_dependent(classify_columns_direct<kFieldUNorm8>, grid, kThreads, 0, st, V);
            case kFieldF32X4: return launch_dependent(classify_columns_direct<kFieldF32X4>, grid, kThreads, 0, st, V);
            default: return launch_dependent(classify_columns_direct<kFieldFunctor>, grid, kThreads, 0, st, V);
        }
    } else {
        const long long nb = V.nblocks;
        const int grid = (int)(nb < (long long)max_ctas ? nb : (long long)max_ctas);
        switch (V.ftype) {
            case kFieldF32: classify_blocks<kFieldF32><<<grid, kThreads, 0, st>>>(V); break;
            case kFieldU8: classify_blocks<kFieldU8><<<grid, kThreads, 0, st>>>(V); break;
            case kFieldUNorm8: classify_blocks<kFieldUNorm8><<<grid, kThreads, 0, st>>>(V); break;
            case kFieldF32X4: classify_blocks<kFieldF32X4><<<grid, kThreads, 0, st>>>(V); break;
            default: classify_blocks<kFieldFunctor><<<grid, kThreads, 0, st>>>(V); break;
        }
    }
    return cudaGetLastError();
}

cudaError_t launch_reduce(const Volume& V, cudaStream_t st) {
    if (V.jtop == kBlockLevel) return launch_dependent(copy_total, 1, 32, 0, st, V);
    int j_in = kBlockLevel;
    while (j_in < V.jtop) {
        // one launch reduces 5 levels per CTA plus up to 6 more in the last CTA
        const int j_stop = (V.jtop - j_in <= 11) ? V.jtop : j_in + 5;
        const long long n_in = level_entries(V.size_l2, j_in);
        const long long grid = (n_in + kReduceChunk - 1) / kReduceChunk;
        cudaError_t e = launch_dependent(reduce_levels, (unsigned)grid, kThreads, 0, st, V, j_in, j_stop);
        if (e != cudaSuccess) return e;
        j_in = j_stop;
    }
    return cudaSuccess;
}

cudaError_t launch_classify_batch(const BatchDev& B, int ftype, unsigned int bricks, cudaStream_t st) {
    if (!bricks) return cudaSuccess;
    if (ftype == kFieldF32)
        classify_batch_tma<kFieldF32><<<bricks, kThreads, kRingBytesF32, st>>>(B);
    else if (ftype == kFieldU8)
        classify_batch_tma<kFieldU8><<<bricks, kThreads, kRingBytesU8, st>>>(B);
    else if (ftype == kFieldUNorm8)
        classify_batch_tma<kFieldUNorm8><<<bricks, kThreads, kRingBytesU8, st>>>(B);
    else
        return cudaErrorInvalidValue;
    return cudaGetLastError();
}

cudaError_t launch_classify_batch_direct(const BatchDev& B, int ftype, unsigned int bricks, cudaStream_t st) {
    if (!bricks) return cudaSuccess;
    if (ftype == kFieldF32)
        classify_batch_direct<kFieldF32><<<bricks, kThreads, 0, st>>>(B);
    else if (ftype == kFieldU8)
        classify_batch_direct<kFieldU8><<<bricks, kThreads, 0, st>>>(B);
    else if (ftype == kFieldUNorm8)
        classify_batch_direct<kFieldUNorm8><<<bricks, kThreads, 0, st>>>(B);
    else
        return cudaErrorInvalidValue;
    return cudaGetLastError();
}

cudaError_t launch_reduce_batch(const BatchDev& B, unsigned int chunks, cudaStream_t st) {
    reduce_batch<<<chunks, kThreads, 0, st>>>(B);
    return cudaGetLastError();
}

void column_smem_opt_in() {
    const auto opt_in = [](auto* kernel, int bytes) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    };
    opt_in(classify_columns<kFieldF32>, kRingBytesF32);
    opt_in(classify_columns<kFieldU8>, kRingBytesU8);
    opt_in(classify_columns<kFieldUNorm8>, kRingBytesU8);
    opt_in(classify_batch_tma<kFieldF32>, kRingBytesF32);
    opt_in(classify_batch_tma<kFieldU8>, kRingBytesU8);
    opt_in(classify_batch_tma<kFieldUNorm8>, kRingBytesU8);
}

}  // namespace hpmc
