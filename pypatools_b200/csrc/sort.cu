// Particle reordering by cell, so that the threads of a warp gather the same
// corner records (one L1 wavefront per corner load instead of one per
// distinct cell).
//
// Counting sort on the particle's map-0 cell: bucket = linear cell index
// (k fastest) modulo 2^22 -- exact for maps up to 4M cells, a hash beyond;
// particles outside the map share one last bucket.  Histogram -> exclusive
// scan -> scatter of whole slots as records -> records back into columns, with
// warp-aggregated atomics (lanes with equal keys combine before touching
// memory).  The
// reordering runs when at least 1/16 of the particles are inside the map, or
// when the warps holding in-map particles exceed the ones those particles
// need by n/512 (a few particles still in the map after the bunch has left,
// spread over many warps: each such warp runs the gather path for one lane).
// Otherwise every kernel after the histogram returns at once: the sort is a
// no-op decided on the device, so the caller's stream never waits.
// Order inside a bucket is arbitrary; `order` records slot -> row so outputs
// land in the caller's row order, and each particle's arithmetic is
// independent of its slot.
#include <cstring>

#include "track_params.cuh"

namespace ppt {

constexpr int kBucketBits = 22;
constexpr int kScanTile = 1024;

struct SortGeom {
    double lo[3];
    double inv_d[3];
    int n[3];           // nodes per axis
    uint32_t n_in;      // buckets for in-map cells
    uint32_t outside;   // bucket of particles outside the map (= n_in)
    int flat[3];        // the map does not vary along the axis: its cell is not part of the key
};

__device__ __forceinline__ bool cell_inside(const SortGeom& G, int c0, int c1, int c2) {
    return (unsigned)c0 <= (unsigned)(G.n[0] - 2) && (unsigned)c1 <= (unsigned)(G.n[1] - 2) &&
           (unsigned)c2 <= (unsigned)(G.n[2] - 2);
}

__device__ __forceinline__ uint32_t bucket_of_cells(const SortGeom& G, int c0, int c1, int c2) {
    if (!cell_inside(G, c0, c1, c2)) return G.outside;
    const uint64_t lin = ((uint64_t)c0 * (uint64_t)(G.n[1] - 1) + (uint64_t)c1) * (uint64_t)(G.n[2] - 1) + (uint64_t)c2;
    return (uint32_t)(lin % G.n_in);
}

// Histogram of the in-map keys (one atomic per distinct key per warp), the
// in-map count and the number of warps with an in-map particle (one atomic
// each per block).  Particles outside the map touch no counter: their
// bucket's size is n minus the in-map count, filled in by the scan, so a
// bunch that has left the map costs no same-address atomics.  Called by every
// thread of the block (full warps).
__device__ __forceinline__ void count_key(uint32_t b, bool inside, uint32_t* count, uint32_t* ctrl) {
    __shared__ unsigned block_in, block_warps;
    if (threadIdx.x == 0) block_in = block_warps = 0;
    __syncthreads();
    if (__any_sync(0xffffffffu, inside) && (threadIdx.x & 31) == 0) atomicAdd(&block_warps, 1u);
    if (inside) {
        const unsigned active = __activemask();
        const unsigned same = __match_any_sync(active, b);
        const int lane = threadIdx.x & 31;
        if (lane == __ffs(same) - 1) {
            atomicAdd(count + b, (uint32_t)__popc(same));
            atomicAdd(&block_in, (unsigned)__popc(same));
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && block_in) {
        atomicAdd(ctrl, block_in);
        atomicAdd(ctrl + 1, block_warps);
    }
}

__global__ void sort_keys_f64(int64_t n, const double* __restrict__ st, SortGeom G, uint32_t* __restrict__ key,
                              uint32_t* __restrict__ count, uint32_t* __restrict__ ctrl) {
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    uint32_t b = G.outside;
    if (s < n) {
        int c[3];
        for (int a = 0; a < 3; ++a) {
            double u = (st[a * n + s] - G.lo[a]) * G.inv_d[a];
            c[a] = (u >= 0.0 && u < 2.0e9) ? (int)u : -1;
        }
        b = bucket_of_cells(G, c[0], c[1], c[2]);
        key[s] = b;
    }
    count_key(b, s < n && b != G.outside, count, ctrl);
}

__global__ void sort_keys_mixed(int64_t n, const int32_t* __restrict__ ci, SortGeom G, uint32_t* __restrict__ key,
                                uint32_t* __restrict__ count, uint32_t* __restrict__ ctrl) {
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    uint32_t b = G.outside;
    if (s < n) {
        // mixed-form cells on an axis the map does not vary along count
        // on their own grid, not the map's single layer
        b = bucket_of_cells(G, G.flat[0] ? 0 : ci[s], G.flat[1] ? 0 : ci[n + s], G.flat[2] ? 0 : ci[2 * n + s]);
        key[s] = b;
    }
    count_key(b, s < n && b != G.outside, count, ctrl);
}

__device__ __forceinline__ bool sort_wanted(const uint32_t* ctrl, int64_t n) {
    const int64_t in = ctrl[0], excess_warps = (int64_t)ctrl[1] - (in + 31) / 32;
    return in * 16 >= n || (in > 0 && excess_warps * 512 >= n);
}

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* sh, uint32_t& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0u;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        sh[lane] = w;   // inclusive warp totals
    }
    __syncthreads();
    total = sh[(blockDim.x >> 5) - 1];
    uint32_t before = warp > 0 ? sh[warp - 1] : 0u;
    uint32_t r = before + x - v;
    __syncthreads();
    return r;
}

__global__ void __launch_bounds__(kScanTile) scan_tiles(int64_t nb, const uint32_t* __restrict__ count,
                                                        uint32_t* __restrict__ offset, uint32_t* __restrict__ tile_sum,
                                                        const uint32_t* __restrict__ ctrl, int64_t n) {
    if (!sort_wanted(ctrl, n)) return;
    __shared__ uint32_t sh[32];
    int64_t i = blockIdx.x * (int64_t)kScanTile + threadIdx.x;
    uint32_t v = i < nb ? count[i] : 0u;
    if (i == nb - 1) v = (uint32_t)(n - (int64_t)ctrl[0]);   // the outside bucket: everything not in the map
    uint32_t total;
    uint32_t ex = block_exclusive_scan(v, sh, total);
    if (i < nb) offset[i] = ex;
    if (threadIdx.x == 0) tile_sum[blockIdx.x] = total;
}

// exclusive scan of the tile sums in one block
__global__ void __launch_bounds__(kScanTile) scan_top(int ntiles, uint32_t* __restrict__ tile_sum,
                                                      const uint32_t* __restrict__ ctrl, int64_t n) {
    if (!sort_wanted(ctrl, n)) return;
    __shared__ uint32_t sh[32];
    uint32_t carry = 0;
    for (int base = 0; base < ntiles; base += kScanTile) {
        int i = base + threadIdx.x;
        uint32_t v = i < ntiles ? tile_sum[i] : 0u;
        uint32_t total;
        uint32_t ex = block_exclusive_scan(v, sh, total);
        if (i < ntiles) tile_sum[i] = ex + carry;
        carry += total;
    }
}

__global__ void scan_add(int64_t nb, uint32_t* __restrict__ offset, const uint32_t* __restrict__ tile_sum,
                         const uint32_t* __restrict__ ctrl, int64_t n) {
    if (!sort_wanted(ctrl, n)) return;
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < nb) offset[i] += tile_sum[i / kScanTile];
}

// A slot as one record: its state (15 words of the mixed form, or 6 doubles),
// row and RF phase, in 16-byte pieces.  Permuting the columns one by one writes
// a 32-byte sector for every 4- or 8-byte word of every slot (17 of them in the
// mixed form) when the order is random; a record takes three or two, and putting
// the records back into columns reads and writes in order, where the permuted
// columns had to be copied back as well.  B200, all sorts of a track, columns ->
// records: 6e6 mixed protons through the RF gap (7 sorts) 3.35 -> 2.52 ms, 5e6 in
// the ring (4) 2.78 -> 2.08, 1e6 float64 through the gap (7) 0.69 -> 0.58.
template <bool F64>
struct Record {
    static constexpr int kWords = F64 ? 16 : 20;
    static constexpr int kOrder = F64 ? 12 : 16;     // first word of the row, then of the phase
};

// Slot s's record to position d.
template <bool F64>
__device__ __forceinline__ void write_record(int64_t n, int64_t s, int64_t d, const uint32_t* __restrict__ src_a,
                                             const uint32_t* __restrict__ src_b, const uint2* __restrict__ order,
                                             const uint2* __restrict__ phase, uint4* __restrict__ records) {
    using R = Record<F64>;
    uint32_t w[R::kWords];
    if constexpr (F64) {
        const uint2* col = reinterpret_cast<const uint2*>(src_a);
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            const uint2 v = col[c * n + s];
            w[2 * c] = v.x;
            w[2 * c + 1] = v.y;
        }
    } else {
        // 3 int32 cell columns, then 12 float32 columns
#pragma unroll
        for (int c = 0; c < 3; ++c) w[c] = src_a[c * n + s];
#pragma unroll
        for (int c = 0; c < 12; ++c) w[3 + c] = src_b[c * n + s];
        w[15] = 0u;
    }
    const uint2 row = order[s], ph = phase ? phase[s] : make_uint2(0u, 0u);
    w[R::kOrder] = row.x;
    w[R::kOrder + 1] = row.y;
    w[R::kOrder + 2] = ph.x;
    w[R::kOrder + 3] = ph.y;
    uint4* out = records + d * (R::kWords / 4);
#pragma unroll
    for (int q = 0; q < R::kWords / 4; ++q) out[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
}

template <bool F64>
__global__ void __launch_bounds__(256) sort_scatter(int64_t n, const uint32_t* __restrict__ key,
                                                    uint32_t* __restrict__ offset, const uint32_t* __restrict__ ctrl,
                                                    const uint32_t* __restrict__ src_a,
                                                    const uint32_t* __restrict__ src_b,
                                                    const uint2* __restrict__ order, const uint2* __restrict__ phase,
                                                    uint4* __restrict__ records) {
    if (!sort_wanted(ctrl, n)) return;
    int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s >= n) return;
    const uint32_t b = key[s];
    const unsigned active = __activemask();
    const unsigned same = __match_any_sync(active, b);
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(same) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(offset + b, (uint32_t)__popc(same));
    base = __shfl_sync(same, base, leader);
    const int64_t d = (int64_t)base + __popc(same & ((1u << lane) - 1u));
    write_record<F64>(n, s, d, src_a, src_b, order, phase, records);
}

// Back to row order: slot s to position order[s].  (order is a permutation of
// 0 .. n-1, kept so by the sorts; a slot with a value outside is skipped.)
// A gather of the columns through the inverse permutation read a 32-byte sector
// for every word of every slot and needed the columns copied back.  B200, gather ->
// records, the random order of a fresh sort: 1e7 mixed slots 3.12 -> 1.35 ms, 1e6
// 0.117 -> 0.101, 20 000 30 -> 13 us, 1e7 float64 1.37 -> 0.87; a 6000-step track
// of 6e6 mixed protons (8 sorts and one return) 4.04 -> 3.47 in all.
template <bool F64>
__global__ void __launch_bounds__(256) restore_scatter(int64_t n, const uint32_t* __restrict__ src_a,
                                                       const uint32_t* __restrict__ src_b,
                                                       const uint2* __restrict__ order,
                                                       const uint2* __restrict__ phase,
                                                       uint4* __restrict__ records) {
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int64_t d = reinterpret_cast<const int64_t*>(order)[s];
    if (d >= 0 && d < n) write_record<F64>(n, s, d, src_a, src_b, order, phase, records);
}

// The permuted records back into the columns (after a sort, ctrl given, only when
// it ran), 128 at a time through shared memory (an odd stride: no bank conflicts).
constexpr int kUnpack = 128;

template <bool F64>
__global__ void __launch_bounds__(kUnpack) sort_unpack(int64_t n, const uint32_t* __restrict__ records,
                                                       const uint32_t* __restrict__ ctrl, uint32_t* __restrict__ dst_a,
                                                       uint32_t* __restrict__ dst_b, uint2* __restrict__ order,
                                                       uint2* __restrict__ phase) {
    using R = Record<F64>;
    if (ctrl && !sort_wanted(ctrl, n)) return;
    __shared__ uint32_t tile[kUnpack * (R::kWords + 1)];
    const int64_t first = blockIdx.x * (int64_t)kUnpack;
    const int here = (int)(n - first < kUnpack ? n - first : kUnpack);
    const uint32_t* from = records + first * R::kWords;
    for (int i = threadIdx.x; i < here * R::kWords; i += kUnpack)
        tile[i / R::kWords * (R::kWords + 1) + i % R::kWords] = from[i];
    __syncthreads();
    const int t = threadIdx.x;
    if (t >= here) return;
    const int64_t s = first + t;
    const uint32_t* w = tile + t * (R::kWords + 1);
    if constexpr (F64) {
        uint2* col = reinterpret_cast<uint2*>(dst_a);
#pragma unroll
        for (int c = 0; c < 6; ++c) col[c * n + s] = make_uint2(w[2 * c], w[2 * c + 1]);
    } else {
#pragma unroll
        for (int c = 0; c < 3; ++c) dst_a[c * n + s] = w[c];
#pragma unroll
        for (int c = 0; c < 12; ++c) dst_b[c * n + s] = w[3 + c];
    }
    // back in row order (no ctrl) every slot is its own row
    order[s] = ctrl ? make_uint2(w[R::kOrder], w[R::kOrder + 1])
                    : make_uint2((uint32_t)s, (uint32_t)((uint64_t)s >> 32));
    if (phase) phase[s] = make_uint2(w[R::kOrder + 2], w[R::kOrder + 3]);
}

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

struct SortLayout {
    size_t key, count, tiles, ctrl, records, total;
};

static SortLayout sort_layout(int64_t n) {
    SortLayout L;
    const size_t nb = ((size_t)1 << kBucketBits) + 1;
    size_t o = 0;
    L.key = o;   o += align256((size_t)n * 4);
    L.count = o; o += align256(nb * 4);
    L.tiles = o; o += align256((nb / kScanTile + 2) * 4);
    L.ctrl = o;  o += 256;
    L.records = o; o += align256((size_t)n * Record<false>::kWords * 4 + 16);   // 16: see records_in
    L.total = o;
    return L;
}

// the records' place in a scratch buffer, on a 16-byte boundary whatever that is on
static uint4* records_in(char* scratch, const SortLayout& L) {
    return reinterpret_cast<uint4*>((reinterpret_cast<uintptr_t>(scratch + L.records) + 15) & ~(uintptr_t)15);
}

// slots -> records -> columns: a sort's permutation, or (key NULL) back to row order
template <bool F64>
static void permute(const ppt_state* st, const uint32_t* key, uint32_t* offset, const uint32_t* ctrl, int64_t* order,
                    double* rf_phase, uint4* records, cudaStream_t s) {
    const int64_t n = st->n;
    uint32_t* a = F64 ? reinterpret_cast<uint32_t*>(st->f64) : reinterpret_cast<uint32_t*>(st->i32);
    uint32_t* b = reinterpret_cast<uint32_t*>(st->f32);
    uint2* row = reinterpret_cast<uint2*>(order);
    uint2* phase = reinterpret_cast<uint2*>(rf_phase);
    if (key) sort_scatter<F64><<<grid_for(n, 256), 256, 0, s>>>(n, key, offset, ctrl, a, b, row, phase, records);
    else restore_scatter<F64><<<grid_for(n, 256), 256, 0, s>>>(n, a, b, row, phase, records);
    sort_unpack<F64><<<grid_for(n, kUnpack), kUnpack, 0, s>>>(n, reinterpret_cast<const uint32_t*>(records), ctrl, a, b,
                                                              row, phase);
}

}  // namespace ppt

using namespace ppt;

extern "C" int64_t ppt_cell_sort_scratch_bytes(int64_t n) {
    if (n < 0) return -1;
    return (int64_t)sort_layout(n).total;
}

extern "C" int ppt_cell_sort(ppt_state* st, const ppt_fields* fields, int64_t* order, double* rf_phase,
                             void* scratch, void* stream) {
    int rc = check_state(st);
    if (rc) return rc;
    if (st->n == 0) return PPT_OK;
    if (st->n > 0x7fffffffLL) return fail(PPT_ERR_UNSUPPORTED, "cell sort handles at most 2^31-1 particles");
    if (!order || !scratch) return fail(PPT_ERR_ARG, "order and scratch must not be NULL");
    FieldsDev F;
    rc = build_fields(fields, &F);
    if (rc) return rc;
    if (F.n_maps == 0) return PPT_OK;   // no map: nothing to be local to
    const MapDev& m = F.maps[0];
    if (!m.all_uniform) return PPT_OK;  // non-uniform maps: no cheap cell key, keep the order
    SortGeom G;
    uint64_t cells = 1;
    for (int a = 0; a < 3; ++a) {
        G.lo[a] = m.ax[a].lo;
        G.inv_d[a] = m.ax[a].inv_d;
        G.n[a] = m.ax[a].n;
        G.flat[a] = axis_is_flat(m.ax[a]) ? 1 : 0;
        cells *= (uint64_t)(m.ax[a].n - 1);
    }
    G.n_in = (uint32_t)(cells < ((uint64_t)1 << kBucketBits) ? cells : ((uint64_t)1 << kBucketBits));
    G.outside = G.n_in;
    const int64_t nb = (int64_t)G.n_in + 1;

    const int64_t n = st->n;
    SortLayout L = sort_layout(n);
    char* base = static_cast<char*>(scratch);
    uint32_t* key = reinterpret_cast<uint32_t*>(base + L.key);
    uint32_t* count = reinterpret_cast<uint32_t*>(base + L.count);
    uint32_t* tiles = reinterpret_cast<uint32_t*>(base + L.tiles);
    uint32_t* ctrl = reinterpret_cast<uint32_t*>(base + L.ctrl);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int block = 256;

    PPT_CUDA_TRY(cudaMemsetAsync(count, 0, (size_t)nb * 4, s));
    PPT_CUDA_TRY(cudaMemsetAsync(ctrl, 0, 8, s));
    if (st->precision == PPT_PREC_F64)
        sort_keys_f64<<<grid_for(n, block), block, 0, s>>>(n, st->f64, G, key, count, ctrl);
    else
        sort_keys_mixed<<<grid_for(n, block), block, 0, s>>>(n, st->i32, G, key, count, ctrl);
    const int ntiles = (int)((nb + kScanTile - 1) / kScanTile);
    scan_tiles<<<ntiles, kScanTile, 0, s>>>(nb, count, count, tiles, ctrl, n);
    scan_top<<<1, kScanTile, 0, s>>>(ntiles, tiles, ctrl, n);
    scan_add<<<grid_for(nb, block), block, 0, s>>>(nb, count, tiles, ctrl, n);
    uint4* records = records_in(base, L);
    if (st->precision == PPT_PREC_F64) permute<true>(st, key, count, ctrl, order, rf_phase, records, s);
    else permute<false>(st, key, count, ctrl, order, rf_phase, records, s);
    PPT_CUDA_TRY(cudaGetLastError());
    return PPT_OK;
}

extern "C" int ppt_restore_order(ppt_state* st, int64_t* order, double* rf_phase, void* scratch, void* stream) {
    int rc = check_state(st);
    if (rc) return rc;
    if (st->n == 0) return PPT_OK;
    if (!order || !scratch) return fail(PPT_ERR_ARG, "order and scratch must not be NULL");
    const int64_t n = st->n;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    uint4* records = records_in(static_cast<char*>(scratch), sort_layout(n));
    if (st->precision == PPT_PREC_F64) permute<true>(st, nullptr, nullptr, nullptr, order, rf_phase, records, s);
    else permute<false>(st, nullptr, nullptr, nullptr, order, rf_phase, records, s);
    PPT_CUDA_TRY(cudaGetLastError());
    return PPT_OK;
}
