// qk_sort.cu -- stable LSD radix sort of (uint32 key, uint32 value) pairs and an exclusive
// int scan, written for the engine's build (Morton codes) and query reordering.
//
// Radix sort: 8-bit digits, tiles of 4096 keys, one kernel per digit:
//   k_rs_hist   counts every pass's digits in one read of the keys (a digit's total does not
//               depend on the order) and clears what the passes count with
//   k_rs_pass   each block takes the next tile from a counter and ranks its keys in input
//               order: __match_any_sync groups lanes holding the same digit, the rank inside a
//               round is the popcount of lower peers, and a per-warp running count carries
//               ranks across rounds.  It publishes the tile's digit counts, adds up those of
//               the tiles before it (one thread per digit, eight tiles per step, until it meets
//               a tile that has published its own sum), publishes its sums, lays the tile out
//               in digit order in shared memory and writes every digit's run with consecutive
//               threads.  Equal digits keep their input order, so the sort is stable.
// Up to one tile of keys is sorted by one block in one launch (k_rs_small).  The chained sums are
// the decoupled look-back of Merrill and Garland (2016), with an end to every wait.
//
// A 30-bit sort of 1,048,576 pairs took 24 launches before (a histogram, three scan kernels and
// a scatter per digit) and takes 5: 143 -> 91 us of kernel time, the cloud's LBVH 361 -> 308 us.
// Stability makes sorting (morton, index) pairs on the 30 Morton bits alone equal to the
// reference's full 64-bit sort of (morton << 32 | index) keys (src/gpu/lbvh.cu:1995-2003).
#include "qk_internal.cuh"

namespace qk {

namespace {

constexpr int kRadix = kSortRadix;
constexpr int kWarps = kBlock / 32;
constexpr int kItems = kSortTile / kBlock;  // 16 keys per thread
static_assert(kItems * kBlock == kSortTile, "tile size");

// ---- warp and block scans (the sort's digit runs and the exclusive scan below) ----
__device__ __forceinline__ int warp_incl_scan(int v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += y;
    }
    return v;
}

// Exclusive block scan of one value per thread; returns the block total in *total.
__device__ __forceinline__ int block_excl_scan(int v, int* total) {
    __shared__ int ws[kBlock / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int inc = warp_incl_scan(v);
    if (lane == 31) ws[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        int s = lane < kBlock / 32 ? ws[lane] : 0;
        s = warp_incl_scan(s);
        if (lane < kBlock / 32) ws[lane] = s;
    }
    __syncthreads();
    const int wprefix = warp > 0 ? ws[warp - 1] : 0;
    *total = ws[kBlock / 32 - 1];
    __syncthreads();
    return wprefix + inc - v;
}

// ---- one tile ----
struct RsTile {
    uint32_t wcount[kWarps][kRadix];  // keys of a digit in each warp, then before each warp
    uint32_t lstart[kRadix];          // a digit's first place in the tile
    uint32_t key[kSortTile];
    uint32_t val[kSortTile];
};

// Ranks the tile's keys (key j of a lane: warp * 512 + 32 j + lane; `m` keys in the tile) by
// the digit at `shift`, stably, and leaves keys and values in digit order in sh.key / sh.val.
// Returns this thread's digit count.
__device__ __forceinline__ uint32_t rs_rank_tile(RsTile& sh, const uint32_t (&key)[kItems],
                                                 const uint32_t (&val)[kItems], int m, int shift) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < kWarps * kRadix; i += kBlock) (&sh.wcount[0][0])[i] = 0;
    __syncthreads();
    const int first = warp * (kSortTile / kWarps) + lane;
    const unsigned lower = (1u << lane) - 1u;
    uint16_t rank[kItems];
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const bool ok = first + 32 * j < m;
        const uint32_t d = ok ? ((key[j] >> shift) & 0xffu) : 0x100u;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const uint32_t before = ok ? sh.wcount[warp][d] : 0u;
        __syncwarp();
        if (ok && lane == __ffs(peers) - 1) sh.wcount[warp][d] = before + __popc(peers);
        __syncwarp();
        rank[j] = static_cast<uint16_t>(before + __popc(peers & lower));
    }
    __syncthreads();
    // per digit: the tile's count, its run's start inside the tile (a block scan over the
    // digits) and every warp's offset inside that run
    static_assert(kRadix == kBlock, "one thread per digit");
    const int d = threadIdx.x;
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        const uint32_t c = sh.wcount[w][d];
        sh.wcount[w][d] = run;
        run += c;
    }
    int total;
    sh.lstart[d] = static_cast<uint32_t>(block_excl_scan(static_cast<int>(run), &total));
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        if (first + 32 * j < m) {
            const uint32_t dj = (key[j] >> shift) & 0xffu;
            const uint32_t at = sh.lstart[dj] + sh.wcount[warp][dj] + rank[j];
            sh.key[at] = key[j];
            sh.val[at] = val[j];
        }
    }
    return run;
}

// What the passes share, cleared before a sort: the next tile of each pass and each pass's
// digit totals.
constexpr int kMaxPasses = kSortPasses;
struct RsCounts {
    int ticket[kMaxPasses];
    int pad[60];
    uint32_t total[kMaxPasses][kRadix];
};

// digit totals of every pass
__global__ __launch_bounds__(kBlock) void k_rs_hist(const uint32_t* __restrict__ keys, int n,
                                                    int passes, RsCounts* __restrict__ c) {
    __shared__ uint32_t h[kMaxPasses][kRadix];
    for (int i = threadIdx.x; i < kMaxPasses * kRadix; i += kBlock) (&h[0][0])[i] = 0;
    __syncthreads();
    for (int i = blockIdx.x * kBlock + threadIdx.x; i < n; i += kBlock * gridDim.x) {
        const uint32_t k = keys[i];
        for (int p = 0; p < passes; ++p) atomicAdd(&h[p][(k >> (8 * p)) & 0xffu], 1u);
    }
    __syncthreads();
    for (int p = 0; p < passes; ++p) {
        const uint32_t v = h[p][threadIdx.x];
        if (v) atomicAdd(&c->total[p][threadIdx.x], v);
    }
}

// A tile's entry for one digit: a count shifted left by two over its state.  S is uint32_t
// while every count fits 30 bits, uint64_t beyond.
constexpr uint32_t kTileCount = 1;  // the tile's own keys
constexpr uint32_t kTileSum = 2;    // with those of every tile before it
constexpr int kLookback = 8;        // tiles read per step

template <class S>
__device__ __forceinline__ S rs_load(const S* p) {
    return *const_cast<const volatile S*>(p);
}
template <class S>
__device__ __forceinline__ void rs_store(S* p, S v) {
    *const_cast<volatile S*>(p) = v;
}

// One digit's pass.  state: tiles x 256 entries of this pass, zero on entry; next_state (null:
// none) the next pass's, cleared tile by tile here.  Tiles are taken in order from a counter,
// so every tile a block waits for has started; a wait that still sees nothing after max_polls
// reads ends by counting the keys before the tile directly, so no block depends on another to
// finish (max_polls < 0: at once).  iota: the values are the keys' positions and vin is not read.
template <class S>
__global__ __launch_bounds__(kBlock) void k_rs_pass(const uint32_t* __restrict__ kin,
                                                    const uint32_t* __restrict__ vin,
                                                    uint32_t* __restrict__ kout,
                                                    uint32_t* __restrict__ vout, int n, int pass,
                                                    RsCounts* __restrict__ c, S* state,
                                                    S* __restrict__ next_state, int iota,
                                                    int max_polls) {
    __shared__ RsTile sh;
    __shared__ uint32_t gbase[kRadix];
    __shared__ int tile_s;
    __shared__ int late;
    const int d = threadIdx.x, lane = d & 31, warp = d >> 5;
    if (d == 0) {
        tile_s = atomicAdd(&c->ticket[pass], 1);
        late = max_polls < 0;
    }
    __syncthreads();
    const int tile = tile_s, shift = 8 * pass;
    const int base = tile * kSortTile;
    const int m = min(kSortTile, n - base);
    uint32_t key[kItems], val[kItems];
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const int i = warp * (kSortTile / kWarps) + 32 * j + lane;
        key[j] = i < m ? kin[base + i] : 0u;
        val[j] = iota ? static_cast<uint32_t>(base + i) : (i < m ? vin[base + i] : 0u);
    }
    const uint32_t total = c->total[pass][d];
    if (next_state) next_state[static_cast<size_t>(tile) * kRadix + d] = 0;
    const uint32_t mine = rs_rank_tile(sh, key, val, m, shift);

    S* own = state + static_cast<size_t>(tile) * kRadix + d;
    if (tile > 0) rs_store(own, static_cast<S>((static_cast<S>(mine) << 2) | kTileCount));
    else rs_store(own, static_cast<S>((static_cast<S>(mine) << 2) | kTileSum));
    int all;
    const uint32_t start = static_cast<uint32_t>(block_excl_scan(static_cast<int>(total), &all));
    uint32_t before = 0;
    int t = max_polls < 0 ? -1 : tile - 1, polls = 0;
    while (t >= 0) {
        S v[kLookback];
#pragma unroll
        for (int j = 0; j < kLookback; ++j)
            v[j] = t - j >= 0 ? rs_load(state + static_cast<size_t>(t - j) * kRadix + d)
                              : static_cast<S>(kTileSum);
        int used = 0;
        bool done = false;
#pragma unroll
        for (int j = 0; j < kLookback; ++j) {
            if (!done && used == j && (v[j] & 3u) != 0) {
                before += static_cast<uint32_t>(v[j] >> 2);
                done = (v[j] & 3u) == kTileSum;
                ++used;
            }
        }
        if (done) break;
        t -= used;
        if (used == 0 && ++polls > max_polls) {
            late = 1;
            break;
        }
    }
    __syncthreads();
    if (late) {
        // the same sums from the keys themselves
        gbase[d] = 0;
        __syncthreads();
        for (int i = d; i < base; i += kBlock) atomicAdd(&gbase[(kin[i] >> shift) & 0xffu], 1u);
        __syncthreads();
        before = gbase[d];
    }
    if (tile > 0) rs_store(own, static_cast<S>((static_cast<S>(before + mine) << 2) | kTileSum));
    gbase[d] = start + before - sh.lstart[d];
    __syncthreads();
    // consecutive threads write consecutive slots of one digit's run
#pragma unroll 4
    for (int i = d; i < m; i += kBlock) {
        const uint32_t k = sh.key[i];
        const uint32_t dst = gbase[(k >> shift) & 0xffu] + static_cast<uint32_t>(i);
        kout[dst] = k;
        vout[dst] = sh.val[i];
    }
}

// every pass of at most one tile of keys, by one block
__global__ __launch_bounds__(kBlock) void k_rs_small(const uint32_t* __restrict__ kin,
                                                     const uint32_t* __restrict__ vin,
                                                     uint32_t* __restrict__ kout,
                                                     uint32_t* __restrict__ vout, int n, int passes,
                                                     int iota) {
    __shared__ RsTile sh;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t key[kItems], val[kItems];
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const int i = warp * (kSortTile / kWarps) + 32 * j + lane;
        key[j] = i < n ? kin[i] : 0u;
        val[j] = iota ? static_cast<uint32_t>(i) : (i < n ? vin[i] : 0u);
    }
    for (int p = 0; p < passes; ++p) {
        rs_rank_tile(sh, key, val, n, 8 * p);
        __syncthreads();
        if (p + 1 == passes) break;
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            const int i = warp * (kSortTile / kWarps) + 32 * j + lane;
            key[j] = i < n ? sh.key[i] : 0u;
            val[j] = i < n ? sh.val[i] : 0u;
        }
        __syncthreads();
    }
    for (int i = threadIdx.x; i < n; i += kBlock) {
        kout[i] = sh.key[i];
        vout[i] = sh.val[i];
    }
}

// ---- exclusive scan: block-local scans, a scan of the block sums, then a fix-up ----
// in and out may alias: each thread reads its own four elements before any write
__global__ __launch_bounds__(kBlock) void k_scan_blocks(const int* in, int* out, int n,
                                                        int* __restrict__ sums) {
    const int base = blockIdx.x * kScanBlock + threadIdx.x * 4;
    int v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = base + j < n ? in[base + j] : 0;
    const int tsum = v[0] + v[1] + v[2] + v[3];
    int total;
    int run = block_excl_scan(tsum, &total);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (base + j < n) out[base + j] = run;
        run += v[j];
    }
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// single block: exclusive scan of the block sums in place, total to *total_out
__global__ __launch_bounds__(kBlock) void k_scan_sums(int* __restrict__ sums, int nb,
                                                      int* __restrict__ total_out) {
    int carry = 0;
    for (int base = 0; base < nb; base += kBlock) {
        const int i = base + threadIdx.x;
        const int v = i < nb ? sums[i] : 0;
        int total;
        const int ex = block_excl_scan(v, &total);
        if (i < nb) sums[i] = carry + ex;
        carry += total;
    }
    if (threadIdx.x == 0 && total_out) *total_out = carry;
}

__global__ __launch_bounds__(kBlock) void k_scan_add(int* __restrict__ out, int n,
                                                     const int* __restrict__ sums) {
    const int b = blockIdx.x;
    if (b == 0) return;
    const int add = sums[b];
    const int base = b * kScanBlock + threadIdx.x * 4;
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (base + j < n) out[base + j] += add;
}

}  // namespace

size_t scan_ws_bytes(int n) {
    return (static_cast<size_t>(blocks_for(n, kScanBlock)) + 1) * sizeof(int) + 256;
}

cudaError_t scan_exclusive(const int* in, int* out, int n, bool write_total, void* ws,
                           cudaStream_t s) {
    if (n <= 0) {
        if (write_total) return cudaMemsetAsync(out, 0, sizeof(int), s);
        return cudaSuccess;
    }
    const int nb = blocks_for(n, kScanBlock);
    int* sums = static_cast<int*>(ws);
    k_scan_blocks<<<nb, kBlock, 0, s>>>(in, out, n, sums);
    k_scan_sums<<<1, kBlock, 0, s>>>(sums, nb, write_total ? out + n : nullptr);
    if (nb > 1) k_scan_add<<<nb, kBlock, 0, s>>>(out, n, sums);
    return cudaGetLastError();
}

// tile states: two passes' worth, each pass clearing the next one's
inline size_t rs_state_bytes(int n, bool wide) {
    return (n < (1 << 30) && !wide ? sizeof(uint32_t) : sizeof(uint64_t)) * kRadix *
           static_cast<size_t>(blocks_for(n, kSortTile));
}

size_t sort_ws_bytes(int n, const SortPaths& paths) {
    Carve c;
    c.take<RsCounts>(1);
    c.take<char>(rs_state_bytes(n, paths.wide_states));
    c.take<char>(rs_state_bytes(n, paths.wide_states));
    return c.used;
}

uint32_t* sort_begin(void* ws, int n, cudaStream_t s, const SortPaths& paths) {
    if (n <= kSortTile) return nullptr;
    Carve c{static_cast<char*>(ws)};
    RsCounts* counts = c.take<RsCounts>(1);
    const size_t bytes = rs_state_bytes(n, paths.wide_states);
    const char* state = c.take<char>(bytes);
    // the counters and the first pass's states are one run of bytes
    cudaMemsetAsync(counts, 0, static_cast<size_t>(state - reinterpret_cast<char*>(counts)) + bytes, s);
    return &counts->total[0][0];
}

template <class S>
static void rs_launch(const uint32_t* sk, const uint32_t* sv, uint32_t* dk, uint32_t* dv, int n,
                      int pass, RsCounts* c, char* state, char* next, bool iota, int max_polls,
                      cudaStream_t s) {
    k_rs_pass<S><<<blocks_for(n, kSortTile), kBlock, 0, s>>>(
        sk, sv, dk, dv, n, pass, c, reinterpret_cast<S*>(state), reinterpret_cast<S*>(next), iota,
        max_polls);
}

// Sorts (kin, vin) by the low `bits` bits.  Passes alternate between the output pair and the
// input pair (pass p writes the output pair when p is even), so kin / vin are clobbered when
// more than one pass runs.  With `sorted` the caller takes the result where it ends (the input
// pair after an even number of passes); without, it is in (kout, vout), copied there if need
// be.  iota: the values are 0..n-1 and vin is only a buffer.
//
// One pass over 1,048,576 pairs (20 us under ncu) is bound by its latency, not by bytes (16 MB):
// 256 tiles on 148 SMs, 16 ranking rounds each, then the earlier tiles' counts.
cudaError_t sort_pairs(const uint32_t* kin, const uint32_t* vin, uint32_t* kout, uint32_t* vout,
                       int n, int bits, void* ws, cudaStream_t s, SortedPairs* sorted, bool iota,
                       bool counted, const SortPaths& paths) {
    if (n <= 0) return cudaSuccess;
    const int passes = bits <= 0 ? 1 : (bits + 7) / 8;
    if (sorted) *sorted = {kout, vout};
    if (n <= kSortTile) {
        k_rs_small<<<1, kBlock, 0, s>>>(kin, vin, kout, vout, n, passes, iota);
        return cudaGetLastError();
    }
    Carve c{static_cast<char*>(ws)};
    RsCounts* counts = c.take<RsCounts>(1);
    char* state[2];
    state[0] = c.take<char>(rs_state_bytes(n, paths.wide_states));
    state[1] = c.take<char>(rs_state_bytes(n, paths.wide_states));
    if (!counted) {
        sort_begin(ws, n, s, paths);
        k_rs_hist<<<min(blocks_for(n, 4 * kBlock), 148 * 4), kBlock, 0, s>>>(kin, n, passes, counts);
    }
    const uint32_t* sk = kin;
    const uint32_t* sv = vin;
    for (int p = 0; p < passes; ++p) {
        uint32_t* dk = (p % 2 == 0) ? kout : const_cast<uint32_t*>(kin);
        uint32_t* dv = (p % 2 == 0) ? vout : const_cast<uint32_t*>(vin);
        char* next = p + 1 < passes ? state[(p + 1) % 2] : nullptr;
        const auto launch = n < (1 << 30) && !paths.wide_states ? rs_launch<uint32_t> : rs_launch<uint64_t>;
        launch(sk, sv, dk, dv, n, p, counts, state[p % 2], next, iota && p == 0, paths.max_polls, s);
        sk = dk;
        sv = dv;
    }
    if (sorted) {
        *sorted = {sk, sv};
    } else if (sk != kout) {
        cudaMemcpyAsync(kout, sk, sizeof(uint32_t) * static_cast<size_t>(n),
                        cudaMemcpyDeviceToDevice, s);
        cudaMemcpyAsync(vout, sv, sizeof(uint32_t) * static_cast<size_t>(n),
                        cudaMemcpyDeviceToDevice, s);
    }
    return cudaGetLastError();
}

}  // namespace qk
