// k_sort.cu — stable LSD radix sort of (63-bit Morton key, u32 body index).
//
// Replaces radixSort (src/main/java/com/grumbo/simulation/BarnesHut.java:358-448)
// and its four kernels (SH/compute/radix/bh_radix.comp:12-166): 16 passes of
// 4-bit digits, each pass histogram -> per-bucket scan -> global scan ->
// scatter with an O(256) serial rank loop.  Any stable LSD sort of the same
// keys yields the same permutation, so this is a onesweep sort (Adinets &
// Merrill 2022): 8 passes of 8-bit digits, one kernel per pass.
//   * The eight digit histograms are accumulated by the encode pass
//     (k_prep_scatter); every block scans its pass's histogram beside its own
//     tile's digit counts, one kernel less than scanning them first.
//   * Up to 4,096 pairs one block does all passes (k_sort_small); above:
//   * Each pass kernel takes a tile ticket, ranks its keys per warp (digit
//     peers from one ballot per digit bit, counts per warp and digit in 16
//     bits), publishes the tile's digit counts, resolves its global digit
//     offsets with a decoupled look-back (bounded spin, error word on
//     timeout), stages the pairs digit-ordered in shared memory (the indices are
//     loaded only now, into the registers that the keys leave) and writes them
//     out with coalesced runs.
// What bounds a pass: no one thing; of 8,388,608 pairs it takes 62 us where its
// 201 MB take 30.  The ballots' integer work holds the ALU pipe 55% busy, the
// shared memory 50%, and the rest is the chain of a tile's phases over 3 to 4
// waves of tiles.  Counts in 16 bits read by every lane (before: 32 bits, an
// atomic by one lane and a shuffle), late index loads and 512 threads a tile:
// 39 -> 31 million warp instructions; sort stage, us: 16,000 pairs 60 ->
// 52, 1,048,576 133 -> 123, 8,388,608 559 ->
// 506, 16,777,216 1,008 -> 934.
#include "gbh_common.cuh"

#define LB_FLAG_AGG 0x40000000u
#define LB_FLAG_INC 0x80000000u
#define LB_COUNT_MASK 0x3FFFFFFFu
#define LB_SPIN_LIMIT (1u << 22)
#ifndef LB_WINDOW
#define LB_WINDOW 4
#endif

// A tile of THREADS x ITEMS pairs.
template <int ITEMS, int THREADS>
struct SortSmem {
    uint16_t warp_hist[THREADS / 32][SORT_RADIX + 2];  // [SORT_RADIX]: sentinel bucket of out-of-range items
    uint32_t block_excl[SORT_RADIX];
    uint32_t delta[SORT_RADIX];
    uint2 warp_tot[SORT_RADIX / 32];
    uint32_t tile;
    unsigned long long keys[THREADS * ITEMS];
    uint32_t vals[THREADS * ITEMS];
};

// Warp-level stable ranking of the items, item rounds in slot order: lanes
// with the same digit from one ballot per digit bit (BITS = 9 in a partial
// tile, whose out-of-range slots carry the sentinel digit 256).  All lanes
// read their digit's count so far, then the lowest lane of each digit writes
// the new one.
template <uint32_t SHIFT, int BITS, int ITEMS>
__device__ __forceinline__ void rank_items(const uint64_t (&key)[ITEMS], uint32_t (&rank)[ITEMS],
                                           uint16_t* warp_hist, uint32_t lane, uint32_t seg, uint32_t n) {
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        uint32_t dig = (uint32_t)(key[i] >> SHIFT) & 0xFFu;
        if (BITS > 8 && seg + i * 32 + lane >= n) dig = SORT_RADIX;
        uint32_t peers = 0xffffffffu;
#pragma unroll
        for (int bit = 0; bit < BITS; ++bit) {
            const bool on = (dig >> bit) & 1u;
            const uint32_t m = __ballot_sync(0xffffffffu, on);
            peers &= on ? m : ~m;
        }
        const uint32_t before = __popc(peers & lanemask_lt());
        const uint32_t prev = warp_hist[dig];
        __syncwarp();
        if (before == 0) warp_hist[dig] = (uint16_t)(prev + __popc(peers));
        __syncwarp();
        rank[i] = prev + before;
    }
}

// resident blocks per SM, by the shared memory and registers of a tile
template <int ITEMS, int THREADS>
struct SortBlocks {
    static constexpr int value = THREADS == 512 ? 3 : ITEMS == 8 ? 5 : 6;
};

// One kernel instance per pass: the digit's bit offset is a constant.
template <uint32_t PASS, int ITEMS, int THREADS>
__global__ __launch_bounds__(THREADS, SortBlocks<ITEMS, THREADS>::value) void k_sort_pass(
    StepBuffers b, const uint64_t* __restrict__ kin, const uint32_t* __restrict__ vin, uint64_t* __restrict__ kout,
    uint32_t* __restrict__ vout) {
    constexpr uint32_t pass = PASS;
    constexpr uint32_t TILE = THREADS * ITEMS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SortSmem<ITEMS, THREADS>& S = *reinterpret_cast<SortSmem<ITEMS, THREADS>*>(smem_raw);
    const uint32_t n = b.st->n_new;
    constexpr uint32_t shift = SORT_BITS * PASS;
    const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
    if (threadIdx.x == 0) S.tile = atomicAdd(&b.st->sort_tiles[pass], 1u);
    for (uint32_t i = threadIdx.x; i < (THREADS / 32) * (SORT_RADIX + 2) / 2; i += THREADS) {
        reinterpret_cast<uint32_t*>(&S.warp_hist[0][0])[i] = 0;
    }
    __syncthreads();
    const uint32_t tile = S.tile;
    const uint32_t base = tile * TILE;
    if (base >= n) return;
    uint32_t* lb = b.lookback + ((size_t)pass * b.sort_tiles_cap) * SORT_RADIX;

    // load: warp w owns slots [base + w*32*ITEMS, +32*ITEMS), item i of lane l at +i*32+l
    const uint32_t seg = base + w * 32 * ITEMS;
    const bool full = base + TILE <= n;  // uniform over the block
    uint64_t key[ITEMS];
    uint32_t rank[ITEMS];
    if (full) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) key[i] = kin[seg + i * 32 + lane];
        rank_items<shift, 8>(key, rank, S.warp_hist[w], lane, seg, n);
    } else {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const uint32_t pos = seg + i * 32 + lane;
            key[i] = pos < n ? kin[pos] : ~0ull;
        }
        rank_items<shift, 9>(key, rank, S.warp_hist[w], lane, seg, n);
    }
    __syncthreads();
    // thread d < 256: exclusive prefix of digit d over warps, tile total
    const uint32_t d = threadIdx.x;
    const bool digit = THREADS == SORT_RADIX || d < SORT_RADIX;  // uniform over a warp
    uint32_t total = 0, digit_count = 0, x = 0, y = 0;
    volatile uint32_t* my = lb + (size_t)tile * SORT_RADIX + d;
    if (digit) {
        digit_count = b.hist[pass * SORT_RADIX + d];
#pragma unroll
        for (int ww = 0; ww < THREADS / 32; ++ww) {
            const uint32_t c = S.warp_hist[ww][d];
            S.warp_hist[ww][d] = (uint16_t)total;
            total += c;
        }
        // publish this tile's count for digit d (inclusive when it is the first tile)
        *my = (tile == 0 ? LB_FLAG_INC : LB_FLAG_AGG) | total;
        // block exclusive scans over the digits: of the tile's totals (block_excl)
        // and of the pass's histogram (where each digit begins in the output)
        x = total;
        y = digit_count;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t px = __shfl_up_sync(0xffffffffu, x, o), py = __shfl_up_sync(0xffffffffu, y, o);
            if (lane >= (uint32_t)o) {
                x += px;
                y += py;
            }
        }
        if (lane == 31) S.warp_tot[w] = make_uint2(x, y);
    }
    __syncthreads();
    uint32_t bucket_base = 0;
    if (digit) {
        uint32_t off = 0;
        for (uint32_t i = 0; i < w; ++i) {
            const uint2 t = S.warp_tot[i];
            off += t.x;
            bucket_base += t.y;
        }
        bucket_base += y - digit_count;
        S.block_excl[d] = off + x - total;
    }
    __syncthreads();
    // stage digit-ordered in shared memory (tile-local offsets only), before
    // the look-back: the items leave the registers, and the predecessors
    // have longer to publish their inclusive counts
    {
        uint32_t val[ITEMS];
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const uint32_t pos = seg + i * 32 + lane;
            const uint32_t dg = (uint32_t)(key[i] >> shift) & 0xFFu;
            rank[i] += S.block_excl[dg] + S.warp_hist[w][dg];
            if (full || pos < n) {
                S.keys[rank[i]] = key[i];
                val[i] = vin[pos];
            }
        }
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
            if (full || seg + i * 32 + lane < n) S.vals[rank[i]] = val[i];
    }
    // decoupled look-back for digit d, LB_WINDOW predecessors per round
    // trip; tile 0 always publishes an inclusive count, so the walk ends
    // there at the latest
    uint32_t prefix = 0;
    if (digit && tile > 0) {
        int32_t j = (int32_t)tile - 1;
        uint32_t spins = 0;
        while (true) {
            uint32_t v[LB_WINDOW];
#pragma unroll
            for (int k = 0; k < LB_WINDOW; ++k)
                v[k] = (j - k >= 0) ? *(volatile uint32_t*)(lb + (size_t)(j - k) * SORT_RADIX + d) : LB_FLAG_INC;
            // aggregates add and continue, an inclusive count adds and ends
            // the walk, a word not yet published ends the round
            uint32_t add = 0, used = 0, state = 0;  // state 1: inclusive found, 2: not yet published
#pragma unroll
            for (int k = 0; k < LB_WINDOW; ++k) {
                if (state == 0) {
                    const uint32_t xv = v[k];
                    if (xv & LB_FLAG_INC) {
                        add += xv & LB_COUNT_MASK;
                        state = 1;
                    } else if (xv & LB_FLAG_AGG) {
                        add += xv & LB_COUNT_MASK;
                        ++used;
                    } else {
                        state = 2;
                    }
                }
            }
            prefix += add;
            if (state == 1) break;
            j -= (int32_t)used;
            if (used == 0) {
                if (++spins > LB_SPIN_LIMIT) {
                    set_error(b.st, GBH_DEVERR_SORT_LOOKBACK);
                    break;
                }
                __nanosleep(20);
            }
        }
        *my = LB_FLAG_INC | (prefix + total);
    }
    if (digit) S.delta[d] = bucket_base + prefix - S.block_excl[d];
    __syncthreads();
    bool bad = false;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const uint32_t j = i * THREADS + threadIdx.x;
        if (!full && base + j >= n) break;
        const uint64_t k = S.keys[j];
        const uint32_t dst = S.delta[(uint32_t)(k >> shift) & 0xFFu] + j;
        if (dst < n) {  // holds whenever the digit histograms describe these keys
            kout[dst] = k;
            vout[dst] = S.vals[j];
        } else {
            bad = true;
        }
    }
    if (bad) set_error(b.st, GBH_DEVERR_SORT_LOOKBACK);
}

#define SMALL_THREADS 1024
#define SMALL_MAX (SMALL_THREADS * 4u)

// The whole sort of up to SMALL_THREADS x ITEMS pairs by one block, pairs in
// registers and shared memory between the passes.
template <int ITEMS>
struct SmallSortSmem {
    uint32_t warp_hist[2][SMALL_THREADS / 32][SORT_RADIX / 2 + 1];  // 16-bit counts, then positions; passes alternate
    uint32_t warp_tot[SMALL_THREADS / 32];
    unsigned long long keys[SMALL_THREADS * ITEMS];
    uint32_t vals[SMALL_THREADS * ITEMS];
};

// What bounds it: the latency of a pass, the ranking and four barriers, 1.7 us
// with one item per thread and 4.3 with four, where a kernel per pass takes 6.
// Sort stage, us, eight kernels -> one: 1,000 pairs 48 -> 17, 2,000 50 -> 24,
// 4,000 51 -> 37; with eight items per thread 6,000 51 -> 49, 8,000 52 -> 61: so
// up to four.  A 1,024-body step with three contexts' steps in flight: 39.8 ->
// 34.2 us.
template <int ITEMS>
__global__ __launch_bounds__(SMALL_THREADS) void k_sort_small(StepBuffers b, uint64_t* __restrict__ keys,
                                                              uint32_t* __restrict__ vals) {
    constexpr int PARTS = SMALL_THREADS / SORT_RADIX;  // threads per digit in the scan
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SmallSortSmem<ITEMS>& S = *reinterpret_cast<SmallSortSmem<ITEMS>*>(smem_raw);
    const uint32_t n = min(b.st->n_new, (uint32_t)(SMALL_THREADS * ITEMS));
    const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
    const uint32_t rounds = (n + SMALL_THREADS - 1) / SMALL_THREADS;  // items of each thread in use
    const uint32_t seg = w * 32 * rounds + lane;                      // item i of the thread at seg + 32 i
    uint64_t key[ITEMS];
    uint32_t val[ITEMS], rank[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
        if (i < rounds && seg + i * 32 < n) {
            key[i] = keys[seg + i * 32];
            val[i] = vals[seg + i * 32];
        }
    for (uint32_t i = threadIdx.x; i < sizeof(S.warp_hist) / 4; i += SMALL_THREADS) (&S.warp_hist[0][0][0])[i] = 0;
    __syncthreads();
#pragma unroll 1
    for (uint32_t pass = 0; pass < SORT_PASSES; ++pass) {
        uint16_t* hist = reinterpret_cast<uint16_t*>(S.warp_hist[pass & 1][w]);
        const uint32_t shift = SORT_BITS * pass;
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            if (i >= rounds) break;
            const bool in = seg + i * 32 < n;
            const uint32_t dig = (uint32_t)(key[i] >> shift) & 0xFFu;
            uint32_t peers = __ballot_sync(0xffffffffu, in);
#pragma unroll
            for (int bit = 0; bit < SORT_BITS; ++bit) {
                const bool on = (dig >> bit) & 1u;
                const uint32_t m = __ballot_sync(0xffffffffu, on);
                peers &= on ? m : ~m;
            }
            const uint32_t before = __popc(peers & lanemask_lt());
            const uint32_t prev = hist[dig];
            __syncwarp();
            if (in && before == 0) hist[dig] = (uint16_t)(prev + __popc(peers));
            __syncwarp();
            rank[i] = prev + before;
        }
        __syncthreads();
        // counts -> positions: one exclusive scan over (digit, warp); each
        // thread holds the counts of a digit in some of the warps
        {
            constexpr int ROWS = SMALL_THREADS / 32 / PARTS;
            const uint32_t d = threadIdx.x / PARTS, first = threadIdx.x % PARTS * ROWS;
            uint32_t sum = 0, c[ROWS];
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                c[r] = reinterpret_cast<const uint16_t*>(S.warp_hist[pass & 1][first + r])[d];
                sum += c[r];
            }
            uint32_t x = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t p = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= (uint32_t)o) x += p;
            }
            if (lane == 31) S.warp_tot[w] = x;
            __syncthreads();
            uint32_t t = lane < SMALL_THREADS / 32 ? S.warp_tot[lane] : 0u;
            const uint32_t own = t;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t p = __shfl_up_sync(0xffffffffu, t, o);
                if (lane >= (uint32_t)o) t += p;
            }
            uint32_t at = __shfl_sync(0xffffffffu, t - own, w) + x - sum;
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                reinterpret_cast<uint16_t*>(S.warp_hist[pass & 1][first + r])[d] = (uint16_t)at;
                at += c[r];
            }
            // the next pass counts in the other buffer, last read a pass ago
            for (uint32_t i = threadIdx.x; i < sizeof(S.warp_hist) / 8; i += SMALL_THREADS)
                (&S.warp_hist[(pass + 1) & 1][0][0])[i] = 0;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            if (i >= rounds) break;
            if (seg + i * 32 < n) {
                const uint32_t pos = hist[(uint32_t)(key[i] >> shift) & 0xFFu] + rank[i];
                if (pass + 1 == SORT_PASSES) {
                    keys[pos] = key[i];
                    vals[pos] = val[i];
                } else {
                    S.keys[pos] = key[i];
                    S.vals[pos] = val[i];
                }
            }
        }
        if (pass + 1 == SORT_PASSES) break;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            if (i >= rounds) break;
            if (seg + i * 32 < n) {
                key[i] = S.keys[seg + i * 32];
                val[i] = S.vals[seg + i * 32];
            }
        }
    }
}

// The eight digit histograms of `n` keys (for a sort whose keys were not
// written by the step's encode pass) and the live count the passes read.
__global__ void k_sort_hist(const uint64_t* __restrict__ keys, uint32_t n, uint32_t* __restrict__ hist,
                            DevState* __restrict__ st) {
    __shared__ uint32_t h[SORT_PASSES * SORT_RADIX];
    for (uint32_t i = threadIdx.x; i < SORT_PASSES * SORT_RADIX; i += blockDim.x) h[i] = 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) st->n_new = n;
    __syncthreads();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint64_t k = keys[i];
#pragma unroll
        for (int p = 0; p < SORT_PASSES; ++p) atomicAdd(&h[p * SORT_RADIX + ((k >> (8 * p)) & 0xFF)], 1u);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < SORT_PASSES * SORT_RADIX; i += blockDim.x)
        if (h[i]) atomicAdd(&hist[i], h[i]);
}

void launch_sort_hist(const uint64_t* keys, uint32_t n, uint32_t* hist, DevState* st, uint32_t num_sms,
                      cudaStream_t s) {
    const uint32_t blocks = min((n + 255) / 256, num_sms * 4u);
    k_sort_hist<<<blocks > 0 ? blocks : 1, 256, 0, s>>>(keys, n, hist, st);
}

// Pairs per tile of a sort of up to `n` pairs, in units of 256.  A small sort is
// eight chains of latency (load, rank item after item, look back, scatter),
// shorter with small tiles, which also reach more SMs; a large one wants long
// runs per digit.  Sort stage of an eager step, us, with 256 threads of 4, 8 and
// 16 items: 1,000 pairs 59, 58, 75; 16,000 64, 75, 91; 150,000 84, 87, 95;
// 300,000 105, 93, 108; 600,000 140, 114, 110.  Tiles of 4,096 pairs are ranked
// by 512 threads (16 items of 256 threads: 127 for 123 us at 1,048,576 pairs,
// 531 for 506 at 8,388,608).  Tiles of 8,192 are faster alone where they fit the
// SMs at once and tiles of 4,096 just do not (170 for 195 us at 2,000,000 pairs,
// but 252 for 240 at 3,000,000), and slower where steps of several contexts
// share the SMs (a 2,000,003-body step 1,610 for 1,587 us).
#define SORT_ONE_BLOCK 32u  // of sort_items: the whole sort by one block (one tile of 8,192 in the counts)
uint32_t sort_items_for(uint32_t n) {
    if (n <= SMALL_MAX) return SORT_ONE_BLOCK;
    return n <= 200000u ? 4u : n <= 500000u ? 8u : 16u;
}

typedef void (*sort_pass_fn)(StepBuffers, const uint64_t*, const uint32_t*, uint64_t*, uint32_t*);
static_assert(SORT_PASSES == 8, "one kernel instance per pass");
template <int ITEMS, int THREADS>
struct SortPasses {
    static constexpr sort_pass_fn fn[SORT_PASSES] = {
        k_sort_pass<0, ITEMS, THREADS>, k_sort_pass<1, ITEMS, THREADS>, k_sort_pass<2, ITEMS, THREADS>,
        k_sort_pass<3, ITEMS, THREADS>, k_sort_pass<4, ITEMS, THREADS>, k_sort_pass<5, ITEMS, THREADS>,
        k_sort_pass<6, ITEMS, THREADS>, k_sort_pass<7, ITEMS, THREADS>};
};

template <int ITEMS, int THREADS>
static void setup_passes() {
    for (sort_pass_fn f : SortPasses<ITEMS, THREADS>::fn)
        cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SortSmem<ITEMS, THREADS>));
}

static const void* small_sort(uint32_t n, uint32_t* smem) {
    if (n <= SMALL_THREADS) return *smem = sizeof(SmallSortSmem<1>), (const void*)k_sort_small<1>;
    return *smem = sizeof(SmallSortSmem<4>), (const void*)k_sort_small<4>;
}

void sort_setup(uint32_t items) {
    if (items == SORT_ONE_BLOCK) {
        for (uint32_t n : {SMALL_THREADS * 1u, SMALL_MAX}) {
            uint32_t smem;
            const void* f = small_sort(n, &smem);
            cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        }
    } else if (items == 4)
        setup_passes<4, 256>();
    else if (items == 8)
        setup_passes<8, 256>();
    else
        setup_passes<8, 512>();
}

template <int ITEMS, int THREADS>
static void launch_passes(const StepBuffers& b, cudaStream_t s) {
    // keys/index of the live bodies are in the *_in buffers (the compaction
    // swap already happened); 8 ping-pong passes through *_out end there again
    const uint64_t* kin = b.keys_in;
    const uint32_t* vin = b.idx_in;
    uint64_t* kt = b.keys_out;
    uint32_t* vt = b.idx_out;
    for (sort_pass_fn f : SortPasses<ITEMS, THREADS>::fn) {
        f<<<b.sort_tiles_cap, THREADS, sizeof(SortSmem<ITEMS, THREADS>), s>>>(b, kin, vin, kt, vt);
        const uint64_t* nk = kt;
        const uint32_t* nv = vt;
        kt = const_cast<uint64_t*>(kin);
        vt = const_cast<uint32_t*>(vin);
        kin = nk;
        vin = nv;
    }
}

void launch_sort(const StepBuffers& b, cudaStream_t s) {
    if (b.sort_items == SORT_ONE_BLOCK) {
        uint32_t smem;
        const void* f = small_sort(b.N, &smem);
        void* args[] = {(void*)&b, (void*)&b.keys_in, (void*)&b.idx_in};
        cudaLaunchKernel(f, dim3(1), dim3(SMALL_THREADS), args, smem, s);
    } else if (b.sort_items == 4)
        launch_passes<4, 256>(b, s);
    else if (b.sort_items == 8)
        launch_passes<8, 256>(b, s);
    else
        launch_passes<8, 512>(b, s);
}
