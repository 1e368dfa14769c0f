// pt_kernels.cu - sm_103a kernels of the PandemicThrust daily simulation step.
//
// Stage map (reference = PandemicThrust/PandemicThrust/PandemicSim.cu):
//   setup   household types/sizes, household scan+scatter, workplace/school draw,
//           workplace buckets                         (setupSim, :146-208)
//   sweep   recover + 16 status bins + ordered infected list, one pass
//           (kernel_countInfectedStatusAndRecover :2097-2192 + copy_if :2207-2224)
//   sched   schedule keys + digit histograms          (:2972-3022 / :2082-2094)
//   bucket  a stable LSD radix sort of the (key, person) entries, whose last pass also
//           writes each bucket's start and size (CUB sort + lower_bound, :1212-1248,
//           :1313-1354)
//   infect  contacts and infection draws; the first attempt in (position, slot)
//           order claims each (victim, strain)        (:3236-3379)
//   apply   winners write status, day, generation     (:3048-3067)
//
// Waits between thread blocks (decoupled look-back) are bounded: after kSpinLimit
// polls the block records an error in Scalars::error and carries on, so a fault in
// the ordering logic surfaces as PT_ERR_TIMEOUT on the host instead of a hang.
#include <cstdio>
#include <climits>
#include <atomic>
#include <tuple>
#include "pt_kernels.h"
#include "pt_device.cuh"
#include "pt_lookback.cuh"

namespace ptk {

static std::atomic<uint64_t> g_launches{0};
uint64_t launches() { return g_launches.load(); }
void add_launches(uint64_t n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
static inline void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

// The next node of a graph's chain.
template <class Add>
static cudaError_t chain_node(DayQueue &q, Add add)
{
    cudaGraphNode_t node = nullptr;
    const cudaError_t e = add(&node, q.last ? &q.last : nullptr, q.last ? 1 : 0);
    if (e == cudaSuccess) q.last = node;
    return e;
}

// A kernel launch to the queue's stream, or its node.
template <class... P, class... A>
static cudaError_t queue_kernel(DayQueue &q, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, const A &...args)
{
    std::tuple<P...> values(args...);   // in the kernel's own types
    return std::apply(
        [&](P &...v) {
            void *params[] = {(void *)&v...};
            if (!q.graph) {
                count_launch();
                return cudaLaunchKernel((const void *)kernel, grid, block, params, smem, q.stream);
            }
            cudaKernelNodeParams n = {};
            n.func = (void *)kernel;
            n.gridDim = grid;
            n.blockDim = block;
            n.sharedMemBytes = (unsigned)smem;
            n.kernelParams = params;
            q.kernels++;
            return chain_node(q, [&](cudaGraphNode_t *node, const cudaGraphNode_t *after, size_t count) {
                return cudaGraphAddKernelNode(node, q.graph, after, count, &n);
            });
        },
        values);
}

// `words` words of `value` at p.
static cudaError_t queue_fill(DayQueue &q, uint32_t *p, uint32_t value, size_t words)
{
    if (!q.graph) return cudaMemsetAsync(p, (int)(value & 0xFFu), words * 4, q.stream);   // (its bytes are alike)
    cudaMemsetParams m = {};
    m.dst = p;
    m.value = value;
    m.elementSize = 4;
    m.width = words;
    m.height = 1;
    return chain_node(q, [&](cudaGraphNode_t *node, const cudaGraphNode_t *after, size_t count) {
        return cudaGraphAddMemsetNode(node, q.graph, after, count, &m);
    });
}

int sm_count()
{
    // initialised once, safely when several host threads drive engines
    static const int n = [] {
        int dev = 0, v = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        return v > 0 ? v : 1;
    }();
    return n;
}

static inline int div_up(long long a, long long b) { return (int)((a + b - 1) / b); }

// ================================================================== setup
// kernel_householdTypeAssignment + hh_peopleCount_functor (PandemicSim.cu:2329-2357,
// :3579-3605): counter g -> households 4g..4g+3.  Writes each household's size and
// counts adults and persons.
__global__ void k_household_types(SimConst c, uint8_t *types, int32_t *sizes, int *adults, int *persons)
{
    const TfKey key = make_key(c);
    int local_adults = 0, local_persons = 0;
    const int G = c.H / 4;
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g <= G; g += gridDim.x * blockDim.x) {
        uint32_t w[4];
        tf2x64(key, (uint64_t)g, w);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            int h = 4 * g + i;
            if (h < c.H) {
                int t = fish_household_type(w[i]);
                types[h] = (uint8_t)t;
                sizes[h] = c_hh_adults[t] + c_hh_children[t];
                local_adults += c_hh_adults[t];
                local_persons += c_hh_adults[t] + c_hh_children[t];
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        local_adults += __shfl_xor_sync(0xffffffffu, local_adults, o);
        local_persons += __shfl_xor_sync(0xffffffffu, local_persons, o);
    }
    if ((threadIdx.x & 31) == 0 && local_adults) atomicAdd(adults, local_adults);
    if ((threadIdx.x & 31) == 0 && local_persons) atomicAdd(persons, local_persons);
}

cudaError_t launch_household_types(const SimConst &c, uint8_t *types, int32_t *sizes, int *adults, int *persons,
                                   cudaStream_t s)
{
    int G = c.H / 4 + 1;
    int blocks = std::min(div_up(G, 256), sm_count() * 16);
    k_household_types<<<blocks, 256, 0, s>>>(c, types, sizes, adults, persons);
    count_launch();
    return cudaGetLastError();
}

// Generic exclusive scan (single pass, decoupled look-back): out[i] = sum in[0..i),
// out[n] = total.  With clear_in the input is zeroed after it is read.  With
// passes > 0, in[] is a histogram over keys 0..n-1 and the scan also accumulates,
// for each radix pass p, the histogram of the key's digit p (dbits bits) weighted by
// the count (digit_hist[p][256]), from which the radix sort takes its digit bases.
constexpr int kScanThreads = 256, kScanItems = 16, kScanTile = kScanThreads * kScanItems;
static_assert(kScanTile == kScanTileEntries, "the host sizes the scan look-back words by kScanTileEntries");
constexpr int kMaxRadixPasses = 4;

__global__ void __launch_bounds__(kScanThreads) k_scan(const int32_t *in, int32_t *out, int n, int clear_in,
                                                       LookBack lb, const int *skip, int passes, int dbits,
                                                       int *digit_hist)
{
    if (skip && *(volatile const int *)skip) return;
    __shared__ int s_dh[kMaxRadixPasses][256];
    if (passes > 0) {
        for (int i = threadIdx.x; i < kMaxRadixPasses * 256; i += blockDim.x) (&s_dh[0][0])[i] = 0;
    }
    int tile;
    unsigned epoch;
    lookback_begin(lb, tile, epoch);
    const long long base = (long long)tile * kScanTile + (long long)threadIdx.x * kScanItems;
    int v[kScanItems];
    int sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        long long i = base + k;
        v[k] = i < n ? in[i] : 0;
        sum += v[k];
    }
    if (clear_in) {
#pragma unroll
        for (int k = 0; k < kScanItems; k++) {
            long long i = base + k;
            if (i < n) ((int32_t *)in)[i] = 0;
        }
    }
    if (passes > 0) {
#pragma unroll
        for (int k = 0; k < kScanItems; k++) {
            if (v[k] > 0) {
                unsigned key = (unsigned)(base + k);
                for (int p = 0; p < passes; p++)
                    atomicAdd(&s_dh[p][(key >> (dbits * p)) & ((1u << dbits) - 1u)], v[k]);
            }
        }
    }
    int total;
    int excl = block_exclusive_scan<kScanThreads, int>(sum, total);
    __shared__ unsigned s_prefix;
    if (threadIdx.x < 32) {
        const unsigned e = lookback_publish_warp(lb, epoch, tile, (unsigned)total);
        if (threadIdx.x == 0) s_prefix = e;
    }
    __syncthreads();
    int run = (int)s_prefix + excl;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        long long i = base + k;
        if (i < n) out[i] = run;
        run += v[k];
    }
    if (tile == (int)gridDim.x - 1 && threadIdx.x == 0) out[n] = (int)s_prefix + total;
    if (passes > 0) {
        for (int p = 0; p < passes; p++) {
            int c = s_dh[p][threadIdx.x];
            if (c) atomicAdd(&digit_hist[p * 256 + threadIdx.x], c);
        }
    }
    lookback_end(lb);
}

cudaError_t launch_scan_exclusive(const int32_t *in, int32_t *out, int n, int clear_in,
                                  unsigned long long *tiles, int *ctl, int *error,
                                  const int *skip, int passes, int dbits, int *digit_hist, cudaStream_t s)
{
    int blocks = std::max(1, div_up(n, kScanTile));
    LookBack lb;
    lb.tiles = tiles;
    lb.ctl = ctl;
    lb.error = error;
    k_scan<<<blocks, kScanThreads, 0, s>>>(in, out, n, clear_in, lb, skip, passes, dbits, digit_hist);
    count_launch();
    return cudaGetLastError();
}

// Exclusive scan of each pass's 256-bin digit histogram -> digit bases; clears the
// histograms for the next sort.
// With stripes > 1 the histograms are split over `stripes` copies of 4 x 256 bins
// (producers spread their updates over the copies); the copies are summed.
__global__ void k_digit_bases(int *digit_hist, int *digit_base, int passes, int stripes, const int *skip)
{
    if (skip && *(volatile const int *)skip) return;
    for (int p = 0; p < passes; p++) {
        int v = 0;
        for (int st = 0; st < stripes; st++) {
            int *h = &digit_hist[(st * kMaxRadixPasses + p) * 256 + threadIdx.x];
            v += *h;
            *h = 0;
        }
        int total;
        int excl = block_exclusive_scan<256, int>(v, total);
        digit_base[p * 256 + threadIdx.x] = excl;
    }
}

// kernel_generateHouseholds (PandemicSim.cu:2490-2531): adults first (AGE_ADULT),
// then children with the AGE_5 placeholder.  Slots of type 0xFF hold an instance's
// padding persons and are skipped.
__global__ void k_generate_households(const uint8_t *types, const int32_t *hh_offset, int slots, int32_t *household,
                                      uint8_t *age)
{
    for (int h = blockIdx.x * blockDim.x + threadIdx.x; h < slots; h += gridDim.x * blockDim.x) {
        int t = types[h];
        if (t > 8) continue;
        int off = hh_offset[h];
        int na = c_hh_adults[t], nc = c_hh_children[t];
        for (int i = 0; i < na + nc; i++) {
            household[off + i] = h;
            age[off + i] = i < na ? 5 : 0;
        }
    }
}

cudaError_t launch_generate_households(const uint8_t *types, const int32_t *hh_offset, int slots, int32_t *household,
                                       uint8_t *age, cudaStream_t s)
{
    int blocks = std::max(1, std::min(div_up(slots, 256), sm_count() * 16));
    k_generate_households<<<blocks, 256, 0, s>>>(types, hh_offset, slots, household, age);
    count_launch();
    return cudaGetLastError();
}

// assignWorkplaceFunctor (PandemicSim.cu:3750-3778): counter W0 + g -> persons
// 4g..4g+3; adults draw a workplace, children an age band and school.  loc_base turns
// the instance's location number into a global one.
__global__ void k_assign_workplaces(SimConst c, uint8_t *age, int32_t *workplace, int loc_base)
{
    const TfKey key = make_key(c);
    const int G = c.N / 4;
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g <= G; g += gridDim.x * blockDim.x) {
        uint32_t w[4];
        tf2x64(key, c.workplace_offset + (uint64_t)g, w);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            int p = 4 * g + i;
            if (p < c.N) {
                int a = age[p];
                if (a == 5) {
                    workplace[p] = loc_base + fish_workplace(c, w[i]);
                } else {
                    workplace[p] = loc_base + fish_school_and_age(c, w[i], &a);
                    age[p] = (uint8_t)a;
                }
            }
        }
    }
}

cudaError_t launch_assign_workplaces(const SimConst &c, uint8_t *age, int32_t *workplace, int loc_base, cudaStream_t s)
{
    int blocks = std::min(div_up(c.N / 4 + 1, 256), sm_count() * 16);
    k_assign_workplaces<<<blocks, 256, 0, s>>>(c, age, workplace, loc_base);
    count_launch();
    return cudaGetLastError();
}

// Padding of a batch, one block per instance.  Without `persons`: the instance's
// last household slot gets type 0xFF and the padding count as its size, so one scan
// of all slots yields tile-aligned person bases.  With `persons`: the padding persons
// get no household, no age and the spare location, which sorts them behind every
// real workplace.
__global__ void k_batch_padding(const InstConst *ic, int K, int P, uint8_t *types, int32_t *sizes,
                                int32_t *household, uint8_t *age, int32_t *workplace, int spare, int persons)
{
    const int k = blockIdx.x;
    if (k >= K) return;
    const InstConst &c = ic[k];
    const int end = k + 1 < K ? ic[k + 1].pbase : P;
    const int first = c.pbase + c.c.N;
    if (!persons) {
        if (threadIdx.x == 0) {
            types[c.hbase + c.c.H] = 0xFF;
            sizes[c.hbase + c.c.H] = end - first;
        }
        return;
    }
    for (int p = first + threadIdx.x; p < end; p += blockDim.x) {
        household[p] = -1;
        age[p] = 0;
        workplace[p] = spare;
    }
}

cudaError_t launch_batch_padding(const DevArrays &d, uint8_t *types, int32_t *sizes, int spare_location, bool persons,
                                 cudaStream_t s)
{
    k_batch_padding<<<d.K, 256, 0, s>>>(d.ic, d.K, d.P, types, sizes, d.household, d.age, d.workplace,
                                        spare_location, persons ? 1 : 0);
    count_launch();
    return cudaGetLastError();
}

__global__ void k_count_keys(const int32_t *keys, int n, int32_t *count)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        atomicAdd(&count[keys[i]], 1);
}

cudaError_t launch_count_keys(const int32_t *keys, int n, int32_t *count, cudaStream_t s)
{
    int blocks = std::min(div_up(n, 256), sm_count() * 16);
    k_count_keys<<<std::max(blocks, 1), 256, 0, s>>>(keys, n, count);
    count_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------------------ radix sort
// Bucket tables: the reference sorts (key, person) pairs stably by key and takes
// lower bounds (CUB radix sort + thrust::lower_bound, PandemicSim.cu:1212-1248,
// :3835-3862), so every bucket lists its persons in ascending id order.  This stable
// LSD radix sort gives the same table: the fewest passes of at most 8 bits, the key's
// bits spread evenly over them.  Entries enter the first pass in ascending person
// order; each pass ranks a tile of 4096 (key, value) pairs by digit (warp-blocked, so
// the rank is stable), places the tile in shared memory in digit order, finds the
// tile's global position per digit by a decoupled look-back over earlier tiles (one
// thread per digit) and writes each digit's run with consecutive threads.
//
// What bounds it (24M pairs on a GB300, each part left out in turn): reading and
// writing 16 bytes an entry 64 us, ranking 50, look-back one tile a step 45, scattered
// instead of linear writes 12.  So the look-back reads four predecessors a step, and
// after the tile is placed, when more of them are ready (143 us instead of 171), and only
// the digits a pass has publish and look (128 of 256 where it sorts 7 bits: weekdays of 48
// instances 77.5 -> 75.2 ms a run); and three blocks of 256 threads an SM (80 registers) do better than four (64, 163 us),
// 16 x 384 or 512 threads (154, 170) or 12 entries a thread (187).  Ranking by ballots
// (160), match (208) or one warp barrier a round with three word sets (160) is slower.
constexpr int kRadixThreads = 256, kRadixItems = 16, kRadixWarps = kRadixThreads / 32;
constexpr int kRadixBlocksPerSm = 3;
constexpr int kRadixTile = kRadixThreads * kRadixItems, kRadixWarpItems = kRadixItems * 32;
static_assert(kRadixTile == kRadixTileEntries, "the host sizes the radix look-back words by kRadixTileEntries");
static_assert(kRadixWarpItems % kRegionChunk == 0, "a warp's entries start at a chunk_region word");
constexpr int kLookBackStep = 4;

// What a pass reads: plain keys with implicit values (entry i is person i); a day's first
// pass (the schedule's regions, or the schedule keys of a dense instance); pairs.
enum RadixIn { kInKeys = 0, kInDay = 1, kInPairs = 2 };
// What it writes: pairs; the values only (the last pass); those and the bucket table
// (a day's last pass).
enum RadixOut { kOutPairs = 0, kOutValues = 1, kOutTable = 2 };
constexpr uint32_t kDropped = 0xFFFFFFFFu;   // value of an entry a pass leaves out (no person id is this)

struct RadixPass {
    const uint32_t *keys;
    const uint2 *in;
    uint2 *out_pairs;
    uint32_t *out_values;
    uint2 *table;
    int E, pass, passes, dbits;
    const int *digit_base;
    RadixSegments sg;
    unsigned long long *status, *ctl;
    int *error;
    const int *skip;
};

// The tile a block works on: its ticket, its segment and what it reads there.
struct RadixTile {
    int tile;               // ticket
    unsigned epoch;         // the launch's
    int seg, stile;         // segment, tile within the segment
    int base, count;        // the segment's first entry slot and entries
    int dense;              // day's first pass: the segment reads the schedule keys
    int nk, pb, bb;         // dense: the instance's persons, first person; bb: its first bucket
    int rlast;              // day's first pass: the segment's last region
};

// Exclusive prefix of the tile's digit d over the segment's earlier tiles: words of
// kLookBackStep predecessors a step, in order, up to the nearest inclusive one.
__device__ __forceinline__ int radix_look_back(volatile unsigned long long *st, unsigned epoch, int tile, int first,
                                               int d, int *error)
{
    int excl = 0, t = tile - 1;
    long long spins = 0;
    for (;;) {
        unsigned long long w[kLookBackStep];
#pragma unroll
        for (int q = 0; q < kLookBackStep; q++)
            w[q] = t - q >= first ? st[(size_t)(t - q) * 256 + d] : lb_word(epoch, 2, 0u);
        int took = 0;
#pragma unroll
        for (int q = 0; q < kLookBackStep; q++) {
            const unsigned flag = (unsigned)(w[q] >> 32) & 3u;
            if (took == q && (unsigned)(w[q] >> 34) == epoch && flag != 0) {
                excl += (int)(unsigned)w[q];
                if (flag == 2) return excl;
                took = q + 1;
            }
        }
        t -= took;
        if (took == 0) {
            if (++spins > kSpinLimit) {
                atomicExch(error, 2);
                return excl;
            }
            __nanosleep(32);
        }
    }
}

// One stable pass over dbits bits of the keys.  Persistent blocks take tiles from a
// ticket in order until the entries run out, so a short input costs no idle blocks.
// Look-back words carry the launch epoch (see lb_word), so they need no reset between
// passes; ticket and epoch are one word, which a block draws from when it starts and,
// while it works on a tile, for its next one.  Every block that takes part draws until
// a ticket is past the last tile, so the draw number tiles + blocks is the launch's last,
// and it sets the ticket back and the epoch on.
//
// A short input is a chain of latencies: 200,000 entries take 10 us, 17 with the ticket
// drawn between tiles, a finish count and an entry's region looked up just before its load.
//
// Segmented sorts (sg.tile_prefix set): segment k's entries lie at
// [ic[k].kbase, ic[k].kbase + is[k].marked) and are ordered within the segment only,
// with digit bases of their own (digit_base[(k * passes + pass) * 256 + d]).  The
// segments' tiles are numbered consecutively (segment k owns tiles
// [tile_prefix[k], tile_prefix[k + 1])), and the look-back of a segment's first tile
// starts from zero.  Unsegmented sorts are one segment [0, E).
template <int IN, int OUT>
__global__ void __launch_bounds__(kRadixThreads, kRadixBlocksPerSm) k_radix_pass(RadixPass a)
{
    const RadixSegments &sg = a.sg;
    const int *const tprefix = IN == kInDay ? sg.tile_prefix0 : sg.tile_prefix;
    const int skip = a.skip ? *(volatile const int *)a.skip : 0;
    const int tiles = sg.tile_prefix ? *(volatile const int *)&tprefix[sg.segments] : (a.E + kRadixTile - 1) / kRadixTile;
    // only as many blocks as there are tiles take part
    const int active = min(tiles, (int)gridDim.x);
    if (skip || (int)blockIdx.x >= active) return;
    extern __shared__ __align__(16) uint8_t radix_smem[];
    uint2 *const s_pair = reinterpret_cast<uint2 *>(radix_smem);                              // kRadixTile
    unsigned *const s_peers = reinterpret_cast<unsigned *>(radix_smem + kRadixTile * 8);      // kRadixWarps x 256
    // counts and places within the tile (at most 4096) fit 16 bits
    uint16_t (*const s_hist)[256] = reinterpret_cast<uint16_t (*)[256]>(radix_smem + kRadixTile * 8 + kRadixWarps * 1024);
    __shared__ RadixTile s_t;
    __shared__ int s_base[256];   // global position of digit d's entries, less its tile-local start
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned bit = 1u << lane, lt = bit - 1u, dmask = (1u << a.dbits) - 1u;
    const int shift = a.dbits * a.pass;
    uint16_t *const hist = s_hist[warp];
    unsigned *const peer = s_peers + warp * 256;   // the lanes of a round holding each digit; zero between rounds
    for (int i = threadIdx.x; i < kRadixWarps * 256; i += kRadixThreads) {
        (&s_hist[0][0])[i] = 0;
        s_peers[i] = 0u;
    }
    unsigned long long drawn = 0;   // warp 0's lane 0: epoch (high half) and next ticket
    if (threadIdx.x == 0) drawn = atomicAdd(a.ctl, 1ull);
    for (;;) {
        if (warp == 0) {
            drawn = __shfl_sync(0xffffffffu, drawn, 0);
            const int t = (int)(unsigned)drawn;
            RadixTile r = {t, (unsigned)(drawn >> 32) & 0x3FFFFFFFu, 0, t, 0, a.E, 0, 0, 0, 0, 0};
            if (sg.tile_prefix && t < tiles) {
                // the segment owning tile t: the last k with tprefix[k] <= t, 32 probes a step
                int lo = 0, hi = sg.segments;   // in [lo, hi)
                while (hi - lo > 1) {
                    const int step = (hi - lo + 31) / 32, i = lo + lane * step;
                    const unsigned below = __ballot_sync(0xffffffffu, i < hi && tprefix[i] <= t);
                    lo += (31 - __clz(below)) * step;   // lane 0's probe always holds
                    hi = min(hi, lo + step);
                }
                const InstConst &k = sg.ic[lo];
                r.seg = lo;
                r.stile = t - tprefix[lo];
                r.base = (int)k.kbase;
                r.count = sg.is[lo].marked;
                if (IN == kInDay || OUT == kOutTable) r.bb = k.bbase[sg.weekend];
                if (IN == kInDay) {
                    r.rlast = k.pend / sg.region_persons - 1;
                    if (sg.is[lo].dense) {
                        r.dense = 1;
                        r.nk = k.c.N;
                        r.pb = k.pbase;
                        r.count = (sg.weekend ? 3 : 2) * r.nk;   // every schedule key of the instance
                    }
                }
            }
            if (lane == 0) s_t = r;
        }
        __syncthreads();   // (also ends the last tile's use of shared memory)
        const int tile = s_t.tile, stile = s_t.stile, sbase = s_t.base, scount = s_t.count, table_base = s_t.bb;
        const int rlast = s_t.rlast;
        const unsigned epoch = s_t.epoch;
        if (tile >= tiles) break;
        if (threadIdx.x == 0) drawn = atomicAdd(a.ctl, 1ull);
        const int first = stile * kRadixTile + warp * kRadixWarpItems + lane;   // index within the segment
        const bool full = (stile + 1) * kRadixTile <= scount;
        bool whole = full;   // every entry of the tile takes part
        uint2 kv[kRadixItems];
        if (IN == kInDay && s_t.dense) {
            // the instance's schedule keys, persons implicit (weekday hour-major: entry
            // i < N is person i's hour-0 key, i >= N person i - N's hour-1 key; weekend
            // person-major, three per person), instance-local bucket keys; an entry of
            // an unmarked bucket gets the value kDropped and is left out
            const int nk = s_t.nk, pb = s_t.pb, bb = s_t.bb;
            whole = false;
#pragma unroll
            for (int j = 0; j < kRadixItems; j++) {
                const int i = first + 32 * j;
                const bool in = full || i < scount;
                const int kg = in ? sg.day_keys[sbase + i] : bb;
                const bool marked = in && ((sg.mark[kg >> 5] >> (kg & 31)) & 1u);
                kv[j].x = (uint32_t)(kg - bb);
                kv[j].y = marked ? (uint32_t)(pb + (sg.weekend ? i / 3 : (i < nk ? i : i - nk))) : kDropped;
            }
        } else if (IN == kInDay) {
            // the schedule's entries, region after region: entry i of the segment is entry
            // i - region_prefix[r] of its region r, whose slots start at 3 C r.  The record
            // of a chunk names the region of its first entry, that region's prefix and the
            // ends of it and of the next one; the records of the warp's chunks are read
            // together, and only entries past those two regions look further.
            constexpr int kChunks = kRadixWarpItems / kRegionChunk, kPer = kRadixItems / kChunks;
            const int c0 = stile * kRadixTile + warp * kRadixWarpItems;
            int4 rec[kChunks];
#pragma unroll
            for (int q = 0; q < kChunks; q++)
                rec[q] = c0 + q * kRegionChunk < scount ? sg.chunk_region[(sbase + c0) / kRegionChunk + q]
                                                        : make_int4(0, 0, INT_MAX, INT_MAX);
            // where each entry lies first, then all loads together
#pragma unroll
            for (int j = 0; j < kRadixItems; j++) {
                const int i = first + 32 * j;
                kv[j] = make_uint2(0u, kDropped);
                if (full || i < scount) {
                    const int4 c = rec[j / kPer];
                    int r = c.x, at = c.y;
                    if (i >= c.z) {
                        r++;
                        at = c.z;
                        if (i >= c.w) {
                            int next = c.w;
                            do {   // ends: the last region's end is scount
                                r++;
                                at = next;
                                next = r < rlast ? sg.region_prefix[r + 1] : scount;
                            } while (i >= next);
                        }
                    }
                    kv[j].x = 3u * (unsigned)r * (unsigned)sg.region_persons + (unsigned)(i - at);
                }
            }
#pragma unroll
            for (int j = 0; j < kRadixItems; j++)
                if (full || first + 32 * j < scount) kv[j] = a.in[kv[j].x];
        } else {
#pragma unroll
            for (int j = 0; j < kRadixItems; j++) {
                const int i = first + 32 * j;
                kv[j] = make_uint2(0u, kDropped);
                if (full || i < scount) kv[j] = IN == kInKeys ? make_uint2(a.keys[sbase + i], (uint32_t)i) : a.in[sbase + i];
            }
        }
        // Rank: each entry's place among the warp's entries of its digit (earlier rounds,
        // then lanes).  The lanes of a round that hold a digit meet in its shared word; the
        // lowest of them clears the word, advances the warp's count of the digit and
        // broadcasts the count before it.
        unsigned place[kRadixItems];
        if (whole) {
#pragma unroll
            for (int j = 0; j < kRadixItems; j++) {
                const unsigned d = (kv[j].x >> shift) & dmask;
                atomicOr(&peer[d], bit);
                __syncwarp();
                const unsigned peers = *(volatile unsigned *)&peer[d];
                const unsigned rank = __popc(peers & lt);
                int before = 0;
                if (rank == 0) before = hist[d];
                __syncwarp();
                if (rank == 0) {
                    peer[d] = 0u;
                    hist[d] = (uint16_t)(before + __popc(peers));
                }
                before = __shfl_sync(0xffffffffu, before, __ffs(peers) - 1);
                __syncwarp();
                place[j] = (unsigned)before + rank;
            }
        } else {
#pragma unroll
            for (int j = 0; j < kRadixItems; j++) {
                const bool ok = kv[j].y != kDropped;
                const unsigned d = (kv[j].x >> shift) & dmask;
                if (ok) atomicOr(&peer[d], bit);
                __syncwarp();
                const unsigned peers = ok ? *(volatile unsigned *)&peer[d] : bit;
                const unsigned rank = __popc(peers & lt);
                int before = 0;
                if (ok && rank == 0) before = hist[d];
                __syncwarp();
                if (ok && rank == 0) {
                    peer[d] = 0u;
                    hist[d] = (uint16_t)(before + __popc(peers));
                }
                before = __shfl_sync(0xffffffffu, before, __ffs(peers) - 1);
                __syncwarp();
                place[j] = (unsigned)before + rank;
            }
        }
        __syncthreads();
        // thread d: the warps' counts of digit d become their first places in the tile's
        // digit order; the tile's count is published for the look-backs of later tiles
        const int d = threadIdx.x;
        int c[kRadixWarps], run = 0;
#pragma unroll
        for (int w = 0; w < kRadixWarps; w++) {
            c[w] = run;
            run += s_hist[w][d];
        }
        volatile unsigned long long *const st = a.status;
        const bool digit = d <= (int)dmask;   // (the others have no entries)
        if (digit) st[(size_t)tile * 256 + d] = lb_word(epoch, stile == 0 ? 2 : 1, (unsigned)run);
        int valid;
        const int toff = block_exclusive_scan<kRadixThreads, int>(run, valid);
#pragma unroll
        for (int w = 0; w < kRadixWarps; w++) s_hist[w][d] = (uint16_t)(c[w] + toff);
        __syncthreads();
        // the tile in shared memory in digit order (stable)
#pragma unroll
        for (int j = 0; j < kRadixItems; j++)
            if (whole || kv[j].y != kDropped) s_pair[hist[(kv[j].x >> shift) & dmask] + place[j]] = kv[j];
        int excl = 0;
        if (digit && stile != 0) {
            excl = radix_look_back(st, epoch, tile, tile - stile, d, a.error);
            st[(size_t)tile * 256 + d] = lb_word(epoch, 2, (unsigned)(excl + run));
        }
        if (digit) s_base[d] = sbase + a.digit_base[((size_t)s_t.seg * a.passes + a.pass) * 256 + d] + excl - toff;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < kRadixWarps; w++) s_hist[w][d] = 0;   // for the next tile (whose barrier follows)
        // each digit's run with consecutive threads (coalesced)
        auto write = [&](int i) {
            const uint2 p = s_pair[i];
            const int pos = s_base[(p.x >> shift) & dmask] + i;
            if (OUT == kOutPairs) a.out_pairs[pos] = p;
            else a.out_values[pos] = p.y;
            if (OUT == kOutTable) {
                // The tile's entries of a digit are in key order, so a bucket's entries here
                // are one run: its first entry offers the bucket's start, first and last
                // together add its length (see BucketSlot).
                uint2 *const slot = a.table + table_base + p.x;
                if (i == 0 || s_pair[i - 1].x != p.x) {
                    atomicMax(&slot->x, kMaxStart - (uint32_t)pos);
                    atomicAdd(&slot->y, (uint32_t)-i);
                }
                if (i == valid - 1 || s_pair[i + 1].x != p.x) atomicAdd(&slot->y, (uint32_t)(i + 1));
            }
        };
        if (valid == kRadixTile) {
#pragma unroll
            for (int j = 0; j < kRadixItems; j++) write(d + j * kRadixThreads);
        } else {
            for (int i = d; i < valid; i += kRadixThreads) write(i);
        }
    }
    if (threadIdx.x == 0 && (int)(unsigned)drawn == tiles + active - 1)
        atomicAdd(a.ctl, (1ull << 32) - (unsigned long long)(tiles + active));
}

static int key_bits(int buckets)
{
    int bits = 0;
    while (bits < 31 && (1ll << bits) < (long long)buckets) bits++;
    return bits;
}

int radix_passes(int buckets) { return std::max(1, (key_bits(buckets) + 7) / 8); }

// The key's bits spread evenly over the passes: fewer digits mean longer runs to write
// and no pass with only a few digits, whose shared words all lanes would meet at.
int radix_digit_bits(int buckets)
{
    const int P = radix_passes(buckets);
    return std::max(1, (key_bits(buckets) + P - 1) / P);
}

constexpr int kRadixSmem = kRadixTile * 8 + kRadixWarps * 256 * (4 + 2);

template <int IN, int OUT>
static cudaError_t radix_launch(const RadixPass &a, int grid, DayQueue &q)
{
    static_assert(kRadixSmem <= 46 * 1024, "with the static part, no more than a launch may ask for without opt-in");
    return queue_kernel(q, k_radix_pass<IN, OUT>, grid, kRadixThreads, kRadixSmem, a);
}

cudaError_t launch_radix_sort(const RadixArgs &r, DayQueue &q)
{
    const int P = radix_passes(r.buckets);
    const int tiles = std::max(1, div_up(r.E, kRadixTile));
    const int grid = std::max(1, std::min(tiles, std::min(r.blocks_per_sm, kRadixBlocksPerSm) * sm_count()));
    RadixPass a;
    a.keys = r.keys;
    a.in = r.in;
    a.out_values = r.out;
    a.table = r.table;
    a.E = r.E;
    a.passes = P;
    a.dbits = radix_digit_bits(r.buckets);
    a.digit_base = r.digit_base;
    a.sg = r.seg;
    a.status = r.status;
    a.ctl = r.ctl;
    a.error = r.error;
    a.skip = r.skip;
    const bool day = r.table != nullptr;
    for (int p = 0; p < P; p++) {
        const bool first = p == 0, last = p == P - 1;
        a.pass = p;
        a.out_pairs = (p & 1) ? r.p1 : r.p0;
        cudaError_t e;
        if (first && day) e = last ? radix_launch<kInDay, kOutTable>(a, grid, q) : radix_launch<kInDay, kOutPairs>(a, grid, q);
        else if (first) e = last ? radix_launch<kInKeys, kOutValues>(a, grid, q) : radix_launch<kInKeys, kOutPairs>(a, grid, q);
        else if (!last) e = radix_launch<kInPairs, kOutPairs>(a, grid, q);
        else e = day ? radix_launch<kInPairs, kOutTable>(a, grid, q) : radix_launch<kInPairs, kOutValues>(a, grid, q);
        if (e != cudaSuccess) return e;
        a.in = a.out_pairs;
    }
    return cudaSuccess;
}

// Count, scan (+digit histograms), digit bases and radix passes: the bucket table of
// `E` keys in [0, buckets).  counts must be zero on entry and is zero on exit.
cudaError_t launch_bucket_table(const RadixArgs &r, int32_t *counts, bool count_keys, int32_t *offset,
                                unsigned long long *tiles, int *lb_ctl, int *digit_hist, cudaStream_t s)
{
    const int P = radix_passes(r.buckets);
    if (count_keys) {
        cudaError_t e = launch_count_keys((const int32_t *)r.keys, r.E, counts, s);
        if (e != cudaSuccess) return e;
    }
    cudaError_t e = launch_scan_exclusive(counts, offset, r.buckets, 1, tiles, lb_ctl, r.error, r.skip, P,
                                          radix_digit_bits(r.buckets), digit_hist, s);
    if (e != cudaSuccess) return e;
    k_digit_bases<<<1, 256, 0, s>>>(digit_hist, (int *)r.digit_base, P, 1, r.skip);
    count_launch();
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    DayQueue q{s};
    return launch_radix_sort(r, q);
}

// setup_initializeStatusArrays (PandemicSim.cu:3654-3664): S/S, day 255/255, gen 255.
__global__ void k_init_status(int N, uint32_t *state, uint8_t *gen_p, uint8_t *gen_s, unsigned long long *claim)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        state[i] = 0x01u | (0x01u << 8) | (0xFFu << 16) | (0xFFu << 24);
        gen_p[i] = 0xFF;
        gen_s[i] = 0xFF;
        claim[2 * (size_t)i] = ~0ull;
        claim[2 * (size_t)i + 1] = ~0ull;
    }
}

cudaError_t launch_init_status(int N, uint32_t *state, uint8_t *gen_p, uint8_t *gen_s,
                               unsigned long long *claim, cudaStream_t s)
{
    int blocks = std::min(div_up(N, 256), sm_count() * 16);
    k_init_status<<<std::max(1, blocks), 256, 0, s>>>(N, state, gen_p, gen_s, claim);
    count_launch();
    return cudaGetLastError();
}

// One block per instance: zero its state words, then set the counter offset.
__global__ void k_reset_instances(const InstConst *ic, InstState *is, int K)
{
    const int k = blockIdx.x;
    if (k >= K) return;
    int *w = reinterpret_cast<int *>(&is[k]);
    for (int i = threadIdx.x; i < (int)(sizeof(InstState) / 4); i += blockDim.x) w[i] = 0;
    __syncthreads();
    if (threadIdx.x == 0)
        is[k].rand_offset = is[k].next_offset[0] =
            (unsigned long long)(ic[k].c.H / 4) + (unsigned long long)(ic[k].c.N / 4);
}

cudaError_t launch_reset_instances(const DevArrays &d, cudaStream_t s)
{
    k_reset_instances<<<d.K, 256, 0, s>>>(d.ic, d.is, d.K);
    count_launch();
    return cudaGetLastError();
}

// Vaccination (an intervention, no reference counterpart): one person tile per block;
// a vaccinated person starts recovered from both strains, never infected.
__global__ void k_vaccinate(const InstConst *ic, const int32_t *tile_inst, uint32_t *state)
{
    const int k = tile_inst[blockIdx.x];
    const InstConst &c = ic[k];
    if (c.vacc_thr == 0) return;
    const int first = blockIdx.x * kPersonTile - c.pbase;
    for (int i = threadIdx.x; i < kPersonTile; i += blockDim.x) {
        const int p = first + i;
        if (p >= c.c.N) break;
        if (intervention_hash(c.c.key0, c.c.key1, kTagVaccinated, 0, p) < c.vacc_thr)
            state[c.pbase + p] = (0xFFu << 16) | (0xFFu << 24);  // status R / R, day 255 / 255
    }
}

cudaError_t launch_vaccinate(const DevArrays &d, cudaStream_t s)
{
    k_vaccinate<<<d.P / kPersonTile, 256, 0, s>>>(d.ic, d.tile_inst, d.state);
    count_launch();
    return cudaGetLastError();
}

// setup_initialInfected (PandemicSim.cu:708-758): the first P seeds get the pandemic
// strain, the next S the seasonal one; status STATUS_INFECTED, day 0, generation 0.
__global__ void k_seed_infected(const int32_t *seeds, int P, int S, uint32_t *state, uint8_t *gen_p, uint8_t *gen_s)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P + S) return;
    int p = seeds[i];
    if (i < P) {
        state[p] = (state[p] & 0xFF00FF00u) | 0x02u;          // status_p = 2, day_p = 0
        gen_p[p] = 0;
    } else {
        state[p] = (state[p] & 0x00FF00FFu) | (0x02u << 8);   // status_s = 2, day_s = 0
        gen_s[p] = 0;
    }
}

cudaError_t launch_seed_infected(const int32_t *seeds, int P, int S, uint32_t *state, uint8_t *gen_p,
                                 uint8_t *gen_s, cudaStream_t s)
{
    if (P + S <= 0) return cudaSuccess;
    k_seed_infected<<<div_up(P + S, 256), 256, 0, s>>>(seeds, P, S, state, gen_p, gen_s);
    count_launch();
    return cudaGetLastError();
}

// The packed per-person records (PersonRec layout in pt_kernels.h): one thread per
// person.  Everything in a record is fixed once the workplace table exists.
__global__ void k_person_records(const InstConst *ic, const int32_t *tile_inst, int P, const int32_t *household,
                                 const int32_t *hh_offset, const int32_t *workplace, const int32_t *wp_offset,
                                 const uint8_t *age, uint4 *prec)
{
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < P; p += gridDim.x * blockDim.x) {
        const int hh = household[p];
        if (hh < 0) {  // padding person
            prec[p] = make_uint4(0u, 0u, 0u, 0u);
            continue;
        }
        const InstConst &k = ic[tile_inst[p / kPersonTile]];
        const int hoff = hh_offset[hh], hcnt = hh_offset[hh + 1] - hoff;
        const int wp = workplace[p];
        const int woff = wp_offset[wp], wcnt = wp_offset[wp + 1] - woff;
        const int loc = wp - k.lbase;
        const uint32_t w = (uint32_t)hcnt | ((uint32_t)age[p] << 4) | ((uint32_t)workplace_max_contacts(k.c, loc) << 8) |
                           ((uint32_t)is_school(k.c, loc) << 10);
        prec[p] = make_uint4((uint32_t)hoff, (uint32_t)woff, (uint32_t)wcnt, w);
    }
}

cudaError_t launch_person_records(const DevArrays &d, cudaStream_t s)
{
    const int blocks = std::max(1, std::min(div_up(d.P, 256), sm_count() * 16));
    k_person_records<<<blocks, 256, 0, s>>>(d.ic, d.tile_inst, d.P, d.household, d.hh_offset, d.workplace,
                                            d.wp_offset, d.age, d.prec);
    count_launch();
    return cudaGetLastError();
}

// ================================================================== day
// Every day kernel covers all instances of a batch in one launch.  Persons are
// global ids; a person tile (kPersonTile persons) belongs to one instance
// (tile_inst), and an infected list position to the instance in infected_inst.

// An instance takes part in a day until a day counts zero infected, and for at
// most its max_days days.
__device__ __forceinline__ bool instance_running(const InstConst &c, const InstState &s, int day)
{
    return !s.done && day < c.max_days;
}

// The day of a launch: its own, or (-1, a launch of a graph that serves every stepped
// day of its kind) the next one to step.
__device__ __forceinline__ int launch_day(int day, const Scalars *sc)
{
    return day >= 0 ? day : *(volatile const int *)&sc->step_day;
}

// R0 of a day whose schedule starts at counter E0.
__device__ __forceinline__ unsigned long long contact_offset(const InstConst &c, unsigned long long E0, bool weekend)
{
    const unsigned long long N = (unsigned long long)c.c.N;
    return E0 + (weekend ? 2ull * N : N / 2ull);
}

// Sweep: one tile of 4096 persons per block; each thread holds 4 rounds of 4
// persons (one 16-byte load per round).  Output order is (round, thread, item),
// which is ascending person order within the tile.
constexpr int kSweepThreads = 256, kSweepRounds = 4, kSweepTile = kSweepThreads * 4 * kSweepRounds;
static_assert(kSweepTile == kPersonTile, "a sweep tile is a person tile");

__device__ __forceinline__ uint32_t recover_word(uint32_t st, int d2r, bool &changed)
{
    uint32_t sp = st & 0xFFu, ss = (st >> 8) & 0xFFu, dp = (st >> 16) & 0xFFu, ds = st >> 24;
    uint32_t out = st;
    if (d2r >= 0 && sp >= 2u && (int)dp <= d2r) out &= ~0xFFu;
    if (d2r >= 0 && ss >= 2u && (int)ds <= d2r) out &= ~0xFF00u;
    changed = out != st;
    return out;
}

// The sweep: kernel_countInfectedStatusAndRecover (PandemicSim.cu:2097-2192), the
// copy_if of the infected (:2207-2224) and runToCompletion's day bookkeeping
// (:891-937) in three launches over every instance:
//   count  a run of person tiles per block (one for small runs): recover, count the
//          instances' 16 status bins (reduced once per block and instance), and
//          record each thread's infected persons as a 16-bit mask and each tile's
//          infected count.  Thread t of a tile holds persons (r * 256 + t) * 4 + j,
//          rounds r = 0..3, items j = 0..3; mask bit 4r + j.
//   scan   one block: exclusive scan of the tile counts, each instance's run
//          [start, list_end) of the infected list and its day bookkeeping.
//   emit   one person tile per warp (per block for small runs): the infected ids,
//          in ascending order, at their list positions.
// The count kernel also clears the day's marks.
// Each launch depends only on the one before, so no block waits for another.
// Person tiles a count block sweeps one after another: as many as make the grid one wave
// of the blocks that fit (kSweepBlocksPerSm), at most what 8-bit status counts hold.
constexpr int kSweepBlocksPerSm = 8, kSweepTilesPerBlock = 255 / (4 * kSweepRounds);
// From this many tiles an SM on, the emit kernel has a warp per tile instead of a block.
constexpr int kSweepEmitTilesPerSm = 32;

// A thread's persons by status.  Most have neither strain now: those take a test and an
// addition each (bytes 0 and 1 of `susceptible`: how many of them are susceptible, status 1
// and not 0, to each strain); the others a byte a status and strain, statuses 0-3 and 4-7.
// (With every person counted the second way the sweep of 24M persons with vaccinations
// took 65 us, now 29, for 100 MB.)
struct SweepBins {
    uint32_t p[2], s[2];
    uint32_t susceptible;
    int healthy;   // persons counted in `susceptible`
};

// One more person of statuses sp, ss (0..7).  (shl gives 0 for shifts of 32 and more, and
// the shift less 32 is such a one when it is negative.)
__device__ __forceinline__ void sweep_count_person(SweepBins &b, uint32_t sp, uint32_t ss)
{
    uint32_t v[4];
    asm("shl.b32 %0, 1, %1;" : "=r"(v[0]) : "r"(8u * sp));
    asm("shl.b32 %0, 1, %1;" : "=r"(v[1]) : "r"(8u * sp - 32u));
    asm("shl.b32 %0, 1, %1;" : "=r"(v[2]) : "r"(8u * ss));
    asm("shl.b32 %0, 1, %1;" : "=r"(v[3]) : "r"(8u * ss - 32u));
    b.p[0] += v[0];
    b.p[1] += v[1];
    b.s[0] += v[2];
    b.s[1] += v[3];
}

// Adds a thread's bins into instance k's row of the day: warp reductions, one shared
// atomic per bin per warp, one global atomic per bin per block.  Block-uniform; clears
// the bins.
__device__ __forceinline__ void sweep_flush_bins(InstState *is, int k, int day, SweepBins &bins, int *s_bins)
{
    // four 16-bit counts a word; a warp's sums stay below 2^13
    auto spread = [](uint32_t v) {
        return (unsigned long long)__byte_perm(v, 0u, 0x4140) | (unsigned long long)__byte_perm(v, 0u, 0x4342) << 32;
    };
    const uint32_t sus_p = bins.susceptible & 0xFFu, sus_s = (bins.susceptible >> 8) & 0xFFu;
    unsigned long long bp_lo = spread(bins.p[0]) + (((uint32_t)bins.healthy - sus_p) | sus_p << 16);
    unsigned long long bs_lo = spread(bins.s[0]) + (((uint32_t)bins.healthy - sus_s) | sus_s << 16);
    unsigned long long bp_hi = spread(bins.p[1]), bs_hi = spread(bins.s[1]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        bp_lo += __shfl_xor_sync(0xffffffffu, bp_lo, o);
        bp_hi += __shfl_xor_sync(0xffffffffu, bp_hi, o);
        bs_lo += __shfl_xor_sync(0xffffffffu, bs_lo, o);
        bs_hi += __shfl_xor_sync(0xffffffffu, bs_hi, o);
    }
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int b = 0; b < 4; b++) {
            int a0 = (int)((bp_lo >> (16 * b)) & 0xFFFF), a1 = (int)((bp_hi >> (16 * b)) & 0xFFFF);
            int a2 = (int)((bs_lo >> (16 * b)) & 0xFFFF), a3 = (int)((bs_hi >> (16 * b)) & 0xFFFF);
            if (a0) atomicAdd(&s_bins[b], a0);
            if (a1) atomicAdd(&s_bins[4 + b], a1);
            if (a2) atomicAdd(&s_bins[8 + b], a2);
            if (a3) atomicAdd(&s_bins[12 + b], a3);
        }
    }
    __syncthreads();
    if (threadIdx.x < 16) {
        if (s_bins[threadIdx.x]) atomicAdd(&is[k].counts[day][threadIdx.x], s_bins[threadIdx.x]);
        s_bins[threadIdx.x] = 0;
    }
    __syncthreads();
    bins = SweepBins{};
}

__global__ void __launch_bounds__(kSweepThreads, kSweepBlocksPerSm) k_sweep_count(const InstConst *ic, InstState *is,
                                                                  const int32_t *tile_inst, int tiles, int per_block,
                                                                  uint32_t *state, uint16_t *flags_out,
                                                                  int32_t *tile_count, uint2 *clear, int clear_n,
                                                                  const Scalars *sc, int day)
{
    day = launch_day(day, sc);
    if (*(volatile const int *)&sc->done) return;
    for (int i = blockIdx.x * kSweepThreads + threadIdx.x; i < clear_n; i += gridDim.x * kSweepThreads)
        clear[i] = make_uint2(0u, 0u);
    const int t0 = blockIdx.x * per_block;
    const int t1 = t0 + per_block < tiles ? t0 + per_block : tiles;
    const int d2r = day - 10;
    __shared__ int s_bins[16];
    __shared__ int s_tc[kSweepTilesPerBlock];   // infected of each of the block's tiles
    if (threadIdx.x < 16) s_bins[threadIdx.x] = 0;
    if (threadIdx.x < kSweepTilesPerBlock) s_tc[threadIdx.x] = 0;
    __syncthreads();
    SweepBins bins = {};   // of the current instance
    int cur = tile_inst[t0];
    for (int tile = t0;; tile++) {
        // after the last tile, or when the tiles move on to the next instance: the bins
        const int k = tile < t1 ? tile_inst[tile] : -1;
        if (k != cur) {
            sweep_flush_bins(is, cur, day, bins, s_bins);  // (ends with a barrier)
            cur = k;
        }
        if (k < 0) break;
        const int first = tile * kSweepTile + 4 * (int)threadIdx.x;
        // end of the tile's persons: none when the instance no longer runs
        const int N = instance_running(ic[k], is[k], day) ? ic[k].pbase + ic[k].c.N : 0;
        uint32_t flags = 0;  // bit (4*round + item)
        auto load = [&](int r) {
            const int p0 = first + r * 4 * kSweepThreads, n = N - p0;   // persons from p0 on
            if (n <= 0) return make_uint4(0u, 0u, 0u, 0u);
            uint4 v = *reinterpret_cast<const uint4 *>(state + p0);     // (padding persons follow)
            if (n < 4) {
                v.w = 0u;
                if (n < 3) v.z = 0u;
                if (n < 2) v.y = 0u;
            }
            bins.healthy += min(n, 4);   // those with a strain are taken off below
            return v;
        };
        uint4 next = load(0);   // a round's load goes before the last round's stores
#pragma unroll
        for (int r = 0; r < kSweepRounds; r++) {
            const uint32_t st[4] = {next.x, next.y, next.z, next.w};
            if (r + 1 < kSweepRounds) next = load(r + 1);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if ((st[j] & 0xFEFEu) == 0u) {   // neither strain (or past the end): nothing to recover
                    bins.susceptible += st[j] & 0x0101u;
                    continue;
                }
                bins.healthy--;
                bool changed;
                const uint32_t out = recover_word(st[j], d2r, changed);
                const uint32_t sp = out & 0xFFu, ss = (out >> 8) & 0xFFu;
                sweep_count_person(bins, sp, ss);
                if (sp >= 2u || ss >= 2u) flags |= 1u << (4 * r + j);
                if (changed) state[first + r * 4 * kSweepThreads + j] = out;
            }
        }
        flags_out[(size_t)tile * kSweepThreads + threadIdx.x] = (uint16_t)flags;
        int cnt = __popc(flags);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(&s_tc[tile - t0], cnt);
    }
    if (threadIdx.x < t1 - t0) tile_count[t0 + threadIdx.x] = s_tc[threadIdx.x];
}

constexpr int kSweepScanThreads = 1024;

// A running instance's day (runToCompletion, PandemicSim.cu:891-937): its run
// [start, end) of the infected list, the statistics row, the stop on zero infected, the
// counter offsets E0 / R0 of the schedule and the contacts.  The day's first counter is
// next_offset[day & 1], which nothing writes that day (k_sweep_list's blocks read it
// while one of them is here).
__device__ __forceinline__ void begin_instance_day(const InstConst &c, InstState &s, int start, int end, int day,
                                                   int dense_level)
{
    const bool weekend = (day % 7) >= 5;  // PandemicSim.h:283-284
    s.start = start;
    s.list_end = end;
    s.marked = 0;
    s.dense = 0;
    if (!instance_running(c, s, day)) {
        s.infected = 0;
        return;
    }
    const int I = end - start;
    s.infected = I;
    // When the infected (each marks one or two buckets) are many against the
    // buckets, most buckets will be read, and the sort can read the schedule keys
    // directly: dense_level 1, 2, 3 take I >= B / 4, I >= B, I >= 2 B; 0 never.
    // Either way the tables are the same.
    const long long B = c.bcount[weekend ? 1 : 0];
    s.dense = dense_level > 0 && 4ll * I >= B * (dense_level == 1 ? 1 : (dense_level == 2 ? 4 : 8)) ? 1 : 0;
    s.infected_per_day[day] = I;
    s.day = day;
    s.days_run = day + 1;
    if (I == 0) {
        s.done = 1;
        return;
    }
    const unsigned long long E0 = s.next_offset[day & 1], R0 = contact_offset(c, E0, weekend);
    s.errand_offset = E0;
    s.infect_offset = R0;
    s.rand_offset = s.next_offset[(day + 1) & 1] = R0 + 6ull * (unsigned long long)I;
}

// The batch's day; done holds the number of days run (so that a block of the launch that
// sets it can tell the day's own end from an earlier one).
__device__ __forceinline__ void begin_day(Scalars *sc, int total, int day)
{
    sc->infected = total;
    sc->day = day;
    sc->new_count = 0;
    if (total == 0) sc->done = day + 1;
}

__global__ void __launch_bounds__(kSweepScanThreads) k_sweep_scan(const InstConst *ic, InstState *is, int K,
                                                                  int32_t *tile_count, int tiles, Scalars *sc,
                                                                  int day, int dense_level)
{
    day = launch_day(day, sc);
    if (*(volatile const int *)&sc->done) return;
    // exclusive scan in place, a contiguous chunk per thread; entry `tiles` = total
    const int per = (tiles + kSweepScanThreads - 1) / kSweepScanThreads;
    const int lo = (int)threadIdx.x * per, hi = lo + per < tiles ? lo + per : tiles;
    int sum = 0;
    for (int i = lo; i < hi; i++) sum += tile_count[i];
    int total;
    int run = block_exclusive_scan<kSweepScanThreads, int>(sum, total);
    for (int i = lo; i < hi; i++) {
        const int v = tile_count[i];
        tile_count[i] = run;
        run += v;
    }
    if (threadIdx.x == 0) tile_count[tiles] = total;
    __syncthreads();
    for (int k = threadIdx.x; k < K; k += kSweepScanThreads)
        begin_instance_day(ic[k], is[k], tile_count[ic[k].pbase / kSweepTile], tile_count[ic[k].pend / kSweepTile], day,
                           dense_level);
    if (threadIdx.x == 0) begin_day(sc, total, day);
}

// Emit for small runs: a block per person tile, a block scan of the threads' packed
// per-round counts (a warp per tile would leave most SMs idle).
__global__ void __launch_bounds__(kSweepThreads) k_sweep_emit_block(const int32_t *tile_inst, const uint16_t *flags_in,
                                                                    const int32_t *tile_prefix, int32_t *infected,
                                                                    int32_t *infected_inst, const Scalars *sc)
{
    if (*(volatile const int *)&sc->done) return;
    const int tile = blockIdx.x;
    const int prefix = tile_prefix[tile];
    if (tile_prefix[tile + 1] == prefix) return;  // no infected in this tile
    const uint32_t f = flags_in[(size_t)tile * kSweepThreads + threadIdx.x];
    unsigned long long packed = 0;
#pragma unroll
    for (int r = 0; r < kSweepRounds; r++) packed |= (unsigned long long)__popc((f >> (4 * r)) & 0xFu) << (16 * r);
    // positions in person order: scan the four per-round counts at once (16-bit fields)
    unsigned long long round_tot;
    const unsigned long long excl = block_exclusive_scan<kSweepThreads, unsigned long long>(packed, round_tot);
    const int k = tile_inst[tile];
    const long long tile_base = (long long)tile * kSweepTile;
    int round_base = prefix;
#pragma unroll
    for (int r = 0; r < kSweepRounds; r++) {
        int pos = round_base + (int)((excl >> (16 * r)) & 0xFFFF);
        const long long p0 = tile_base + ((long long)r * kSweepThreads + threadIdx.x) * 4;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (f & (1u << (4 * r + j))) {
                infected[pos] = (int32_t)(p0 + j);
                infected_inst[pos] = k;
                pos++;
            }
        }
        round_base += (int)((round_tot >> (16 * r)) & 0xFFFF);
    }
}

constexpr int kEmitWarps = 8;   // person tiles per emit block, one warp each

// Emit: a warp per person tile.  Lane l reads the masks of count-kernel threads
// 8l .. 8l+7 in one 16-byte load; per round, a warp scan of the lanes' counts places
// them, so the ids come out in (round, thread, item) order: ascending persons.
__global__ void __launch_bounds__(kEmitWarps * 32) k_sweep_emit(const int32_t *tile_inst, int tiles,
                                                                const uint16_t *flags_in,
                                                                const int32_t *tile_prefix, int32_t *infected,
                                                                int32_t *infected_inst, const Scalars *sc)
{
    if (*(volatile const int *)&sc->done) return;
    const int lane = threadIdx.x & 31;
    const int tile = blockIdx.x * kEmitWarps + (threadIdx.x >> 5);
    if (tile >= tiles) return;
    const int prefix = tile_prefix[tile];
    if (tile_prefix[tile + 1] == prefix) return;  // no infected in this tile
    const uint4 raw = *reinterpret_cast<const uint4 *>(flags_in + (size_t)tile * kSweepThreads + 8 * lane);
    const uint32_t wd[4] = {raw.x, raw.y, raw.z, raw.w};  // masks of threads 8l + 2i (low half), 8l + 2i + 1
    const int k = tile_inst[tile];
    const long long tile_base = (long long)tile * kSweepTile;
    int round_base = prefix;
#pragma unroll
    for (int r = 0; r < kSweepRounds; r++) {
        int c = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) c += __popc((wd[i] >> (4 * r)) & 0xFu) + __popc((wd[i] >> (16 + 4 * r)) & 0xFu);
        const int incl = warp_inclusive_scan(c);
        int pos = round_base + incl - c;
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const uint32_t m = (wd[q >> 1] >> (16 * (q & 1) + 4 * r)) & 0xFu;
            if (m) {
                const long long p0 = tile_base + ((long long)r * kSweepThreads + 8 * lane + q) * 4;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    if ((m >> j) & 1u) {
                        infected[pos] = (int32_t)(p0 + j);
                        infected_inst[pos] = k;
                        pos++;
                    }
                }
            }
        }
        round_base += __shfl_sync(0xffffffffu, incl, 31);
    }
}

// ------------------------------------------------------------------ schedules
// Weekday schedule (kernel_assignWeekdayAfterschoolAndErrands, PandemicSim.cu:2972-3022):
// counter E0 + g -> the instance's persons 2g, 2g+1.  Hour-0 keys at [0,N), hour-1
// keys at [N,2N) of the instance's key slots.  Weekday destinations lie in [lo, L),
// lo = first location of type 8 (afterschool), so the instance's bucket is
// hour * R + dest - lo with R = L - lo (order-preserving); the global bucket adds the
// instance's weekday bucket base.
__device__ __forceinline__ void weekday_pair_keys(const SimConst &c, const uint32_t w[4], int k, bool adult, int lo,
                                                  int R, int &k1, int &k2)
{
    // the second errand is drawn for every lane and kept for adults (no divergence)
    const int d1 = fish_weekday_dest(c, w[2 * k], adult);
    const int e2 = fish_weekday_dest(c, w[2 * k + 1], true);
    const int d2 = adult ? e2 : d1;
    k1 = d1 - lo;
    k2 = R + d2 - lo;
}

// mark word of bucket b, its bit shifted to bit 0 (the others follow)
__device__ __forceinline__ uint32_t mark_bit(const uint32_t *mark, uint32_t b)
{
    return __funnelshift_r(mark[b >> 5], 0u, b);
}

// Fire-and-forget global updates (PTX red): the thread does not wait for the result.
__device__ __forceinline__ void red_add(int *p, int v)
{
    asm volatile("red.relaxed.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ void red_or(uint32_t *p, uint32_t v)
{
    asm volatile("red.relaxed.gpu.global.or.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Sets bucket b's bit.
__device__ __forceinline__ void mark_bucket(uint32_t *mark, int b) { red_or(&mark[b >> 5], 1u << (b & 31)); }

// The same into a block's copy of the bitmap (s_mark), which is merged at the end.
__device__ __forceinline__ void mark_bucket_shared(uint32_t *s_mark, int b)
{
    const uint32_t bit = 1u << (b & 31);
    if (!(*(volatile uint32_t *)&s_mark[b >> 5] & bit)) atomicOr(&s_mark[b >> 5], bit);
}

// The buckets (global) that today's contact draws of an infected person read, -1 for
// none: `person` global, lpos its place in its instance's infected list.  They are kept in
// list order (d.read) for the infection kernels, which would otherwise gather them from
// every person's keys and draw the adults' profile again; so nobody's keys are written
// unless the sort reads them (a dense instance).  Weekdays a person's two errand contacts
// go to the first bucket, the second or one each; weekends one each, in slot order.
__device__ __forceinline__ int2 read_buckets(const InstConst &ik, const uint8_t *age, int weekend, unsigned long long E0,
                                             unsigned long long R0, int person, int lpos)
{
    const SimConst &c = ik.c;
    const TfKey key = make_key(c);
    const int me = person - ik.pbase;   // the instance's person number
    uint32_t w[4];
    if (weekend) {
        const int lo = c.type_offset[9], R = c.L - lo;
        int d[3];
        weekend_errands(c, key, E0 + 2ull * (unsigned long long)me, lo, R, d);
        tf2x64(key, R0 + 6ull * (unsigned long long)lpos, w);
        const int prof = (int)(w[3] % 6u);
        return make_int2(ik.bbase[1] + d[c_weekend_assign[prof][0]], ik.bbase[1] + d[c_weekend_assign[prof][1]]);
    }
    const int lo = c.type_offset[8], R = c.L - lo;
    tf2x64(key, E0 + (uint64_t)(me / 2), w);
    const bool adult = age[person] == 5;
    const int slot = 2 * (me & 1);
    int k1, k2;
    weekday_pair_keys(c, w, me & 1, adult, lo, R, k1, k2);
    const int prof = adult ? (int)((w[slot] ^ w[slot + 1]) % 3u) : 3;
    return make_int2(c_weekday_assign[prof][0] > 0 ? ik.bbase[0] + k1 : -1,
                     c_weekday_assign[prof][1] > 0 ? ik.bbase[0] + k2 : -1);
}

// Marks the errand buckets today's contact draws will read: the only buckets that
// must be materialised.  Destinations are regenerated from the schedule counter, as
// the reference's device_recalc_* functions do (PandemicSim.cu:3667-3705,
// :3742-3746), and only the hours / errands the person's contact profile uses are
// marked: weekday hours whose profile wants contacts (the adult profile comes from
// the same Threefry block, :3697-3702; children use the afterschool profile), and on
// weekends the two errand slots picked by word 3 of the infection counter's block
// (:1892, :1909, :1929).
//
// On a dense day the infected far outnumber the bitmap's words, and updates of one
// word are served one after another: 2M infected over 640 words took 400 us.  So when
// the bitmap fits a block's shared memory (kMarkSharedWords) and the infected are at
// least kMarkSharedPerWord to a word, each block marks a copy of its own and merges the
// words it set.  Below that the merge (a word per block) would cost more than it saves.
// Where the bitmap does not fit and there are kMarkSeenPerWord to a word, a warp looks
// before it marks: a batch's list goes instance by instance, so all blocks mark the few
// hundred words of one instance at a time, most of them set (weekends of 48 instances:
// list and marks 10.6 -> 7.1 ms a run; at four to a word 50M persons lost 0.2 of 2.1 ms).
constexpr int kMarkSharedWords = 8192, kMarkSharedPerWord = 64, kMarkSeenPerWord = 32;
constexpr int kMarkThreads = 256, kMarkBlocksPerSm = 4;

__global__ void __launch_bounds__(kMarkThreads) k_mark_buckets(const InstConst *ic, const InstState *is,
                                                               const uint8_t *age, const int32_t *infected,
                                                               const int32_t *infected_inst, int weekend,
                                                               int2 *read, uint32_t *mark, int words, const Scalars *sc)
{
    if (sc->done) return;
    const int I = sc->infected;
    __shared__ uint32_t s_mark[kMarkSharedWords];
    const bool shared = words <= kMarkSharedWords && I >= kMarkSharedPerWord * words;
    const bool seen = I >= kMarkSeenPerWord * words;
    if (shared) {
        for (int i = threadIdx.x; i < words; i += blockDim.x) s_mark[i] = 0u;
        __syncthreads();
    }
    for (int pos = blockIdx.x * blockDim.x + threadIdx.x; pos < I; pos += gridDim.x * blockDim.x) {
        const int k = infected_inst[pos];
        const InstState &s = is[k];
        const int2 b = read_buckets(ic[k], age, weekend, s.errand_offset, s.infect_offset, infected[pos], pos - s.start);
        read[pos] = b;
        if (shared) {
            if (b.x >= 0) mark_bucket_shared(s_mark, b.x);
            if (b.y >= 0) mark_bucket_shared(s_mark, b.y);
        } else {
            if (b.x >= 0 && !(seen && (__ldcg(&mark[b.x >> 5]) >> (b.x & 31) & 1u))) mark_bucket(mark, b.x);
            if (b.y >= 0 && !(seen && (__ldcg(&mark[b.y >> 5]) >> (b.y & 31) & 1u))) mark_bucket(mark, b.y);
        }
    }
    if (shared) {
        __syncthreads();
        // blocks start at different words, so they do not queue at the same one
        const int first = (int)((long long)words * blockIdx.x / gridDim.x);
        for (int i = threadIdx.x; i < words; i += blockDim.x) {
            const int w = first + i < words ? first + i : first + i - words;
            if (s_mark[w]) red_or(&mark[w], s_mark[w]);
        }
    }
}

// A small run's list and marks in one launch instead of three (scan, emit, mark): a block
// per person tile sums the counts of the tiles itself, emits its part of the list and
// marks its persons' buckets.  The block of an instance's first tile begins the
// instance's day, the last tile's block the batch's; no block waits for another.  Small
// runs are bound by their launches: a day of 100,000 persons has seven of 3 to 10 us.
// Up to kListTiles tiles (4M persons) the sums are four loads a thread: 30 days of 1.2M and
// 3.9M persons 2.60 and 3.41 ms, 2.87 and 3.71 with the three launches.  With sixteen loads
// (to 16M persons) everything below 4M is 1% slower and 4 to 9M 3 to 0.5% faster; at 16M
// the three launches are faster by 1%.
constexpr int kListTiles = 4 * kSweepThreads;
constexpr int kListMarkWords = 2048;   // a bitmap this small is marked in shared memory and merged once a block

__global__ void __launch_bounds__(kSweepThreads) k_sweep_list(const InstConst *ic, InstState *is, const int32_t *tile_inst,
                                                              int tiles, const uint16_t *flags_in,
                                                              const int32_t *tile_count, int32_t *infected,
                                                              int32_t *infected_inst, int2 *read, const uint8_t *age,
                                                              uint32_t *mark,
                                                              int words, int mark_all, Scalars *sc, int day,
                                                              int dense_level)
{
    day = launch_day(day, sc);
    const int ended = *(volatile const int *)&sc->done;
    if (ended != 0 && ended != day + 1) return;
    const bool weekend = (day % 7) >= 5;
    const int tile = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t f = flags_in[(size_t)tile * kSweepThreads + t];
    const int k = tile_inst[tile], n = tile_count[tile];
    const InstConst &ik = ic[k];
    const unsigned long long E0 = is[k].next_offset[day & 1];
    const int first = ik.pbase / kSweepTile, end = ik.pend / kSweepTile;
    // infected before the instance, in it before the tile, in it from the tile on, behind it
    int sum[4] = {0, 0, 0, 0};
#pragma unroll
    for (int q = 0; q < kListTiles / kSweepThreads; q++) {
        const int i = t + q * kSweepThreads;
        const int c = i < tiles ? tile_count[i] : 0;
        if (i < first) sum[0] += c;
        else if (i < tile) sum[1] += c;
        else if (i < end) sum[2] += c;
        else sum[3] += c;
    }
    __shared__ int s_sum[kSweepThreads / 32][4];
    __shared__ uint16_t s_list[kSweepTile];
    __shared__ uint32_t s_mark[kListMarkWords];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int v = __reduce_add_sync(0xffffffffu, sum[q]);
        if (lane == 0) s_sum[warp][q] = v;
    }
    const bool shared = words <= kListMarkWords;
    if (n > 0 && shared && !mark_all)
        for (int i = t; i < words; i += kSweepThreads) s_mark[i] = 0u;
    __syncthreads();
    int start = 0, prefix = 0, list_end = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kSweepThreads / 32; w++) {
        start += s_sum[w][0];
        prefix += s_sum[w][1];
        list_end += s_sum[w][2];
        total += s_sum[w][3];
    }
    prefix += start;
    list_end += prefix;
    total += list_end;
    if (t == 0 && tile == first) begin_instance_day(ik, is[k], start, list_end, day, dense_level);
    if (t == 0 && tile == tiles - 1) begin_day(sc, total, day);
    if (n == 0) return;
    unsigned long long packed = 0;
#pragma unroll
    for (int r = 0; r < kSweepRounds; r++) packed |= (unsigned long long)__popc((f >> (4 * r)) & 0xFu) << (16 * r);
    // positions in person order: scan the four per-round counts at once (16-bit fields)
    unsigned long long round_tot;
    const unsigned long long excl = block_exclusive_scan<kSweepThreads, unsigned long long>(packed, round_tot);
    int round_base = 0;
#pragma unroll
    for (int r = 0; r < kSweepRounds; r++) {
        int at = round_base + (int)((excl >> (16 * r)) & 0xFFFF);
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (f & (1u << (4 * r + j))) s_list[at++] = (uint16_t)((r * kSweepThreads + t) * 4 + j);
        round_base += (int)((round_tot >> (16 * r)) & 0xFFFF);
    }
    __syncthreads();
    const unsigned long long R0 = contact_offset(ik, E0, weekend);
    for (int i = t; i < n; i += kSweepThreads) {
        const int person = tile * kSweepTile + s_list[i];
        infected[prefix + i] = person;
        infected_inst[prefix + i] = k;
        const int2 b = read_buckets(ik, age, weekend, E0, R0, person, prefix + i - start);
        read[prefix + i] = b;
        if (mark_all) continue;
        if (shared) {
            if (b.x >= 0) mark_bucket_shared(s_mark, b.x);
            if (b.y >= 0) mark_bucket_shared(s_mark, b.y);
        } else {
            if (b.x >= 0) mark_bucket(mark, b.x);
            if (b.y >= 0) mark_bucket(mark, b.y);
        }
    }
    if (mark_all || !shared) return;
    __syncthreads();
    for (int i = t; i < words; i += kSweepThreads)
        if (s_mark[i]) red_or(&mark[i], s_mark[i]);
}

// Words of the day's mark bitmap.
static int mark_words(const DevArrays &d, bool weekend) { return d.buckets[weekend ? 1 : 0] / 32 + 1; }

cudaError_t launch_sweep(const DevArrays &d, bool weekend, int day, DayQueue &q)
{
    const int tiles = d.P / kSweepTile;
    const int per_block = std::min(div_up(tiles, kSweepBlocksPerSm * sm_count()), kSweepTilesPerBlock);
    const cudaError_t e = queue_kernel(q, k_sweep_count, div_up(tiles, per_block), kSweepThreads, 0, d.ic, d.is, d.tile_inst,
                                       tiles, per_block, d.state, d.sweep_flags, d.sweep_tiles,
                                       reinterpret_cast<uint2 *>(d.mark), (mark_words(d, weekend) + 1) / 2, d.sc, day);
    if (e != cudaSuccess || tiles <= kListTiles) return e;
    return queue_kernel(q, k_sweep_scan, 1, kSweepScanThreads, 0, d.ic, d.is, d.K, d.sweep_tiles, tiles, d.sc, day,
                        d.tune.dense_level);
}

// The infected list and the marks of the buckets that its persons read (every bucket's
// for complete tables).
cudaError_t launch_infected_list(const DevArrays &d, bool weekend, int day, bool full_tables, DayQueue &q)
{
    const int tiles = d.P / kSweepTile, words = mark_words(d, weekend);
    if (full_tables) {
        const cudaError_t e = queue_fill(q, d.mark, 0xFFFFFFFFu, (size_t)words);
        if (e != cudaSuccess) return e;
    }
    if (tiles <= kListTiles)
        return queue_kernel(q, k_sweep_list, tiles, kSweepThreads, 0, d.ic, d.is, d.tile_inst, tiles, d.sweep_flags,
                            d.sweep_tiles, d.infected, d.infected_inst, d.read, d.age, d.mark, words,
                            full_tables ? 1 : 0, d.sc, day, d.tune.dense_level);
    const cudaError_t e =
        tiles >= kSweepEmitTilesPerSm * sm_count()
            ? queue_kernel(q, k_sweep_emit, div_up(tiles, kEmitWarps), kEmitWarps * 32, 0, d.tile_inst, tiles,
                           d.sweep_flags, d.sweep_tiles, d.infected, d.infected_inst, d.sc)
            : queue_kernel(q, k_sweep_emit_block, tiles, kSweepThreads, 0, d.tile_inst, d.sweep_flags, d.sweep_tiles,
                           d.infected, d.infected_inst, d.sc);
    if (e != cudaSuccess) return e;
    return queue_kernel(q, k_mark_buckets, sm_count() * kMarkBlocksPerSm, kMarkThreads, 0, d.ic, d.is, d.age, d.infected,
                        d.infected_inst, weekend ? 1 : 0, d.read, d.mark, words, d.sc);
}

// Schedule kernel.  The persons are cut into regions of C consecutive ones (64 to 1024,
// launch_schedule), each inside one instance.  A persistent block owns a run of regions
// and its warps take them one by one; a warp walks its region in rounds (weekday: 64
// persons a round, a pair per lane, one Threefry block per pair; weekend: 32 persons a
// round, one per lane).  The kernel keeps the entries of marked buckets, compacted in
// ascending person order, in the warp's part of shared memory; full parts are added to
// the block's radix digit histograms and copied, as (instance-local key, person), to the
// region's slots of the entry array (3C from 3C times the region's number), or, for a
// dense instance, every person's keys are written instead.  The sort's first pass reads the regions of an instance
// one after another (k_day_digit_bases scans their counts): the order its stability needs.
//
// No warp waits for another within an instance.  A form that placed the entries of
// all tiles contiguously by a decoupled look-back spent two thirds of its issue slots
// waiting: at this rate of tiles (80 per microsecond) a look-back of 32 tiles per
// round trip cannot keep up.  What is left is the integer pipe (62-71% busy) and
// instruction issue, so the work around the Threefry blocks is kept small: a
// destination is one table row found on the floating-point pipe (errand_bucket), marks
// cost a ballot per bit of a lane's count, and the per-entry work runs over compacted
// entries with all lanes busy.  At 50M persons: 400 us a weekday and 930 us a weekend day
// with marking, 620 and 1,250 before (look-back, selects, add / add-with-carry Threefry).
constexpr int kSchedThreads = 256, kSchedWarps = kSchedThreads / 32;
constexpr int kSchedPart = 256;       // persons whose entries a warp's part holds (a person's place fits a byte)
constexpr int kSchedBlocksPerSm = 5;  // 47 and 48 registers; 6 (40) and 7 (32, spills) cost 15% and 21% more on weekends
                                      // and 5% and 55% more on weekdays at 50M persons

// Adds the block's histograms to instance k's stripe of the day's digit histograms
// and clears them.  Block-uniform; the caller separates it from other uses of s_dh by barriers.
__device__ __forceinline__ void sched_flush_digits(int (*s_dh)[256], int passes, int *digit_hist, int k)
{
    int *h = digit_hist + ((size_t)k * kDigitStripes + blockIdx.x % kDigitStripes) * kMaxRadixPasses * 256;
    for (int p = 0; p < passes; p++) {
        const int v = s_dh[p][threadIdx.x];
        if (v) red_add(&h[p * 256 + threadIdx.x], v);
        s_dh[p][threadIdx.x] = 0;
    }
}

// The warp's part of `n` entries: into the digit histograms, and (unless the instance is
// dense) to `entries`.
__device__ __forceinline__ void sched_flush_entries(const uint32_t *my_key, const uint8_t *my_who, int n, int lane,
                                                    uint32_t bb, uint32_t first, int (*s_dh)[256], int passes,
                                                    int dbits, bool dense, uint2 *entries)
{
    const uint32_t dmask = (1u << dbits) - 1u;
    __syncwarp();
    for (int e = lane; e < n; e += 32) {
        const uint32_t b = my_key[e] - bb;
#pragma unroll
        for (int p = 0; p < kMaxRadixPasses; p++)
            if (p < passes) atomicAdd(&s_dh[p][(b >> (dbits * p)) & dmask], 1);
        if (!dense) entries[e] = make_uint2(b, first + my_who[e]);
    }
    __syncwarp();
}

template <bool WEEKEND>
__global__ void __launch_bounds__(kSchedThreads, kSchedBlocksPerSm)
    k_sched(const InstConst *ic, InstState *is, const int32_t *tile_inst, int regions, int C, const uint8_t *age,
            const uint32_t *mark, int32_t *keys, int *digit_hist, int passes, int dbits, uint2 *entries,
            int32_t *region_count, uint2 *slot, int slots, const Scalars *sc, int day)
{
    day = launch_day(day, sc);
    if (*(volatile const int *)&sc->done) return;
    // the day's bucket slots, for the sort (only on a day that goes on: the tables of the
    // last day with infected stay)
    for (int i = blockIdx.x * kSchedThreads + threadIdx.x; i < slots; i += gridDim.x * kSchedThreads)
        slot[i] = make_uint2(0u, 0u);
    static_assert(kSchedThreads == 256, "one thread per digit in sched_flush_digits");
    constexpr int kPer = WEEKEND ? 3 : 2;                       // keys per person
    constexpr int kCap = kPer * kSchedPart;                     // entries of a warp's part at most
    constexpr int kRound = WEEKEND ? 32 : 64;                   // persons per round
    __shared__ __align__(16) uint32_t s_key[kSchedWarps][kCap]; // marked keys of the warp's persons (global buckets)
    __shared__ uint8_t s_who[kSchedWarps][kCap];                // their persons, numbered within the part
    __shared__ int s_dh[kMaxRadixPasses][256];                  // digit histograms of the current instance's entries
    __shared__ ErrandRow s_row[2 * kErrandRows];                // errand tables (weekday: hour 0, hour 1)
    __shared__ int s_next;                                      // next region of the block's run
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    uint32_t *const my_key = s_key[warp];
    uint8_t *const my_who = s_who[warp];
    for (int i = threadIdx.x; i < kMaxRadixPasses * 256; i += kSchedThreads) (&s_dh[0][0])[i] = 0;
    const int r1 = (int)((long long)regions * (blockIdx.x + 1) / gridDim.x);
    for (int r = (int)((long long)regions * blockIdx.x / gridDim.x); r < r1;) {
        // the block's regions of one instance: [r, end)
        const int inst = tile_inst[(long long)r * C / kPersonTile];
        const InstConst &ik = ic[inst];
        const int end = min(r1, ik.pend / C);
        if (!instance_running(ik, is[inst], day)) {
            r = end;
            continue;
        }
        const TfKey key = make_key(ik.c);
        const int pbase = ik.pbase, N = ik.c.N;
        const int bb = ik.bbase[WEEKEND ? 1 : 0];
        const int lo = ik.c.type_offset[WEEKEND ? 9 : 8], R = ik.c.L - lo;
        int32_t *const kk = keys + ik.kbase;   // the instance's key slots: weekday hour 0 at [0, N), hour 1 at [N, 2N)
        const bool dense = is[inst].dense != 0;
        const unsigned long long E0 = is[inst].errand_offset;
        if (threadIdx.x < 2 * kErrandRows) {
            const int hour = threadIdx.x / kErrandRows;
            s_row[threadIdx.x] = errand_table_row<WEEKEND>(ik.c, threadIdx.x % kErrandRows, bb + hour * R, lo);
        }
        if (threadIdx.x == 0) s_next = r;
        __syncthreads();
        for (;;) {
            int q = 0;
            if (lane == 0) q = atomicAdd(&s_next, 1);
            q = __shfl_sync(0xffffffffu, q, 0);
            if (q >= end) break;
            const int rp = q * C - pbase;                       // the region's first person, instance numbering
            const int rend = min(rp + C, N);                    // (below rp when the region is all padding)
            uint2 *const mine = entries + 3 * (size_t)q * C;    // the region's slots
            int run = 0, part = rp, written = 0;                // entries in the part, its first person, entries flushed
#pragma unroll 1
            for (int p0 = rp; p0 < rend; p0 += kRound) {
                if (p0 - part >= kSchedPart) {
                    sched_flush_entries(my_key, my_who, run, lane, (uint32_t)bb, (uint32_t)(pbase + part), s_dh, passes,
                                        dbits, dense, mine + written);
                    written += run;
                    run = 0;
                    part = p0;
                }
                if (WEEKEND) {
                    // kernel_assignWeekendErrands (PandemicSim.cu:2082-2094): counters E0 + 2p, E0 + 2p + 1
                    const int p = p0 + lane;
                    uint32_t w[8];
                    tf2x64(key, E0 + 2ull * (unsigned long long)p, w);
                    tf2x64(key, E0 + 2ull * (unsigned long long)p + 1ull, w + 4);
                    int h[3];
                    weekend_hours(w, h[0], h[1], h[2]);
                    uint32_t kb[3];
#pragma unroll
                    for (int k = 0; k < 3; k++)
                        kb[k] = (uint32_t)(errand_bucket<true>(s_row, w[3 + k], errand_p9<true>(true), 0) + h[k] * R);
                    if (dense) {
                        // the round's 96 key slots, written in whole 16-byte pieces through the
                        // unused end of the warp's part (run <= 3 (p0 - part))
                        uint32_t *const stage = my_key + 3 * (p0 - part);
#pragma unroll
                        for (int k = 0; k < 3; k++) stage[3 * lane + k] = kb[k];
                        __syncwarp();
                        if (p0 + 32 <= N) {
                            if (lane < 24)
                                *reinterpret_cast<uint4 *>(kk + 3 * (size_t)p0 + 4 * lane) =
                                    *reinterpret_cast<const uint4 *>(stage + 4 * lane);
                        } else {
                            for (int i = lane; i < 3 * (N - p0); i += 32) kk[3 * (size_t)p0 + i] = (int32_t)stage[i];
                        }
                        __syncwarp();   // the stage is read before the entries below reach it
                    }
                    const uint32_t in = p < N ? 1u : 0u;
                    uint32_t mk[3];
#pragma unroll
                    for (int k = 0; k < 3; k++) mk[k] = mark_bit(mark, kb[k]) & in;
                    const uint32_t cnt = mk[0] + mk[1] + mk[2];
                    const unsigned b0 = __ballot_sync(0xffffffffu, cnt & 1u), b1 = __ballot_sync(0xffffffffu, cnt & 2u);
                    if ((b0 | b1) == 0) continue;
                    int pos = run + __popc(b0 & lt) + 2 * __popc(b1 & lt);
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        if (mk[k]) {
                            my_key[pos] = kb[k];
                            my_who[pos] = (uint8_t)(p - part);
                        }
                        pos += (int)mk[k];
                    }
                    run += __popc(b0) + 2 * __popc(b1);
                } else {
                    // kernel_assignWeekdayAfterschoolAndErrands (PandemicSim.cu:2972-3022): counter E0 + p / 2
                    const int p = p0 + 2 * lane;
                    uint32_t w[4];
                    const uchar2 ag = *reinterpret_cast<const uchar2 *>(age + pbase + p);
                    tf2x64(key, E0 + (uint64_t)(p / 2), w);
                    const bool ad[2] = {ag.x == 5, ag.y == 5};
                    // a child's second draw is its first (one afterschool place)
                    w[1] = ad[0] ? w[1] : w[0];
                    w[3] = ad[1] ? w[3] : w[2];
                    constexpr int kChild = (kErrandRows - 1) * (int)sizeof(ErrandRow);
                    const float p9[2] = {errand_p9<false>(ad[0]), errand_p9<false>(ad[1])};
                    const int base[2] = {ad[0] ? 0 : kChild, ad[1] ? 0 : kChild};
                    uint32_t kb[4];   // [person][hour]
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        kb[k] = (uint32_t)errand_bucket<false>(s_row + (k & 1) * kErrandRows, w[k], p9[k >> 1], base[k >> 1]);
                    const uint32_t in[2] = {p < N ? 1u : 0u, p + 1 < N ? 1u : 0u};
                    uint32_t mk[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) mk[k] = mark_bit(mark, kb[k]) & in[k >> 1];
                    if (dense && p + 1 < N) {
                        *reinterpret_cast<int2 *>(kk + p) = make_int2((int)kb[0], (int)kb[2]);
                        if ((N & 1) == 0) {   // hour 1's slots start 8-byte aligned
                            *reinterpret_cast<int2 *>(kk + (size_t)N + p) = make_int2((int)kb[1], (int)kb[3]);
                        } else {
                            kk[(size_t)N + p] = (int)kb[1];
                            kk[(size_t)N + p + 1] = (int)kb[3];
                        }
                    } else if (dense && p < N) {
                        kk[p] = (int)kb[0];
                        kk[(size_t)N + p] = (int)kb[1];
                    }
                    const uint32_t cnt = mk[0] + mk[1] + mk[2] + mk[3];
                    const unsigned b0 = __ballot_sync(0xffffffffu, cnt & 1u), b1 = __ballot_sync(0xffffffffu, cnt & 2u),
                                   b2 = __ballot_sync(0xffffffffu, cnt & 4u);
                    if ((b0 | b1 | b2) == 0) continue;
                    int pos = run + __popc(b0 & lt) + 2 * __popc(b1 & lt) + 4 * __popc(b2 & lt);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        if (mk[k]) {
                            my_key[pos] = kb[k];
                            my_who[pos] = (uint8_t)(p + (k >> 1) - part);
                        }
                        pos += (int)mk[k];
                    }
                    run += __popc(b0) + 2 * __popc(b1) + 4 * __popc(b2);
                }
            }
            sched_flush_entries(my_key, my_who, run, lane, (uint32_t)bb, (uint32_t)(pbase + part), s_dh, passes, dbits,
                                dense, mine + written);
            written += run;
            if (lane == 0) {
                region_count[q] = written;
                if (written) red_add(&is[inst].marked, written);
            }
        }
        __syncthreads();
        sched_flush_digits(s_dh, passes, digit_hist, inst);
        __syncthreads();
        r = end;
    }
}

// Every person's schedule keys of the last day run, as the sort numbers them.
__global__ void k_day_keys(const InstConst *ic, const InstState *is, const uint8_t *age, int weekend, int32_t *keys)
{
    const int k = blockIdx.y;
    const InstConst &ik = ic[k];
    const SimConst &c = ik.c;
    const TfKey key = make_key(c);
    const unsigned long long E0 = is[k].errand_offset;
    int32_t *const kk = keys + ik.kbase;
    const int lo = c.type_offset[weekend ? 9 : 8], R = c.L - lo, bb = ik.bbase[weekend ? 1 : 0];
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < c.N; p += gridDim.x * blockDim.x) {
        if (weekend) {
            int d[3];
            weekend_errands(c, key, E0 + 2ull * (unsigned long long)p, lo, R, d);
            for (int j = 0; j < 3; j++) kk[3 * (size_t)p + j] = bb + d[j];
        } else {
            uint32_t w[4];
            tf2x64(key, E0 + (uint64_t)(p / 2), w);
            int k1, k2;
            weekday_pair_keys(c, w, p & 1, age[ik.pbase + p] == 5, lo, R, k1, k2);
            kk[p] = bb + k1;
            kk[(size_t)c.N + p] = bb + k2;
        }
    }
}

cudaError_t launch_day_keys(const DevArrays &d, bool weekend, cudaStream_t s)
{
    k_day_keys<<<dim3(std::min(div_up(d.persons_max, 256), 8 * sm_count()), d.K), 256, 0, s>>>(d.ic, d.is, d.age,
                                                                                         weekend ? 1 : 0, d.keys);
    count_launch();
    return cudaGetLastError();
}

int day_buckets(const SimConst &c, bool weekend)
{
    return weekend ? 10 * (c.L - c.type_offset[9]) : 2 * (c.L - c.type_offset[8]);
}

// Persons per region of the schedule kernel: the largest power of two that still
// leaves two regions for every resident warp (small simulations spread over the SMs,
// large ones have fewer counts to scan and longer runs of entries per region: a run of
// 24 instances of 1M persons, most of them with few infected, takes 72 ms, with four
// regions a warp 76, because the sort looks up twice as many regions an entry).
static int sched_region_persons(long long P)
{
    int C = kSchedMaxRegion;
    while (C > kSchedMinRegion && P / C < 2ll * kSchedWarps * kSchedBlocksPerSm * sm_count()) C /= 2;
    return C;
}

cudaError_t launch_schedule(const DevArrays &d, bool weekend, int day, DayQueue &q)
{
    const int C = sched_region_persons(d.P), regions = d.P / C;
    const int blocks = std::min(div_up(regions, kSchedWarps), kSchedBlocksPerSm * sm_count());
    const int passes = radix_passes(d.bucket_max[weekend ? 1 : 0]), dbits = radix_digit_bits(d.bucket_max[weekend ? 1 : 0]);
    return queue_kernel(q, weekend ? k_sched<true> : k_sched<false>, blocks, kSchedThreads, 0, d.ic, d.is, d.tile_inst,
                        regions, C, d.age, d.mark, d.keys, d.digit_hist, passes, dbits, d.rp1, d.region_count, d.bkt,
                        d.buckets[weekend ? 1 : 0], d.sc, day);
}

// The day's radix sort: one sorted segment per instance, keys local to the instance,
// so the passes cover the largest instance's buckets only.  A segment's first pass
// reads the marked entries the schedule wrote region by region to the instance's part of rp1
// in person order, or, for an instance dense today, every schedule key (keeping the
// marked ones).  Equal keys come from one hour, in person order, in both inputs, so
// the sorted tables are the same.
static RadixArgs day_radix_args(const DevArrays &d, bool weekend)
{
    RadixArgs r;
    r.in = d.rp1;
    r.E = 3 * d.P;   // at most (sizes the persistent grid)
    r.buckets = d.bucket_max[weekend ? 1 : 0];
    r.p0 = d.rp0;
    r.p1 = d.rp1;
    r.out = (uint32_t *)d.bkt_people;
    r.table = d.bkt;
    r.digit_base = d.digit_base;
    r.seg.tile_prefix = d.tile_prefix;
    r.seg.ic = d.ic;
    r.seg.is = d.is;
    r.seg.segments = d.K;
    r.seg.region_prefix = d.region_prefix;
    r.seg.chunk_region = d.chunk_region;
    r.seg.region_persons = sched_region_persons(d.P);
    r.seg.day_keys = d.keys;
    r.seg.tile_prefix0 = d.tile_prefix0;
    r.seg.mark = d.mark;
    r.seg.weekend = weekend ? 1 : 0;
    r.status = d.radix_status;
    r.ctl = d.radix_ctl;
    r.error = &d.sc->error;
    r.skip = &d.sc->done;
    r.blocks_per_sm = d.tune.radix_blocks_per_sm;
    return r;
}

// The day's sort tables, a row of blocks per instance (blockIdx.y), every block with one
// task and no wait for another.
//  * Block 0: the digit bases of the instance's segment from the digit histograms the
//    schedule kernel accumulated (summing the stripes, clearing them).  Every entry has
//    a digit in every pass, so the passes' totals are equal and one scan over all
//    passes' digits gives every pass's.
//  * Block 1, of the first row: the numbers of the segments' radix tiles (tile_prefix),
//    and the day's materialised entries added to the running total.
//  * The others: 4096 regions of the instance each.  Their place in the segment is an
//    exclusive scan of the regions' entry counts; a block sums the counts before its
//    own itself (at most a few hundred KB from L2) rather than wait for the others.
//    Output: region_prefix, and for every kRegionChunk entries of the segment the region
//    the first of them lies in, its prefix, its end and the next one's (chunk_region).
constexpr int kBasesThreads = 1024, kBasesRegions = 4 * kBasesThreads, kBasesTasks = 2;
static_assert(kBasesThreads == kMaxRadixPasses * 256, "a thread per digit of every pass");

__global__ void __launch_bounds__(kBasesThreads) k_day_digit_bases(int *digit_hist, int *digit_base, int passes,
                                                                   const InstConst *ic, const InstState *is, int K,
                                                                   int weekend, int C, const int32_t *region_count,
                                                                   int32_t *region_prefix, int4 *chunk_region,
                                                                   int32_t *tile_prefix, int32_t *tile_prefix0,
                                                                   Scalars *sc)
{
    if (*(volatile const int *)&sc->done) return;
    const int k = blockIdx.y, t = threadIdx.x, task = (int)blockIdx.x - kBasesTasks;
    if (task >= 0) {
        // regions of the block (an instance starts on a person tile, and 4 C persons divide one)
        const int r0 = ic[k].pbase / C, r1 = ic[k].pend / C, rb = r0 + task * kBasesRegions;
        if (rb >= r1 || is[k].marked == 0 || is[k].dense) return;
        int before = 0;
        for (int r = r0 + 4 * t; r < rb; r += kBasesRegions) {
            const int4 c = *reinterpret_cast<const int4 *>(region_count + r);
            before += c.x + c.y + c.z + c.w;
        }
        int4 c = make_int4(0, 0, 0, 0);
        const int r = rb + 4 * t;
        if (r < r1) c = *reinterpret_cast<const int4 *>(region_count + r);
        int carry = 0, total;
        if (task > 0) block_exclusive_scan<kBasesThreads, int>(before, carry);
        int at = carry + block_exclusive_scan<kBasesThreads, int>(c.x + c.y + c.z + c.w, total);
        if (r < r1) {
            int4 *const chunks = chunk_region + ic[k].kbase / kRegionChunk;
            const int n[5] = {c.x, c.y, c.z, c.w, r + 4 < r1 ? region_count[r + 4] : 0};
            int pre[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                pre[j] = at;
                at += n[j];
                for (int m = (pre[j] + kRegionChunk - 1) / kRegionChunk; m * kRegionChunk < at; m++)
                    chunks[m] = make_int4(r + j, pre[j], at, at + n[j + 1]);
            }
            *reinterpret_cast<int4 *>(region_prefix + r) = make_int4(pre[0], pre[1], pre[2], pre[3]);
        }
        return;
    }
    if (task == -kBasesTasks) {
        const int p = t / 256;
        unsigned v = 0;
        if (p < passes) {
            int *const h = digit_hist + (size_t)k * kDigitStripes * kMaxRadixPasses * 256 + t;
            int x[kDigitStripes];   // all loads before the first store
#pragma unroll
            for (int st = 0; st < kDigitStripes; st++) x[st] = h[st * kMaxRadixPasses * 256];
#pragma unroll
            for (int st = 0; st < kDigitStripes; st++) {
                v += (unsigned)x[st];
                h[st * kMaxRadixPasses * 256] = 0;
            }
        }
        unsigned total;
        const unsigned excl = block_exclusive_scan<kBasesThreads, unsigned>(v, total);
        // (modulo 2^32, like the scan)
        if (p < passes)
            digit_base[((size_t)k * passes + p) * 256 + t % 256] = (int)(excl - (unsigned)is[k].marked * (unsigned)p);
        return;
    }
    if (k != 0) return;
    int carry = 0, carry0 = 0;
    unsigned long long entries = 0;
    for (int b = 0; b < K; b += kBasesThreads) {
        const int i = b + t;
        const int m = i < K ? is[i].marked : 0;
        // the first pass reads every key of a dense instance, the appended entries otherwise
        const int m0 = (i < K && is[i].dense) ? (weekend ? 3 : 2) * ic[i].c.N : m;
        int total;
        const int excl = block_exclusive_scan<kBasesThreads, int>((m + kRadixTile - 1) / kRadixTile, total);
        if (i < K) tile_prefix[i] = carry + excl;
        carry += total;
        int total0;
        const int excl0 = block_exclusive_scan<kBasesThreads, int>((m0 + kRadixTile - 1) / kRadixTile, total0);
        if (i < K) tile_prefix0[i] = carry0 + excl0;
        carry0 += total0;
        int msum;
        block_exclusive_scan<kBasesThreads, int>(m, msum);
        entries += (unsigned long long)msum;
    }
    if (t == 0) {
        tile_prefix[K] = carry;
        tile_prefix0[K] = carry0;
        sc->materialised_sum += entries;
    }
}

cudaError_t launch_bucket_scan(const DevArrays &d, bool weekend, DayQueue &q)
{
    const int P = radix_passes(d.bucket_max[weekend ? 1 : 0]);
    const int C = sched_region_persons(d.P);
    const dim3 grid(kBasesTasks + std::max(1, div_up(d.persons_max / C, kBasesRegions)), d.K);
    return queue_kernel(q, k_day_digit_bases, grid, kBasesThreads, 0, d.digit_hist, d.digit_base, P, d.ic, d.is, d.K,
                        weekend ? 1 : 0, C, d.region_count, d.region_prefix, d.chunk_region, d.tile_prefix,
                        d.tile_prefix0, d.sc);
}

cudaError_t launch_bucket_sort(const DevArrays &d, bool weekend, DayQueue &q)
{
    return launch_radix_sort(day_radix_args(d, weekend), q);
}

// ------------------------------------------------------------------ infection
// device_selectRandomPersonFromLocation (PandemicSim.cu:2028-2071).  A location with
// at most one person gives victim = count and type NONE (kappa 0).  Without a table the
// location's persons are off, off + 1, ... (a household).
__device__ __forceinline__ int select_victim(int self, int off, int count, uint32_t r, int &victim,
                                             const int32_t *table = nullptr)
{
    if (count <= 1) {
        victim = count;
        return 0;
    }
    int o = (int)(r % (uint32_t)count);
    int v = table ? table[off + o] : off + o;
    if (v == self) {
        o = (o + 1) % count;
        v = table ? table[off + o] : off + o;
    }
    victim = v;
    return 1;
}

// The same for NC locations with tables, the tables' loads together.
template <int NC>
__device__ __forceinline__ void select_victims(int self, const int (&off)[NC], const int (&cnt)[NC],
                                               const int32_t *const (&table)[NC], const uint32_t *r, int *victim,
                                               int *kv)
{
    int o[NC];
#pragma unroll
    for (int j = 0; j < NC; j++) {
        kv[j] = cnt[j] > 1 ? 1 : 0;
        victim[j] = cnt[j];
        if (kv[j]) {
            o[j] = (int)(r[j] % (uint32_t)cnt[j]);
            victim[j] = table[j][off[j] + o[j]];
        }
    }
#pragma unroll
    for (int j = 0; j < NC; j++)
        if (kv[j] && victim[j] == self) victim[j] = table[j][off[j] + (o[j] + 1) % cnt[j]];
}

// First claims of the day, collected per warp in shared memory and appended to the
// day's list in runs: one update of the list's length for every run.  (One update per
// claim made all claims of a dense day queue at that one address, 0.3 of the 0.45 ms
// of a weekday at 12M persons.)  Claims past the queue's end go to the list directly.
constexpr int kQueueLen = 96, kQueueRun = 32;

struct ClaimQueue {
    int32_t *entry;   // kQueueLen
    int *count;       // claims pushed since the last run (may exceed kQueueLen)
    int32_t *new_list;
    Scalars *sc;

    __device__ __forceinline__ void push(int32_t e) const
    {
        const int i = atomicAdd(count, 1);
        if (i < kQueueLen) entry[i] = e;
        else new_list[atomicAdd(&sc->new_count, 1)] = e;
    }

    // Appends the queue when it holds at least `run` claims; called by the whole warp.
    __device__ __forceinline__ void flush(int run, int lane) const
    {
        __syncwarp();
        // lane 0's count for all: no lane may push before every lane has decided
        int n = lane == 0 ? *(volatile int *)count : 0;
        n = min(__shfl_sync(0xffffffffu, n, 0), kQueueLen);
        if (n < run) return;
        int at = 0;
        if (lane == 0) at = atomicAdd(&sc->new_count, n);
        at = __shfl_sync(0xffffffffu, at, 0);
        for (int i = lane; i < n; i += 32) new_list[at + i] = entry[i];
        __syncwarp();
        if (lane == 0) *count = 0;
        __syncwarp();
    }
};

// The calling warp's queue of a block of WARPS warps, empty.
template <int WARPS>
__device__ __forceinline__ ClaimQueue claim_queue(int32_t *new_list, Scalars *sc)
{
    __shared__ int32_t s_entry[WARPS][kQueueLen];
    __shared__ int s_count[WARPS];
    const int warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) s_count[warp] = 0;
    __syncwarp();
    return {s_entry[warp], &s_count[warp], new_list, sc};
}

struct Infector {
    int me, pos;   // global person id, position in the batch's infected list
    float prob[2];
    int gen[2];
};

// device_processContacts (PandemicSim.cu:3106-3233) with the claim rule: a
// successful draw on a victim whose strain status was susceptible at the start of
// the day claims (victim, strain) with key (position, slot); the smallest key wins.
// A victim is only ever drawn by infectors of its own instance, whose list positions
// keep the instance's order.
//
// The draws come first, then the loads of every victim drawn, then a strain's claims:
// one after the other, each waits for its own load and its own atomic.
template <int NC>
__device__ __forceinline__ void process_contacts(const SimConst &c, const TfKey &key, const Infector &inf,
                                                 unsigned long long ctr, const int (&victims)[NC],
                                                 const int (&kv)[NC], const uint32_t *state,
                                                 unsigned long long *claim, const ClaimQueue &queue)
{
    uint32_t w[16];
    tf2x64(key, ctr + 0, w + 0);
    tf2x64(key, ctr + 1, w + 4);
    tf2x64(key, ctr + 2, w + 8);
    tf2x64(key, ctr + 3, w + 12);
    unsigned hits = 0;   // bit 2 j + strain
#pragma unroll
    for (int j = 0; j < NC; j++) {
        const float kf = __int2float_rn(kv[j]);
#pragma unroll
        for (int strain = 0; strain < 2; strain++)
            if (to_unit(w[2 * j + strain]) < __fmul_rn(inf.prob[strain], kf)) hits |= 1u << (2 * j + strain);
    }
    uint32_t st[NC];
#pragma unroll
    for (int j = 0; j < NC; j++) {
        st[j] = 0u;
        if ((hits >> (2 * j)) & 3u) st[j] = state[victims[j]];
    }
#pragma unroll
    for (int strain = 0; strain < 2; strain++) {
        unsigned long long old[NC];
#pragma unroll
        for (int j = 0; j < NC; j++) {
            const int u = 2 * j + strain;
            old[j] = 0ull;
            if (((hits >> u) & 1u) && ((st[j] >> (8 * strain)) & 0xFFu) == 1u) {
                const int profile = infection_profile(c, w[u] ^ w[(u + 1) & 15]);
                const unsigned long long k =
                    ((unsigned long long)((long long)inf.pos * 8 + j) << 16) | ((unsigned long long)profile << 8) |
                    (unsigned long long)(inf.gen[strain] & 0xFF);
                old[j] = atomicMin(&claim[2 * (size_t)victims[j] + strain], k);
            }
        }
#pragma unroll
        for (int j = 0; j < NC; j++)
            if (old[j] == ~0ull) queue.push(2 * victims[j] + strain);
    }
}

// The generation of its victims, of each strain the infector (status word st) has.
__device__ __forceinline__ void infector_gens(Infector &inf, uint32_t st, const uint8_t *gen_p, const uint8_t *gen_s)
{
    inf.gen[0] = (st & 0xFFu) >= 2u ? gen_p[inf.me] + 1 : 0xFF;
    inf.gen[1] = ((st >> 8) & 0xFFu) >= 2u ? gen_s[inf.me] + 1 : 0xFF;
}

// Infection probability of each strain (device_calculateInfectionProbability); -1
// when the strain is not infectious today.
__device__ __forceinline__ void infector_probs(const SimConst &c, uint32_t st, int day, int ksum, float prob[2])
{
#pragma unroll
    for (int strain = 0; strain < 2; strain++) {
        const uint32_t status = strain ? ((st >> 8) & 0xFFu) : (st & 0xFFu);
        const uint32_t dday = strain ? (st >> 24) : ((st >> 16) & 0xFFu);
        prob[strain] = -1.f;
        if (status >= 2u) {
            const int pd = day - (int)dday;
            if (pd >= 0 && pd < 10) prob[strain] = infection_probability(c, (int)status - 2, pd, strain, ksum);
        }
    }
}

struct InfectArgs {
    const InstConst *ic;
    const InstState *is;
    const uint32_t *state;
    const uint8_t *gen_p, *gen_s, *age;
    const uint4 *prec;
    const int32_t *wp_people;
    const uint2 *bkt;
    const int32_t *bkt_people, *infected, *infected_inst;
    const int2 *read;   // the buckets an infector's contacts read (read_buckets)
    unsigned long long *claim;
    int32_t *new_list;
    Scalars *sc;
    int coop_most;   // up to this many infectors, eight lanes work on one
};

// Errand contacts of a weekday infector that go to its first bucket, of two.
__device__ __forceinline__ int first_errands(int2 read) { return read.x < 0 ? 0 : (read.y < 0 ? 2 : 1); }

// An infector's packed record: one 128-bit read-only load.
__device__ __forceinline__ uint4 load_record(const uint4 *prec, int me) { return __ldg(&prec[me]); }

// ---------------------------------------------------- warp-cooperative contacts
// The same draws with eight lanes per infector (four infectors per warp round).  Lane
// j of a group first computes one Threefry block of the infector's draws, all in
// parallel:
//   weekday  j = 0, 1: contact words (counters R + 6 pos, +1); j = 2..5: infection
//            words (+2..+5)
//   weekend  j = 0: contact words; j = 1: the Threefry-2x32 errand block; j = 2..5:
//            infection words
// then picks contact slot j's victim (its own gather chain) and draws slot j's two
// infections.  The words reach the lanes that use them by shuffles; the contact sum
// is a shuffle reduction over the group.  Every draw, victim and claim key equals the
// one-thread-per-infector kernels' (same counters, same words, same slots).
constexpr unsigned kFull = 0xffffffffu;
// The thread-per-infector kernels work this way themselves on a day of at most
// kCoopPerSm infectors an SM, where a thread's seven Threefry blocks in a row take longer
// than the chip is busy: 10 us instead of 13 for a weekday of 100,000 persons, 1.12 ms
// instead of 1.31 for the weekdays of a 1M run (64, 192 and 320 an SM: 1.19, 1.18, 1.23);
// on larger days one thread an infector is faster (12M: 10 ms, 17.5 this way).
constexpr int kCoopPerSm = 128;

__device__ __forceinline__ uint32_t pick4(int i, uint32_t q0, uint32_t q1, uint32_t q2, uint32_t q3)
{
    return i == 0 ? q0 : (i == 1 ? q1 : (i == 2 ? q2 : q3));
}

// Slot j's infection draws: words W[2j], W[2j+1], W[(2j+2) & 15] of the four
// infection blocks, which lanes 2..5 of the group hold.
__device__ __forceinline__ void infection_words(const uint32_t blk[4], int gl, int j, uint32_t &w0, uint32_t &w1,
                                                uint32_t &w2)
{
    const int sa = gl + 2 + (j >> 1), sb = gl + 2 + (((j + 1) & 7) >> 1);
    const uint32_t a0 = __shfl_sync(kFull, blk[0], sa), a1 = __shfl_sync(kFull, blk[1], sa);
    const uint32_t a2 = __shfl_sync(kFull, blk[2], sa), a3 = __shfl_sync(kFull, blk[3], sa);
    const uint32_t b0 = __shfl_sync(kFull, blk[0], sb), b2 = __shfl_sync(kFull, blk[2], sb);
    w0 = (j & 1) ? a2 : a0;
    w1 = (j & 1) ? a3 : a1;
    w2 = ((j + 1) & 1) ? b2 : b0;
}

// Slot j's two infection draws against its victim (process_contacts for one slot).
__device__ __forceinline__ void claim_slot(const SimConst &c, const InfectArgs &a, int pos, int j, int me, int victim,
                                           int kv, const float prob[2], uint32_t w0, uint32_t w1, uint32_t w2,
                                           const ClaimQueue &queue)
{
    const float kf = __int2float_rn(kv);
#pragma unroll
    for (int strain = 0; strain < 2; strain++) {
        const float y = to_unit(strain ? w1 : w0);
        if (y < __fmul_rn(prob[strain], kf)) {
            const uint32_t st = a.state[victim];
            const uint32_t vstatus = strain ? ((st >> 8) & 0xFFu) : (st & 0xFFu);
            if (vstatus == 1u) {
                const int profile = infection_profile(c, strain ? (w1 ^ w2) : (w0 ^ w1));
                const int gen = ((strain ? a.gen_s[me] : a.gen_p[me]) + 1) & 0xFF;
                const unsigned long long k = ((unsigned long long)((long long)pos * 8 + j) << 16) |
                                             ((unsigned long long)profile << 8) | (unsigned long long)gen;
                const unsigned long long old = atomicMin(&a.claim[2 * (size_t)victim + strain], k);
                if (old == ~0ull) queue.push(2 * victim + strain);
            }
        }
    }
}

template <bool WEEKEND>
__device__ __forceinline__ void infect_coop(const InfectArgs &a, int day, int I, const ClaimQueue &queue)
{
    const int lane = threadIdx.x & 31, j = lane & 7, gl = lane & ~7;
    const int gwarp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int nwarps = (int)((gridDim.x * blockDim.x) >> 5);
    for (int base = gwarp * 4; base < I; base += nwarps * 4) {   // warp-uniform
        const int pos0 = base + (lane >> 3);
        const bool act = pos0 < I;       // groups past the list's end shadow its last entry
        const int pos = act ? pos0 : I - 1;
        const int inst = a.infected_inst[pos];
        const InstConst &ik = a.ic[inst];
        const SimConst &c = ik.c;
        const InstState &s = a.is[inst];
        const int me = a.infected[pos];
        const int lme = me - ik.pbase;
        const unsigned long long ctr = s.infect_offset + 6ull * (unsigned long long)(pos - s.start);
        const TfKey key = make_key(c);
        const uint4 rec = load_record(a.prec, me);
        const int2 read = a.read[pos];
        // one Threefry block per lane
        uint32_t blk[4] = {0u, 0u, 0u, 0u};
        if (WEEKEND && j == 1) {
            tf2x32(key, (uint32_t)(ctr + 1), blk);   // :1895-1901, counter truncated to 32 bits
        } else {
            tf2x64(key, ctr + (uint64_t)j, blk);
        }
        // contact words: W[j] of blocks R, R + 1 (weekday), W[j] of block R (weekend)
        const int csrc = WEEKEND ? gl : gl + (j >> 2);
        const uint32_t q0 = __shfl_sync(kFull, blk[0], csrc), q1 = __shfl_sync(kFull, blk[1], csrc);
        const uint32_t q2 = __shfl_sync(kFull, blk[2], csrc), q3 = __shfl_sync(kFull, blk[3], csrc);
        const uint32_t wc = pick4(j & 3, q0, q1, q2, q3);
        int victim = -1, kv = 0;
        const int hoff = (int)rec.x, hcnt = prec_household_size(rec.w);
        if (WEEKEND) {
            const uint32_t v0 = __shfl_sync(kFull, blk[0], gl + 1), v1 = __shfl_sync(kFull, blk[1], gl + 1);
            if (j < 3) {
                kv = select_victim(me, hoff, hcnt, wc, victim);
            } else if (j < 5) {
                const uint2 slot = a.bkt[j == 3 ? read.x : read.y];
                const int eoff = bucket_start(slot), ecnt = bucket_count(slot);
                kv = select_victim(me, eoff, ecnt, j == 3 ? v0 : v1, victim, a.bkt_people);
            }
        } else {
            const int desired = prec_desired(rec.w);
            if (j < 3) {
                kv = select_victim(me, hoff, hcnt, wc, victim);
            } else if (j < 3 + desired) {
                kv = select_victim(me, (int)rec.y, (int)rec.z, wc, victim, a.wp_people);
            } else {
                const int e = j - 3 - desired;   // the infector's e-th errand contact of two
                if (e < 2) {
                    const uint2 slot = a.bkt[e < first_errands(read) ? read.x : read.y];
                    const int eoff = bucket_start(slot), ecnt = bucket_count(slot);
                    kv = select_victim(me, eoff, ecnt, wc, victim, a.bkt_people);
                }
            }
        }
        // the contact sum over the group's slots
        int ksum = kv;
        ksum += __shfl_xor_sync(kFull, ksum, 4);
        ksum += __shfl_xor_sync(kFull, ksum, 2);
        ksum += __shfl_xor_sync(kFull, ksum, 1);
        if (!WEEKEND && j >= 3 && j < 3 + prec_desired(rec.w) && kv != 0 &&
            (ik.absent_thr != 0 || (day >= ik.closure_start && day < ik.closure_end))) {
            // interventions void a workplace / school contact after it counted in ksum
            const bool closed = day >= ik.closure_start && day < ik.closure_end && prec_school(rec.w);
            const bool me_absent = prec_age(rec.w) == 5 &&
                                   intervention_hash(c.key0, c.key1, kTagAbsent, day, lme) < ik.absent_thr;
            const bool v_absent = ik.absent_thr != 0 && a.age[victim] == 5 &&
                                  intervention_hash(c.key0, c.key1, kTagAbsent, day, victim - ik.pbase) <
                                      ik.absent_thr;
            if (closed || me_absent || v_absent) kv = 0;
        }
        float prob[2];
        infector_probs(c, a.state[me], day, ksum, prob);
        uint32_t w0, w1, w2;
        infection_words(blk, gl, j, w0, w1, w2);
        if (act && kv != 0 && j < (WEEKEND ? 5 : 8)) 
            claim_slot(c, a, pos, j, me, victim, kv, prob, w0, w1, w2, queue);
        queue.flush(kQueueRun, lane);
    }
    queue.flush(1, lane);
}

template <bool WEEKEND>
__global__ void __launch_bounds__(256) k_infect_coop(InfectArgs a, int day)
{
    Scalars *sc = a.sc;
    day = launch_day(day, sc);
    if (sc->done) return;
    infect_coop<WEEKEND>(a, day, sc->infected, claim_queue<8>(a.new_list, sc));
}

// kernel_doWeekday + device_makeContacts_weekday (PandemicSim.cu:3236-3308, :1669-1829),
// one thread per infector.  Bound by random 32-byte sectors (record, keys, bucket
// slots, tables, victims, claims) and by how many a warp has in flight, so each kind is
// loaded for all contacts together: 36 ms of a 48-instance run's weekdays on a GB300, 42
// with every contact's loads after the last one's.  Eight blocks an SM (64 registers) are
// as good as six (80) there and better than ten (38 ms) or twelve (43).
__global__ void __launch_bounds__(128, 8) k_infect_weekday(InfectArgs a, int day)
{
    Scalars *sc = a.sc;
    day = launch_day(day, sc);
    if (sc->done) return;
    const int I = sc->infected;
    const ClaimQueue queue = claim_queue<4>(a.new_list, sc);
    if (I <= a.coop_most) {
        infect_coop<false>(a, day, I, queue);
        return;
    }
    const int lane = threadIdx.x & 31;
    for (int base = blockIdx.x * blockDim.x + threadIdx.x - lane; base < I; base += gridDim.x * blockDim.x) {
        queue.flush(kQueueRun, lane);
        const int pos = base + lane;
        if (pos >= I) continue;   // (the last round; the warp meets again at the flush)
        const int inst = a.infected_inst[pos];
        const InstConst &ik = a.ic[inst];
        const SimConst &c = ik.c;
        const InstState &s = a.is[inst];
        const TfKey key = make_key(c);
        Infector inf;
        inf.pos = pos;
        inf.me = a.infected[pos];
        const int me = inf.me;
        const int lme = me - ik.pbase;  // the instance's person number
        const unsigned long long ctr = s.infect_offset + 6ull * (unsigned long long)(pos - s.start);
        const uint4 rec = load_record(a.prec, me);
        uint32_t w[8];
        tf2x64(key, ctr, w);
        tf2x64(key, ctr + 1, w + 4);
        const bool adult = prec_age(rec.w) == 5;
        const uint32_t mine = a.state[me];
        // errands / afterschool
        const int2 read = a.read[pos];
        const uint2 none = make_uint2(0u, 0u);
        const uint2 slot0 = read.x >= 0 ? a.bkt[read.x] : none, slot1 = read.y >= 0 ? a.bkt[read.y] : none;
        infector_gens(inf, mine, a.gen_p, a.gen_s);
        int victims[8], kv[8];
        // household: offset + r % count, the household table is the identity
        const int hoff = (int)rec.x, hcnt = prec_household_size(rec.w);
#pragma unroll
        for (int j = 0; j < 3; j++) kv[j] = select_victim(me, hoff, hcnt, w[j], victims[j]);
        // then the workplace's or school's max-contacts, then each errand hour's
        const int desired = prec_desired(rec.w);
        const int want0 = first_errands(read);
        int off[5], cnt[5];
        const int32_t *table[5];
#pragma unroll
        for (int j = 0; j < 5; j++) {
            const int e = j - desired;
            const uint2 slot = e < want0 ? slot0 : slot1;
            off[j] = e < 0 ? (int)rec.y : bucket_start(slot);
            cnt[j] = e < 0 ? (int)rec.z : (e < 2 ? bucket_count(slot) : 0);
            table[j] = e < 0 ? a.wp_people : a.bkt_people;
        }
        select_victims<5>(me, off, cnt, table, w + 3, victims + 3, kv + 3);
        int ksum = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) ksum += kv[j];
        infector_probs(c, mine, day, ksum, inf.prob);
        // interventions: a closed school or an absent adult voids the workplace / school
        // contacts; they keep their share of ksum, so the contact does not happen
        // rather than passing its weight to the others
        if (desired > 0 && (ik.absent_thr != 0 || (day >= ik.closure_start && day < ik.closure_end))) {
            const bool closed = day >= ik.closure_start && day < ik.closure_end && prec_school(rec.w);
            const bool me_absent =
                adult && intervention_hash(c.key0, c.key1, kTagAbsent, day, lme) < ik.absent_thr;
            int age[3];
#pragma unroll
            for (int j = 0; j < 3; j++) {
                age[j] = 0;
                if (j < desired && kv[3 + j] != 0 && ik.absent_thr != 0) age[j] = a.age[victims[3 + j]];
            }
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const bool v_absent = age[j] == 5 && intervention_hash(c.key0, c.key1, kTagAbsent, day,
                                                                       victims[3 + j] - ik.pbase) < ik.absent_thr;
                if (j < desired && (closed || me_absent || v_absent)) kv[3 + j] = 0;
            }
        }
        process_contacts<8>(c, key, inf, ctr + 2, victims, kv, a.state, a.claim, queue);
    }
    queue.flush(1, lane);
}

// kernel_doWeekend + device_makeContacts_weekend (PandemicSim.cu:3311-3379, :1833-1950)
__global__ void __launch_bounds__(128, 8) k_infect_weekend(InfectArgs a, int day)
{
    Scalars *sc = a.sc;
    day = launch_day(day, sc);
    if (sc->done) return;
    const int I = sc->infected;
    const ClaimQueue queue = claim_queue<4>(a.new_list, sc);
    if (I <= a.coop_most) {
        infect_coop<true>(a, day, I, queue);
        return;
    }
    const int lane = threadIdx.x & 31;
    for (int base = blockIdx.x * blockDim.x + threadIdx.x - lane; base < I; base += gridDim.x * blockDim.x) {
        queue.flush(kQueueRun, lane);
        const int pos = base + lane;
        if (pos >= I) continue;   // (the last round; the warp meets again at the flush)
        const int inst = a.infected_inst[pos];
        const InstConst &ik = a.ic[inst];
        const SimConst &c = ik.c;
        const InstState &s = a.is[inst];
        const TfKey key = make_key(c);
        Infector inf;
        inf.pos = pos;
        inf.me = a.infected[pos];
        const int me = inf.me;
        const unsigned long long ctr = s.infect_offset + 6ull * (unsigned long long)(pos - s.start);
        const uint4 rec = load_record(a.prec, me);
        const uint32_t mine = a.state[me];
        uint32_t w[4];
        tf2x64(key, ctr, w);
        const int2 read = a.read[pos];
        const uint2 slot0 = a.bkt[read.x], slot1 = a.bkt[read.y];
        infector_gens(inf, mine, a.gen_p, a.gen_s);
        // Threefry-2x32 on the low seed words with counter (u32)(ctr + 1) (:1895-1901)
        uint32_t v2[2];
        tf2x32(key, (uint32_t)(ctr + 1), v2);
        int victims[5], kv[5];
        const int hoff = (int)rec.x, hcnt = prec_household_size(rec.w);
#pragma unroll
        for (int j = 0; j < 3; j++) kv[j] = select_victim(me, hoff, hcnt, w[j], victims[j]);
        const int off[2] = {bucket_start(slot0), bucket_start(slot1)};
        const int cnt[2] = {bucket_count(slot0), bucket_count(slot1)};
        const int32_t *const table[2] = {a.bkt_people, a.bkt_people};
        select_victims<2>(me, off, cnt, table, v2, victims + 3, kv + 3);
        infector_probs(c, mine, day, kv[0] + kv[1] + kv[2] + kv[3] + kv[4], inf.prob);
        process_contacts<5>(c, key, inf, ctr + 2, victims, kv, a.state, a.claim, queue);
    }
    queue.flush(1, lane);
}

cudaError_t launch_infect(const DevArrays &d, bool weekend, int day, DayQueue &q)
{
    InfectArgs a;
    a.ic = d.ic; a.is = d.is;
    a.state = d.state; a.gen_p = d.gen_p; a.gen_s = d.gen_s; a.age = d.age;
    a.prec = d.prec;
    a.wp_people = d.wp_people; a.read = d.read;
    a.bkt = d.bkt; a.bkt_people = d.bkt_people; a.infected = d.infected;
    a.infected_inst = d.infected_inst;
    a.claim = d.claim; a.new_list = d.new_list; a.sc = d.sc;
    const Tuning &t = d.tune;
    a.coop_most = kCoopPerSm * sm_count();
    const int blocks = sm_count() * t.infect_blocks_per_sm;
    if (t.infect_coop) return queue_kernel(q, weekend ? k_infect_coop<true> : k_infect_coop<false>, blocks, 256, 0, a, day);
    return queue_kernel(q, weekend ? k_infect_weekend : k_infect_weekday, 2 * blocks, 128, 0, a, day);
}

// device_setInfectionStatus (PandemicSim.cu:3048-3067) for the winning claims:
// status = profile, day = today + 1 (8-bit), generation = infector's + 1.
__global__ void k_apply(uint32_t *state, uint8_t *gen_p, uint8_t *gen_s, unsigned long long *claim,
                        const int32_t *new_list, Scalars *sc, int day)
{
    day = launch_day(day, sc);
    if (sc->done) return;
    const int n = sc->new_count;
    const uint8_t dset = (uint8_t)(day + 1);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int e = new_list[i];
        const int v = e >> 1, strain = e & 1;
        unsigned long long *cp = &claim[2 * (size_t)v + strain];
        const unsigned long long cl = *cp;
        *cp = ~0ull;
        const uint8_t profile = (uint8_t)(cl >> 8), gen = (uint8_t)cl;
        // the strain's two bytes of the status word; the other strain's may be written now too
        uint8_t *const st = reinterpret_cast<uint8_t *>(state + v) + strain;
        st[0] = profile;
        st[2] = dset;
        if (strain) gen_s[v] = gen;
        else gen_p[v] = gen;
    }
}

cudaError_t launch_apply(const DevArrays &d, int day, DayQueue &q)
{
    return queue_kernel(q, k_apply, sm_count() * 8, 256, 0, d.state, d.gen_p, d.gen_s, d.claim, d.new_list, d.sc, day);
}

// Four persons a thread; the persons up to the next multiple of four are padding.
__global__ void k_unpack_state(const uint32_t *state, int n, size_t plane, uint8_t *out)
{
    const int i = 4 * (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= n) return;
    const uint4 v = *reinterpret_cast<const uint4 *>(state + i);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint32_t lo = __byte_perm(v.x, v.y, k | (4 + k) << 4), hi = __byte_perm(v.z, v.w, k | (4 + k) << 4);
        *reinterpret_cast<uint32_t *>(out + k * plane + i) = __byte_perm(lo, hi, 0x5410);
    }
}

uint8_t *state_planes(const DevArrays &d) { return reinterpret_cast<uint8_t *>(d.new_list); }

cudaError_t launch_unpack_state(const DevArrays &d, int first, int n, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    k_unpack_state<<<div_up(n, 4 * 256), 256, 0, s>>>(d.state + first, n, state_plane((size_t)n), state_planes(d));
    count_launch();
    return cudaGetLastError();
}

// Also moves the next stepped day on, which nothing here reads: the day is the one that the
// list has begun.  As many blocks as there are rows for: with one block a step of 4,096
// instances took 1,272 us, now 1,203.
__global__ void __launch_bounds__(256) k_day_rows(const InstState *is, int K, Scalars *sc, int *out)
{
    const int day = sc->day, i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < K * kDayRow) {
        const InstState &s = is[i / kDayRow];
        const int f = i % kDayRow;
        out[1 + i] = f < 16 ? s.counts[day][f] : (f == 16 ? s.infected_per_day[day] : s.days_run);
    }
    if (i == 0) {
        out[0] = sc->error;
        sc->step_day = day + 1;
    }
}

cudaError_t launch_day_rows(const DevArrays &d, int *out, DayQueue &q)
{
    const int n = d.K * kDayRow, threads = std::min(256, div_up(n, 32) * 32);
    return queue_kernel(q, k_day_rows, div_up(n, threads), threads, 0, d.is, d.K, d.sc, out);
}

// ================================================================== bounded-wait probe
// The look-back wait above, in isolation: one warp plays tile 1 of a fresh look-back
// (epoch 1, words zeroed by the host) and waits for tile 0.  With publish_first the
// warp writes tile 0's inclusive prefix (1234) before waiting, and the wait returns it
// at once.  Without it nothing ever writes tile 0's word: the wait polls spin_limit
// times, records the error word and returns, and the kernel ends normally.
__global__ void k_wait_probe(LookBack lb, int publish_first, long long spin_limit, unsigned *prefix_out)
{
    constexpr unsigned kEpoch = 1;
    if (publish_first && threadIdx.x == 0) {
        *(volatile unsigned long long *)&lb.tiles[0] = lb_word(kEpoch, 2, 1234u);
        __threadfence();
    }
    __syncwarp();
    const unsigned excl = lookback_publish_warp(lb, kEpoch, 1, 5u, false, spin_limit);
    if (threadIdx.x == 0) *prefix_out = excl;
}

cudaError_t launch_wait_probe(unsigned long long *tiles, int *error, int publish_first, long long spin_limit,
                              unsigned *prefix_out, cudaStream_t s)
{
    LookBack lb;
    lb.tiles = tiles;
    lb.ctl = nullptr;   // the probe takes no ticket
    lb.error = error;
    k_wait_probe<<<1, 32, 0, s>>>(lb, publish_first, spin_limit, prefix_out);
    count_launch();
    return cudaGetLastError();
}

long long max_spin_limit() { return kSpinLimit; }

// ================================================================== errand-lookup self-test
// The schedule kernels' branch-free errand search (errand_row) against the reference's
// loop and IEEE division (errand_row_loop), on every 32-bit random word the schedule
// can draw: counts[0] weekday and counts[1] weekend words whose row or quotient bits
// differ.  counts[2]: floats x in the domain the search divides, 0 and [2^-32, 1]
// (a draw is 0 or at least 2^-32, a remainder after a subtraction at least 2^-28), and
// errand rows r in {9, 11, 12, 13} of both tables where div_rn_recip(x, pdf[r], rcp[r])
// differs from __fdiv_rn(x, pdf[r]).  (Below about 2^-100 the correction step's
// remainder underflows and the two can differ; no draw gets there.)  counts[3]:
// reciprocal table entries that differ from __frcp_rn of their probability.
// The schedule kernel's table form (errand_step and the scaled quotient) against the
// same loop; `rows` holds the errand table of the day type.
template <bool WEEKEND>
__device__ bool errand_table_differs(uint32_t r, const ErrandRow *rows)
{
    constexpr int kRow = (int)sizeof(ErrandRow);
    float x, want;
    const int at = errand_step<WEEKEND>(__uint2float_rn(r), errand_p9<WEEKEND>(true), 0, x);
    const int row = errand_row_loop<WEEKEND>(to_unit(r), want);
    bool bad = at % kRow != 0 || at < 0 || at > 3 * kRow;
    if (bad) return true;
    const ErrandRow &e = rows[at / kRow];
    bad = (at == 0 ? 9 : 10 + at / kRow) != row || __float_as_uint(div_rn_recip(x, e.d, e.r)) != __float_as_uint(want);
    if (!WEEKEND) {
        // a child's row: the quotient is the draw
        const int c = errand_step<false>(__uint2float_rn(r), errand_p9<false>(false), 4 * kRow, x);
        bad |= c != 4 * kRow || __float_as_uint(div_rn_recip(x, rows[4].d, rows[4].r)) != __float_as_uint(to_unit(r));
    }
    return bad;
}

__global__ void k_errand_selftest(unsigned long long *counts)
{
    __shared__ SimConst s_none;   // the tables' locations do not matter here
    __shared__ ErrandRow rows[2 * kErrandRows];
    for (int i = threadIdx.x; i < (int)(sizeof(SimConst) / 4); i += blockDim.x) reinterpret_cast<int *>(&s_none)[i] = 0;
    __syncthreads();
    if (threadIdx.x < 2 * kErrandRows)
        rows[threadIdx.x] = threadIdx.x < kErrandRows ? errand_table_row<false>(s_none, threadIdx.x, 0, 0)
                                                      : errand_table_row<true>(s_none, threadIdx.x - kErrandRows, 0, 0);
    __syncthreads();
    unsigned long long bad_wd = 0, bad_we = 0, bad_div = 0;
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < (1ull << 32);
         i += stride) {
        const float y = to_unit((uint32_t)i);
        float a, b;
        int ra = errand_row<false>(y, a), rb = errand_row_loop<false>(y, b);
        bad_wd += (ra != rb || __float_as_uint(a) != __float_as_uint(b)) ? 1 : 0;
        ra = errand_row<true>(y, a);
        rb = errand_row_loop<true>(y, b);
        bad_we += (ra != rb || __float_as_uint(a) != __float_as_uint(b)) ? 1 : 0;
        bad_wd += errand_table_differs<false>((uint32_t)i, rows) ? 1 : 0;
        bad_we += errand_table_differs<true>((uint32_t)i, rows + kErrandRows) ? 1 : 0;
        if (i == 0 || (i >= 0x2F800000ull && i <= 0x3F800000ull)) {   // 0 and [2^-32, 1]
            const float x = __uint_as_float((uint32_t)i);
            const int rows[4] = {9, 11, 12, 13};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int r = rows[k];
                bad_div += __float_as_uint(div_rn_recip(x, c_weekday_errand_pdf[r], c_weekday_errand_rcp[r])) !=
                                   __float_as_uint(__fdiv_rn(x, c_weekday_errand_pdf[r]))
                               ? 1
                               : 0;
                bad_div += __float_as_uint(div_rn_recip(x, c_weekend_errand_pdf[r], c_weekend_errand_rcp[r])) !=
                                   __float_as_uint(__fdiv_rn(x, c_weekend_errand_pdf[r]))
                               ? 1
                               : 0;
            }
        }
    }
    if (bad_wd) atomicAdd(&counts[0], bad_wd);
    if (bad_we) atomicAdd(&counts[1], bad_we);
    if (bad_div) atomicAdd(&counts[2], bad_div);
    if (blockIdx.x == 0 && threadIdx.x < kTypes) {
        const int t = threadIdx.x;
        unsigned long long bad = 0;
        if (c_weekday_errand_pdf[t] > 0.f && c_weekday_errand_rcp[t] != __frcp_rn(c_weekday_errand_pdf[t])) bad++;
        if (c_weekend_errand_pdf[t] > 0.f && c_weekend_errand_rcp[t] != __frcp_rn(c_weekend_errand_pdf[t])) bad++;
        if (bad) atomicAdd(&counts[3], bad);
    }
}

cudaError_t launch_errand_selftest(unsigned long long *counts, cudaStream_t s)
{
    k_errand_selftest<<<sm_count() * 8, 256, 0, s>>>(counts);
    count_launch();
    return cudaGetLastError();
}

// ================================================================== final
// final_countReproduction's generation counts (PandemicSim.cu:2227-2304) for every
// instance: one block per person tile, histogram in shared memory.
__global__ void k_gen_hist(const InstConst *ic, const int32_t *tile_inst, const uint8_t *gen_p, const uint8_t *gen_s,
                           int *hist)
{
    __shared__ int h[512];
    for (int i = threadIdx.x; i < 512; i += blockDim.x) h[i] = 0;
    __syncthreads();
    const int k = tile_inst[blockIdx.x];
    const long long first = (long long)blockIdx.x * kPersonTile;
    const long long end = (long long)ic[k].pbase + ic[k].c.N;
    for (long long i = first + threadIdx.x; i < first + kPersonTile && i < end; i += blockDim.x) {
        atomicAdd(&h[gen_p[i]], 1);
        atomicAdd(&h[256 + gen_s[i]], 1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 512; i += blockDim.x)
        if (h[i]) atomicAdd(&hist[(size_t)k * 512 + i], h[i]);
}

cudaError_t launch_gen_hist(const DevArrays &d, int *hist, cudaStream_t s)
{
    cudaError_t e = cudaMemsetAsync(hist, 0, (size_t)d.K * 512 * sizeof(int), s);
    if (e != cudaSuccess) return e;
    k_gen_hist<<<d.P / kPersonTile, 256, 0, s>>>(d.ic, d.tile_inst, d.gen_p, d.gen_s, hist);
    count_launch();
    return cudaGetLastError();
}

}  // namespace ptk
