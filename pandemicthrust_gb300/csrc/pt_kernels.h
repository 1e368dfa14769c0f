// pt_kernels.h - kernel launchers and the device data model of the simulation.
// Shared by the CUDA translation unit (pt_kernels.cu) and the host orchestration
// (pt_sim.cpp); no CUDA-specific types beyond cudaStream_t appear here.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace ptk {

constexpr int kTypes = 14;
constexpr int kMaxDays = 256;

constexpr int kPersonTile = 4096;  // persons per sweep / schedule tile
constexpr int kRadixTileEntries = 4096;  // entries per radix-pass tile (256 look-back words each)
constexpr int kScanTileEntries = 4096;   // values per scan tile (one look-back word each)
constexpr int kSchedMinRegion = 64, kSchedMaxRegion = 1024;   // persons per region of the schedule kernel
constexpr int kRegionChunk = 256;  // entries per chunk_region word (a radix warp's entries are whole chunks)
constexpr int kDigitStripes = 16;  // copies of the day's radix digit histograms (spreads the updates)

// Constants of one simulation (setup kernels take them by value; the day kernels
// read them from the InstConst array).
struct SimConst {
    int N, H, L;
    int type_count[kTypes];
    int type_offset[kTypes];
    float shedding[6][10];
    float infectiousness[2];
    float pct_sympt;
    uint64_t key0, key1;           // {(long)SEED[0], (long)SEED[1]}
    uint64_t workplace_offset;     // W0: counter base of the workplace draws
};

// One simulation of a batch and where its rows sit in the batch-wide arrays.  Every
// instance's persons start on a person-tile boundary, so a sweep or schedule tile
// belongs to exactly one instance; the persons up to the next boundary are padding
// (never infected, never counted, in no table).
struct InstConst {
    SimConst c;            // c.N = the instance's persons
    int pbase;             // first global person (a multiple of kPersonTile)
    int pend;              // end of its persons and padding (the next instance's pbase)
    int hbase;             // first global household slot; H + 1 slots, the last one
                           // holds the padding persons
    int lbase;             // first global location
    int bbase[2];          // first global bucket of the weekday / weekend errand tables
    int bcount[2];         // the instance's weekday / weekend buckets; one more global
                           // slot follows them (the end offset of its last bucket)
    int max_days;
    long long kbase;       // first schedule-key slot (3 * pbase)
    // interventions (build-defined extensions; all zero reproduces the reference)
    int closure_start, closure_end;  // school-type locations closed on days [start, end)
    uint64_t absent_thr;             // an adult is absent from work when intervention_hash < this
    uint64_t vacc_thr;               // a person starts vaccinated when intervention_hash < this
};

constexpr uint64_t kTagAbsent = 1, kTagVaccinated = 2;

// Device-resident state of one simulation.  The day loop reads and updates it on
// the device, so a whole run needs no host round trip.
struct InstState {
    unsigned long long rand_offset;     // next free Random123 counter
    unsigned long long next_offset[2];  // the same, of an even and an odd day's start
    unsigned long long errand_offset;   // E0 of the current day's schedule
    unsigned long long infect_offset;   // R0 of the current day's contacts
    int infected;                       // infected count of the current day
    int start;                          // their first position in the batch's infected list
    int list_end;                       // one past their last position
    int marked;                         // today's schedule entries in materialised buckets
    int dense;                          // today's sort reads the schedule keys directly (most
                                        // buckets are read) instead of entries the schedule appended
    int done;                           // set once a day counts zero infected
    int days_run;                       // statistics rows written
    int day;                            // last day run
    int counts[kMaxDays][16];           // per-day status bins
    int infected_per_day[kMaxDays];
};

// Batch-wide device scalars.
struct Scalars {
    unsigned long long materialised_sum;  // schedule entries written to bucket tables, all days
    int infected;                         // length of today's infected list (all instances)
    int done;                             // the number of days once a day finds no instance with infected
    int day;                              // current day index
    int new_count;                        // entries in the new-infection list
    int error;                            // nonzero: a bounded device wait gave up
    int error_site;
    int step_day;                         // next day to step (launches with day -1 read it)
};

// Launch shapes chosen at run time (the engine's tuner picks them per engine; every
// choice gives bit-identical results, only the speed differs).
struct Tuning {
    int infect_coop = 0;            // 1: eight lanes per infector on every day, 0: on days of few
    int infect_blocks_per_sm = 8;   // infection grid: 256-thread blocks per SM (twice as
                                    // many 128-thread blocks for the thread-per-infector kernels)
    int radix_blocks_per_sm = 4;    // persistent blocks of a day's radix pass per SM (1..4;
                                    // three fit, more act as three)
    int sched_tf = 0;               // accepted (0..2) and kept, without effect: one form of the
                                    // Threefry arithmetic is the fastest everywhere (tf2x64)
    int dense_level = 0;            // when a day's sort reads the schedule keys directly:
                                    // 0 never; 1, 2, 3: infected >= buckets / 4, x 1, x 2
    int radix_threads = 256;        // accepted (256, 512) and kept, without effect
};

// Device pointers of a batch of simulations (one simulation is a batch of one).
// Person, household, location and bucket ids are global: an instance's ids are its
// local ids plus its bases.
struct DevArrays {
    uint32_t *state;          // P: status_p | status_s<<8 | day_p<<16 | day_s<<24
    uint8_t *gen_p, *gen_s;   // P
    uint8_t *age;             // P
    int32_t *household;       // P
    int32_t *hh_offset;       // household slots + 1
    int32_t *workplace;       // P
    int32_t *wp_people;       // P (padding persons last, in the spare bucket)
    int32_t *wp_offset;       // locations + 2
    uint4 *prec;              // P packed per-person records for the contact draws (see PersonRec)
    int32_t *keys;            // 3P schedule keys (global bucket indices) of dense instances (launch_day_keys: of all)
    uint2 *bkt;               // today's buckets: start and size (BucketSlot below)
    int32_t *bkt_count;       // the workplace histogram of the setup, zero between uses
    int32_t *bkt_people;      // 3P person ids bucket by bucket, ascending in each
    uint2 *rp0, *rp1;         // 3P each: radix ping-pong (key, value) pairs
    unsigned long long *radix_status;  // ceil(3P/4096) x 256 epoch-tagged look-back words
    unsigned long long *radix_ctl;   // epoch (high half) and ticket
    int *digit_hist;          // K x kDigitStripes x 4 x 256 (the first 4 x 256 also serve the setup sorts)
    int *digit_base;          // K x 4 x 256
    int32_t *tile_prefix;     // K + 1: radix tiles of the instances' segments
    int32_t *tile_prefix0;    // K + 1: the same for the first pass (a dense segment's input is all its keys)
    int32_t *region_count;    // P / kSchedMinRegion: entries the schedule kernel wrote in each region
    int32_t *region_prefix;   // P / kSchedMinRegion: their exclusive prefix within the instance
    int4 *chunk_region;       // 3P / kRegionChunk: region of every kRegionChunk-th entry of a segment (RadixSegments)
    uint32_t *mark;           // bitmap over today's buckets: 1 = materialise
    int32_t *infected;        // P ascending infected ids
    int32_t *infected_inst;   // P: instance of each infected list position
    int2 *read;               // P: the buckets that position's contacts read today, -1 for none
    uint16_t *sweep_flags;    // P / 16: the sweep's per-thread infected masks
    int32_t *sweep_tiles;     // P / kPersonTile + 1: infected per person tile, then their prefix
    unsigned long long *claim;// 2P (victim, strain) -> min attempt key
    int32_t *new_list;        // 2P first claims of the day
    unsigned long long *tiles;// look-back tile status words
    int tiles_cap;
    const InstConst *ic;      // K
    InstState *is;            // K
    const int32_t *tile_inst; // P / kPersonTile: instance of each person tile
    int K;
    int P;                    // persons including padding, a multiple of kPersonTile
    int persons_max;          // of the largest instance, including padding
    int buckets[2];           // weekday / weekend bucket slots over all instances
    int bucket_max[2];        // largest weekday / weekend bucket count of one instance
    int locations;            // locations over all instances
    Scalars *sc;
    Tuning tune;
};

// BucketSlot: a bucket of the day's errand table, one 8-byte load.  x: kMaxStart less the
// place of its first person in bkt_people (0: no entries); y: its persons.  Cleared to
// zero each day that finds infected; the sort's last pass raises x to the largest offer (the smallest
// place) and adds up y.
constexpr uint32_t kMaxStart = 0x7FFFFFFFu;   // above every place, so a bucket with entries has x > 0
__host__ __device__ inline int bucket_start(uint2 slot) { return (int)(kMaxStart - slot.x); }
__host__ __device__ inline int bucket_count(uint2 slot) { return (int)slot.y; }

// The static part of a person that the contact draws read, packed in 16 bytes so an
// infector's own data is one 128-bit load (built once at setup, after the workplace
// table):
//   x  first person of the person's household (household victims are x + r % size)
//   y  start of the person's workplace / school in the workplace table
//   z  persons in that workplace / school
//   w  bits 0-3 household size, 4-7 age code, 8-9 workplace contacts (the type's
//      maximum, PandemicSim.cu:3492-3511), bit 10 the location is a school (types 3-7)
// Padding persons have an all-zero record (they are never infected).
__host__ __device__ inline int prec_household_size(uint32_t w) { return (int)(w & 15u); }
__host__ __device__ inline int prec_age(uint32_t w) { return (int)((w >> 4) & 15u); }
__host__ __device__ inline int prec_desired(uint32_t w) { return (int)((w >> 8) & 3u); }
__host__ __device__ inline bool prec_school(uint32_t w) { return ((w >> 10) & 1u) != 0; }

// Launch configuration helpers
int sm_count();

// Where a day's launches go: to a stream, or (graph set) to a graph, as nodes one behind
// the other.  (Not by capturing the stream: while a stream is captured, a thread that waits
// for the device is refused and ends the capture.)
struct DayQueue {
    cudaStream_t stream = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphNode_t last = nullptr;   // the graph's last node
    uint64_t kernels = 0;             // kernel nodes
};

// ---- setup
cudaError_t launch_household_types(const SimConst &c, uint8_t *types, int32_t *sizes, int *adults,
                                   int *persons, cudaStream_t s);
cudaError_t launch_scan_exclusive(const int32_t *in, int32_t *out, int n, int clear_in,
                                  unsigned long long *tiles, int *ctl, int *error,
                                  const int *skip, int passes, int dbits, int *digit_hist, cudaStream_t s);
cudaError_t launch_generate_households(const uint8_t *types, const int32_t *hh_offset, int slots,
                                       int32_t *household, uint8_t *age, cudaStream_t s);
cudaError_t launch_assign_workplaces(const SimConst &c, uint8_t *age, int32_t *workplace, int loc_base,
                                     cudaStream_t s);
// household slots of the padding persons, and the padding persons themselves
cudaError_t launch_batch_padding(const DevArrays &d, uint8_t *types, int32_t *sizes, int spare_location,
                                 bool persons, cudaStream_t s);
cudaError_t launch_count_keys(const int32_t *keys, int n, int32_t *count, cudaStream_t s);

// Segments of a day's sort: segment k (instance k) holds its entries at
// [ic[k].kbase, ic[k].kbase + is[k].marked), keys local to the instance, sorted within
// the segment; its tiles are [tile_prefix[k], tile_prefix[k + 1]).  tile_prefix ==
// nullptr: one segment [0, E).
struct RadixSegments {
    const int *tile_prefix = nullptr;   // segments + 1, on the device
    const InstConst *ic = nullptr;
    const InstState *is = nullptr;
    int segments = 0;
    // The first pass of a day's sort reads the entries the schedule kernel wrote region by
    // region (see k_sched): region r's at 3 region_persons r, its first one entry
    // region_prefix[r] of the segment; chunk_region[(kbase + i) / kRegionChunk] is the
    // region of entry i (a multiple of kRegionChunk) of the segment at kbase, that region's
    // prefix, its end and the end of the next one.
    const int32_t *region_prefix = nullptr;
    const int4 *chunk_region = nullptr;
    int region_persons = 0;
    // The day's sort: in its first pass a segment whose instance is dense today reads
    // its entries straight from the schedule keys (global bucket ids at
    // day_keys[kbase ...], 2N weekday hour-major / 3N weekend person-major, persons
    // implicit), keeping those of marked buckets; the other segments read the
    // entries the schedule appended.  tile_prefix0 numbers the first pass's tiles.
    const int32_t *day_keys = nullptr;
    const int *tile_prefix0 = nullptr;
    const uint32_t *mark = nullptr;
    int weekend = 0;
};

// Stable LSD radix sort of E keys in [0, buckets).  Without `table`: plain keys, entry i
// has the value i.  With it, a day's sort (seg): see RadixSegments; the sorted persons
// go to `out`, the buckets' starts and sizes to `table`.
struct RadixArgs {
    const uint32_t *keys = nullptr;
    const uint2 *in = nullptr;    // a day's entries (key, person), in the schedule's regions
    int E, buckets;
    uint2 *p0, *p1;               // ping-pong pairs, E each (in may be p1)
    uint32_t *out;
    uint2 *table = nullptr;
    const int *digit_base;        // [segment][pass][256]
    RadixSegments seg;
    unsigned long long *status;   // look-back words, ceil(E/4096) x 256, epoch-tagged
    unsigned long long *ctl;      // epoch (high half) and ticket
    int *error;
    const int *skip;
    int blocks_per_sm = 4;        // persistent blocks per SM, at most what fits
};
int radix_passes(int buckets);
int radix_digit_bits(int buckets);   // bits of a pass's digit
cudaError_t launch_radix_sort(const RadixArgs &r, DayQueue &q);
// count (optional) + scan + digit bases + radix passes: a complete bucket table
cudaError_t launch_bucket_table(const RadixArgs &r, int32_t *counts, bool count_keys, int32_t *offset,
                                unsigned long long *tiles, int *lb_ctl, int *digit_hist, cudaStream_t s);
cudaError_t launch_init_status(int N, uint32_t *state, uint8_t *gen_p, uint8_t *gen_s,
                               unsigned long long *claim, cudaStream_t s);
// every instance's device state back to "set up, day 0": rand_offset after setup is
// H/4 (household types) + N/4 (workplaces)
cudaError_t launch_reset_instances(const DevArrays &d, cudaStream_t s);
// vaccinated persons start recovered from both strains (only when some instance
// has a vaccination coverage)
cudaError_t launch_vaccinate(const DevArrays &d, cudaStream_t s);
cudaError_t launch_seed_infected(const int32_t *seeds, int P, int S, uint32_t *state, uint8_t *gen_p,
                                 uint8_t *gen_s, cudaStream_t s);
// the packed per-person records (after households, workplaces and the workplace table)
cudaError_t launch_person_records(const DevArrays &d, cudaStream_t s);

// ---- day (every instance of the batch in each launch)
cudaError_t launch_sweep(const DevArrays &d, bool weekend, int day, DayQueue &q);   // recover, count, bookkeeping
cudaError_t launch_infected_list(const DevArrays &d, bool weekend, int day, bool full_tables,
                                 DayQueue &q);                                        // the ordered list, the marks
cudaError_t launch_schedule(const DevArrays &d, bool weekend, int day, DayQueue &q);
cudaError_t launch_day_keys(const DevArrays &d, bool weekend, cudaStream_t s);        // for inspection
cudaError_t launch_bucket_scan(const DevArrays &d, bool weekend, DayQueue &q);
cudaError_t launch_bucket_sort(const DevArrays &d, bool weekend, DayQueue &q);
cudaError_t launch_infect(const DevArrays &d, bool weekend, int day, DayQueue &q);
cudaError_t launch_apply(const DevArrays &d, int day, DayQueue &q);
// A day's rows of every instance to mapped host memory: out[0] the device error word, then
// per instance its 16 counts, infected and days run.
constexpr int kDayRow = 18;
// The state words of n persons from `first` on (a tile boundary) as four planes of bytes, each
// state_plane(n) long, in the day's claim list (free between days): status_p, status_s, day_p, day_s.
inline size_t state_plane(size_t n) { return (n + 15) / 16 * 16; }
uint8_t *state_planes(const DevArrays &d);
cudaError_t launch_unpack_state(const DevArrays &d, int first, int n, cudaStream_t s);
cudaError_t launch_day_rows(const DevArrays &d, int *out, DayQueue &q);
// weekday / weekend buckets of one instance (compact keys hour * R + dest - lo)
int day_buckets(const SimConst &c, bool weekend);

// ---- final: per-instance generation histograms, K x 512 (pandemic 0..255, seasonal 256..511)
cudaError_t launch_gen_hist(const DevArrays &d, int *hist, cudaStream_t s);

// ---- the bounded look-back wait in isolation (tiles: 2 zeroed words; error: zeroed)
cudaError_t launch_wait_probe(unsigned long long *tiles, int *error, int publish_first, long long spin_limit,
                              unsigned *prefix_out, cudaStream_t s);
// The errand-lookup self-test: counts[4] (zeroed by the caller) receive mismatch counts.
cudaError_t launch_errand_selftest(unsigned long long *counts, cudaStream_t s);
long long max_spin_limit();   // the polls every wait of the simulation allows

uint64_t launches();
void add_launches(uint64_t n);  // kernels run by a replayed graph

}  // namespace ptk
