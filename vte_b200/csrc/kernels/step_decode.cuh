// A whole decode step in one launch (included by decode_attention.cu): attention of every layer, sequence and KV head of
// a step whose inputs are all there before it starts, with this step's K and V rows appended on the way.
//
// A run is the positions of one (layer, group of `hg` KV heads, sequence), in tiles of `tile` positions.  All runs are laid end to
// end and cut into one equal share of tiles per CTA, one CTA an SM.  A warp fetches K and V tiles in turn, one tensor-map copy
// each, into a ring; `wph` warps serve a KV head, a 16-position block of every tile each (block arithmetic of lean_decode.cuh,
// fp32 sums).  At the end of a run the warps' states meet in the tile they have just done with, while the rest of the ring keeps
// filling.  A run that lies in one share is normalised and stored.  Of one that was cut, each CTA but the last leaves its state
// on a board, in 64-bit words that carry the number of the launch (each written and read in one relaxed access, so valid exactly
// when it carries it, without a fence), and the last merges them, bounded, in their order; it waits for CTAs with lower numbers only.
//
// What bounds it: HBM, and about 9 us of launch, start (2), first tile (1.3), merges (1.3 a run) and finish (2 to 2.5).  us a step,
// launches per layer / one launch, in turn on one machine, 12 heads on 2 KV heads of 128, one sequence: 28 layers of 1,531 positions
// 105 / 15.9, of 11,003 183 / 55.5, four of a million 654 / 634 (6.8 TB/s); 8 ragged sequences of 32 heads on 8 of 64, ten layers 254 / 208; eight
// of 32 on 2 of 128, eight layers 90 / 47; one of 24,001, 256-wide, eight layers 115 / 72.  Machines differ by 5 % where HBM is the
// bound (the million 602 to 637, the eight ragged ones 192 to 209).  Nine to sixteen query heads per KV head are bound by block
// arithmetic: an SM takes 43 B/ns, its share of HBM is 45.  What was measured:
//   128 KB of tiles in flight an SM, not 192: with more, the SMs of the two largest clusters of SMs get 15 % less than the others
//     and every share waits for them (a million positions 676 / 614, 28 layers of 32,768 174 / 164);
//   one copy a tile in place of one per 64 channels: the warp that fetches was the limit (an SM alone, 64-wide heads 52 / 58
//     B/ns, 256-wide 59 / 70); 16-byte asynchronous copies by every warp 5.8 TB/s on 64 ragged sequences of 64-wide heads (6.5);
//   64-wide heads: twelve warps (8: 40 B/ns an SM, below its share of HBM), four heads a CTA (rows of 512 bytes; 128: 6.0 TB/s);
//   256-wide heads: two teams of three warps that take tiles in turn: 24 KB a tile, five in flight (48 KB, three: 209 / 205);
//   tagged words in place of a fence, a counter and a reload: 28.6 / 22.6 for 28 layers of 1,531 (as relaxed 64-bit accesses, with the
//     fetching warp's last wait: 15.6 / 15.7);
//   up to sixteen states merged at once, not eight, and the fetching warp ahead of the others: one of 24,001, 256-wide, eight layers
//     71.9 / 71.2, 28 layers of 1,531 16.1 / 15.6;
//   two runs of 128-wide heads: seven computing warps and the fetching one have 255 registers each, eight and one 168 and spill (8
//     sequences of 32 heads on 2, eight layers: 51.2 / 47.4).
#pragma once

struct StepLayer {
    KvTensorMap k_map, v_map;                             // of the caches: boxes of `tile` positions x hg * D / 64 columns
    const __half* q; __half* k_cache; __half* v_cache;
    const __half* k_new; const __half* v_new;             // this step's projections [B, Hkv, D]; null: the newest row is in the cache
    void* output;
    void* mirror; void* unused;                           // a step whose outputs go to the host: pinned memory that they are stored to as well; else null
};
constexpr int kStepMaxLayers = 64;                        // a launch
constexpr int kStepOffsets = 64;                          // sequences whose offsets may come with the launch
struct StepArgs {
    StepLayer layer[kStepMaxLayers];
    const int* kv_offsets; const __half* rope_cos; const __half* rope_sin;
    ulonglong2* boards; unsigned* launches; int* status;  // [CTAs][hg * group][D / 2 + 1]: the state of a cut run, two tagged words an entry; [CTAs]: launches so far
    int* status_mirror;                                   // the same for what `status` says
    __half* keep_q; int* keep_offsets; void* unused[7];
    int offsets[kStepOffsets]; int offsets_here;          // 1: the kv offsets are these, and go to kv_offsets for whoever reads them there
    int keep_layer;                                       // keep_q, keep_offsets: a copy of that layer's Q and of the offsets, from which partials can be had; -1: none
    int num_layers, batch, num_q_heads, num_kv_heads, kv_batch_stride, out_kind, rope_type, rotary_dim;
    int hg, hg_log2, wph, group, groups, group_inv;        // of the plan: KV heads a CTA serves at once, warps of a team, query heads of a KV
                                                          // head, runs of a sequence and layer, ceil(65536 / group)
    float scale; int fan; int unused_too[14];
};

static_assert(sizeof(StepLayer) == 320 && sizeof(StepArgs) == kStepMaxLayers * 320 + 512, "mirrored by the host");

__host__ __device__ constexpr int step_warps(int D, int NV) { return D == 256 ? 6 : D == 128 && NV == 2 ? 7 : D == 64 && NV == 1 ? 12 : 8; }     // that compute; one more fetches
__host__ __device__ constexpr int step_teams(int D) { return D == 256 ? 2 : 1; }           // that take tiles in turn
__host__ __device__ constexpr int step_tile_bytes(int D, int NV) { return step_warps(D, NV) / step_teams(D) * 32 * D; }    // a 16-position block for every warp of a team
__host__ __device__ constexpr int step_slots(int D, int NV) { return (128 << 10) / step_tile_bytes(D, NV); }   // K or V tiles in flight: 128 KB
constexpr int kStepStatePad = 4;                          // floats after o[D] in a kept state: m, l, 2 unused
constexpr int kStepMaxBatch = 1024;
constexpr int kStepMostFan = 16;                          // CTAs whose states of one run are merged at once, where shared memory holds as many
constexpr int kStepFew = 7;                               // of a run, where more would have less than three tiles each
// Tiles a CTA up to which a run has no more states than are merged at once: the second merge costs more than the CTAs left idle.  One
// sequence, 32 heads on 2 of 128, four layers, us without / with (launches per layer): 4,096 positions 34.1 / 26.4 (26.7), 8,192 36.3 / 29.3
// (32.8), 9,000 38.0 / 31.9 (34.5).  Up to four: 36.3 / 39.0 for the second; up to sixteen: 25.2 / 31.3 for 32,768 of 16 heads on 1 of 64.
constexpr unsigned kStepOnce = 8;
constexpr int kStepCtrlBytes = 256;                       // barriers (full, empty: 24 at most), abort word

// What a launch needs.  ok = 0: a geometry or batch that it does not cover.  hg 0: rows of 256 bytes and more are read in full wherever
// they lie, so wider heads go one a CTA (fewer rows to merge: 12 heads on 2 of 128, two a CTA 26.6 / 22.6 us); 64-wide heads up to four.
struct StepPlan { int ok, threads, smem_bytes, hg, state_bytes, max_layers, hg_log2, wph, tile, fan; };
__host__ __device__ inline StepPlan make_step_plan(int num_q_heads, int num_kv_heads, int head_dim, int batch, int n_ctas, int hg = 0) {
    StepPlan p = {0, 0, 0, 0, 0, kStepMaxLayers, 0, 0, 0, 0};
    if ((head_dim != 64 && head_dim != 128 && head_dim != 256) || num_kv_heads <= 0 || num_q_heads <= 0 || num_q_heads % num_kv_heads ||
        batch < 1 || batch > kStepMaxBatch || n_ctas < 1) return p;
    const int group = num_q_heads / num_kv_heads, runs = group > 8 ? 2 : 1, warps = step_warps(head_dim, runs), team = warps / step_teams(head_dim);
    if (group > 16 || (runs > 1 && head_dim == 256)) return p;
    if (!hg) {
        hg = 1;
        for (int d = 1; d <= team; d *= 2)
            if (num_kv_heads % d == 0 && team % d == 0 && d * head_dim <= 256 && (head_dim == 64 || d == 1)) hg = d;
    }
    if (hg < 1 || hg & (hg - 1) || num_kv_heads % hg || team % hg || hg * head_dim > 512) return p;
    p.hg = hg;
    p.wph = team / hg;
    p.tile = 16 * p.wph;
    while (1 << p.hg_log2 < hg) ++p.hg_log2;
    p.threads = (warps + 1) * 32;
    p.state_bytes = n_ctas * hg * group * (head_dim / 2 + 1) * 16;
    p.smem_bytes = 1024 + step_slots(head_dim, runs) * (step_tile_bytes(head_dim, runs) + hg * head_dim * 2) + hg * runs * (head_dim / 8) * 128 +
                   warps * runs * 8 * 16 + kStepCtrlBytes + hg * group * (head_dim + kStepStatePad) * 4 + vteb::vteb_round_up((2 * batch + 1) * 4, 16);
    // states that the ring holds at once, less two for parts merged before (32 heads on 2 of 128, one of 16,384 positions, four layers,
    // 19 CTAs a run: 63 us with sixteen, which take two goes)
    p.fan = step_slots(head_dim, runs) * step_tile_bytes(head_dim, runs) / (hg * group * (head_dim + kStepStatePad) * 4) - 2;
    p.fan = p.fan < 4 ? 4 : p.fan > kStepMostFan ? kStepMostFan : p.fan;
    p.ok = p.smem_bytes <= 227 * 1024;
    return p;
}

// A run and where it lies among all tiles of the step.
struct StepRun {
    int l, h, b, start, end;
    __device__ __forceinline__ void next(const int* pre, int batch, int groups) {
        if (++b == batch) {
            b = 0;
            if (++h == groups) { h = 0; ++l; }
        }
        start = end;
        end += pre[b + 1] - pre[b];
    }
};

// An entry of a board: two fp32 values, each in a 64-bit word with the launch's number above it.  A vector access is as many scalar
// ones in no order, so the elements are the words: a number seen has come with its value.
__device__ __forceinline__ void store_entry(ulonglong2* p, float x, float y, unsigned tag) {
    const unsigned long long up = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(up | __float_as_uint(x)), "l"(up | __float_as_uint(y)) : "memory");
}
__device__ __forceinline__ ulonglong2 load_entry(const ulonglong2* p) {
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool entry_of(const ulonglong2& v, unsigned tag) { return (unsigned)(v.x >> 32) == tag && (unsigned)(v.y >> 32) == tag; }
template <int THREADS> __device__ __forceinline__ void step_sync() { asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory"); }   // of the warps that compute

template <int D, int NV>
__device__ __forceinline__ void step_body(const StepArgs& a)
{
    constexpr int CW = step_warps(D, NV), TEAMS = step_teams(D), TB = CW / TEAMS, SLOTS = step_slots(D, NV), TILE = step_tile_bytes(D, NV), THREADS = CW * 32;
    constexpr int CPR = D / 8, SP = D + kStepStatePad;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char* ring = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    unsigned char* fresh = ring + SLOTS * TILE;                      // [slot]: the newest row of the slot's heads
    const int hg = a.hg, group = a.group, rows = hg * group, groups = a.groups, wph = a.wph;
    uint32_t* q_store = reinterpret_cast<uint32_t*>(fresh + SLOTS * hg * D * 2);    // Q as mma fragments: [hg][run][chunk / 4][head, word][chunk % 4]
    const int q_words = NV * CPR * 32;                               // of a KV head
    float4* stats = reinterpret_cast<float4*>(q_store + hg * q_words);              // [warp][NV * 8]: m, l, true maximum, the slots with its state (0: none)
    unsigned char* ctrl = reinterpret_cast<unsigned char*>(stats + CW * NV * 8);
    const uint32_t full0 = smem_u32(ctrl), empty0 = full0 + 8 * TEAMS * SLOTS;
    volatile int* abort_word = reinterpret_cast<volatile int*>(ctrl + 200);
    float* kept = reinterpret_cast<float*>(ctrl + kStepCtrlBytes);  // [rows][SP]: this CTA's state of the run that it finishes for others
    int* lens = reinterpret_cast<int*>(kept + rows * SP);
    int* pre = lens + a.batch;                                       // tiles of the sequences in front
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int team = TEAMS == 1 ? 0 : warp / TB, kvh = (warp - team * TB) & (hg - 1), wt = (warp - team * TB) >> a.hg_log2;
    const int tile = 16 * wph;                                       // positions
    const auto gave_up = [&](int code) {
        raise_abort(abort_word, a.status, code);
        if (lane == 0 && a.status_mirror != nullptr) *a.status_mirror = code;
    };

    // The warp that fetches goes ahead: it sets up the barriers and adds up the lengths, and starts on its tiles while the others still
    // prepare Q's fragments.
    unsigned tag = 0;
    if (warp == CW) {
        if (lane == 0) {
            for (int i = 0; i < TEAMS * SLOTS; ++i) mbar_init(full0 + 8 * i, 1);
            for (int i = 0; i < SLOTS; ++i) mbar_init(empty0 + 8 * i, TB);
            *abort_word = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        grid_dependency_wait();                                      // and no early release: a CTA of the launch behind has no room beside this one (17.2 / 16.1 us)
        if (a.status_mirror != nullptr && blockIdx.x == 0 && lane == 0 && *a.status != 0) *a.status_mirror = *a.status;
        int sum = 0;
        for (int b0 = 0; b0 < a.batch; b0 += 32) {
            const int b = b0 + lane, len = b >= a.batch ? 0 : max((a.offsets_here ? a.offsets[b] : a.kv_offsets[b]) + 1, 0);
            int n = b < a.batch ? max((len + tile - 1) / tile, 1) : 0;
            if (b < a.batch) lens[b] = len;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, n, off);
                if (lane >= off) n += up;
            }
            if (b < a.batch) pre[b + 1] = sum + n;
            sum += __shfl_sync(0xffffffffu, n, 31);
        }
        if (lane == 0) pre[0] = 0;
        __syncwarp();
        asm volatile("bar.arrive 2, %0;" ::"n"(THREADS + 32) : "memory");
    } else {
        for (int i = tid; i < hg * q_words / 4; i += THREADS) reinterpret_cast<uint4*>(q_store)[i] = make_uint4(0u, 0u, 0u, 0u);
        grid_dependency_wait();
        tag = a.launches[blockIdx.x] + 1;                            // every CTA counts the launches: all have the same number
        asm volatile("bar.sync 2, %0;" ::"n"(THREADS + 32) : "memory");
    }

    const int N = pre[a.batch], T = a.num_layers * groups * N, cta = blockIdx.x;
    // Few states to merge for a run where that costs a CTA up to three tiles, and no more than one merge takes where it costs up to eight.
    const int runs = a.num_layers * groups * a.batch, few = runs * kStepFew, once = runs * a.fan;
    const int G = min(min((int)gridDim.x, T), T <= 3 * few ? few : (unsigned)T <= kStepOnce * (unsigned)once ? once : T);
    if (tid == 0) a.launches[cta] = tag;
    if (cta >= G) return;
    // CTA c's share starts at floor(c T / G).  Divisions by way of floats: quotients below 2^20 are at most one off.
    const float per_cta = __fdividef(1.f, (float)G);
    const auto over_g = [&](int x) {
        const int q = (int)((float)x * per_cta), r = x - q * G;
        return q + (r >= G) - (r < 0);
    };
    const int whole = over_g(T), rest = T - whole * G, extra = over_g(cta * rest);
    const int x0 = cta * whole + extra, x1 = x0 + whole + (cta * rest - extra * G + rest >= G);
    const auto kv_head_of = [&](int j) { return (j * a.group_inv) >> 16; };  // j / group: both are small

    StepRun run;                                                     // the run that is worked through
    {
        int lh = (int)__fdividef((float)x0, (float)N);
        lh += (x0 - lh * N >= N) - (x0 < lh * N);
        const int r = x0 - lh * N;
        int lo = 0, hi = a.batch - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (pre[mid] <= r) lo = mid; else hi = mid - 1;
        }
        run.l = groups == 1 ? lh : lh / groups; run.h = lh - run.l * groups; run.b = lo;
        run.start = lh * N + pre[lo]; run.end = lh * N + pre[lo + 1];
    }
    const long long pos_stride = (long long)a.num_kv_heads * D;      // halves between positions

    if (warp == CW) {
        // ---- the tiles of the share, K and V in turn, one tensor-map box each (`tile` positions of the heads' columns of 64 halves).  A team's copies complete on
        // barriers of their own, one after another: a warp waits for every phase of the barriers that it looks at.
        const int seq_rows = a.kv_batch_stride / (a.num_kv_heads * D);
        const auto full_of = [&](int n) {                            // of the n-th copy
            const int j = TEAMS == 1 ? n : 2 * ((n >> 1) / TEAMS) + (n & 1), at = j % SLOTS;
            return full0 + 8 * ((TEAMS == 1 ? 0 : (n >> 1) % TEAMS) * SLOTS + at) + (((j / SLOTS) & 1) << 31);      // and its parity
        };
        int slot = 0, sent = 0, team_at[TEAMS] = {};
        uint32_t phase = 0;
        bool ok = true;
#pragma unroll 1
        for (int t = x0; ok && t < x1; ++t) {
            while (t >= run.end) run.next(pre, a.batch, groups);
            const StepLayer& L = a.layer[run.l];
            const int y = run.b * seq_rows + (t - run.start) * tile, x = run.h * hg * D;
            const bool newest = t == run.end - 1 && L.k_new != nullptr;
#pragma unroll 1
            for (int kv = 0; kv < 2; ++kv) {
                // a tile given back by a warp that gave up may have a copy under way to it still
                if (sent >= SLOTS && __any_sync(0xffffffffu, !mbar_wait_bounded(empty0 + 8 * slot, phase ^ 1, abort_word) || *abort_word != 0)) {
                    gave_up(kStatusEmptyTimeout);
                    ok = false;
                    break;
                }
                int& at = team_at[TEAMS == 1 ? 0 : (t - x0) % TEAMS];
                const uint32_t bar = full0 + 8 * ((TEAMS == 1 ? 0 : (t - x0) % TEAMS) * SLOTS + at);
                if (++at == SLOTS) at = 0;
                if (lane == 0) {
                    mbar_arrive_expect_tx(bar, TILE + (newest ? hg * D * 2 : 0));
                    tma_load_box_columns(smem_u32(ring) + slot * TILE, kv ? &L.v_map : &L.k_map, x / 64, y, bar);
                    if (newest)
                        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                     ::"r"(smem_u32(fresh) + slot * hg * D * 2), "l"((kv ? L.v_new : L.k_new) + (long long)run.b * pos_stride + x), "r"(hg * D * 2), "r"(bar) : "memory");
                }
                __syncwarp();
                ++sent;
                if (++slot == SLOTS) { slot = 0; phase ^= 1; }
            }
        }
        if (a.offsets_here && cta == 0)                              // for whoever reads them there; not in front: a path of one CTA's own is slow to fetch
            for (int b = lane; b < a.batch; b += 32) const_cast<int*>(a.kv_offsets)[b] = a.offsets[b];
        // Every copy lands before this warp, and with it the CTA, ends: the computing warps may have given up.
        for (int i = 1; i <= min(sent, SLOTS); ++i) {
            const uint32_t bar = full_of(sent - i);
            mbar_wait_bounded(bar & 0x7fffffffu, bar >> 31, nullptr);
        }
        return;
    }

    // ---- Q of a run's heads as mma fragments, one 16-byte chunk a thread at a time (the same chunk of every head): asked for a
    // run ahead, put in place when every warp has done with the run before
    const int q_chunk = tid % CPR, q_row = tid / CPR;
    constexpr int QR = THREADS / CPR;                                // heads at a time
    static_assert(THREADS % CPR == 0, "one chunk per thread");
    uint4 q_next[2];
    RopeWords words;
    const bool rotate = rope_touches(a.rope_type, a.rotary_dim, q_chunk * 8);
    const auto ask_q = [&](const StepRun& r) {
        const __half* row = a.layer[r.l].q + ((long long)r.b * a.num_q_heads + r.h * rows + q_row) * D + q_chunk * 8;
#pragma unroll
        for (int i = 0; i < 2; ++i)
            if (q_row + i * QR < rows) q_next[i] = *reinterpret_cast<const uint4*>(row + (long long)i * QR * D);
        if (rotate) words = rope_words(a.rope_cos, a.rope_sin, lens[r.b] - 1, a.rope_type, a.rotary_dim, D, q_chunk * 8);
    };
    const auto put_q = [&](const StepRun& r) {
#pragma unroll 1
        for (int i = 0, hh = q_row; hh < rows; ++i, hh += QR) {
            const __half* row = a.layer[r.l].q + ((long long)r.b * a.num_q_heads + r.h * rows + hh) * D;
            uint4 x = i == 0 ? q_next[0] : i == 1 ? q_next[1] : *reinterpret_cast<const uint4*>(row + q_chunk * 8);
            if (rotate) x = rope_chunk(x, row, q_chunk * 8, words, a.rope_type, a.rotary_dim, D);
            const int k = kv_head_of(hh), r8 = hh - k * group;
            uint32_t* dst = q_store + k * q_words + ((r8 >> 3) * CPR + (q_chunk & ~3)) * 32 + (r8 & 7) * 16 + (q_chunk & 3);
            dst[0] = x.x; dst[4] = x.y; dst[8] = x.z; dst[12] = x.w;
        }
    };
    ask_q(run);
    put_q(run);
    step_sync<THREADS>();

    // This warp's block of a tile: rows 16 wt .. of the column blocks of its head.  128-byte swizzle: 16-byte chunk c of row r at c ^ (r & 7).
    const int g = lane >> 2, t4 = lane & 3, col_bytes = tile * 128;
    const float scale2 = a.scale * kLog2e;
    const uint32_t own = (kvh * (D / 64) * tile + 16 * wt) * 128;
    const uint32_t k_off = own + ((lane & 7) + ((lane >> 4) << 3)) * 128 + ((((lane >> 3) & 1) ^ (lane & 7)) << 4);
    const uint32_t v_off = own + ((lane & 7) + (((lane >> 3) & 1) << 3)) * 128 + (((lane >> 4) ^ (lane & 7)) << 4);
    // Row r of a warp's state, D floats, in the memory of the tile that only that warp has read: rows 8 .. 15 in the K tile, the others in
    // the V tile; columns at c ^ 8 (r / 2 % 4)
    constexpr int RP = 512 / D;                                      // rows in the 2 KB that a block has of a column block
    const auto state_row = [&](int w_own, int slot_k, int slot_v, int r) {
        const int r8 = r & 7;
        return reinterpret_cast<float*>(ring + (NV == 2 && r >= 8 ? slot_k : slot_v) * TILE + w_own + (r8 / RP) * col_bytes + (r8 % RP) * 4 * D);
    };
    const auto store_out = [&](const StepRun& r, int j, int q4, const float4& acc, float sum) {
        const float inv = fmaxf(sum, 1e-20f);
        const float4 y = make_float4(acc.x / inv, acc.y / inv, acc.z / inv, acc.w / inv);
        const long long at = ((long long)r.b * a.num_q_heads + r.h * rows + j) * D + q4 * 4;
        const StepLayer& L = a.layer[r.l];
        if (a.out_kind == 2) {
            *reinterpret_cast<float4*>(reinterpret_cast<float*>(L.output) + at) = y;
            if (L.mirror != nullptr) *reinterpret_cast<float4*>(reinterpret_cast<float*>(L.mirror) + at) = y;
        } else {
            const uint2 h = make_uint2(pack_half2(y.x, y.y), pack_half2(y.z, y.w));
            *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(L.output) + at) = h;
            if (L.mirror != nullptr) *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(L.mirror) + at) = h;
        }
    };
    const auto cta_of = [&](int x) {                                 // whose share the tile is in
        int c = min((int)((float)x * (float)G * __fdividef(1.f, (float)T)), G - 1);
        while (c * whole + over_g(c * rest) > x) --c;
        while ((c + 1) * whole + over_g((c + 1) * rest) <= x) ++c;
        return c;
    };
    const auto push = [&](int j, int q4, const float4& acc, float m, float l) {      // to the CTA that finishes the run or the part
        ulonglong2* const to = a.boards + ((long long)cta * rows + j) * (D / 2 + 1);
        store_entry(to + 2 * q4, acc.x, acc.y, tag);
        store_entry(to + 2 * q4 + 1, acc.z, acc.w, tag);
        if (q4 == 0) store_entry(to + D / 2, m, l, tag);
    };
    const StepRun head = run;                                        // the run that was cut at the share's start, if any was
    int finish = 0;                                                  // 1: a run that CTAs in front began, 2: a part of one that goes on
    bool alive = true;
    int slot = 2 * team, landed = 0;                                 // where the team's next tile goes; which of its barriers says that it is there
    uint32_t phase = 0;

    for (int n = 0;; ++n) {
        const int s0 = max(run.start, x0), s1 = min(run.end, x1), len = lens[run.b];
        const StepLayer& L = a.layer[run.l];
        const uint32_t* q_frag = q_store + kvh * q_words + lane * 4;
        StepRun next = run;
        const bool more = run.end < x1;
        if (more) {
            next.next(pre, a.batch, groups);
            ask_q(next);
        }
        ConsumerStateT<D / 16> st[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) st[v].reset();
        const int t0 = s0 + (TEAMS == 1 ? 0 : (s0 - x0 + team) % TEAMS);   // the team's first tile of the run
        int pos = ((t0 - run.start) * wph + wt) * kBlockPos;         // of this warp's block
        const int first = pos;
        int slot_k = 0, slot_v = 0;
#pragma unroll 1
        for (int t = t0; t < s1; t += TEAMS, pos += TEAMS * tile) {
            const int left = len - pos;                              // positions of the block that count
            const bool last = t + TEAMS >= s1;
            const int r_new = L.k_new != nullptr && t == run.end - 1 && left > 0 && left <= kBlockPos ? left - 1 : -1;
            // the newest row: from the projections into the tile, rotated if asked to, and into the cache
            const auto put_newest = [&](int kv, int s) {
                const int head_at = run.h * hg + kvh;
                __half* cache = (kv ? L.v_cache : L.k_cache) + (long long)run.b * a.kv_batch_stride + (len - 1) * pos_stride + head_at * D;
                if (lane < CPR && *abort_word == 0) {                // where a wait was given up the row may not be here
                    uint4 w = reinterpret_cast<const uint4*>(fresh + (s * hg + kvh) * D * 2)[lane];
                    if (!kv && rope_touches(a.rope_type, a.rotary_dim, lane * 8))
                        w = rope_chunk(w, L.k_new + (long long)run.b * pos_stride + head_at * D, lane * 8,
                                       rope_words(a.rope_cos, a.rope_sin, len - 1, a.rope_type, a.rotary_dim, D, lane * 8), a.rope_type, a.rotary_dim, D);
                    *reinterpret_cast<uint4*>(ring + s * TILE + own + (lane >> 3) * col_bytes + r_new * 128 + (((lane & 7) ^ (r_new & 7)) << 4)) = w;
                    reinterpret_cast<uint4*>(cache)[lane] = w;
                }
                __syncwarp();
            };
            const auto release = [&](int s, bool written) {
                if (written) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(empty0 + 8 * s);
            };
            const auto arrived = [&]() {
                if (alive && !mbar_wait_bounded(full0 + 8 * (team * SLOTS + landed), phase, abort_word)) {
                    gave_up(kStatusFullTimeout);
                    alive = false;                                   // walks on without waiting: nobody is left alone at a barrier
                }
                __syncwarp();
                if (++landed == SLOTS) { landed = 0; phase ^= 1; }
            };
            const auto advance = [&](int by) { slot += by; if (slot >= SLOTS) slot -= SLOTS; };

            float s[NV][4];
            arrived();
            slot_k = slot;
            if (left > 0) {
                if (r_new >= 0) put_newest(0, slot);
                lean_scores<D, NV, true>(q_frag, smem_u32(ring) + slot * TILE + k_off, s, col_bytes);
            }
            if (NV == 1 || !last) release(slot, r_new >= 0);
            advance(1);
            arrived();
            slot_v = slot;
            if (left > 0) {
                if (left < kBlockPos || r_new >= 0) {                // rows past the end are zeros
                    for (int i = max(left, 0) * CPR + lane; i < kBlockPos * CPR; i += 32) {
                        const int r = i / CPR, c = i % CPR;
                        *reinterpret_cast<uint4*>(ring + slot * TILE + own + (c >> 3) * col_bytes + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = make_uint4(0u, 0u, 0u, 0u);
                    }
                    if (r_new >= 0) put_newest(1, slot);
                    __syncwarp();
                }
                lean_softmax_pv<D, NV, true>(st, s, smem_u32(ring) + slot * TILE + v_off, left, scale2, g, col_bytes);
            }
            if (!last) release(slot, left < kBlockPos || r_new >= 0);
            advance(2 * TEAMS - 1);
        }
        const bool held = t0 < s1, any = held && first < len;

        // ---- the warps' states meet
        if (any) {
            float probe[4] = {0.f, 0.f, 0.f, 0.f};                   // NaN if any sum is (and sometimes if some are infinite)
            __syncwarp();
#pragma unroll
            for (int v = 0; v < NV; ++v)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = v * 8 + 2 * t4 + h;
                    const float l_head = sum_over_g(st[v].l[h]), m_head = max_over_g(st[v].mt[h]);
                    if (r < group) {
                        float* dst = state_row(own, slot_k, slot_v, r);
#pragma unroll
                        for (int mt = 0; mt < D / 16; ++mt) {
                            dst[(mt * 16 + g) ^ (t4 << 3)] = st[v].o[mt][h];
                            dst[(mt * 16 + g + 8) ^ (t4 << 3)] = st[v].o[mt][2 + h];
                            probe[2 * h] += st[v].o[mt][h];
                            probe[2 * h + 1] += st[v].o[mt][2 + h];
                        }
                        if (g == 0) stats[warp * NV * 8 + r] = make_float4(st[v].m[h], l_head, m_head, __int_as_float(1 + slot_v + (slot_k << 8)));
                    }
                }
            const float all = (probe[0] + probe[1]) + (probe[2] + probe[3]);
            if (__any_sync(0xffffffffu, all != all)) {
                const int head_at = run.h * hg + kvh;
#pragma unroll 1
                for (int r = 0; r < group; ++r)
                    redo_rows_fp32<D>(state_row(own, slot_k, slot_v, r), 1, D, &stats[warp * NV * 8 + r].x, 4,
                                      QueryFragments<D>{smem_u32(q_store + kvh * q_words + QueryFragments<D>::row(r))}, L.k_cache + (long long)run.b * a.kv_batch_stride + head_at * D,
                                      L.v_cache + (long long)run.b * a.kv_batch_stride + head_at * D, pos_stride, first, min((s1 - run.start) * tile, len), TEAMS * tile, scale2, ((r >> 1) & 3) << 3);
            }
        } else if (lane < group) stats[warp * NV * 8 + lane] = make_float4(kNeutralM, 0.f, kNeutralM, 0.f);
        step_sync<THREADS>();
        if (more) put_q(next);
        const bool goes_on = s1 != run.end, was_begun = s0 != run.start;
        bool keep = was_begun && !goes_on;                           // the state stays here, until this CTA finishes the run or a part of it
        if (goes_on && was_begun) {
            const int k = cta - cta_of(run.start);
            keep = (k + 1) % a.fan == 0 && cta_of(run.end - 1) - cta + k >= a.fan;
        }
        if (keep) finish = goes_on ? 2 : 1;
        for (int idx = tid; idx < rows * (D / 4); idx += THREADS) {
            const int j = idx / (D / 4), q4 = idx - j * (D / 4), k = kv_head_of(j), r = j - k * group;
            const float4* const sv = stats + k * NV * 8 + r;
            const int stride = hg * NV * 8, parts = TEAMS * wph;
            float mm = kNeutralM, ll = 0.f;
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int i = 0; i < parts; ++i) mm = fmaxf(mm, sv[i * stride].z);
            for (int i0 = 0; i0 < parts; i0 += 4) {                  // four warps' states at once
                float4 x[4], o[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) x[e] = sv[min(i0 + e, parts - 1) * stride];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int i = min(i0 + e, parts - 1), at = max(__float_as_int(x[e].w), 1), in_team = TEAMS == 2 && i >= wph ? i - wph : i;
                    o[e] = *reinterpret_cast<const float4*>(state_row((k * (D / 64) * tile + 16 * in_team) * 128, at >> 8, (at & 255) - 1, r) + ((q4 * 4) ^ (((r >> 1) & 3) << 3)));
                }
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (i0 + e < parts && __float_as_int(x[e].w) != 0) {
                        const float wgt = fast_exp2(x[e].x - mm);
                        ll = fmaf(x[e].y, wgt, ll);
                        acc.x = fmaf(o[e].x, wgt, acc.x); acc.y = fmaf(o[e].y, wgt, acc.y); acc.z = fmaf(o[e].z, wgt, acc.z); acc.w = fmaf(o[e].w, wgt, acc.w);
                    }
            }
            if (keep) {
                *reinterpret_cast<float4*>(kept + j * SP + q4 * 4) = acc;
                if (q4 == 0) *reinterpret_cast<float2*>(kept + j * SP + D) = make_float2(mm, ll);
            } else if (goes_on) push(j, q4, acc, mm, ll);
            else store_out(run, j, q4, acc, ll);
        }
        if (run.l == a.keep_layer && s0 == run.start) {
            const long long from = ((long long)run.b * a.num_q_heads + run.h * rows) * D;
            for (int i = tid; i < rows * CPR; i += THREADS)
                reinterpret_cast<uint4*>(a.keep_q + from)[i] = reinterpret_cast<const uint4*>(L.q + from)[i];
            if (run.h == 0 && tid == 0) a.keep_offsets[run.b] = len - 1;
        }
        if (!more) break;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // the states lie where the next tiles go
        step_sync<THREADS>();
        if (held && lane == 0) {
            if (NV == 2) mbar_arrive(empty0 + 8 * slot_k);
            mbar_arrive(empty0 + 8 * slot_v);
        }
        run = next;
    }
    if (!finish) return;
    step_sync<THREADS>();
    // ---- a cut run: the states of the CTAs in front, in order, then this CTA's.  Only CTAs with lower numbers are waited for: they run or
    // are done.  Of more than `fan` CTAs in a run, every fan-th merges what lies between the one before it and itself.
    const StepRun& r = finish == 2 ? run : head;
    const int c0 = cta_of(r.start), k = cta - c0;
    const int fan = a.fan, parts = finish == 2 || k < fan ? 0 : k / fan, from = finish == 2 ? k + 1 - fan : parts * fan, sources = parts + k - from;
    const auto source = [&](int i) { return c0 + (i < parts ? (i + 1) * fan - 1 : from + i - parts); };
    const long long t_start = clock64();
    bool in_time = true;
    constexpr int ENTRIES = D / 2 + 1, AT_ONCE = 8;
    const int entries = rows * ENTRIES, at_most = SLOTS * TILE / (rows * SP * 4), items = rows * (D / 4);
#pragma unroll 1
    for (int idx = tid; idx - tid < items; idx += THREADS) {
        const int j = idx / (D / 4), q4 = idx - j * (D / 4);
        float mm = kNeutralM, ll = 0.f;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
        for (int i0 = 0; i0 <= sources; i0 += at_most) {             // as many as shared memory holds; the last of all is this CTA's own
            const int n = min(at_most, sources - i0);
            if (idx == tid || sources >= at_most) {
                if (idx != tid || i0 != 0) step_sync<THREADS>();
                int e = tid, i = 0;                                  // an entry of a source; eight of them at once
                const auto settle = [&]() { for (; e >= entries; e -= entries) ++i; };
                settle();
#pragma unroll 1
                while (i < n) {
                    ulonglong2 w[AT_ONCE];
                    const ulonglong2* from_at[AT_ONCE];
                    float* to[AT_ONCE];
#pragma unroll
                    for (int u = 0; u < AT_ONCE; ++u) {
                        to[u] = nullptr;
                        if (i < n) {
                            const int row = e / ENTRIES;
                            from_at[u] = a.boards + (long long)source(i0 + i) * entries + e;
                            to[u] = reinterpret_cast<float*>(ring) + (i * rows + row) * SP + 2 * (e - row * ENTRIES);
                            w[u] = load_entry(from_at[u]);
                            e += THREADS;
                            settle();
                        }
                    }
#pragma unroll
                    for (int u = 0; u < AT_ONCE; ++u)
                        if (to[u] != nullptr) {
                            while (!entry_of(w[u], tag) && in_time) {
                                w[u] = load_entry(from_at[u]);
                                if (clock64() - t_start > kWaitLimitCycles) in_time = false;
                            }
                            *reinterpret_cast<float2*>(to[u]) = make_float2(__uint_as_float((unsigned)w[u].x), __uint_as_float((unsigned)w[u].y));
                        }
                }
                step_sync<THREADS>();
            }
            if (idx < items) {
                const bool own_too = i0 + at_most > sources;
                const float* at = reinterpret_cast<const float*>(ring) + j * SP;
#pragma unroll 2
                for (int i = 0; i < n + own_too; ++i, at += rows * SP) {
                    if (i == n) at = kept + j * SP;
                    const float2 ml = *reinterpret_cast<const float2*>(at + D);
                    const float4 o = *reinterpret_cast<const float4*>(at + q4 * 4);
                    const float top = fmaxf(mm, ml.x), down = fast_exp2(mm - top), up = fast_exp2(ml.x - top);
                    mm = top;
                    ll = fmaf(ml.y, up, ll * down);
                    acc.x = fmaf(o.x, up, acc.x * down); acc.y = fmaf(o.y, up, acc.y * down);
                    acc.z = fmaf(o.z, up, acc.z * down); acc.w = fmaf(o.w, up, acc.w * down);
                }
            }
        }
        if (idx < items) {
            if (finish == 2) push(j, q4, acc, mm, ll);
            else store_out(r, j, q4, acc, ll);
        }
    }
    if (!in_time) {
        atomicCAS(a.status, 0, kStatusGridTimeout);
        if (a.status_mirror != nullptr) *a.status_mirror = kStatusGridTimeout;
    }
}

#define VTEB_STEP_KERNEL(NAME, DIM, NV)                                                                              \
    extern "C" __global__ void __launch_bounds__((step_warps(DIM, NV) + 1) * 32, 1) NAME(const __grid_constant__ StepArgs a) { \
        step_body<DIM, NV>(a);                                                                                       \
    }

VTEB_STEP_KERNEL(vteb_decode_step_d64_kernel, 64, 1)
VTEB_STEP_KERNEL(vteb_decode_step_d128_kernel, 128, 1)
VTEB_STEP_KERNEL(vteb_decode_step_d256_kernel, 256, 1)
VTEB_STEP_KERNEL(vteb_decode_step_2_d64_kernel, 64, 2)
VTEB_STEP_KERNEL(vteb_decode_step_2_d128_kernel, 128, 2)
