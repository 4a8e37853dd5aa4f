// Decode attention with one work item per CTA (included by decode_attention.cu): every warp of a CTA fetches and
// works through 16-position blocks of its own, so nothing is handed from warp to warp before the merge.
//
// An item is part `c` of `N` of one sequence's positions for ONE KV head and its whole group of query heads.  Two
// kinds of kernel share the body:
//   cluster (`vteb_decode_cluster_...`): the N parts of a (sequence, KV head) are one thread-block cluster; each CTA
//     sends its merged state, 32 columns of a query head at a time, into the shared memory of the CTA that owns those
//     columns (st.async, counted in bytes on the owner's mbarrier), which merges the N states and stores the
//     normalised output.  A layer is ONE launch: no partials in memory, no combine launch, no work words.
//   split (`vteb_split_kv_lean_...`): each CTA stores its state to partial_m / partial_l / partial_o for a combine
//     launch, as the persistent split kernel does.
//
// What bounds them, us: a cluster layer of one sequence of 1,531 positions (12 heads on 2 KV heads of 128) takes 3.3 (7.1
// with append, split and combine): 1.5 between the end of one launch and the end of the next one's wait, 0.4 block
// arithmetic, 0.5 the warps' exchange, 0.6 merge and send, 0.4 last merge and store.  A CTA alone streams about 72 B/ns, two
// warps a scheduler (568 instructions a block before the copies' addresses and Q's words were simplified: 24.8 -> 23.0 for 6,000
// positions on two CTAs); with every SM busy HBM bounds them: 64 (sequence, KV head) pairs of 6,000 positions 33, 6.5 TB/s
// while streaming.  A lean split layer takes 4.6 plus its bytes at 6.6 TB/s: 6.3 for 11,003 positions (8.5), 9.6 for 32,768 (9.9).
// Rings are as deep as the longest part needs, three blocks a warp (two of 256-wide heads) at most: 192 KB in flight an SM.
// Half blocks (four or three warps, two CTAs an SM) serve more pairs than whole-SM clusters fit at once: 40 sequences of 8
// heads 42.4 -> 35.8, 37 of 300 positions 24.3 -> 15.4, 32 sequences of 28 heads on 4 27.3 -> 26.6.
//
// Either way this step's K and V rows may be handed over (`k_new`, `v_new`): the warp whose block ends with the newest
// position puts them, rotated if asked to, into the cache and into its block; no append launch.
#pragma once

#include <cmath>

struct LeanArgs {
    const __half* q; __half* k_cache; __half* v_cache;
    float* partial_m; float* partial_l; float* partial_o;
    int num_q_heads, num_kv_heads; float scale; const int* kv_offsets; int kv_batch_stride; int n_parts;
    int depth;
    const __half* k_new; const __half* v_new;             // this step's projections [B, Hkv, D]; null: the newest row is in the cache
    void* output; int out_kind;                           // cluster kernels: 1 fp16, 2 fp32
    int flags; int* status;
    const __half* next_k_cache; const __half* next_v_cache;   // split kernels, optional: the next layer's caches, for L2;
                                                              // with kLeanKeep: where Q and the offsets are kept instead
    const __half* rope_cos; const __half* rope_sin; int rope_type, rotary_dim;   // rope_type < 0: Q and K arrive rotated
};

__host__ __device__ constexpr int lean_warps(int D) { return D == 256 ? 6 : 8; }
__host__ __device__ constexpr int lean_half_warps(int D) { return D == 256 ? 3 : 4; }  // two CTAs an SM with rings of full depth
__host__ __device__ constexpr int lean_depth(int D) { return D == 256 ? 2 : 3; }      // most blocks a warp has in flight

constexpr int kLeanSplit = 0, kLeanCluster = 1, kLeanHalf = 2;      // split and combine; clusters; clusters of CTAs of half the warps

// What a launch of these kernels needs; `context` is the longest sequence.  A ring no deeper than its blocks need leaves
// room on the SM for the CTAs of the launch behind.  ok = 0: a geometry the kernels do not cover.
struct LeanPlan { int ok, threads, smem_bytes, depth; };
__host__ __device__ inline LeanPlan make_lean_plan(int num_q_heads, int num_kv_heads, int head_dim, int n_parts, long long context, int kind) {
    const bool cluster = kind != kLeanSplit;
    LeanPlan p = {0, 0, 0, 0};
    if ((head_dim != 64 && head_dim != 128 && head_dim != 256) || num_kv_heads <= 0 || num_q_heads <= 0 ||
        num_q_heads % num_kv_heads || n_parts < 1 || kind < kLeanSplit || kind > kLeanHalf || (kind == kLeanHalf && head_dim == 64) || (cluster && (n_parts < 2 || n_parts > 16)) || context < 1) return p;
    const int group = num_q_heads / num_kv_heads, runs = group > 8 ? 2 : 1, block = 64 * head_dim;
    const int warps = kind == kLeanHalf ? lean_half_warps(head_dim) : lean_warps(head_dim);
    if (group > 16 || (runs > 1 && (head_dim == 256 || !cluster))) return p;
    const long long blocks = (vteb::vteb_round_up((int)((context + n_parts - 1) / n_parts), vteb::kBlockPos) / vteb::kBlockPos + warps - 1) / warps;
    p.depth = blocks < lean_depth(head_dim) ? (int)blocks : lean_depth(head_dim);
    while (p.depth * block < group * (head_dim + vteb::kMergePad) * 4) ++p.depth;      // a warp's exchange rows lie in its blocks' memory
    p.threads = warps * 32;
    p.smem_bytes = 128 + runs * (head_dim / 8) * 128 + warps * p.depth * block;
    if (cluster) p.smem_bytes += (group * (head_dim / 32) + n_parts - 1) / n_parts * n_parts * 144;
    p.ok = 1;
    return p;
}

// Estimated microseconds of one layer, by which a route is chosen; `kind` -1: the append / split / combine launches
// these kernels compete with (without the append, 2 us).  `resident`: clusters the device runs at once.  `context`: room in
// the cache, of which a sequence is expected to use three quarters (a batch's mean: half).
// The figures are fitted to 971 steps of 12 head geometries, 1 to 64 sequences of 130 to 80,000 positions (the shortest down to
// a twentieth of the longest) in caches with room for 1 to 2.5 times the longest, 14 routes timed on each.  The choice
// is within 3.5 % of the best route on the whole and takes 0.61 times as long as the launches of kind -1, at most 1.08
// times (above 1.03 in 3 of them).
//   per_position: K and V rows of one KV head through one CTA alone, us; CTAs of an SM share its rate, so a launch lasts as
//   long as its longest part or as all positions spread over the SMs, whichever is longer, but no less than the
//   bytes; a second wave starts when the first one's clusters end.
inline double lean_estimate_us(int kind, int n_parts, int num_q_heads, int num_kv_heads, int head_dim, int batch, long long context,
                               int resident, int num_sms) {
    (void)num_q_heads;
    const double pairs = (double)batch * num_kv_heads;
    const double longest = (batch == 1 ? 0.765 : 0.72) * (double)context, mean = batch == 1 ? longest : 0.504 * (double)context;
    const double bytes = pairs * mean * 4.0 * head_dim;
    const double per_position = head_dim == 64 ? 0.0045 : head_dim == 128 ? 0.00706 : 0.0168;
    if (kind < 0) return batch == 1 ? 9.0 + bytes / 8.2e6 : 12.0 + bytes / 5.5e6;
    if (kind == kLeanSplit) {
        const double stream = bytes / 8.0e6, walk = 0.62 * per_position * longest / n_parts;
        return 4.8 + 0.0117 * head_dim + (stream > walk ? stream : walk);
    }
    const double waves = resident > 0 ? std::ceil(pairs / resident) : 1e9;
    const double part = per_position * (kind == kLeanHalf ? 1.7 : 1.0) * longest / n_parts, spread = 0.96 * per_position * mean * pairs / num_sms;
    const double walk = waves > 1.0 ? 0.84 * part + spread : part > spread ? part : spread;
    return 3.5 + 0.2 * std::log2((double)n_parts) + 2.6 * (waves - 1.0) + std::pow(std::pow(bytes / 6.1e6, 4.0) + std::pow(walk, 4.0), 0.25);
}
constexpr double kLeanMargin = 0.95;       // a route has to be estimated this much below kind -1 (MARGIN in core/lean_route.py)

// The same where the lengths are known: the longest sequence has `longest` positions, all together `total`, in caches with room
// for `capacity`.  Fitted to 3,444 steps of 8 head geometries, 1 to 64 sequences, room for 16 to 65,536 positions, lengths
// all the same, uniform, one or a quarter of them long and the others a fiftieth to a twentieth of it, up to 19 routes timed on
// each: 90 % within a sixth.  Of 2,340 batches in caches above 128 positions, the clusters chosen by capacity took up to 3.3
// times as long as kind -1 and longer than 1.03 times in 248; where every step takes the one that this finds shorter, at
// most 1.37 times and in 42 (and longer than 1.03 times the clusters in 15).
//   a cluster layer: its longest part, the starts of all clusters and the bytes overlap (a p-norm); every further wave costs as
//   much again; merges and starts grow with the query heads of a KV head
//   kind -1: bytes over a rate, what grows with the work items and with the longest over the mean length; up to 128 positions it
//   is one launch that stores the output itself
struct LeanStepFit { double base, per_position, per_pair, wave, bytes_per_us, norm, base_8, per_pair_8, wave_8; };   // _8: for eight query heads a KV head
struct PlainStepFit { double base, bytes_per_us, per_pair_log, per_row, skew, longest_log; };
inline double lean_step_us(int kind, int n_parts, int num_q_heads, int num_kv_heads, int head_dim, int batch, long long capacity, long long longest,
                           double total, int resident) {
    const int runs = num_q_heads > 8 * num_kv_heads ? 1 : 0, d = head_dim == 64 ? 0 : head_dim == 128 ? 1 : 2;
    const double pairs = (double)batch * num_kv_heads, bytes = total * num_kv_heads * 4.0 * head_dim, g = num_q_heads / (8.0 * num_kv_heads);
    if (kind < 0 && capacity <= 128) {
        static const double kSmall[2][3][5] = {{{2.55, .0205, .10, 0., 0.}, {3.4, .0135, .09, .26, .045}, {3.2, .0145, .30, 0., 0.}},
                                               {{3.2, .0045, .06, 0., 0.}, {4.25, .011, .25, .3, 0.}, {4.25, .011, .25, .3, 0.}}};
        const double* c = kSmall[runs][d];
        return c[0] + c[1] * (double)longest + c[2] * std::log2((double)batch) + c[3] * pairs / 148.0 + c[4] * (num_q_heads > 12 ? num_q_heads - 12 : 0);
    }
    if (kind < 0) {
        static const PlainStepFit kOne[2][3] = {{{3.52, 6.87e6, .25, .0027, 0., .25}, {4.42, 7.41e6, .01, .0557, 0., .31}, {5.44, 7.88e6, 0., 0., 0., .36}},
                                                {{5.88, 7.37e6, .25, .002, 0., .50}, {6.42, 7.36e6, .64, .006, 0., .75}, {6.42, 7.36e6, .64, .006, 0., .75}}};
        static const PlainStepFit kBatch[2][3] = {{{3.37, 7.20e6, .89, .0005, .65, .42}, {7.28, 7.13e6, .25, .0057, .80, .48}, {9.51, 7.32e6, .04, .0102, 1.20, .32}},
                                                  {{6.94, 4.02e6, .66, .0023, .66, .26}, {7.89, 5.75e6, 1.15, 0., .83, .68}, {7.89, 5.75e6, 1.15, 0., .83, .68}}};
        const PlainStepFit& c = batch == 1 ? kOne[runs][d] : kBatch[runs][d];
        const double skew = (double)longest * batch / total;
        return c.base + bytes / c.bytes_per_us + c.per_pair_log * std::log2(pairs) + c.per_row * batch * num_q_heads +
               c.skew * std::log2(skew > 1.0 ? skew : 1.0) + c.longest_log * std::log2(longest > 512 ? longest / 512.0 : 1.0);
    }
    if (kind == kLeanSplit) {
        const double stream = bytes / 8.0e6, walk = 0.62 * (d == 0 ? 0.0045 : d == 1 ? 0.00706 : 0.0168) * (double)longest / n_parts;
        return 4.8 + 0.0117 * head_dim + (stream > walk ? stream : walk);
    }
    static const LeanStepFit kCluster[2][3] = {{{2.84, .0038, .0057, 2.80, 6.56e6, 2.0, .29, .0014, .14}, {2.96, .0055, .0062, 2.95, 6.66e6, 3.2, .61, .0118, .56},
                                                {2.99, .0121, .0147, 2.93, 5.95e6, 3.4, 1.51, .0329, .95}},
                                               {{2.90, .0060, .0194, 2.34, 4.39e6, 2.0, .34, .0035, .44}, {3.25, .0080, .0051, 2.99, 5.24e6, 2.8, .73, .0149, .59},
                                                {3.25, .0080, .0051, 2.99, 5.24e6, 2.8, .73, .0149, .59}}};
    static const LeanStepFit kHalf[2][2] = {{{2.76, .0078, .0046, 2.41, 7.00e6, 2.0, .66, .0139, .84}, {3.35, .0165, .0048, 2.93, 6.53e6, 2.0, 1.67, .0417, 1.30}},
                                            {{3.24, .0125, .0092, 2.92, 6.60e6, 3.0, .80, .0143, .76}, {3.24, .0125, .0092, 2.92, 6.60e6, 3.0, .80, .0143, .76}}};
    const LeanStepFit& c = kind == kLeanHalf ? kHalf[runs][d == 2 ? 1 : 0] : kCluster[runs][d];
    const double waves = resident > 0 ? std::ceil(pairs / resident) : 1e9;
    const double part = c.per_position * (double)longest / n_parts, start = (c.per_pair + c.per_pair_8 * g) * pairs, stream = bytes / c.bytes_per_us;
    return c.base + c.base_8 * g + std::pow(std::pow(part, c.norm) + std::pow(start, c.norm) + std::pow(stream, c.norm), 1.0 / c.norm) +
           (c.wave + c.wave_8 * g) * (waves - 1.0);
}

// Where a launch without a status word of its own (flash_attention_kernel's arguments have none) reports a wait that ran
// out; read by vteb_module_check_status.
extern "C" { __device__ int vteb_lean_status = 0; }

constexpr int kLeanRowsFinal = 64;      // flag: the newest row is in the cache before the launch in front starts
constexpr int kLeanKeep = 128;          // flag: Q as it came goes to next_k_cache [B, Hq, D], the offsets to next_v_cache [B], so that
                                        // the partials of this launch can be had later
constexpr int kLeanCtrlBytes = 128;     // barriers and the abort word
constexpr int kLeanUnit = 36;           // floats a CTA sends per 32 output columns: o[32], m, l, 2 unused

__device__ __forceinline__ void cp_async_16_zfill(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// For threads of a warp that may have parted.
__device__ __forceinline__ void cluster_rejoin() { asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ int cluster_size() {
    int n;
    asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n));
    return n;
}
// The address of `addr` (this CTA's shared memory) in the shared memory of CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_map(uint32_t addr, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_send4(uint32_t dst, uint32_t bar, float4 v) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(dst), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar) : "memory");
}

// Eight channels of a row at one position, rotated: `x` = channels d0 .. d0 + 7 of `row`.  The arithmetic of
// rope_channel on 16-byte pieces; cos and sin words are fetched by rope_words ahead of time.
struct RopeWords { uint32_t c[4], s[4]; };
__device__ __forceinline__ bool rope_touches(int rope_type, int rotary_dim, int d0) {
    return rope_type >= 0 && (rope_type != 2 || d0 < rotary_dim);
}
__device__ __forceinline__ RopeWords rope_words(const __half* cos_table, const __half* sin_table, int pos, int rope_type,
                                                int rotary_dim, int D, int d0) {
    RopeWords w;
    const int rot = (rope_type == 2) ? rotary_dim : D, half = rot >> 1;
    const long long at = rope_type == 1 ? (long long)pos * D + (d0 >> 1) : (long long)pos * rot + (d0 < half ? d0 : d0 - half);
    const uint32_t* c = reinterpret_cast<const uint32_t*>(cos_table + at);
    const uint32_t* s = reinterpret_cast<const uint32_t*>(sin_table + at);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const bool on = rope_type != 1 || i < 2;        // adjacent pairs: four entries for eight channels
        w.c[i] = on ? c[i] : 0u;
        w.s[i] = on ? s[i] : 0u;
    }
    return w;
}
__device__ __forceinline__ uint4 rope_chunk(uint4 x, const __half* row, int d0, const RopeWords& w, int rope_type, int rotary_dim, int D) {
    uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4];
    if (rope_type == 1) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 p = unpack_half2(xs[i]), c = unpack_half2(w.c[i >> 1]), s = unpack_half2(w.s[i >> 1]);
            float y0, y1;
            rope_pair(p.x, p.y, (i & 1) ? c.y : c.x, (i & 1) ? s.y : s.x, y0, y1);
            ys[i] = pack_half2(y0, y1);
        }
    } else {
        const int half = ((rope_type == 2) ? rotary_dim : D) >> 1;
        const bool low = d0 < half;
        const uint4 other = *reinterpret_cast<const uint4*>(row + (low ? d0 + half : d0 - half));
        const uint32_t os[4] = {other.x, other.y, other.z, other.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 a = unpack_half2(low ? xs[i] : os[i]), b = unpack_half2(low ? os[i] : xs[i]);
            const float2 c = unpack_half2(w.c[i]), s = unpack_half2(w.s[i]);
            float a0, b0, a1, b1;
            rope_pair(a.x, b.x, c.x, s.x, a0, b0);
            rope_pair(a.y, b.y, c.y, s.y, a1, b1);
            ys[i] = low ? pack_half2(a0, a1) : pack_half2(b0, b1);
        }
    }
    return make_uint4(ys[0], ys[1], ys[2], ys[3]);
}

// Scores of a 16-position block for NV runs of up to eight query heads, K fragments shared by the runs (transposed form
// of consumer_block.cuh); `col_bytes` between 64 channels and the next 64 of a row.  kFresh: products of one k-step start from zero and are summed in fp32 registers.
template <int D, int NV, bool kFresh>
__device__ __forceinline__ void lean_scores(const uint32_t* q_frag, uint32_t kaddr, float (&s)[NV][4], uint32_t col_bytes = 128) {
    constexpr int KS = D / 16, CH = kFresh ? 4 : 2;
    float acc[NV][CH][4];
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            s[v][i] = 0.f;
#pragma unroll
            for (int c = 0; c < CH; ++c) acc[v][c][i] = 0.f;
        }
#pragma unroll
    for (int kc = 0; kc < KS; kc += 4) {
        uint32_t kf[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) ldmatrix_x4((kaddr ^ (i << 5)) + (kc >> 2) * col_bytes, kf[i][0], kf[i][1], kf[i][2], kf[i][3]);
#pragma unroll
        for (int i = 0; i < 4; i += 2)
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const uint4 qv = *reinterpret_cast<const uint4*>(q_frag + (v * (D / 8) + 2 * (kc + i)) * 32);    // k-steps kc + i, kc + i + 1
                if constexpr (kFresh) {
                    mma_alone(acc[v][i], kf[i][0], kf[i][2], kf[i][1], kf[i][3], qv.x, qv.y);
                    mma_alone(acc[v][i + 1], kf[i + 1][0], kf[i + 1][2], kf[i + 1][1], kf[i + 1][3], qv.z, qv.w);
                } else {
                    mma_full(acc[v][i % CH], kf[i][0], kf[i][2], kf[i][1], kf[i][3], qv.x, qv.y);
                    mma_full(acc[v][(i + 1) % CH], kf[i + 1][0], kf[i + 1][2], kf[i + 1][1], kf[i + 1][3], qv.z, qv.w);
                }
            }
        if constexpr (kFresh) {
#pragma unroll
            for (int v = 0; v < NV; ++v)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[v][j] += (acc[v][0][j] + acc[v][1][j]) + (acc[v][2][j] + acc[v][3][j]);
        }
    }
    if constexpr (!kFresh) {
#pragma unroll
        for (int v = 0; v < NV; ++v)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[v][j] = acc[v][0][j] + acc[v][1][j];
    }
}

// Softmax step and O^T += V^T P^T for NV runs, V fragments shared by the runs; `st[v]` as in softmax_pv_t.
template <int D, int NV, bool kFresh>
__device__ __forceinline__ void lean_softmax_pv(ConsumerStateT<D / 16> (&st)[NV], const float (&sraw)[NV][4], uint32_t vaddr,
                                                int left, float scale2, int g, uint32_t col_bytes = 128) {
    constexpr int NVC = D / 64;                  // chunks of 64 output columns
    uint32_t vf[2][4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) ldmatrix_x4_trans(vaddr ^ (i << 5), vf[0][i][0], vf[0][i][1], vf[0][i][2], vf[0][i][3]);
    const bool valid[2] = {g < left, g + 8 < left};
    constexpr float kSlack = VTEB_LAZY_MAX;
    uint32_t bh[NV][2], bl[NV][2];
    float s[NV][4], p[NV][4], mx[NV][2];
    bool up = false;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
#pragma unroll
        for (int i = 0; i < 4; ++i) s[v][i] = valid[i >> 1] ? sraw[v][i] * scale2 : kNeutralM;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            mx[v][h] = fmaxf(s[v][h], s[v][2 + h]);
            st[v].mt[h] = fmaxf(st[v].mt[h], mx[v][h]);
            up = up || mx[v][h] > st[v].m[h] + kSlack;
        }
    }
    if (__any_sync(0xffffffffu, up)) {                               // one branch for all runs: their arithmetic overlaps
#pragma unroll
        for (int v = 0; v < NV; ++v)
            if (NV == 1 || __any_sync(0xffffffffu, (mx[v][0] > st[v].m[0] + kSlack) | (mx[v][1] > st[v].m[1] + kSlack))) {
                float corr[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float m_up = fmaxf(st[v].m[h], max_over_g(mx[v][h]));
                    corr[h] = fast_exp2(st[v].m[h] - m_up);
                    st[v].l[h] *= corr[h];
                    st[v].m[h] = m_up;
                }
#pragma unroll
                for (int i = 0; i < D / 16; ++i) { st[v].o[i][0] *= corr[0]; st[v].o[i][1] *= corr[1]; st[v].o[i][2] *= corr[0]; st[v].o[i][3] *= corr[1]; }
            }
    }
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
        for (int i = 0; i < 4; ++i) p[v][i] = valid[i >> 1] ? fast_exp2(s[v][i] - st[v].m[i & 1]) : 0.f;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        st[v].l[0] += p[v][0] + p[v][2];
        st[v].l[1] += p[v][1] + p[v][3];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            if constexpr (kFresh) { p[v][2 * r] *= kFreshUp; p[v][2 * r + 1] *= kFreshUp; }
            const __half2 hi = __floats2half2_rn(p[v][2 * r], p[v][2 * r + 1]);
            const float2 hif = __half22float2(hi);
            bh[v][r] = movmatrix_trans(*reinterpret_cast<const uint32_t*>(&hi));
            constexpr float lo_up = kFresh ? kFreshLoUp : 1.f;
            bl[v][r] = movmatrix_trans(pack_half2((p[v][2 * r] - hif.x) * lo_up, (p[v][2 * r + 1] - hif.y) * lo_up));
        }
    }
#pragma unroll
    for (int ch = 0; ch < NVC; ++ch) {
        if (ch + 1 < NVC) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                ldmatrix_x4_trans((vaddr ^ (i << 5)) + (ch + 1) * col_bytes, vf[(ch + 1) & 1][i][0], vf[(ch + 1) & 1][i][1],
                                  vf[(ch + 1) & 1][i][2], vf[(ch + 1) & 1][i][3]);
        }
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            if constexpr (kFresh) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t* f = vf[ch & 1][i];
                    float hi[4], lo[4];
                    mma_alone(hi, f[0], f[2], f[1], f[3], bh[v][0], bh[v][1]);
                    mma_alone(lo, f[0], f[2], f[1], f[3], bl[v][0], bl[v][1]);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        st[v].o[ch * 4 + i][j] = fmaf(fmaf(lo[j], kFreshLoDown, hi[j]), kFreshDown, st[v].o[ch * 4 + i][j]);
                }
            } else if constexpr (D == 64) {                              // the low parts' products on their own, added in fp32
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t* f = vf[ch & 1][i];
                    float lo[4] = {0.f, 0.f, 0.f, 0.f};
                    mma_full(st[v].o[ch * 4 + i], f[0], f[2], f[1], f[3], bh[v][0], bh[v][1]);
                    mma_full(lo, f[0], f[2], f[1], f[3], bl[v][0], bl[v][1]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) st[v].o[ch * 4 + i][j] += lo[j];
                }
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t* f = vf[ch & 1][i];
                    mma_full(st[v].o[ch * 4 + i], f[0], f[2], f[1], f[3], bh[v][0], bh[v][1]);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t* f = vf[ch & 1][i];
                    mma_full(st[v].o[ch * 4 + i], f[0], f[2], f[1], f[3], bl[v][0], bl[v][1]);
                }
            }
        }
    }
}

// Q as redo_rows_fp32 takes it: the fragments at their place in shared memory, with no register spent on it.
template <int D> struct LeanQueries {
    __device__ __forceinline__ float operator()(int r, int d) const {
        extern __shared__ __align__(128) unsigned char smem_raw[];
        return QueryFragments<D>{smem_u32(smem_raw) + kLeanCtrlBytes}(r, d);
    }
};

// D: head width; NV: runs of eight query heads a warp serves; CW: warps.
template <int D, int NV, int CW, bool kFresh, bool kCluster>
__device__ __forceinline__ void lean_body(const LeanArgs& a)
{
    constexpr int P = lean_depth(D);
    constexpr int ROW = 2 * D, CPR = D / 8, BLK = 2 * 16 * ROW;      // bytes of a row, its 16-byte chunks, bytes of a block (K, then V)
    constexpr int PITCH = D + kMergePad;                             // floats of an exchange row: o[D], 4 unused, m, l, true maximum, 1 unused
    constexpr int THREADS = CW * 32;
    const int depth = a.depth;                                       // blocks a warp has in flight, at most P; the host sizes the ring for it
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const uint32_t bar_recv = smem_u32(smem_raw);
    volatile int* abort_word = reinterpret_cast<volatile int*>(smem_raw + 8);
    uint32_t* q_store = reinterpret_cast<uint32_t*>(smem_raw + kLeanCtrlBytes);              // Q as mma fragments: [run][chunk / 4][head, word][chunk % 4]
    unsigned char* ring = smem_raw + kLeanCtrlBytes + NV * CPR * 128;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int group = a.num_q_heads / a.num_kv_heads, N = a.n_parts;
    float* recv = reinterpret_cast<float*>(ring + CW * depth * BLK);     // cluster kernels: [owned unit][sender][kLeanUnit]

    int b, kv_head, part;
    if constexpr (kCluster) {                                        // the parts of a pair are neighbours: one cluster
        const int pair = blockIdx.x / N;
        part = blockIdx.x - pair * N;
        b = pair / a.num_kv_heads; kv_head = pair - b * a.num_kv_heads;
    } else {                                                         // the KV heads of a part are neighbours: their rows alternate in memory
        const int rest = blockIdx.x / a.num_kv_heads;
        kv_head = blockIdx.x - rest * a.num_kv_heads;
        b = rest / N; part = rest - b * N;
    }
    if constexpr (kCluster) {
        // Launched with other clusters than its parts (or without any, where st.async is an illegal instruction): refuse.
        if (cluster_size() != N) {
            if (threadIdx.x == 0) atomicCAS(a.status, 0, kStatusGridTimeout);
            return;
        }
    }
    // With kFlagWaitFirst nothing is read before the launch in front is done; what needs no memory is set up before that (28
    // launches of four sequences of 100 to 1,500 positions, each behind the one in front: 161.7 -> 144.1 us).
    const bool wait_first = a.flags & kFlagWaitFirst;
    int total = wait_first ? 0 : a.kv_offsets[b] + 1;
    const int units = group * (D / 32), my_units = kCluster && part < units ? (units - part + N - 1) / N : 0;
    if (threadIdx.x == 0) {
        mbar_init(bar_recv, 1);
        *abort_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (my_units > 0) mbar_arrive_expect_tx(bar_recv, my_units * N * kLeanUnit * 4);
    }
    for (int i = threadIdx.x; i < NV * CPR * 8; i += THREADS) reinterpret_cast<uint4*>(q_store)[i] = make_uint4(0u, 0u, 0u, 0u);
    if (wait_first) {
        if constexpr (kCluster) cluster_arrive();
        grid_dependency_wait();
        total = a.kv_offsets[b] + 1;
    }
    __syncthreads();
    grid_launch_dependents();
    if constexpr (kCluster) { if (!wait_first) cluster_arrive(); }
    const int chunk = vteb_round_up((total + N - 1) / N, kBlockPos);
    const int start = (int)min((long long)part * chunk, (long long)total), end = min(start + chunk, total);
    const int nblk = (end - start + kBlockPos - 1) / kBlockPos;
    // The newest row may be written by the launch in front (or comes from k_new): this CTA's last block gets it after the wait.
    const bool late = end > start && end == total && !((a.flags & kLeanRowsFinal) && a.k_new == nullptr);
    const int load_end = late ? end - 1 : end;
    const long long pos_stride = (long long)a.num_kv_heads * D;      // halves between positions
    const long long base = (long long)b * a.kv_batch_stride + (long long)kv_head * D;

    // ---- this warp's blocks: warp, warp + CW, ...; block i in slot i % depth.  Swizzled rows: chunk c of row r at c ^ (r & 7).
    const uint32_t ring_w = smem_u32(ring) + warp * depth * BLK;
    constexpr int RPI = 32 / CPR;                                    // rows per copy instruction of the warp (a power of two)
    const int row_l = lane / CPR, c_l = lane % CPR;
    const uint32_t at_l = row_l * ROW + (((c_l & ~7) | ((c_l ^ row_l) & 7)) << 4);
    const long long step = RPI * pos_stride;
    auto fetch = [&](int i, int slot) {
        const int blk = warp + i * CW;
        if (blk < nblk) {
            const int row0 = start + blk * kBlockPos;
            const uint32_t dst = ring_w + slot * BLK + at_l;
            const long long off = base + (row0 + row_l) * pos_stride + c_l * 8;
            const __half* ks = a.k_cache + off;
            const __half* vs = a.v_cache + off;
            if (row0 + kBlockPos <= load_end) {
#pragma unroll
                for (int s = 0; s < 16 / RPI; ++s) {
                    const uint32_t at = (dst ^ (((s * RPI) & 7) << 4)) + s * RPI * ROW;
                    async_copy_16(at, ks);
                    async_copy_16(at + 16 * ROW, vs);
                    ks += step; vs += step;
                }
            } else {                                                 // rows past the end are zeros
#pragma unroll 1
                for (int s = 0; s < 16 / RPI; ++s) {
                    const bool on = row0 + s * RPI + row_l < load_end;
                    const uint32_t at = (dst ^ (((s * RPI) & 7) << 4)) + s * RPI * ROW;
                    cp_async_16_zfill(at, on ? ks : a.k_cache + base, on);
                    cp_async_16_zfill(at + 16 * ROW, on ? vs : a.v_cache + base, on);
                    ks += step; vs += step;
                }
            }
        }
        cp_async_commit();
    };
#pragma unroll
    for (int i = 0; i < P; ++i)
        if (i < depth) fetch(i, i);

    // the next layer's rows of this part
    bool ahead = !kCluster && a.next_k_cache != nullptr && !(a.flags & kLeanKeep) && warp < 2 && end > start &&
                 (long long)total * pos_stride * 2 <= kL2PrefetchMaxBytes;
    auto fetch_ahead = [&]() {
        ahead = false;
        const long long bytes = (long long)(end - start) * ROW;      // this KV head's share of the part's full rows
        prefetch_range_l2(reinterpret_cast<const unsigned char*>(warp == 0 ? a.next_k_cache : a.next_v_cache) +
                              2 * ((long long)b * a.kv_batch_stride + (long long)start * pos_stride) + kv_head * bytes, bytes, lane);
    };
    const bool my_late = late && (nblk - 1) % CW == warp;
    const bool rotate = a.rope_type >= 0;
    const int q_chunk = threadIdx.x % CPR;                           // THREADS is a multiple of CPR: the same chunk of every head
    static_assert(THREADS % CPR == 0, "one chunk per thread");
    RopeWords q_words, k_words;
    constexpr int LATE = (2 * CPR + 31) / 32;                        // 16-byte pieces of the newest K and V rows per lane
    if (rotate) {
        if (rope_touches(a.rope_type, a.rotary_dim, q_chunk * 8))
            q_words = rope_words(a.rope_cos, a.rope_sin, total - 1, a.rope_type, a.rotary_dim, D, q_chunk * 8);
        if (my_late && a.k_new != nullptr && lane < CPR && rope_touches(a.rope_type, a.rotary_dim, lane * 8))
            k_words = rope_words(a.rope_cos, a.rope_sin, total - 1, a.rope_type, a.rotary_dim, D, lane * 8);
    }
    if ((a.flags & kFlagPrefetchQ) && threadIdx.x == 0 && part == 0) {
        const __half* q0 = a.q + ((long long)b * a.num_q_heads + (long long)kv_head * group) * D;
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(q0), "r"((unsigned)(group * D * 2)) : "memory");
    }
    if constexpr (kCluster) cluster_wait();                          // every CTA's barriers are set up
    grid_dependency_wait();

    // ---- the newest row's pieces (K: 0 .. CPR - 1, V: CPR .. 2 CPR - 1), then Q
    uint4 fresh[LATE];
    const long long new_row = ((long long)b * a.num_kv_heads + kv_head) * D, cache_row = base + (long long)(total - 1) * pos_stride;
    if (my_late) {
#pragma unroll
        for (int i = 0; i < LATE; ++i) {
            const int p = lane + 32 * i, c = p % CPR;
            if (p < 2 * CPR) {
                const __half* src = p < CPR ? (a.k_new ? a.k_new + new_row : a.k_cache + cache_row)
                                            : (a.k_new ? a.v_new + new_row : a.v_cache + cache_row);
                fresh[i] = *reinterpret_cast<const uint4*>(src + c * 8);
            }
        }
    }
    for (int h = threadIdx.x / CPR; h < group; h += THREADS / CPR) {
        const __half* row = a.q + ((long long)b * a.num_q_heads + (long long)kv_head * group + h) * D;
        uint4 x = *reinterpret_cast<const uint4*>(row + q_chunk * 8);
        if (rotate && rope_touches(a.rope_type, a.rotary_dim, q_chunk * 8))
            x = rope_chunk(x, row, q_chunk * 8, q_words, a.rope_type, a.rotary_dim, D);
        uint32_t* dst = q_store + ((h >> 3) * CPR + (q_chunk & ~3)) * 32 + (h & 7) * 16 + (q_chunk & 3);
        dst[0] = x.x; dst[4] = x.y; dst[8] = x.z; dst[12] = x.w;
    }
    if (my_late && a.k_new != nullptr) {
        if (rotate && lane < CPR && rope_touches(a.rope_type, a.rotary_dim, lane * 8))
            fresh[0] = rope_chunk(fresh[0], a.k_new + new_row, lane * 8, k_words, a.rope_type, a.rotary_dim, D);
#pragma unroll
        for (int i = 0; i < LATE; ++i) {
            const int p = lane + 32 * i, c = p % CPR;
            if (p < 2 * CPR) *reinterpret_cast<uint4*>((p < CPR ? a.k_cache : a.v_cache) + cache_row + c * 8) = fresh[i];
        }
    }
    __syncthreads();                                                 // Q is in place

    const int g = lane >> 2, t = lane & 3;
    const float scale2 = a.scale * kLog2e;
    const uint32_t* q_frag = q_store + lane * 4;
    const uint32_t k_off = ((lane & 7) + ((lane >> 4) << 3)) * ROW + ((((lane >> 3) & 1) ^ (lane & 7)) << 4);
    const uint32_t v_off = ((lane & 7) + (((lane >> 3) & 1) << 3)) * ROW + (((lane >> 4) ^ (lane & 7)) << 4) + 16 * ROW;
    ConsumerStateT<D / 16> st[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) st[v].reset();

    for (int i = 0, slot = 0, blk = warp; blk < nblk; ++i, blk += CW) {
        if (depth == 1) cp_async_wait<0>();
        else if (depth == 2) cp_async_wait<1>();
        else cp_async_wait<2>();
        __syncwarp();
        const uint32_t at = ring_w + slot * BLK;
        if (my_late && blk == nblk - 1) {
            const int r = (end - 1 - start) & (kBlockPos - 1);
#pragma unroll
            for (int j = 0; j < LATE; ++j) {
                const int p = lane + 32 * j, c = p % CPR;
                if (p < 2 * CPR) {
                    const uint32_t dst = at + (p < CPR ? 0 : 16 * ROW) + r * ROW + (((c & ~7) | ((c ^ r) & 7)) << 4);
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(fresh[j].x), "r"(fresh[j].y), "r"(fresh[j].z), "r"(fresh[j].w) : "memory");
                }
            }
            __syncwarp();
        }
        if (ahead && blk + depth * CW >= nblk) fetch_ahead();
        float s[NV][4];
        lean_scores<D, NV, kFresh>(q_frag, at + k_off, s);
        lean_softmax_pv<D, NV, kFresh>(st, s, at + v_off, end - start - blk * kBlockPos, scale2, g);
        __syncwarp();
        fetch(i + depth, slot);
        slot = slot + 1 == depth ? 0 : slot + 1;
    }
    cp_async_wait<0>();
    __syncwarp();

    // ---- the warps' states meet in shared memory: row h of warp w lies in warp w's own blocks' memory
    float* const mine = reinterpret_cast<float*>(ring + (size_t)warp * depth * BLK);
    float probe[4] = {0.f, 0.f, 0.f, 0.f};                           // NaN if any sum is (and sometimes if some are infinite)
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = v * 8 + 2 * t + h;
            const float l_head = sum_over_g(st[v].l[h]), m_head = max_over_g(st[v].mt[h]);
            if (r < group) {
                float* dst = mine + r * PITCH;
#pragma unroll
                for (int mt = 0; mt < D / 16; ++mt) {
                    dst[mt * 16 + g] = st[v].o[mt][h];
                    dst[mt * 16 + g + 8] = st[v].o[mt][2 + h];
                    if constexpr (kFresh) { probe[2 * h] += st[v].o[mt][h]; probe[2 * h + 1] += st[v].o[mt][2 + h]; }
                }
                if (g == 0) { dst[D + 4] = st[v].m[h]; dst[D + 5] = l_head; dst[D + kMergeTrueMax] = m_head; }
            }
        }
    if constexpr (kFresh) {
        const float all = (probe[0] + probe[1]) + (probe[2] + probe[3]);
        if (__any_sync(0xffffffffu, all != all))
            redo_rows_fp32<D>(mine, group, PITCH, mine + D + 4, PITCH, LeanQueries<D>{}, a.k_cache + (long long)b * a.kv_batch_stride + (long long)kv_head * D,
                              a.v_cache + (long long)b * a.kv_batch_stride + (long long)kv_head * D, pos_stride, start + warp * kBlockPos, end, CW * kBlockPos, scale2);
    }
    __syncthreads();

    // What kLeanKeep asks for.  The place is by measurement: beside the load of Q the test cost every launch 0.1 us; clusters take
    // it best behind their sends (28 layers of 1,531 positions 103.9 us, here 105.5), the split of 256-wide heads here
    // (8 layers of 24,001 positions 112.4, at the end 115 to 117).
    const auto keep_inputs = [&]() {
        if (a.flags & kLeanKeep) {
            const long long from = ((long long)b * a.num_q_heads + (long long)kv_head * group) * D;
#pragma unroll 1
            for (int i = threadIdx.x; part == 0 && i < group * CPR; i += THREADS)
                reinterpret_cast<uint4*>(const_cast<__half*>(a.next_k_cache) + from)[i] = reinterpret_cast<const uint4*>(a.q + from)[i];
            if (part == 0 && kv_head == 0 && threadIdx.x == 0) reinterpret_cast<int*>(const_cast<__half*>(a.next_v_cache))[b] = total - 1;
        }
    };
    if constexpr (!kCluster) keep_inputs();
    const long long head0 = (long long)b * a.num_q_heads + (long long)kv_head * group;
    for (int idx = threadIdx.x; idx < group * (D / 4); idx += THREADS) {
        const int h = idx / (D / 4), q4 = idx - h * (D / 4);
        const float* row = reinterpret_cast<const float*>(ring) + h * PITCH;
        const int WS = depth * BLK / 4;                              // floats between two warps' rows
        float mm = kNeutralM;
#pragma unroll
        for (int w = 0; w < CW; ++w) mm = fmaxf(mm, row[w * WS + D + kMergeTrueMax]);
        float ll = 0.f;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < CW; ++w) {
            const float wt = fast_exp2(row[w * WS + D + 4] - mm);
            const float4 o = *reinterpret_cast<const float4*>(row + w * WS + q4 * 4);
            ll = fmaf(row[w * WS + D + 5], wt, ll);
            acc.x = fmaf(o.x, wt, acc.x); acc.y = fmaf(o.y, wt, acc.y); acc.z = fmaf(o.z, wt, acc.z); acc.w = fmaf(o.w, wt, acc.w);
        }
        if constexpr (kCluster) {
            const int unit = h * (D / 32) + (q4 >> 3), owner = unit % N, slot = unit / N;
            const uint32_t dst = cluster_map(smem_u32(recv + (slot * N + part) * kLeanUnit), owner), bar = cluster_map(bar_recv, owner);
            cluster_send4(dst + (q4 & 7) * 16, bar, acc);
            if ((q4 & 7) == 0) cluster_send4(dst + 128, bar, make_float4(mm, ll, 0.f, 0.f));
        } else {
            const long long stat = (head0 + h) * N + part;
            *reinterpret_cast<float4*>(a.partial_o + stat * D + q4 * 4) = acc;
            if (q4 == 0) {
                a.partial_m[stat] = end > start ? mm * kLn2 : kNeutralM;
                a.partial_l[stat] = end > start ? ll : 0.f;
            }
        }
    }
    if constexpr (kCluster) keep_inputs();
    if constexpr (kCluster) {
        if (my_units == 0) return;
        if (!mbar_wait_bounded(bar_recv, 0, abort_word)) {           // nobody leaves while another CTA may still send to it
            raise_abort(abort_word, a.status, kStatusGridTimeout);
            cluster_rejoin();                                        // every state that comes has been sent, but may not have arrived
            mbar_wait_bounded(bar_recv, 0, nullptr, 1LL << 31);
            return;
        }
        for (int slot = warp; slot < my_units; slot += CW) {
            const float* src = recv + slot * N * kLeanUnit;
            // every lane takes all the weights itself: broadcast reads instead of shuffles
            float m[16], top = kNeutralM, sum = 0.f, acc = 0.f;
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                m[k] = k < N ? src[k * kLeanUnit + 32] : kNeutralM;
                top = fmaxf(top, m[k]);
            }
#pragma unroll
            for (int k = 0; k < 16; ++k)
                if (k < N) {
                    const float wt = fast_exp2(m[k] - top);
                    sum = fmaf(src[k * kLeanUnit + 33], wt, sum);
                    acc = fmaf(src[k * kLeanUnit + lane], wt, acc);
                }
            const int unit = slot * N + part, h = unit / (D / 32);
            const long long at = (head0 + h) * D + (unit - h * (D / 32)) * 32 + lane;
            const float v = acc / fmaxf(sum, 1e-20f);
            if (a.out_kind == 2) reinterpret_cast<float*>(a.output)[at] = v;
            else reinterpret_cast<__half*>(a.output)[at] = __float2half(v);
        }
    }
}

#define VTEB_LEAN_KERNEL(NAME, DIM, NV, WARPS, FRESH, CLUSTER, BOUNDS)                                                  \
    extern "C" __global__ void BOUNDS NAME(                                                                             \
        const __half* __restrict__ q, __half* k_cache, __half* v_cache, float* __restrict__ partial_m,                  \
        float* __restrict__ partial_l, float* __restrict__ partial_o, int num_q_heads, int num_kv_heads, int head_dim,  \
        float scale, const int* __restrict__ kv_cache_offset_ptr, int kv_batch_stride, int n_parts,                     \
        const __half* __restrict__ k_new, const __half* __restrict__ v_new, void* __restrict__ output, int out_kind,    \
        int flags, int depth, int* __restrict__ status, const __half* __restrict__ next_k_cache,                        \
        const __half* __restrict__ next_v_cache, const __half* __restrict__ cos_cache,                                  \
        const __half* __restrict__ sin_cache, int rope_type, int rotary_dim)                                            \
    {                                                                                                                   \
        (void)head_dim;                                                                                                 \
        LeanArgs a;                                                                                                     \
        a.q = q; a.k_cache = k_cache; a.v_cache = v_cache;                                                              \
        a.partial_m = partial_m; a.partial_l = partial_l; a.partial_o = partial_o;                                      \
        a.num_q_heads = num_q_heads; a.num_kv_heads = num_kv_heads; a.scale = scale;                                    \
        a.kv_offsets = kv_cache_offset_ptr; a.kv_batch_stride = kv_batch_stride; a.n_parts = n_parts;                   \
        a.k_new = k_new; a.v_new = v_new; a.output = output; a.out_kind = out_kind; a.flags = flags; a.status = status ? status : &vteb_lean_status; \
        a.depth = depth;                                                                                                    \
        a.next_k_cache = next_k_cache; a.next_v_cache = next_v_cache;                                                   \
        a.rope_cos = cos_cache; a.rope_sin = sin_cache; a.rope_type = rope_type; a.rotary_dim = rotary_dim;             \
        lean_body<DIM, NV, WARPS, FRESH, CLUSTER>(a);                                                                   \
    }

VTEB_LEAN_KERNEL(vteb_decode_cluster_d64_kernel, 64, 1, lean_warps(64), true, true, __launch_bounds__(256, 2))
VTEB_LEAN_KERNEL(vteb_decode_cluster_d128_kernel, 128, 1, lean_warps(128), true, true, __launch_bounds__(256, 2))
VTEB_LEAN_KERNEL(vteb_decode_cluster_d256_kernel, 256, 1, lean_warps(256), true, true, __launch_bounds__(192, 1))
VTEB_LEAN_KERNEL(vteb_decode_cluster_2_d64_kernel, 64, 2, lean_warps(64), true, true, __launch_bounds__(256, 2))
VTEB_LEAN_KERNEL(vteb_decode_cluster_2_d128_kernel, 128, 2, lean_warps(128), true, true, __launch_bounds__(256, 1))
VTEB_LEAN_KERNEL(vteb_decode_cluster_half_d128_kernel, 128, 1, lean_half_warps(128), true, true, __launch_bounds__(128, 3))
VTEB_LEAN_KERNEL(vteb_decode_cluster_half_d256_kernel, 256, 1, lean_half_warps(256), true, true, __launch_bounds__(96, 2))
VTEB_LEAN_KERNEL(vteb_decode_cluster_half_2_d128_kernel, 128, 2, lean_half_warps(128), true, true, __launch_bounds__(128, 2))
VTEB_LEAN_KERNEL(vteb_split_kv_lean_d64_kernel, 64, 1, lean_warps(64), false, false, __maxnreg__(160))
VTEB_LEAN_KERNEL(vteb_split_kv_lean_d128_kernel, 128, 1, lean_warps(128), false, false, __maxnreg__(160))
VTEB_LEAN_KERNEL(vteb_split_kv_lean_d256_kernel, 256, 1, lean_warps(256), true, false, __maxnreg__(168))
