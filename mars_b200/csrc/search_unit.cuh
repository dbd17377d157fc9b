// The unit-vector correlation of the small block sizes (4 and 8), included by search_tc.cu
// inside its anonymous namespace.
//
// At these sizes a candidate fit is few multiply-adds, so the correlation is bound by what
// follows the accumulator, not by the tensor pipe: the integer form (process_item) spends 13
// of its 26 instructions per 8 fits on one threshold per (domain lane, range).  Here the
// operands are normalised instead, so that the threshold depends on the range alone:
//   A row (domain) = 64 (D - mean) / |D - mean|, f16, the S x S contracted window;
//   B row (range, isometry) = 64 (r - mean) / |r - mean|, f16, the permuted block;
//   accumulator (f32) = 4096 rho, rho = Nrd / sqrt(Ndd Nrr), the cosine of the two.
// A candidate of a range whose champion has W = Nrr - n T > 0 (fit.cuh) can only survive with
// Nrd >= sqrt(W Ndd), that is rho >= sqrt(W / Nrr): one number per range, republished when the
// champion improves.  W > 0 also means that the qalfa = 0 class cannot win (its SSE is at least
// Nrr / n > T), so nothing else has to be looked at.
//
// The filter stays exact.  Rounding to f16 moves a row by at most 2^-11 of its length (the
// factor 64 keeps what a flushed subnormal could add below 2^-17), so rho is off by at most
// 2^-10 + 2^-22 from the operands and, |products| summing to at most 1, by less than 2^-14 from
// f32 accumulation, 0.00104 together; thresholds are lowered by 4.5 / 4096 = 0.0011.  (2^-9 let
// twice as many pass where a step edge meets many like it.)  What passes is evaluated again from
// the integers: the exact correlation, the full bound of fit.cuh with the largest contrast added,
// then the f64 fit.  So the winners, their rms bits and the tie order are the integer path's.
//
// Ranges whose champion is no better than the flat fit have no such number: a candidate of
// contrast 0 ties with that fit, and wins if its domain comes first.  They take the per-lane bound
// of fit.cuh on Nrd = rho sqrt(Ndd Nrr), the full form, until their champion improves or is of
// the first domain, which the seeds see to (seed_small_kernel); from then on W <= 0 leaves the
// tile's contrast alone to give a threshold (unit_tile_threshold).  A tile whose threshold is low
// takes the full form too.  (A checkerboard of 4 x 4 squares, 1024 x 1024 at S = 8, stride 4, where
// nothing beats the flat fit: 1.8 ms, 13.1 with every tile in the full form; the integer form 2.8.)
//
// Survivors leave the scan at once: a scan warp appends (domain, range) to its own ring in
// shared memory, and the fit warp of its column half evaluates them, up to 32 at a time, so the
// scan does not wait for window loads and f64 divisions; at the end of an item the scan warps
// evaluate what is left in theirs.  (Evaluated by the scan warps throughout, the registers kept
// around it cost every tile more than the evaluation.)  A scan warp whose ring is full evaluates
// some of it: the ranges of highest contrast are step edges that a thousand domains match nearly
// alike, and two fit warps alone took 2.2 ms over such a tile of a 640 x 480 plane at stride 4,
// ten times a usual tile and more than everything after it: every node of that plane alone
// took 3.2 to 4.3 ms, 2.0 to 2.2 so.
// Champions are guarded by a sequence lock per range, a ring's takers by a lock; every wait is
// bounded.
//
// Domains and ranges are sorted by contrast (sqrt Ndd, sqrt Nrr; order_* kernels).  The contrast a
// fit may apply is limited to a_min..a_max, so against a domain much flatter, or much rougher,
// than the range the needed rho is higher than sqrt(W / Nrr), past 1 when the two cannot match at
// all.  In sorted order a tile of 128 domains has nearly one contrast, and the load warp takes
// the bound at it per (tile, range): tiles that none of the 32 ranges can use are never loaded
// (a tenth at 512 x 512, S = 4; nearly all for high-contrast ranges), and the others' thresholds
// are the tile's.
//
// Most survivors of a plain sweep come early, while the champions are the seeds.  So an item
// whose ranges no other split has searched yet starts with a preview: every 16th tile (or 8 of
// them, or all) is correlated once without thresholds, keeping each range's best candidate,
// which the fit warp evaluates.
//
// Bound: the maxima and comparisons after the accumulator (5 ALU instructions per 8 fits, a half-
// rate pipe) and the survivors.  Measured on one B200 at stride 2, sizes 32..4: the search of a
// 512 x 512 plane 3.70 -> 2.35 ms, of a 1024 x 1024 plane 49.8 -> 27.3 ms (before the lower
// allowance and the help with full rings: an encode of 512 x 512 by 14 % and of 1536 x 1024 by 9 %
// faster with them); a 128 x 256 tile at
// S = 4 takes 1,150 cycles with its survivors, the integer form's 2,900, the bare pipeline (MMA,
// accumulator reads, maxima) 550.

// Warp roles (384 threads): load, MMA, 8 scan warps (4 TMEM lane quadrants x 2 column halves), 2
// fit warps.  (Two groups of 8 scan warps taking alternate tiles were no faster: their maxima
// share the same ALU pipes, and at 96 registers the evaluation spills.)
constexpr int kScanWarps = 8;
constexpr int kFitWarps = 2;                               // one per column half
constexpr int kHalfWarps = kScanWarps / kFitWarps;         // scan warps of a half
constexpr int kUnitThreads = 32 * (2 + kScanWarps + kFitWarps);
constexpr int kRing = 64;                                  // slots of a scan warp's ring
constexpr int kPreview = 16;                               // the preview's tile stride,
constexpr int kPreviewLeast = 8;                           // and the tiles it has at least
constexpr int kSlots = 16;                                 // tiles announced ahead
constexpr int kGroup = 8;                                  // tiles that share their thresholds
constexpr int kSets = 32;                                  // sets of thresholds in use
constexpr float kUnitScale = 4096.0f;                      // 64 x 64
constexpr float kUnitSlack = 4.5f;                         // the filter's allowance
constexpr float kUnitLeast = kUnitScale / 64.0f;           // a tile's threshold below: full form
constexpr float kUnitAlike = 1.1f;                         // the contrasts of tiles that are alike
constexpr float kUnitNone = 1e-30f;                        // a champion's W gives no threshold

// A tile as the load warp announces it: what to do, which domains, and the set of thresholds its
// ranges take there.  The load warp is at most kMaxStages tiles ahead of the MMAs and those two
// ahead of the scan, so a slot, or a set, is rewritten only when its tiles are through.
enum SlotKind : int { kSlotScan = 0, kSlotPreview = 1, kSlotEvaluate = 2, kSlotEnd = 3 };
struct __align__(16) Slot {
    int tile;
    int kind_set;    // kind | threshold set << 8
    float contrast;  // the tile's largest sqrt(Ndd)
    uint32_t full;   // the ranges that take the full form there, a bit each
};

struct USmem {
    uint64_t full[kMaxStages];
    uint64_t empty[kMaxStages];
    uint64_t tfull[2];
    uint64_t tempty[2];
    uint64_t bres;
    uint32_t tmem_base;
    int abort_flag;
    int item;  // the all-levels launch: this CTA's current work item
    int last;  // this CTA finished the last split of its range tile
    ThrRec thr[kRangesPerTile];          // the full form's records (unit_publish)
    Champ ch[kRangesPerTile];
    float uscan[kRangesPerTile];         // the scan's state of each range (scan_state.cuh)
    int udone[2];                        // per half: scan warps through with the item
    uint32_t useq[kRangesPerTile];       // the champions' sequence locks
    uint32_t utail[kScanWarps];          // the rings' next slots to take, and
    uint32_t ulock[kScanWarps];          // their takers' locks
    uint32_t udirty, uexact;             // ranges with an unshared champion; fits made
    // The preview: whether there is one; per half the warps whose best are in, and one more once
    // they are evaluated; each range's 1 / sqrt(Nrr) and best (share of its energy, position).
    int upreview, ukeyed[2];
    float uinv[kRangesPerTile];
    unsigned long long ukey[kRangesPerTile];
    uint32_t urange[kRangesPerTile];     // the tile's ranges (indices into the level's)
    Slot slot[kSlots];
    alignas(16) float set[kSets][kRangesPerTile];
    unsigned long long ring[kScanWarps][kRing];  // zero between items
};
constexpr size_t kUnitHead = (sizeof(USmem) + 1023) / 1024 * 1024;

template <int S>
struct UCfg {
    static constexpr int N = S * S;
    static constexpr int KG = N / 8;             // 16-byte k-groups of a row
    static constexpr int kStage = KG * kM * 16;  // A bytes of a tile, one pipeline stage
    static constexpr int kB = KG * kN * 16;      // resident B tile
    static constexpr int kStages = S == 8 ? 5 : 6;
    static constexpr int kPix = kRangesPerTile * 8 * N;  // the ranges' pixels, per isometry
    static constexpr size_t kBytes = (size_t)kStages * kStage + kB + kPix;
    static_assert(S == 4 || S == 8, "block sizes of the unit form");
    static_assert(kStages <= kMaxStages, "pipeline depth");
};
// A ring entry: domain position in contrast order | range of the tile << 32 | 1 << 63 (a free slot
// is zero).
__device__ __forceinline__ unsigned long long unit_entry(int pos, int rl) {
    return 1ull << 63 | (unsigned long long)rl << 32 | (uint32_t)pos;
}

struct ScanWords {
    float* at;
    __device__ float load(int i) const { return *(volatile const float*)(at + i); }
    __device__ void store(int i, float v) const { *(volatile float*)(at + i) = v; }
};

// The pruning records of range rl from its champion: the full form's (sqrt W, W / (2 a_min),
// sqrt Nrr rounded up, tie domain), then the scan's state: its threshold, or the full form.
__device__ __forceinline__ void unit_publish(USmem& sm, int rl, const FitParams& fp, int n) {
    const Champ& C = sm.ch[rl];
    const ScanWords words{sm.uscan};
    if (!C.valid || C.nrr == 0) {
        sm.thr[rl] = ThrRec{INFINITY, INFINITY, 0.0f, -1};
        scan_publish(words, rl, false, kScanNothing);
        return;
    }
    const Threshold th = make_threshold(C.sum, C.rms, C.idx >> 3, C.rms0, C.nrr, n, fp);
    const float snrr = __fsqrt_ru(__ll2float_ru(C.nrr));
    // Whether no candidate of contrast 0 can win any more: the champion is better than the flat
    // fit, or as good and of the first domain, whose candidates the seed was chosen among.
    const bool settled = th.mode == 2 || (th.mode == 1 && th.tie_dom == 0);
    ThrRec t;
    t.sqrt_w = th.wpos ? th.sqrt_w : -INFINITY;
    t.w2a = th.w2a;
    t.c = snrr;
    t.tie = settled ? -1 : (th.mode == 1 ? (int32_t)th.tie_dom : INT32_MAX);
    sm.thr[rl] = t;
    const float u = th.wpos ? __fdiv_rd(th.sqrt_w, snrr) * kUnitScale - kUnitSlack : 0.0f;
    scan_publish(words, rl, !settled, fmaxf(u, kUnitNone));
}

// fit.cuh's bound on Nrd for one (range record, domain), every step rounded toward -inf, with
// the contrast's upper limit added: among the contrasts a_min..a_max the SSE's minimum lies at
// sqrt(W / Ndd) clamped to them, so past a_max the bound is W / (2 a_max) + a_max Ndd / 2.
__device__ __forceinline__ float unit_tau(const ThrRec& t, int dom, float detf, float sdetf,
                                          const FitParams& fp) {
    const float g1 = __fmul_rd(t.sqrt_w, sdetf);
    if (dom <= t.tie) return g1;
    const float ad = __fmul_rd(fp.a_min, detf);
    float tau = fminf(__fadd_rd(t.w2a, __fmul_rd(fp.a_half, detf)), fmaxf(g1, ad));
    if (t.sqrt_w > 1.0001f * fp.a_max * sdetf)
        tau = fmaxf(tau, __fadd_rd(__fmul_rd(t.w2a, fp.min_over_max), __fmul_rd(fp.max_half, detf)));
    return tau;
}

// Whether (rms, idx) beats range rl's champion, read without the lock: a torn read says yes.
__device__ __forceinline__ bool unit_better(USmem& sm, int rl, double rms, uint32_t idx) {
    volatile Champ* C = &sm.ch[rl];
    const uint32_t s0 = *(volatile uint32_t*)&sm.useq[rl];
    __threadfence_block();
    const double r = C->rms;
    const uint32_t i = C->idx;
    __threadfence_block();
    const uint32_t s1 = *(volatile uint32_t*)&sm.useq[rl];
    return s0 != s1 || (s0 & 1u) || rms < r || (rms == r && idx < i);
}

// One lane of a warp at a time: replaces range rl's champion by (rms, sum, idx, t1) if that is
// better, under the range's lock (bounded: a holder only does arithmetic).  True when it was replaced.
__device__ bool unit_replace(USmem& sm, int rl, const FitParams& fp, int n, double rms, double sum,
                             uint32_t idx, int32_t t1, int* err) {
    for (int spin = 0; spin < (1 << 22); ++spin) {
        const uint32_t s = *(volatile uint32_t*)&sm.useq[rl];
        if ((s & 1u) || atomicCAS(&sm.useq[rl], s, s + 1u) != s) continue;
        __threadfence_block();
        Champ& C = sm.ch[rl];
        const double r = *(volatile double*)&C.rms;
        const bool better = rms < r || (rms == r && idx < *(volatile uint32_t*)&C.idx);
        if (better) {
            *(volatile double*)&C.rms = rms;
            *(volatile double*)&C.sum = sum;
            *(volatile uint32_t*)&C.idx = idx;
            *(volatile int32_t*)&C.t1x4 = t1;
            __threadfence_block();
            unit_publish(sm, rl, fp, n);
        }
        __threadfence_block();
        atomicExch(&sm.useq[rl], s + 2u);
        return better;
    }
    *(volatile int*)&sm.abort_flag = 1;
    atomicOr(err, 64);
    return false;
}

// A 16-byte shared-memory read that is made where it stands (another warp may rewrite the
// record; a v4 access moves whole).
__device__ __forceinline__ float4 lds_f4(const void* p) {
    float4 v;
    asm volatile("ld.volatile.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(smem_u32(p))
                 : "memory");
    return v;
}

// The exact correlations t1_x4 of each lane's entry (domain position pos, range rl) under the eight
// isometries: 16 samples of the window at a time, in pairs of 16 bits (they are at most 1020),
// against the range's permuted bytes.  The windows lie beside the A operand in its order, so 16
// bytes a load, and those of the neighbouring domains that survive together share lines.  (Sample
// by sample from the contracted plane, 64 loads of as many lines at S = 8, a 1024 x 1024 ramp,
// whose blocks all match, took 31.7 ms at stride 8; 26.1 so, the integer form 25.2.)  Compact on purpose:
// this code runs rarely, and what a cold instruction costs to fetch exceeds what it computes.
template <int S>
__device__ __forceinline__ void unit_correlate(const ItemArgs& a, const uint8_t* pix, bool act,
                                               uint32_t pos, int rl, uint32_t (&t1)[8]) {
    constexpr int N = S * S;
#pragma unroll
    for (int k = 0; k < 8; ++k) t1[k] = 0u;
    if (!act) return;
    const uint4* dw = a.unit.windows + (size_t)(pos / 8) * N + pos % 8;
    const uint4* rr = reinterpret_cast<const uint4*>(pix + rl * 8 * N);
#pragma unroll 1
    for (int c = 0; c < N / 16; ++c) {
        const uint4 lo = __ldg(dw), hi = __ldg(dw + 8);
        const uint32_t d[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
        dw += 16;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint4 r = rr[k * (N / 16) + c];
            const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                t1[k] = __dp2a_lo(d[2 * i], w[i], t1[k]);
                t1[k] = __dp2a_hi(d[2 * i + 1], w[i], t1[k]);
            }
        }
    }
}

// Evaluates up to 32 entries, one a lane (zero: none): the exact correlations, the full bound,
// the exact fits, and the champions.  best_only: the entry's largest correlation alone.  All 32
// lanes call this.
template <int S>
__device__ __noinline__ void unit_fit(const ItemArgs& a, USmem& sm, const uint8_t* pix,
                                      unsigned long long entry, bool best_only, int* err) {
    constexpr int N = S * S;
    const int lane = threadIdx.x & 31;
    const bool act = entry != 0ull;
    const uint32_t dom = act ? a.unit.domains[(uint32_t)entry] : 0u;
    const int rl = (int)(entry >> 32) & 31;
    // The candidate's statistics are in flight with its window.
    int s1 = 0;
    int64_t s2 = 0;
    float detf = 0.0f, sdetf = 0.0f;
    if (act) {
        s1 = a.ds.s1x4[dom];
        s2 = a.ds.s2x16[dom];
        detf = a.ds.detf[dom];
        sdetf = a.ds.sdetf[dom];
    }
    uint32_t t1s[8];
    unit_correlate<S>(a, pix, act, (uint32_t)entry, rl, t1s);
    const int32_t t0 = sm.ch[rl].t0, t2 = sm.ch[rl].t2;
    uint32_t isos = act ? 0xFFu : 0u;
    if (best_only && act) {
        uint32_t most = t1s[0];
        isos = 1u;
#pragma unroll
        for (int c = 1; c < 8; ++c)
            if (t1s[c] > most) {
                most = t1s[c];
                isos = 1u << c;
            }
    }
    for (;;) {
        // The lane's next isometry that the range's present bound lets through: t1_x4 at least
        // (s1_x4 t0 + 4 tau) / n, rounded down.
        const float4 rr = lds_f4(&sm.thr[rl]);
        const ThrRec rec{rr.x, rr.y, rr.z, __float_as_int(rr.w)};
        const float tau = unit_tau(rec, (int)dom, detf, sdetf, a.fp);
        const float least =
            __fmul_rd(__fmaf_rd((float)s1, (float)t0, __fmul_rd(4.0f, tau)), 1.0f / (float)N);
        const int32_t floor_t1 = __float2int_rd(least);
        int k = 0;
        int32_t t1 = 0;
        bool take = false;
#pragma unroll
        for (int c = 0; c < 8; ++c)
            if ((isos >> c & 1u) && !take) {
                if ((int32_t)t1s[c] >= floor_t1) {
                    take = true;
                    k = c;
                    t1 = (int32_t)t1s[c];
                }
                isos &= ~(1u << c);
            }
        if (!__any_sync(0xffffffffu, take)) break;
        double rms = 0.0, sum = 0.0;
        bool better = false;
        const uint32_t idx = dom * 8u + (uint32_t)k;
        if (take) {
            const FitResult f = fit_exact(N, s1, s2, t0, t1, t2, a.fp);
            rms = f.rms;
            sum = f.sum;
            better = unit_better(sm, rl, rms, idx);
        }
        // One lane a range takes the lock: the best of the warp's, so lanes never wait for each
        // other there.
        uint32_t pend = __ballot_sync(0xffffffffu, better);
        while (pend) {
            const int r0 = __shfl_sync(0xffffffffu, rl, __ffs(pend) - 1);
            const bool same = better && rl == r0;
            pend &= ~__ballot_sync(0xffffffffu, same);
            // rms >= 0: its bits order as integers.
            const unsigned long long bits =
                same ? (unsigned long long)__double_as_longlong(rms) : ~0ull;
            const uint32_t hi = __reduce_min_sync(0xffffffffu, (uint32_t)(bits >> 32));
            const uint32_t lo = __reduce_min_sync(
                0xffffffffu, (uint32_t)(bits >> 32) == hi ? (uint32_t)bits : UINT32_MAX);
            const bool top = same && (uint32_t)(bits >> 32) == hi && (uint32_t)bits == lo;
            const uint32_t first = __reduce_min_sync(0xffffffffu, top ? idx : UINT32_MAX);
            if (top && idx == first && unit_replace(sm, rl, a.fp, N, rms, sum, idx, t1, err))
                atomicOr(&sm.udirty, 1u << rl);
            __syncwarp();
        }
        const uint32_t nfit = __popc(__ballot_sync(0xffffffffu, take));
        if (lane == 0) atomicAdd(&sm.uexact, nfit);
    }
    __syncwarp();
}

// Shares improved champions with the ranges' other splits through the 128-bit records (rms
// bits, index, t1_x4), and takes theirs when better.  Lanes 0..15: the ranges of column half
// `part`.
template <int S>
__device__ __noinline__ void unit_share(const ItemArgs& a, USmem& sm, int part, int* err) {
    const int lane = threadIdx.x & 31;
    uint32_t bits = 0u;
    if (lane == 0) bits = atomicAnd(&sm.udirty, ~(0xFFFFu << (16 * part)));
    bits = __shfl_sync(0xffffffffu, bits, 0) >> (16 * part) & 0xFFFFu;
    if (a.gch && lane < 16 && (bits >> lane & 1u)) {
        const int rl = part * 16 + lane;
        unsigned long long* grec = a.gch + 2 * (size_t)sm.urange[rl];
        volatile Champ* C = &sm.ch[rl];
        unsigned long long clo, chi;
        cas128(grec, 0ull, 0ull, 0ull, 0ull, clo, chi);
        for (int tries = 0; tries < 64; ++tries) {
            // The champion as one consistent triple.
            const uint32_t q0 = *(volatile uint32_t*)&sm.useq[rl];
            __threadfence_block();
            const unsigned long long mlo = (unsigned long long)__double_as_longlong(C->rms);
            const uint32_t idx = C->idx;
            const int32_t mt1 = C->t1x4;
            __threadfence_block();
            if ((q0 & 1u) || *(volatile uint32_t*)&sm.useq[rl] != q0) continue;
            const uint32_t gidx = (uint32_t)chi;
            if (mlo < clo || (mlo == clo && idx < gidx)) {
                const unsigned long long vhi =
                    (unsigned long long)idx | (unsigned long long)(uint32_t)mt1 << 32;
                unsigned long long olo, ohi;
                cas128(grec, clo, chi, mlo, vhi, olo, ohi);
                if (olo == clo && ohi == chi) break;
                clo = olo;
                chi = ohi;
            } else {
                if (clo < mlo || gidx < idx) {
                    const uint32_t d = gidx >> 3;
                    const int32_t gt1 = (int32_t)(uint32_t)(chi >> 32);
                    const FitResult f = fit_exact(S * S, a.ds.s1x4[d], a.ds.s2x16[d], C->t0, gt1,
                                                  C->t2, a.fp);
                    unit_replace(sm, rl, a.fp, S * S, f.rms, f.sum, gidx, gt1, err);
                }
                break;
            }
        }
    }
    __syncwarp();
}

// Takes the oldest entries of 32 / PER rings: lane l looks at slot l % PER past the tail of ring
// first + l / PER.  A ring that another warp is taking from is left out this time.  All 32 lanes
// call this; each gets an entry or zero.
template <int PER>
__device__ __forceinline__ unsigned long long unit_take(USmem& sm, int first) {
    const int lane = threadIdx.x & 31, off = lane % PER, lead = lane - off;
    const int w = first + lane / PER;
    // Looked at before it is locked: an empty ring costs one read.
    uint32_t tail = *(volatile uint32_t*)&sm.utail[w];
    bool mine = false;
    if (off == 0 && *(volatile unsigned long long*)&sm.ring[w][tail & (kRing - 1)])
        mine = atomicCAS(&sm.ulock[w], 0u, 1u) == 0u;
    if (!__any_sync(0xffffffffu, mine)) return 0ull;
    mine = __shfl_sync(0xffffffffu, mine, lead);
    __threadfence_block();
    volatile unsigned long long* slot = nullptr;
    unsigned long long e = 0ull;
    if (mine) {
        tail = *(volatile uint32_t*)&sm.utail[w];
        slot = &sm.ring[w][(tail + (uint32_t)off) & (kRing - 1)];
        e = *slot;
    }
    // The written slots from the tail on, without a gap.
    const uint32_t bal = __ballot_sync(0xffffffffu, e != 0ull);
    const uint32_t own = PER == 32 ? bal : (bal >> lead) & ((1u << (PER & 31)) - 1u);
    const int count = ~own ? __ffs(~own) - 1 : 32;
    if (off >= count) e = 0ull;
    if (e) *slot = 0ull;
    __threadfence_block();
    __syncwarp();
    if (mine && off == 0) {
        *(volatile uint32_t*)&sm.utail[w] = tail + (uint32_t)count;
        __threadfence_block();
        atomicExch(&sm.ulock[w], 0u);
    }
    return e;
}

// Appends the warp's entries (lanes with `act`) to its own ring; while they do not fit, evaluates
// some of it, or waits (bounded) for the fit warp that holds it: false when the wait gave up.  head
// is the ring's next slot, tail the last tail read.
template <int S>
__device__ __forceinline__ bool unit_push(const ItemArgs& a, USmem& sm, const uint8_t* pix, int w,
                                          bool act, unsigned long long entry, uint32_t& head,
                                          uint32_t& tail, int* err) {
    volatile int* abort_flag = &sm.abort_flag;
    const uint32_t bal = __ballot_sync(0xffffffffu, act);
    const uint32_t count = __popc(bal);
    if (head + count - tail > (uint32_t)kRing) {
        const long long t0 = clock64();
        for (;;) {
            tail = __shfl_sync(0xffffffffu, *(volatile uint32_t*)&sm.utail[w], 0);
            if (head + count - tail <= (uint32_t)kRing) break;
            const unsigned long long mine = unit_take<32>(sm, w);
            if (__any_sync(0xffffffffu, mine != 0ull)) {
                unit_fit<S>(a, sm, pix, mine, false, err);
                continue;
            }
            if (clock64() - t0 > kWaitCycles) {
                *abort_flag = 1;
                atomicOr(err, 128);
            }
            if (__any_sync(0xffffffffu, *abort_flag != 0)) return false;
            __nanosleep(100);
        }
    }
    if (act)
        *(volatile unsigned long long*)&sm
             .ring[w][(head + __popc(bal & ((1u << (threadIdx.x & 31)) - 1u))) & (kRing - 1)] =
            entry;
    head += count;
    return true;
}

__device__ __forceinline__ void tmem_ld64(uint32_t taddr, int32_t (&v)[64]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x64.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
        "%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32,%33,%34,"
        "%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47,%48,%49,%50,%51,%52,%53,%54,%55,"
        "%56,%57,%58,%59,%60,%61,%62,%63}, [%64];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
          "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
          "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
          "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]),
          "=r"(v[31]), "=r"(v[32]), "=r"(v[33]), "=r"(v[34]), "=r"(v[35]), "=r"(v[36]),
          "=r"(v[37]), "=r"(v[38]), "=r"(v[39]), "=r"(v[40]), "=r"(v[41]), "=r"(v[42]),
          "=r"(v[43]), "=r"(v[44]), "=r"(v[45]), "=r"(v[46]), "=r"(v[47]), "=r"(v[48]),
          "=r"(v[49]), "=r"(v[50]), "=r"(v[51]), "=r"(v[52]), "=r"(v[53]), "=r"(v[54]),
          "=r"(v[55]), "=r"(v[56]), "=r"(v[57]), "=r"(v[58]), "=r"(v[59]), "=r"(v[60]),
          "=r"(v[61]), "=r"(v[62]), "=r"(v[63])
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, int32_t (&v)[8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
          "=r"(v[7])
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait8(int32_t (&v)[8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) asm volatile("" : "+r"(v[i]));
}

__device__ __forceinline__ void tmem_wait64(int32_t (&v)[64]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    // No consumer of the loaded registers moves ahead of the wait.
#pragma unroll
    for (int i = 0; i < 64; ++i) asm volatile("" : "+r"(v[i]));
}

// Maximum of a range's 8 columns (positive floats order as integers; a negative one is a
// negative integer).
template <int W>
__device__ __forceinline__ int32_t unit_top(const int32_t (&v)[W], int o) {
    return __vimax3_s32(__vimax3_s32(v[o], v[o + 1], v[o + 2]),
                        __vimax3_s32(v[o + 3], v[o + 4], v[o + 5]), max(v[o + 6], v[o + 7]));
}

// Ranges in the full form (bits of `full`, from range rb) that domain position pos may survive:
// Nrd is at most (rho + slack) sqrt(Ndd) sqrt(Nrr), rho the lane's maxima `top`.
__device__ __noinline__ uint32_t unit_look_full(const ItemArgs& a, USmem& sm, uint32_t full, int rb,
                                                uint32_t tcol, int pos, int ndom) {
    const bool inside = pos < ndom;
    const int dom = inside ? (int)a.unit.domains[pos] : 0;
    const float detf = inside ? a.ds.detf[dom] : 0.0f, sdetf = inside ? a.ds.sdetf[dom] : 0.0f;
    uint32_t mask = 0u;
#pragma unroll 1
    for (int q = 0; q < 8; ++q) {
        if (!(full >> q & 1u)) continue;
        int32_t v[8];
        tmem_ld8(tcol + 8u * q, v);
        tmem_wait8(v);
        const float4 rr = lds_f4(&sm.thr[rb + q]);
        const ThrRec rec{rr.x, rr.y, rr.z, __float_as_int(rr.w)};
        const float len = __fmul_ru(__fmul_ru(sdetf, 1.000001f), rec.c) * (1.0f / kUnitScale);
        const float most = __fadd_ru(__int_as_float(max(unit_top(v, 0), 0)), kUnitSlack);
        if (inside && __fmul_ru(most, len) >= unit_tau(rec, dom, detf, sdetf, a.fp)) mask |= 1u << q;
    }
    return mask;
}

// The scan's threshold of a range in a tile of contrasts lo..hi (sqrt Ndd, rounded down; ilo and
// ihi their reciprocals): the smallest rho that a fit with a contrast in a_min..a_max needs
// there, in accumulator units.  It is u = sqrt(W / Nrr) where the best contrast
// sqrt(W) / sqrt(Ndd) is allowed, and grows away from there, so the tile's end nearest to that
// counts; with W <= 0 it grows with the contrast.  rr: the range's record (sqrt W, W / (2 a_min)),
// inv: 1 / sqrt(Nrr).  The steps' rounding, and reciprocals good to a few units in the last place,
// stay far below the 1e-5 taken off.
__device__ __forceinline__ float unit_tile_threshold(const float4& rr, float u, float inv, float lo,
                                                     float hi, float ilo, float ihi,
                                                     const FitParams& fp) {
    const float weak = rr.y * fp.min_over_max * ihi + fp.max_half * hi;
    // (W <= 0: what the two terms' rounding could leave of their difference is taken off the first.)
    const float strong = fminf(rr.y, rr.y * 1.00001f) * ilo + fp.a_half * lo;
    // Nrd needed over sqrt(Ndd)
    const float tau = rr.x > 1.0001f * fp.a_max * hi
                          ? weak
                          : (rr.x * 1.0001f < fp.a_min * lo ? strong : 0.0f);
    return fmaxf(u, tau * inv * (kUnitScale * 0.99999f) - kUnitSlack);
}

// An item's tiles: every msplit-th group of kGroup, from group `split` on, so that each split meets
// domains of every contrast (in bands of their own, a split of flat domains kept poor champions
// and let everything through).  Tile t of the item, and how many it has.
__device__ __forceinline__ int unit_tile(const ItemArgs& a, int split, int t) {
    return (t / kGroup * a.msplit + split) * kGroup + t % kGroup;
}

__device__ __forceinline__ int unit_tile_count(const ItemArgs& a, int split) {
    const int groups = (a.m_tiles + kGroup - 1) / kGroup;
    if (split >= groups) return 0;
    const int mine = (groups - 1 - split) / a.msplit + 1;
    const bool ends = (groups - 1 - split) % a.msplit == 0;  // has the last, maybe partial one
    return mine * kGroup - (ends ? groups * kGroup - a.m_tiles : 0);
}

// ---- the roles of a work item (each warp runs one; out of line, so that each gets its own
// register allocation) ----

// Load warp: the B tile, then the item's tiles in contrast order -- the preview's, then those that
// some range can use -- each announced in a slot with its thresholds.  Lane = range.
template <int S>
__device__ __noinline__ void unit_load_role(const ItemArgs& a, USmem& sm, int ntile, int split,
                                            int count, unsigned char* stages, PipeState& state,
                                            int* err) {
    using C_ = UCfg<S>;
    PipeState ps = state;  // in registers
    const int lane = threadIdx.x & 31;
    volatile int* abort_flag = &sm.abort_flag;
    unsigned char* stA = stages;
    unsigned char* stB = stages + C_::kStages * C_::kStage;
    if (lane == 0) {
        mbar_expect_tx(&sm.bres, C_::kB);
        bulk_load(stB, a.bglob + (size_t)ntile * C_::kB, C_::kB, &sm.bres);
    }
    const int n_pre = sm.upreview ? max(count / kPreview, min(count, kPreviewLeast)) : 0;
    int s = 0, seq = 0;
    // One slot (lane 0): a tile to correlate, or a word to the other roles (tile < 0).
    auto announce = [&](int kind_set, int tile, float contrast, uint32_t full) {
        const uint32_t bit = 1u << s;
        if ((ps.stage_used & bit) &&
            !mbar_wait(&sm.empty[s], (ps.stage_par & bit) ? 0u : 1u, abort_flag, err, 1))
            return false;
        sm.slot[seq++ % kSlots] = Slot{tile, kind_set, contrast, full};
        if (tile >= 0) {
            mbar_expect_tx(&sm.full[s], C_::kStage);
            bulk_load(stA + s * C_::kStage, a.unit.aglob + (size_t)tile * C_::kStage, C_::kStage,
                      &sm.full[s]);
        } else {
            mbar_arrive(&sm.full[s]);
        }
        ps.stage_used |= bit;
        ps.stage_par ^= bit;
        if (++s == C_::kStages) s = 0;
        return true;
    };
    bool ok = true;
    int sets = 0;
    // The item's tiles begin, begin + step, ... (n of them), `group` at a time with common
    // thresholds: those that some range can use (no accumulator is above kUnitScale by more than
    // rounding).
    auto sweep = [&](int kind, int begin, int step, int n, int group) {
        const float inv = sm.uinv[lane];
        for (int base = 0; ok && base < n; base += 32) {
            // The contrasts of 32 tiles at a time.
            const float2 c = __ldg(a.unit.contrasts +
                                   unit_tile(a, split, begin + min(base + lane, n - 1) * step));
            const int m = min(32, n - base);
            for (int t = 0; ok && t < m; t += group) {
                // Tiles are in contrast order up to a class's width: the group's range is its
                // first and last tiles'.
                float lo = INFINITY, hi = 0.0f;
                for (int q = t; q < min(t + group, m); ++q) {
                    lo = fminf(lo, __shfl_sync(0xffffffffu, c.x, q));
                    hi = fmaxf(hi, __shfl_sync(0xffffffffu, c.y, q));
                }
                // The record may be of an earlier or a later champion than the state: any
                // champion's bounds hold.
                const float4 rr = lds_f4(&sm.thr[lane]);
                const ScanState st = scan_read(ScanWords{sm.uscan}, lane);
                float thr = unit_tile_threshold(rr, st.threshold, inv, lo, hi, __fdividef(1.0f, lo),
                                                __fdividef(1.0f, hi), a.fp);
                // Where the contrast alone gives the threshold, only tiles of one contrast scan.
                const bool full = st.full || thr < kUnitLeast ||
                                  (st.threshold < kUnitLeast && hi > kUnitAlike * lo);
                const uint32_t fulls = __ballot_sync(0xffffffffu, full);
                if (full) thr = INFINITY;
                if (!fulls && !__any_sync(0xffffffffu, thr <= kUnitScale * 1.002f)) continue;
                const int set = sets++ % kSets;
                sm.set[set][lane] = thr;
                __syncwarp();
                if (lane == 0)
                    for (int q = t; ok && q < min(t + group, m); ++q)
                        ok = announce(kind | set << 8, unit_tile(a, split, begin + (base + q) * step),
                                      hi, fulls);
                ok = __shfl_sync(0xffffffffu, ok, 0);
            }
        }
    };
    auto word = [&](int kind) {
        if (ok && lane == 0) ok = announce(kind, -1, 0.0f, 0u);
        ok = __shfl_sync(0xffffffffu, ok, 0);
    };
    if (n_pre) {
        const int step = count / n_pre;
        sweep(kSlotPreview, step / 2, step, n_pre, 1);
        word(kSlotEvaluate);
        // The thresholds that follow are those of the preview's champions.
        const long long t0 = clock64();
        while (ok && (*(volatile int*)&sm.ukeyed[0] <= kHalfWarps ||
                      *(volatile int*)&sm.ukeyed[1] <= kHalfWarps)) {
            if (*abort_flag || clock64() - t0 > kWaitCycles) break;  // others report it
            __nanosleep(100);
        }
        __syncwarp();
    }
    sweep(kSlotScan, 0, 1, count, kGroup);
    word(kSlotEnd);
    if (!ok && lane == 0) {
        // Given up: wait (bounded) for the loads still in flight before leaving.
        for (int s2 = 0; s2 < kMaxStages; ++s2) {
            const uint32_t bit = 1u << s2;
            if (!(ps.stage_used & bit)) continue;
            const uint32_t par = (ps.stage_par & bit) ? 0u : 1u;
            const long long t0 = clock64();
            while (!mbar_try_wait(&sm.full[s2], par) && clock64() - t0 < kWaitCycles) {
            }
        }
        const long long t0 = clock64();
        while (!mbar_try_wait(&sm.bres, ps.bres & 1u) && clock64() - t0 < kWaitCycles) {
        }
    }
    ++ps.bres;
    state = ps;
    __syncwarp();
}

// MMA warp's elected lane: a tile's products into the TMEM buffers in turn; a slot without a tile
// passes through them the same way.
template <int S>
__device__ __noinline__ void unit_mma_role(USmem& sm, unsigned char* stages, uint32_t tmem,
                                           PipeState& state, int* err) {
    using C_ = UCfg<S>;
    PipeState ps = state;  // in registers
    constexpr uint32_t kSbo = C_::KG * 128;
    volatile int* abort_flag = &sm.abort_flag;
    const uint32_t a0 = smem_u32(stages), b0 = a0 + C_::kStages * C_::kStage;
    int s = 0;
    bool ok = mbar_wait(&sm.bres, ps.bres & 1u, abort_flag, err, 2);
    ++ps.bres;
    for (int seq = 0; ok; ++seq) {
        const uint32_t i = ps.tiles;
        const int b = (int)(i & 1u);
        if (i >= 2 && !mbar_wait(&sm.tempty[b], ((i >> 1) & 1u) ^ 1u, abort_flag, err, 4)) break;
        const uint32_t bit = 1u << s;
        if (!mbar_wait(&sm.full[s], (ps.stage_par & bit) ? 1u : 0u, abort_flag, err, 8)) break;
        ps.stage_par ^= bit;
        ++ps.tiles;
        tmem_fence_after();
        const int kind = *(volatile int*)&sm.slot[seq % kSlots].kind_set & 0xFF;
        if (kind <= kSlotPreview) {
            const uint32_t a_addr = a0 + (uint32_t)(s * C_::kStage);
#pragma unroll
            for (int kk = 0; kk < C_::KG / 2; ++kk)
                mma_f16<kN>(tmem + (uint32_t)(b * kN), smem_desc(a_addr + kk * 256, kSbo),
                            smem_desc(b0 + kk * 256, kSbo), kk > 0 ? 1u : 0u);
        }
        mma_commit(&sm.empty[s]);
        mma_commit(&sm.tfull[b]);
        if (++s == C_::kStages) s = 0;
        ok = kind != kSlotEnd;
    }
    state = ps;
}

// The preview's part of a scan warp: the best candidate of each of its 16 ranges, by the share of
// the range's energy its fit explains, over the slots up to kSlotEvaluate; handed to the fit
// warp, whose evaluation it waits for.  Returns the next slot, or -1 when given up.
__device__ __noinline__ int unit_preview(const ItemArgs& a, USmem& sm, uint32_t tcol0, int part,
                                         int m, PipeState& ps, int* err) {
    volatile int* abort_flag = &sm.abort_flag;
    const int lane = threadIdx.x & 31;
    float best[16];
    int where[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        best[q] = 0.0f;
        where[q] = -1;
    }
    int seq = 0;
    bool ok = true;
    for (;; ++seq) {
        const uint32_t i = ps.tiles;
        const int b = (int)(i & 1u);
        if (!mbar_wait(&sm.tfull[b], (i >> 1) & 1u, abort_flag, err, 16)) {
            ok = false;
            break;
        }
        ++ps.tiles;
        __syncwarp();
        tmem_fence_after();
        const Slot& sl = sm.slot[seq % kSlots];
        const bool last = (*(volatile const int*)&sl.kind_set & 0xFF) == kSlotEvaluate;
        if (!last) {
            const float amax_d = a.fp.a_max * kUnitScale * *(volatile const float*)&sl.contrast;
            const int pos = *(volatile const int*)&sl.tile * kM + m;
#pragma unroll
            for (int ch = 0; ch < 4; ++ch) {
                int32_t v[32];
                tmem_ld32(tcol0 + (uint32_t)(b * kN) + 32u * ch, v);
                tmem_wait(v);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    // With x = a_max sqrt(Ndd / Nrr), the explained share is rho^2, or past the
                    // largest contrast (rho > x) x (2 rho - x).
                    const float x = amax_d * sm.uinv[part * 16 + ch * 4 + q];
                    const float r = fmaxf(__int_as_float(unit_top(v, 8 * q)), 0.0f);
                    const float z = fminf(r, x);
                    const float share = z * (2.0f * r - z);
                    if (share > best[ch * 4 + q]) {
                        best[ch * 4 + q] = share;
                        where[ch * 4 + q] = pos;
                    }
                }
            }
        }
        tmem_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_n(&sm.tempty[b], 32u);
        if (last) break;
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        const uint32_t key = __float_as_uint(best[q]);
        const uint32_t high = __reduce_max_sync(0xffffffffu, key);
        const int pos = __reduce_max_sync(0xffffffffu, key == high ? where[q] : -1);
        if (lane == 0 && pos >= 0)
            atomicMax(&sm.ukey[part * 16 + q], (unsigned long long)high << 32 | (uint32_t)pos);
    }
    __threadfence_block();
    __syncwarp();
    if (lane == 0) atomicAdd(&sm.ukeyed[part], 1);
    const long long t0 = clock64();
    while (ok && *(volatile int*)&sm.ukeyed[part] <= kHalfWarps) {
        if (*abort_flag) break;
        if (clock64() - t0 > kWaitCycles) {
            *abort_flag = 1;
            atomicOr(err, 32);
            break;
        }
        __nanosleep(200);
    }
    __syncwarp();
    return ok ? seq + 1 : -1;
}

// Scan warp: its quadrant's 32 domains x its column half of every tile against the slot's
// thresholds.
template <int S>
__device__ __noinline__ void unit_scan_role(const ItemArgs& a, USmem& sm, const uint8_t* pix,
                                            uint32_t tmem, PipeState& ps, int* err) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int e = warp & 3;
    const int part = (warp - 2) >> 2;
    const int m = e * 32 + lane;
    const int w = part * kHalfWarps + e;  // this warp's ring: a half's are neighbours
    const int ndom = a.g.nrow_d * a.g.ncol_d;
    const uint32_t tcol0 = tmem + ((uint32_t)(e * 32) << 16) + (uint32_t)(part * (kN / 2));
    volatile int* abort_flag = &sm.abort_flag;
    uint32_t head = 0u, tail = 0u;
    int seq = 0;
    if (sm.upreview) seq = unit_preview(a, sm, tcol0, part, m, ps, err);
    uint32_t i = ps.tiles;
    for (; seq >= 0; ++seq) {
        const int b = (int)(i & 1u);
        if (!mbar_wait(&sm.tfull[b], (i >> 1) & 1u, abort_flag, err, 16)) break;
        ++i;
        __syncwarp();
        tmem_fence_after();
        const float4 sl = lds_f4(&sm.slot[seq % kSlots]);
        const float* thr = sm.set[__float_as_int(sl.y) >> 8];
        const bool last = (__float_as_int(sl.y) & 0xFF) == kSlotEnd;  // nothing was correlated
        const int pos = __float_as_int(sl.x) * kM + m;
        const uint32_t full = __float_as_uint(sl.w) >> (16 * part) & 0xFFFFu;
        const uint32_t tcol = tcol0 + (uint32_t)(b * kN);
        // Survivors are pushed right here: out of line, and so out of the instruction cache, the
        // same few instructions took 2,000 cycles a time.
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            int32_t v[64], top[8];
            tmem_ld64(tcol + 64u * hf, v);
            const int rb = part * 16 + hf * 8;  // the half's 8 ranges
            const float4 ta = lds_f4(thr + rb), tb = lds_f4(thr + rb + 4);
            const float th[8] = {ta.x, ta.y, ta.z, ta.w, tb.x, tb.y, tb.z, tb.w};
            tmem_wait64(v);
            // Thresholds are positive, so the float comparison is the integers'.  Lanes past the
            // last domain hold zeros.
            bool pass = false;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                top[q] = unit_top(v, 8 * q);
                pass |= top[q] >= __float_as_int(th[q]);
            }
            const uint32_t slow = full >> (8 * hf) & 0xFFu;
            if (last || !(__any_sync(0xffffffffu, pass) || slow)) continue;
            uint32_t mask = 0u;  // surviving ranges
#pragma unroll
            for (int q = 0; q < 8; ++q) mask |= (top[q] >= __float_as_int(th[q]) ? 1u : 0u) << q;
            if (slow) mask |= unit_look_full(a, sm, slow, rb, tcol + 64u * hf, pos, ndom);
            while (__any_sync(0xffffffffu, mask != 0u)) {
                if (!unit_push<S>(a, sm, pix, w, mask != 0u, unit_entry(pos, rb + __ffs(mask) - 1),
                                  head, tail, err))
                    break;
                mask &= mask - 1u;
            }
        }
        // The accumulator has been read completely: hand it back to the MMA warp.
        tmem_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_n(&sm.tempty[b], 32u);
        if (last) break;
    }
    ps.tiles = i;
    // Through with the tiles: help with what is left in this warp's ring.
    __syncwarp();
    for (;;) {
        const unsigned long long entry = unit_take<32>(sm, w);
        if (!__any_sync(0xffffffffu, entry != 0ull)) break;
        unit_fit<S>(a, sm, pix, entry, false, err);
    }
    __threadfence_block();
    __syncwarp();
    if (lane == 0) atomicAdd(&sm.udone[part], 1);
}

// Fit warp of a column half: the preview's candidates, then the rings' entries as they come.
template <int S>
__device__ __noinline__ void unit_fit_role(const ItemArgs& a, USmem& sm, const uint8_t* pix,
                                           int* err) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int part = warp - (2 + kScanWarps);
    volatile int* abort_flag = &sm.abort_flag;
    if (sm.upreview) {
        const long long t0 = clock64();
        bool ok = true;
        while (*(volatile int*)&sm.ukeyed[part] < kHalfWarps) {
            if (*abort_flag || clock64() - t0 > kWaitCycles) {
                ok = false;  // the scan warps' own wait reports it
                break;
            }
            __nanosleep(200);
        }
        if (__all_sync(0xffffffffu, ok)) {
            __threadfence_block();
            const int rl = part * 16 + (lane & 15);
            const unsigned long long key = *(volatile unsigned long long*)&sm.ukey[rl];
            unit_fit<S>(a, sm, pix, lane < 16 && key ? unit_entry((int)(uint32_t)key, rl) : 0ull,
                        true, err);
            __threadfence_block();
            __syncwarp();
            if (lane == 0) atomicAdd(&sm.ukeyed[part], 1);
            unit_share<S>(a, sm, part, err);
        }
    }
    for (uint32_t turn = 0;; ++turn) {
        // Read before the rings: once all scan warps are done, nothing is appended.
        const int done = __shfl_sync(0xffffffffu, *(volatile int*)&sm.udone[part], 0);
        __threadfence_block();
        const unsigned long long entry = unit_take<32 / kHalfWarps>(sm, part * kHalfWarps);
        if (!__any_sync(0xffffffffu, entry != 0ull)) {
            if (*(volatile uint32_t*)&sm.udirty >> (16 * part) & 0xFFFFu)
                unit_share<S>(a, sm, part, err);
            if (done == kHalfWarps || __any_sync(0xffffffffu, *abort_flag != 0)) break;
            __nanosleep(64);
            continue;
        }
        unit_fit<S>(a, sm, pix, entry, false, err);
        if ((turn & 15u) == 15u) unit_share<S>(a, sm, part, err);
    }
}

// One work item of the unit form: range tile `ntile` (32 ranges) against domain tiles
// of split `split` (unit_tile), 128 domains each in contrast order.  The contract is
// process_item's: every thread of the CTA (kUnitThreads) calls it, it begins and ends with a CTA
// barrier, and the pipelines' phases carry over in `ps`.
template <int S>
__device__ __forceinline__ void process_unit_item(const ItemArgs& a, int ntile, int split, USmem& sm,
                                                  unsigned char* stages, uint32_t tmem,
                                                  PipeState& ps, int* err,
                                                  unsigned long long& exact) {
    using C_ = UCfg<S>;
    constexpr int N = C_::N;
    constexpr int RT = kRangesPerTile;

    unsigned char* stA = stages;
    unsigned char* stB = stages + C_::kStages * C_::kStage;
    uint8_t* pix = stB + C_::kB;

    const LevelGeom& g = a.g;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int count = unit_tile_count(a, split);
    const int rbase = ntile * RT;

    if (warp == 0) {
        // A lane per range: its seed, or the range's shared champion when the splits before
        // this one found a better one.
        bool fresh = true;  // no split has shared a champion yet
        Champ& C = sm.ch[lane];
        const int r = rbase + lane < a.nranges ? (int)a.unit.ranges[rbase + lane] : a.nranges;
        sm.urange[lane] = (uint32_t)r;
        C.valid = r < a.nranges && load_seed(a.seeds + r).idx != UINT32_MAX;
        if (C.valid) {
            C.t0 = a.rs.t0[r];
            C.t2 = a.rs.t2[r];
            C.nrr = a.rs.nrr[r];
            C.rms0 = a.rs.rms0[r];
            const SeedOut sd = load_seed(a.seeds + r);
            C.rms = sd.rms;
            C.sum = sd.sum;
            C.idx = sd.idx;
            C.t1x4 = sd.t1x4;
            if (C.nrr == 0) {
                // A flat block: every candidate's contrast is 0 and its fit the same, so the
                // first in reference order wins; there is nothing to scan for.
                C.rms = C.rms0;
                C.sum = a.rs.sum0[r];
                C.idx = 0u;
                C.t1x4 = a.ds.s1x4[0] * (C.t0 / N);
            } else if (a.gch) {
                unsigned long long clo, chi;
                cas128(a.gch + 2 * (size_t)r, 0ull, 0ull, 0ull, 0ull, clo, chi);
                fresh = clo == ~0ull;
                const uint32_t gidx = (uint32_t)chi;
                const unsigned long long mlo = (unsigned long long)__double_as_longlong(C.rms);
                if (clo < mlo || (clo == mlo && gidx < C.idx)) {
                    const uint32_t dom = gidx >> 3;
                    C.rms = __longlong_as_double((long long)clo);
                    C.idx = gidx;
                    C.t1x4 = (int32_t)(uint32_t)(chi >> 32);
                    C.sum = fit_exact(N, a.ds.s1x4[dom], a.ds.s2x16[dom], C.t0, (int64_t)C.t1x4,
                                      C.t2, a.fp).sum;
                }
            }
        } else {
            C.rms = INFINITY;
            C.sum = 0.0;
            C.idx = UINT32_MAX;
            C.t1x4 = 0;
        }
        sm.ukey[lane] = 0ull;
        sm.uinv[lane] = C.valid && C.nrr > 0 ? rsqrtf((float)C.nrr) : 0.0f;
        sm.useq[lane] = 0u;
        unit_publish(sm, lane, a.fp, N);
        const uint32_t unseen = __ballot_sync(0xffffffffu, C.valid && C.nrr > 0 && fresh);
        if (lane < 2) {
            sm.udone[lane] = 0;
            sm.ukeyed[lane] = 0;
        }
        if (lane < kScanWarps) {
            sm.utail[lane] = 0u;
            sm.ulock[lane] = 0u;
        }
        if (lane == 0) {
            sm.udirty = 0u;
            sm.uexact = 0u;
            sm.upreview = unseen && count > 0;
        }
    } else {
        // The range tile's pixels, a thread per row of a block (into the still unused stages).
        for (int i = threadIdx.x - 32; i < RT * S; i += kUnitThreads - 32) {
            const int u = i % S;
            bool in = rbase + i / S < a.nranges;
            const uint8_t* from = a.unit.plane;
            if (in) {
                const uint32_t r = a.unit.ranges[rbase + i / S];
                const uint32_t row = a.unit.rows[r], col = a.unit.cols[r];
                in = row + (uint32_t)S <= (uint32_t)g.h && col + (uint32_t)S <= (uint32_t)g.w;
                from += in ? (size_t)(row + u) * g.w + col : 0;
            }
#pragma unroll
            for (int v = 0; v < S; ++v) stA[i * S + v] = in ? __ldg(from + v) : (uint8_t)0;
        }
    }
    __syncthreads();
    // Under each isometry, for the survivors' exact correlations: a thread per four samples.
    for (int i = threadIdx.x; i < RT * 8 * N / 4; i += kUnitThreads) {
        // iso_src_rt(k, u, v, S) = base + u * du + v * dv: rows run backwards for odd k, columns
        // for k = 2, 3, 4, 7, and u walks columns for k = 1, 2, 6, 7.
        const int e = i % (N / 4) * 4, k = i / (N / 4) % 8;
        const bool tr = (0xC6u >> k) & 1u, rev_i = k & 1, rev_j = (0x9Cu >> k) & 1u;
        const int step_i = rev_i ? -S : S, step_j = rev_j ? -1 : 1;
        const int du = tr ? step_j : step_i, dv = tr ? step_i : step_j;
        const unsigned char* from = stA + i / (8 * N / 4) * N + (rev_i ? (S - 1) * S : 0) +
                                    (rev_j ? S - 1 : 0) + e / S * du + e % S * dv;
        uint32_t w = 0u;
#pragma unroll
        for (int c = 0; c < 4; ++c) w |= (uint32_t)from[c * dv] << (8 * c);
        reinterpret_cast<uint32_t*>(pix)[i] = w;
    }
    fence_proxy_async();
    __syncthreads();
    if (warp == 0)
        unit_load_role<S>(a, sm, ntile, split, count, stages, ps, err);
    else if (warp == 1) {
        if (lane == 0) unit_mma_role<S>(sm, stages, tmem, ps, err);
        __syncwarp();
    } else if (warp < 2 + kScanWarps)
        unit_scan_role<S>(a, sm, pix, tmem, ps, err);
    else
        unit_fit_role<S>(a, sm, pix, err);

    // ---------------------------------------------------------------- item end
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    if (threadIdx.x == 0) exact += sm.uexact;
    const int r = threadIdx.x < RT ? (int)sm.urange[threadIdx.x] : a.nranges;
    finish_item(a, sm, ntile, split, r);
}

__device__ __forceinline__ uint32_t pack_f16(float lo, float hi) {
    return (uint32_t)__half_as_ushort(__float2half_rn(lo)) |
           (uint32_t)__half_as_ushort(__float2half_rn(hi)) << 16;
}

// A operand of one level, in contrast order: groups of 8 domains, each KG k-groups x (8 rows x
// 16 B); a tile is 16 groups.  One thread per (domain, k-group): 8 samples of the contracted
// window, centred and scaled to length 64; zero rows for flat domains and past the last one.
// windows: the samples themselves, 16 bits each, in the same order.
template <int S>
__global__ void __launch_bounds__(256) unit_a_kernel(const int32_t* __restrict__ D, LevelGeom g,
                                                     DomainStats ds,
                                                     const uint32_t* __restrict__ domains,
                                                     long long total, uint4* __restrict__ out,
                                                     uint4* __restrict__ windows) {
    using C_ = UCfg<S>;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    // t runs over the output: row group, k-group, row.
    const int r8 = (int)(t & 7);
    const long long rest = t >> 3;
    const int kg = (int)(rest % C_::KG);
    const long long pos = rest / C_::KG * 8 + r8;
    uint4 pk = make_uint4(0u, 0u, 0u, 0u), win = pk;
    if (pos < (long long)g.nrow_d * g.ncol_d) {
        const uint32_t dom = domains[pos];
        const int s1 = ds.s1x4[dom];
        const int64_t det = (int64_t)C_::N * ds.s2x16[dom] - (int64_t)s1 * s1;
        // |N D - s1|^2 = N det
        const float inv = det > 0 ? 64.0f * rsqrtf((float)C_::N * (float)det) : 0.0f;
        const int32_t* db = D + (size_t)(dom / (uint32_t)g.ncol_d) * g.step_c * g.dw +
                            (size_t)(dom % (uint32_t)g.ncol_d) * g.step_c;
        uint32_t h[4], d[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float x[2];
            d[i] = 0u;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int e = kg * 8 + 2 * i + c;
                const int v = __ldg(db + (size_t)(e / S) * g.dw + e % S);
                d[i] |= (uint32_t)v << (16 * c);
                x[c] = (float)(C_::N * v - s1) * inv;
            }
            h[i] = det > 0 ? pack_f16(x[0], x[1]) : 0u;
        }
        pk = make_uint4(h[0], h[1], h[2], h[3]);
        win = make_uint4(d[0], d[1], d[2], d[3]);
    }
    windows[t] = win;
    out[t] = pk;
}

// B operand of one level, in contrast order: per range a row group of its 8 isometries, KG k-groups
// x (8 rows x 16 B); a tile is 32 ranges.  One thread per (row, k-group); zero rows for flat blocks, blocks
// outside the plane and padding.
template <int S>
__global__ void __launch_bounds__(256) unit_b_kernel(const uint8_t* __restrict__ plane, int w, int h,
                                                     const uint32_t* __restrict__ rows,
                                                     const uint32_t* __restrict__ cols, int nranges,
                                                     RangeStats rs,
                                                     const uint32_t* __restrict__ ranges,
                                                     long long total,
                                                     uint4* __restrict__ out) {
    using C_ = UCfg<S>;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const int r8 = (int)(t & 7);  // the isometry: 8 rows a range
    const long long rest = t >> 3;
    const int kg = (int)(rest % C_::KG);
    const long long at = rest / C_::KG;
    uint4 pk = make_uint4(0u, 0u, 0u, 0u);
    const uint32_t r = at < nranges ? ranges[at] : 0u;
    if (at < nranges && rows[r] + (uint32_t)S <= (uint32_t)h && cols[r] + (uint32_t)S <= (uint32_t)w) {
        const int t0 = rs.t0[r];
        const int64_t nrr = rs.nrr[r];
        if (nrr > 0) {
            // |N r - t0|^2 = N Nrr
            const float inv = 64.0f * rsqrtf((float)C_::N * (float)nrr);
            const uint8_t* rb = plane + (size_t)rows[r] * w + cols[r];
            uint32_t hv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float x[2];
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int e = kg * 8 + 2 * i + c;
                    const int src = iso_src_rt(r8, e / S, e % S, S);
                    x[c] = (float)(C_::N * (int)rb[(size_t)(src / S) * w + src % S] - t0) * inv;
                }
                hv[i] = pack_f16(x[0], x[1]);
            }
            pk = make_uint4(hv[0], hv[1], hv[2], hv[3]);
        }
    }
    out[t] = pk;
}

// ---- contrast order: a counting sort of n keys into kBins classes of their float's leading bits
// (5 % wide in sqrt Ndd or sqrt Nrr); the order inside a class is the scheduler's, which no
// result depends on.  Bins of one warp-sized work item each would be finer than a tile needs.

constexpr int kBins = 1024;
constexpr int kOrderItems = 4096;  // keys a CTA counts and scatters

// Ndd or Nrr as a bin: exponent and three mantissa bits, 2^-16 at the bottom; 0 (flat) first.
__device__ __forceinline__ int contrast_bin(float x) {
    if (!(x > 0.0f) || x > 1e37f) return 0;  // flat domains carry +huge
    return min(max((int)(__float_as_uint(x) >> 20) - ((127 - 16) << 3), 1), kBins - 1);
}

template <bool RANGES>
__device__ __forceinline__ int order_bin(const DomainStats& ds, const RangeStats& rs, int i) {
    return contrast_bin(RANGES ? (float)rs.nrr[i] : ds.detf[i]);
}

template <bool RANGES>
__global__ void __launch_bounds__(1024) order_count_kernel(DomainStats ds, RangeStats rs, int n,
                                                           uint32_t* __restrict__ bins) {
    __shared__ uint32_t h[kBins];
    for (int i = threadIdx.x; i < kBins; i += blockDim.x) h[i] = 0u;
    __syncthreads();
    const int end = min(n, (int)(blockIdx.x + 1) * kOrderItems);
    for (int i = blockIdx.x * kOrderItems + threadIdx.x; i < end; i += blockDim.x)
        atomicAdd(&h[order_bin<RANGES>(ds, rs, i)], 1u);
    __syncthreads();
    for (int i = threadIdx.x; i < kBins; i += blockDim.x)
        if (h[i]) atomicAdd(&bins[i], h[i]);
}

// bins[0..kBins): the counts; bins[kBins..2 kBins): zero, the slots given out so far.
template <bool RANGES>
__global__ void __launch_bounds__(1024) order_scatter_kernel(DomainStats ds, RangeStats rs, int n,
                                                             uint32_t* __restrict__ bins,
                                                             uint32_t* __restrict__ order) {
    __shared__ uint32_t h[kBins], base[kBins], sums[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    h[t] = 0u;
    // Exclusive scan of the counts (one bin a thread).
    const uint32_t c = bins[t];
    uint32_t x = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sums[warp] = x;
    __syncthreads();
    uint32_t before = 0u;
    for (int k = 0; k < warp; ++k) before += sums[k];
    base[t] = before + x - c;
    const int begin = blockIdx.x * kOrderItems, end = min(n, begin + kOrderItems);
    for (int i = begin + t; i < end; i += blockDim.x)
        atomicAdd(&h[order_bin<RANGES>(ds, rs, i)], 1u);
    __syncthreads();
    // This CTA's run in each bin, then its keys into it.
    if (h[t]) base[t] += atomicAdd(&bins[kBins + t], h[t]);
    __syncthreads();
    for (int i = begin + t; i < end; i += blockDim.x)
        order[atomicAdd(&base[order_bin<RANGES>(ds, rs, i)], 1u)] = (uint32_t)i;
}

// The smallest and largest sqrt(Ndd) of each tile of 128 domains in order (0 for flat ones), a
// warp a tile.
__global__ void __launch_bounds__(256) tile_contrast_kernel(DomainStats ds,
                                                            const uint32_t* __restrict__ domains,
                                                            int ndom, int tiles,
                                                            float2* __restrict__ out) {
    const int tile = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (tile >= tiles) return;
    float lo = INFINITY, hi = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int pos = tile * kM + 32 * k + lane;
        if (pos >= ndom) break;
        const float s = ds.sdetf[domains[pos]], c = s > 1e18f ? 0.0f : s;
        lo = fminf(lo, c);
        hi = fmaxf(hi, c);
    }
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (lane == 0) out[tile] = make_float2(lo, hi);
}

__device__ __forceinline__ USmem& unit_record(unsigned char* raw) {
    return *reinterpret_cast<USmem*>(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
}

// CTA set-up: mbarriers, empty rings, TMEM (all 512 columns, held until unit_teardown).
__device__ __forceinline__ uint32_t unit_setup(USmem& sm) {
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kMaxStages; ++s) {
            mbar_init(&sm.full[s], 1);
            mbar_init(&sm.empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&sm.tfull[b], 1);
            mbar_init(&sm.tempty[b], 32 * kScanWarps);
        }
        mbar_init(&sm.bres, 1);
        sm.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = threadIdx.x; i < kScanWarps * kRing; i += kUnitThreads) sm.ring[0][i] = 0ull;
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&sm.tmem_base)),
                     "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    return sm.tmem_base;
}

__device__ __forceinline__ void unit_teardown(uint32_t tmem, unsigned long long exact,
                                              unsigned long long* exact_counter) {
    if (exact_counter && exact) atomicAdd(exact_counter, exact);
    tmem_fence_before();
    __syncthreads();
    if ((threadIdx.x >> 5) == 1) {
        tmem_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
    }
}

// Every unit level of a plane, or one level alone, in one persistent launch: the work items of
// corr_tc_all_kernel (level job, range tile, split), taken from a counter by one CTA per SM.
struct UnitLevels {
    ItemArgs args[kMaxLevelJobs];
    int size[kMaxLevelJobs];
    int tile_begin[kMaxLevelJobs];
    int tile_count[kMaxLevelJobs];
    int item_begin[kMaxLevelJobs + 1];
    int njobs;
};

__global__ void __launch_bounds__(kUnitThreads, 1)
    corr_unit_all_kernel(const __grid_constant__ UnitLevels L, int* __restrict__ work,
                         int* __restrict__ err, unsigned long long* __restrict__ exact_counter) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    USmem& sm = unit_record(smem_raw);
    unsigned char* stages = reinterpret_cast<unsigned char*>(&sm) + kUnitHead;
    const uint32_t tmem = unit_setup(sm);
    PipeState ps;
    unsigned long long exact = 0;
    const int nitems = L.item_begin[L.njobs];
    volatile int* abort_flag = &sm.abort_flag;
    if (threadIdx.x == 0) sm.item = atomicAdd(work, 1);
    __syncthreads();
    for (;;) {
        const int item = sm.item;
        if (item >= nitems || *abort_flag) break;
        int j = 0;
        while (j + 1 < L.njobs && item >= L.item_begin[j + 1]) ++j;
        const ItemArgs& a = L.args[j];
        // Split-major within a job: a range tile's later splits start after its earlier ones
        // have finished and begin from their champions (the shared records).
        // The range tiles of either end of the contrast order are the slow ones (flat blocks in
        // the full form, step edges with many survivors): both ends first.
        const int local = item - L.item_begin[j];
        const int turn = local % L.tile_count[j];
        const int ntile = L.tile_begin[j] + (turn & 1 ? turn / 2 : L.tile_count[j] - 1 - turn / 2);
        const int split = local / L.tile_count[j];
        if (L.size[j] == 4)
            process_unit_item<4>(a, ntile, split, sm, stages, tmem, ps, err, exact);
        else
            process_unit_item<8>(a, ntile, split, sm, stages, tmem, ps, err, exact);
        if (threadIdx.x == 0) sm.item = atomicAdd(work, 1);
        __syncthreads();
    }
    unit_teardown(tmem, exact, exact_counter);
}
