// sllg_tcr.cu -- mixed-precision Heun sLLG for clusters of 65 to 126 particles:
// the dipolar field on the tensor cores, D resident in tensor memory, the
// moments of a member tile in every CTA's shared memory.
//
// The split is sllg_tcc.cu's: a thread-block cluster of T = 2 or 3 CTAs takes NB
// members that share one cluster geometry, CTA r owns particles [42 r, 42 r + 42)
// and the 128 rows of D of their components.  At this size a D tile (both FP16
// splits) fills 384 of the 512 tensor-memory columns and is loaded once.
//
// The NB members are two groups, each with its own B tile, accumulators and
// field tile, and a stage of one group's integration runs while the other's
// moments are exchanged and multiplied.  Per group and stage:
//   1. integrating warps: wait for the group's MMAs (`acc`), move the
//      accumulators to the field tile, integrate the CTA's particles (one pair
//      of one member a thread, both particles in one packed instruction), and,
//      when the peers have multiplied what they were sent last (`free`), write
//      the FP16 split of the new moments into the CTA's K slab of its own B tile
//      (`slab`);
//   2. copy warp: one bulk copy of the slab into each peer's B tile, completed
//      on the peer's `peer` barrier;
//   3. the group's MMA warp: multiply the own slab as soon as it is written, the peers' when
//      they have arrived, and commit (`acc`).
//
// What bounds it: the chain of one group's stage (125 particles, 40 members:
// ~5900 clocks: 750 of increments and field tile, 1500 of integration and
// writing, 300 to start the copies, 700 for them, 2000 for the MMAs, 24 k-steps
// of 3 G columns), with the other group's beside it.  As one group it was 9100
// clocks in a row.  Bulk copies between the CTAs' shared memories need no fence
// at either end beyond the slab's own; plain remote stores took 1200 clocks to
// issue, 900 to fence and 1500 for two releasing arrivals, and a multicast of
// the slabs from global memory was slower than each CTA reading the whole tile.
// The MMAs are a warp a group: the issue takes 35 to 40 clocks an MMA beside the
// integrating warps.  us a step (512 members; 125 x 1638; 125 x 4096): 65
// particles 9.16 -> 4.57, 126 particles 10.1 -> 5.1, 10.6 -> 6.3, 24.8 -> 12.8.
// The step loop's code counts as in sllg_tc.cu: with the MMA chain written out
// for each slab as well, 147 CTAs took 7.1 us where 48 took 5.1 (32 members).
//
// Every wait is bounded.  The wait for a product has the plan's limit; one that
// runs out marks the CTA (sErr bit 0), waits on with the long limit, and the
// cluster stops together at its next check (every 64 steps, and once after the
// last).  A wait that exceeds the long limit marks it for good (bit 1): no wait
// polls long, nothing is sent or multiplied any more until that check.  When a
// CTA leaves the loop every copy sent to it has been waited for, and the MMA warps
// wait for everything they issued before tensor memory is released.
#include "common.cuh"
#include "llg32.cuh"
#include "llg64.cuh"
#include "tcc_common.cuh"

namespace magpy {

namespace {

constexpr int KMAX = 384;         // K of three CTAs
constexpr int FIELD_BLOCK = 64;   // steps of applied field computed at a time (two per lane)
constexpr int CHECK = 64;         // steps between the cluster's checks (FIELD_BLOCK relies on it)
static_assert(FIELD_BLOCK == CHECK, "a field block is published by the next check");

// Members of the two groups (multiples of 8, G0 >= G1).
template <int G0, int G1> struct Cfg {
    static constexpr int NB = G0 + G1;
    static constexpr int IT = PAIRS * G0;               // integrating threads
    static constexpr int IW = (IT + 31) / 32;           // integrating warps (>= EPI_WARPS)
    static constexpr int MMA = IW;                      // MMA-issuing warps, one per group
    static constexpr int COPY = IW + 2;                 // copying warp
    static constexpr int THREADS = 32 * (IW + 3);
    static constexpr bool LO_SMEM = NB <= 48;           // states' low words in shared memory
    // tensor memory: accumulators of the groups, then D
    static constexpr uint32_t ACC1 = tcc_acc_cols(G0), D = ACC1 + tcc_acc_cols(G1);
    static_assert(D + KMAX <= 512, "tensor memory");
    static_assert(IW >= EPI_WARPS, "epilogue warps");
    // shared memory (bytes)
    static constexpr size_t B1 = (size_t)KMAX * 2 * G0 * 2, F0 = B1 + (size_t)KMAX * 2 * G1 * 2;
    static constexpr size_t F1 = F0 + (size_t)RT * (G0 + 4) * 4;
    static constexpr size_t AW = F1 + (size_t)RT * (G1 + 4) * 4;
    static constexpr size_t XL = AW + (size_t)2 * 3 * IT * 16;
    static constexpr size_t PAR = XL + (LO_SMEM ? (size_t)2 * 3 * IT * 8 : 0);
    static constexpr size_t SR = PAR + (size_t)PAIRS * 32;
    static constexpr size_t SEED = SR + (size_t)PAIRS * 8;
    static constexpr size_t NOFF = SEED + (size_t)NB * 8;
    static constexpr size_t FLD = NOFF + (size_t)NB * 8;
    static constexpr size_t BAR = FLD + (size_t)2 * FIELD_BLOCK * 8;
    static constexpr size_t FLAG = BAR + 10 * 8;        // 9 mbarriers, the tensor-memory address
    static constexpr size_t TOTAL = FLAG + (size_t)4 * (NB + 1);
    static_assert(TOTAL <= 232448, "shared memory");
    // never two on an SM: each takes all of the tensor memory, and clusters that
    // waited for one another's would not end
    static_assert(TOTAL > 114 * 1024, "one CTA an SM");
};

// Named barrier of the integrating warps.
template <class C> __device__ inline void integ_sync()
{
    __syncwarp();
    asm volatile("bar.sync 1, %0;" ::"n"(32 * C::IW) : "memory");
}

// Element offset of (row, k) in a group's B tile (2 G rows: B_hi, then B_lo).
template <int G> __device__ inline uint32_t b_off(uint32_t row, uint32_t k)
{
    return (k >> 3) * (16 * G) + ((row >> 3) << 6) + ((row & 7) << 3) + (k & 7);
}

// One word of B_hi and of B_lo: x ~ hi + lo / 2048 for two K elements.
template <int G> __device__ inline void put_word(__half *bt, uint32_t o, float a, float b)
{
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn((a - f.x) * tc::SPLIT_SCALE, (b - f.y) * tc::SPLIT_SCALE);
    *reinterpret_cast<__half2 *>(bt + o) = h;
    *reinterpret_cast<__half2 *>(bt + o + 8 * G) = l;
}

// The moments of pair p (particles 2 p, 2 p + 1 of the CTA) of member j into the
// CTA's slab.  A warp's 8 members x 4 pairs write 32 different banks.  A particle
// past the cluster leaves its words zero.
template <int G>
__device__ inline void put_pair(__half *slab, int p, int j, bool two, const float2 m[3])
{
    put_word<G>(slab, b_off<G>(j, 6 * p), m[0].x, m[1].x);
    put_word<G>(slab, b_off<G>(j, 6 * p + 2), m[2].x, two ? m[0].y : 0.f);
    if (two) put_word<G>(slab, b_off<G>(j, 6 * p + 4), m[1].y, m[2].y);
}

// Injected increments of a pair (not inlined: rarely used).
__device__ __noinline__ PairNormals injected_pair(const double *w, bool two)
{
    PairNormals o;
    for (int c = 0; c < 6; c++) o.n[c] = c < 3 || two ? (float)w[c] : 0.f;
    return o;
}

// The applied field of steps FIELD_BLOCK b + 1 + lane + 32 i, at t or (second)
// t + dt.
__device__ __noinline__ void field_block(float2 *sF2, const MemberDev *md, int64_t b, int64_t K,
                                         int second)
{
    const int lane = threadIdx.x & 31;
    for (int i = lane; i < FIELD_BLOCK; i += 32) {
        const int64_t k = FIELD_BLOCK * b + 1 + i;
        if (k <= K)
            reinterpret_cast<float *>(sF2 + FIELD_BLOCK * (b & 1) + i)[second] =
                f64::heun_field_f32(md->shape, md->dt, md->happ, md->fapp, k, second);
    }
}

// A group's product with CTA sl's slab of its B tile.
template <int G>
__device__ inline void mma_slab(uint32_t acc, uint32_t d, int K, uint32_t B, int sl, bool first)
{
    constexpr uint32_t b_lbo = Idesc<G>::B_LBO;
    const uint64_t bd = tc::smem_desc(B + (uint32_t)(RT / 8) * b_lbo * sl, b_lbo, 128);
    const uint32_t hi = d + (uint32_t)(RT / 2) * sl, lo = hi + (uint32_t)(K / 2);
#pragma unroll
    for (int s = 0; s < RT / 16; s++) {
        const uint64_t b = bd + (uint64_t)((2 * b_lbo * s) >> 4);
        tc::mma_f16_ta_warp(acc, hi + 8u * s, b, Idesc<G>::MAIN, first && s == 0 ? 0u : 1u);
        tc::mma_f16_ta_warp(acc + G, lo + 8u * s, b, Idesc<G>::CORR, 1u);
    }
}

// Wait for a phase; false (and marked) if `limit` polls are not enough or the
// CTA is marked for good.
__device__ inline bool wait_phase(uint64_t *bar, uint32_t parity, int *sErr, uint32_t limit,
                                  int mark)
{
    for (uint32_t i = 0; i < limit; i++) {
        if (tc::mbar_try_wait(bar, parity)) return true;
        if ((i & 255u) == 255u && (*(volatile int *)sErr & 2)) break;
    }
    atomicOr(sErr, mark);
    return false;
}

template <int G0, int G1>
__global__ void __launch_bounds__(Cfg<G0, G1>::THREADS, 1)
    sllg_tcr_kernel(DevPlan p, const __half *dglob)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    using C = Cfg<G0, G1>;
    const int n = p.n, T = (n + PPC - 1) / PPC, KD = RT * T;
    const int r = (int)tc::cluster_ctarank();
    const int64_t base = (int64_t)(blockIdx.x / T) * C::NB;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const MemberDev *m0d = p.members;  // members of a launch share their parameters
    const int64_t P = p.P;

    float4 *sPar = (float4 *)(sm + C::PAR);  // per pair: (ax, ax', ay, ay'), (az, az', K, K')
    float2 *sSr = (float2 *)(sm + C::SR);    // per pair: sqrt(dt) x noise scale
    uint64_t *sSeed = (uint64_t *)(sm + C::SEED);
    int64_t *sNoff = (int64_t *)(sm + C::NOFF);
    // applied field of step k, (h(k dt), h(k dt + dt)), in slot ((k - 1) / 64) % 2
    float2 *sF2 = (float2 *)(sm + C::FLD);
    uint64_t *bars = (uint64_t *)(sm + C::BAR);
    uint64_t *slab_b = bars, *peer_b = bars + 2, *free_b = bars + 4, *acc_b = bars + 6;
    uint64_t *drain_b = bars + 8;
    uint32_t *slot = (uint32_t *)(bars + 9);
    int *sFlag = (int *)(sm + C::FLAG);      // [NB] member status bits
    int *sErr = sFlag + C::NB;               // this CTA's watchdog word

    // padding rows, absent particles and members of the B tiles stay zero
    for (int i = threadIdx.x; i < (int)(C::F0 / 16); i += C::THREADS)
        reinterpret_cast<uint4 *>(sm)[i] = make_uint4(0, 0, 0, 0);
    for (int i = threadIdx.x; i < PAIRS; i += C::THREADS) {
        float a[2][4], s[2];
        for (int k = 0; k < 2; k++) {
            const int q = PPC * r + 2 * i + k;
            const int64_t gq = m0d->pbase + (q < n ? q : 0);
            for (int c = 0; c < 3; c++) a[k][c] = (float)p.axes[c * P + gq];
            a[k][3] = (float)p.k_red[gq];
            s[k] = (float)m0d->sqrt_dt * (float)p.sr[gq];
        }
        sPar[2 * i] = make_float4(a[0][0], a[1][0], a[0][1], a[1][1]);
        sPar[2 * i + 1] = make_float4(a[0][2], a[1][2], a[0][3], a[1][3]);
        sSr[i] = make_float2(s[0], s[1]);
    }
    for (int i = threadIdx.x; i < C::NB; i += C::THREADS) {
        const bool ok = base + i < p.E;
        sFlag[i] = 0;
        sSeed[i] = ok ? p.members[base + i].seed : 0;
        sNoff[i] = ok ? p.members[base + i].noise_off : 0;
    }
    if (threadIdx.x == 0) {
        *sErr = 0;
        for (int g = 0; g < 2; g++) {
            tc::mbar_init(&slab_b[g], C::IW);
            tc::mbar_init(&peer_b[g], 1);  // and the peers' bytes
            tc::mbar_init(&free_b[g], (uint32_t)(T - 1));
            tc::mbar_init(&acc_b[g], 1);
        }
        tc::mbar_init(drain_b, 2);
    }
    if (threadIdx.x < 32) tc::tmem_alloc(slot, 512);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *slot;
    tcc_load_d_tmem(tmem + C::D, KD, dglob + (size_t)r * RT * KD * 2, warp, lane);

    const float dt = (float)m0d->dt, alpha = (float)m0d->alpha;
    const bool renorm = m0d->renorm != 0;
    const int64_t S = p.S;
    const int64_t *sched = p.sched + m0d->sched_off;
    const int64_t K = S > 1 ? sched[S - 1] : 0;
    const int64_t per_step = 3 * (int64_t)n;
    const int64_t noise_steps = p.noise ? m0d->noise_len / per_step : K;

    // thread t integrates pair pp of member j of both groups: eight consecutive
    // threads serve eight members, the next eight the next pair (a warp's reads
    // of the field tile, rows 6 (G + 4) floats apart, hit 32 different banks)
    const bool integ = (int)threadIdx.x < C::IT;
    const int j = 8 * ((int)threadIdx.x / (8 * PAIRS)) + ((int)threadIdx.x & 7);
    const int pp = ((int)threadIdx.x >> 3) % PAIRS;
    const int q0 = PPC * r + 2 * pp;
    const bool live = integ && q0 < n, two = q0 + 1 < n;
    const auto member = [&](int g) { return base + (g ? G0 : 0) + j; };
    const auto valid = [&](int g) { return live && j < (g ? G1 : G0) && member(g) < p.E; };
    const auto slab_of = [&](int g) {
        return (__half *)(sm + (g ? C::B1 : 0)) + (size_t)r * RT * 2 * (g ? G1 : G0);
    };
    // state: float-float, components of both particles side by side; the high
    // words xh in registers, the low words (used once per step) in shared memory
    float2 xh[2][3], xlr[C::LO_SMEM ? 1 : 2][3];
    const auto xl = [&](int g, int c) -> float2 & {
        if constexpr (C::LO_SMEM)
            return reinterpret_cast<float2 *>(sm + C::XL)[(3 * g + c) * C::IT + threadIdx.x];
        else
            return xlr[C::LO_SMEM ? 0 : g][c];
    };
    const auto record = [&](int64_t smp, int g) {
        const int64_t o = smp * P + member(g) * n + q0;
        const double sc = p.out_scale[member(g)];
        const float2 l0 = xl(g, 0), l1 = xl(g, 1), l2 = xl(g, 2);
        tcc_write_sample(p.mx, p.my, p.mz, o, sc, xh[g][0].x, l0.x, xh[g][1].x, l1.x, xh[g][2].x,
                         l2.x);
        if (two)
            tcc_write_sample(p.mx, p.my, p.mz, o + 1, sc, xh[g][0].y, l0.y, xh[g][1].y, l1.y,
                             xh[g][2].y, l2.y);
    };
#pragma unroll
    for (int g = 0; g < 2; g++) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            float h[2] = {0.f, 0.f}, l[2] = {0.f, 0.f};
            for (int k = 0; k < 2; k++)
                if (valid(g) && (k == 0 || two)) {
                    const double v = p.m0[c * P + member(g) * n + q0 + k];
                    h[k] = (float)v;
                    l[k] = (float)(v - (double)h[k]);
                }
            xh[g][c] = make_float2(h[0], h[1]);
            if (integ) xl(g, c) = make_float2(l[0], l[1]);
        }
        if (valid(g)) {
            if (g == 0) put_pair<G0>(slab_of(0), pp, j, two, xh[0]);
            else put_pair<G1>(slab_of(1), pp, j, two, xh[1]);
            if (p.mx) record(0, g);  // the initial state (lib/simulation.cpp:212-219)
        }
    }
    if (warp == C::COPY || warp == C::MMA + 1) field_block(sF2, m0d, 0, K, warp == C::COPY);
    tc::fence_proxy_async();
    tc::fence_before_sync();
    // every CTA's tiles are zeroed and its barriers initialised
    tc::cluster_sync();
    __syncthreads();
    tc::fence_after_sync();

    int32_t status = ST_OK;
    int64_t s_next = 1, next_sample = S > 1 ? sched[1] : -1;
    int64_t step;
    bool stop = false;
    if (warp < C::IW && lane == 0 && K > 0)
        for (int g = 0; g < 2; g++) tc::mbar_arrive(&slab_b[g]);
    // a wait with the long limit
    const auto wait = [&](uint64_t *bar, uint32_t parity) {
        return wait_phase(bar, parity, sErr, DRAIN_LIMIT, 3);
    };
    for (step = 1; step <= K; step++) {
        // every thread of the cluster comes here with the same step: whether to
        // go on is decided together
        if ((step - 1) % CHECK == 0 && cluster_check(sErr, T, (step - 1) / CHECK)) {
            status |= ST_WATCHDOG;
            stop = true;
        }
        if (!stop && step > noise_steps) { status |= ST_NOISE_EXHAUSTED; stop = true; }
        if (stop) break;
        // every barrier below completes a phase per stage, two a step: its parity
        // is the stage
        // the next block of the applied field: its slot was last read before this
        // check, and the next check publishes it
        if (warp > C::MMA && (step - 1) % CHECK == 0)
            field_block(sF2, m0d, (step - 1) / FIELD_BLOCK + 1, K, warp == C::COPY);
        if (warp == C::COPY) {
            if (lane == 0)
#pragma unroll
                for (int ph = 0; ph < 4; ph++) {
                    const int g = ph & 1;
                    if (!wait(&slab_b[g], ph >> 1)) continue;
                    const uint32_t sl = tc::smem_addr(slab_of(g)), bar = tc::smem_addr(&peer_b[g]);
                    for (int k = 1; k < T; k++) {
                        const uint32_t rr = (uint32_t)(r + k < T ? r + k : r + k - T);
                        tc::bulk_s2s(tc::mapa(sl, rr), slab_of(g), RT * 4 * (g ? G1 : G0),
                                     tc::mapa(bar, rr));
                    }
                }
            __syncwarp();
            continue;
        }
        if (warp >= C::MMA) {  // warp MMA + g: group g
            const int g = warp - C::MMA;
            const uint32_t acc = tmem + (g ? C::ACC1 : 0u);
            const uint32_t B = tc::smem_addr(sm + (g ? C::B1 : 0));
#pragma unroll 1
            for (int st = 0; st < 2; st++) {
                // (the whole warp takes each decision)
                if (!__all_sync(0xffffffffu, wait(&slab_b[g], st))) continue;
                if (lane == 0)
                    tc::mbar_arrive_expect_tx(&peer_b[g],
                                              (uint32_t)((T - 1) * RT * 4 * (g ? G1 : G0)));
                __syncwarp();
                tc::fence_after_sync();
                bool in = true;
#pragma unroll 1
                for (int k = 0; k < T; k++) {
                    if (k == 1) {
                        in = __all_sync(0xffffffffu, wait(&peer_b[g], st));
                        if (!in) break;
                        tc::fence_after_sync();
                    }
                    const int sl = r + k < T ? r + k : r + k - T;
                    if (G0 == G1 || g == 0) mma_slab<G0>(acc, tmem + C::D, KD, B, sl, k == 0);
                    else mma_slab<G1>(acc, tmem + C::D, KD, B, sl, k == 0);
                }
                if (in) tc::mma_commit_warp(&acc_b[g]);
            }
            continue;
        }
        // integrating warps
        while (next_sample == step) {  // the state after step - 1 steps
            if (p.mx)
#pragma unroll
                for (int g = 0; g < 2; g++)
                    if (valid(g)) record(s_next, g);
            s_next++;
            next_sample = s_next < S ? sched[s_next] : -1;
        }
        const float2 hf = sF2[(step - 1) % (2 * FIELD_BLOCK)];
#pragma unroll
        for (int st = 0; st < 2; st++)
#pragma unroll
            for (int g = 0; g < 2; g++) {
                constexpr int FS0 = G0 + 4, FS1 = G1 + 4;
                float *F = (float *)(sm + (g ? C::F1 : C::F0));
                if (warp < EPI_WARPS) {
                    const bool ok = __all_sync(
                        0xffffffffu, wait_phase(&acc_b[g], st, sErr, p.wait_limit, 1) ||
                                         wait(&acc_b[g], st));
                    tc::fence_after_sync();
                    // the tile has been read: peers may write their parts again
                    if (ok && threadIdx.x == 0)
                        for (int k = 1; k < T; k++)
                            tc::mbar_arrive_remote_relaxed(
                                tc::mapa(tc::smem_addr(&free_b[g]),
                                         (uint32_t)(r + k < T ? r + k : r + k - T)));
                    if (ok) {
                        if (g == 0) tcc_field_tile<G0>(tmem, F, warp, lane);
                        else tcc_field_tile<G1>(tmem + C::ACC1, F, warp, lane);
                    }
                    tc::fence_before_sync();
                }
                // the increments need no field
                PairNormals wn;
                if (st == 0 && valid(g)) {
                    const int sl = (g ? G0 : 0) + j;
                    if (!p.noise)
                        wn = wiener_pair(sSeed[sl], (uint64_t)step,
                                         (uint32_t)(PAIRS * r + pp));
                    else
                        wn = injected_pair(p.noise + sNoff[sl] + (step - 1) * per_step + 3 * q0,
                                           two);
                }
                integ_sync<C>();
                float2 out[3];
                if (valid(g)) {
                    const int FS = g ? FS1 : FS0;
                    const float *ha = F + 6 * pp * FS + j;
                    const float *hb = ha + 3 * FS;
                    const float hz = st == 0 ? hf.x : hf.y;
                    const float4 pxy = sPar[2 * pp], pzk = sPar[2 * pp + 1];
                    const float2 ax = make_float2(pxy.x, pxy.y), ay = make_float2(pxy.z, pxy.w);
                    const float2 az = make_float2(pzk.x, pzk.y), ak = make_float2(pzk.z, pzk.w);
                    const float2 ssr = sSr[pp];
                    const float2 hd[3] = {make_float2(ha[0], hb[0]), make_float2(ha[FS], hb[FS]),
                                          make_float2(ha[2 * FS], hb[2 * FS])};
                    float4 *aw = (float4 *)(sm + C::AW) + 3 * g * C::IT + threadIdx.x;
                    float2 w[3], A[3], m[3];
                    if (st == 0) {
                        for (int c = 0; c < 3; c++) {
                            w[c] = make_float2(wn.n[c], wn.n[3 + c]);
                            m[c] = xh[g][c];
                        }
                    } else {
                        const float4 a01 = aw[0], a2w0 = aw[C::IT], w12 = aw[2 * C::IT];
                        A[0] = make_float2(a01.x, a01.y);
                        A[1] = make_float2(a01.z, a01.w);
                        A[2] = make_float2(a2w0.x, a2w0.y);
                        w[0] = make_float2(a2w0.z, a2w0.w);
                        w[1] = make_float2(w12.x, w12.y);
                        w[2] = make_float2(w12.z, w12.w);
                        // the predictor x~ = x + dt a + sqrt(dt) B w
                        for (int c = 0; c < 3; c++) m[c] = fma2(f2(2.f), A[c], xh[g][c]);
                    }
                    const float2 dot = mul2(fma2(m[2], az, fma2(m[1], ay, mul2(m[0], ax))), ak);
                    const float2 v[3] = {
                        fma2(f2(dt), fma2(dot, ax, hd[0]), mul2(ssr, w[0])),
                        fma2(f2(dt), fma2(dot, ay, hd[1]), mul2(ssr, w[1])),
                        fma2(f2(dt), fma2(dot, az, add2(hd[2], f2(hz))), mul2(ssr, w[2]))};
                    float2 inc[3];
                    llg_F2(inc, m, f2(alpha), v);
                    if (st == 0) {
                        for (int c = 0; c < 3; c++) {
                            A[c] = mul2(f2(0.5f), inc[c]);
                            out[c] = add2(m[c], inc[c]);
                        }
                        aw[0] = make_float4(A[0].x, A[0].y, A[1].x, A[1].y);
                        aw[C::IT] = make_float4(A[2].x, A[2].y, w[0].x, w[0].y);
                        aw[2 * C::IT] = make_float4(w[1].x, w[1].y, w[2].x, w[2].y);
                    } else {
                        float2 lo[3];
                        for (int c = 0; c < 3; c++) {
                            lo[c] = xl(g, c);
                            dd_add_ts2(xh[g][c], lo[c], fma2(f2(0.5f), inc[c], A[c]));
                        }
                        if (renorm) {
                            const float2 n2 =
                                fma2(xh[g][2], xh[g][2],
                                     fma2(xh[g][1], xh[g][1], mul2(xh[g][0], xh[g][0])));
                            const float2 inv =
                                make_float2(1.0f / sqrtf(n2.x), 1.0f / sqrtf(n2.y));
                            for (int c = 0; c < 3; c++) {
                                xh[g][c] = mul2(xh[g][c], inv);
                                lo[c] = mul2(lo[c], inv);
                            }
                        }
                        for (int c = 0; c < 3; c++) {
                            if (!two) xh[g][c].y = lo[c].y = 0.f;
                            xl(g, c) = lo[c];
                            out[c] = xh[g][c];
                        }
                    }
                }
                // the copies of the last slab have been read where they went
                wait(&free_b[g], st);
                if (valid(g)) {
                    if (g == 0) put_pair<G0>(slab_of(0), pp, j, two, out);
                    else put_pair<G1>(slab_of(1), pp, j, two, out);
                }
                // the last step's moments are not multiplied
                if (st == 0 || step < K) {
                    tc::fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(&slab_b[g]);
                }
            }
    }
    // the loop leaves `step` one past the last completed step
    step -= 1;
    __syncwarp();
    if (warp == C::MMA || warp == C::MMA + 1) {
        // everything issued has completed before the tensor memory is released
        tc::mma_commit_warp(drain_b);
        tc::mbar_wait_bounded(drain_b, 0, DRAIN_LIMIT);
    }
    if (cluster_last_check(sErr, T)) status |= ST_WATCHDOG;
#pragma unroll
    for (int g = 0; g < 2; g++)
        if (valid(g)) {
            if (p.mx)  // samples a stopped member never reached
                for (int64_t s = s_next; s < S; s++)
                    for (int k = 0; k < (two ? 2 : 1); k++) {
                        const int64_t o = s * P + member(g) * n + q0 + k;
                        p.mx[o] = NAN; p.my[o] = NAN; p.mz[o] = NAN;
                    }
            bool bad = false;
            for (int c = 0; c < 3; c++) bad |= !(isfinite(xh[g][c].x) && isfinite(xh[g][c].y));
            if (bad) atomicOr(&sFlag[(g ? G0 : 0) + j], ST_NONFINITE);
        }
    tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x < 32) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, 512);
    }
    // member status: the OR over the cluster's CTAs, written by CTA 0
    tc::cluster_sync();
    if (r == 0 && threadIdx.x < C::NB && base + threadIdx.x < p.E) {
        const int64_t em = base + threadIdx.x;
        int32_t st = status;
        const uint32_t fl = tc::smem_addr(&sFlag[threadIdx.x]);
        for (int rr = 0; rr < T; rr++) st |= tc::ld_cluster_s32(tc::mapa(fl, (uint32_t)rr));
        if (p.status) p.status[em] = st;
        if (p.steps) p.steps[em] = step;
    }
    tc::cluster_sync();  // no CTA leaves while another may use its shared memory
}

template <int G0, int G1>
cudaError_t launch_form(const DevPlan &p, const __half *d, cudaStream_t stream)
{
    using C = Cfg<G0, G1>;
    return tcc_launch(sllg_tcr_kernel<G0, G1>, (p.n + PPC - 1) / PPC, C::TOTAL, C::THREADS,
                      (p.E + C::NB - 1) / C::NB, stream, p, d);
}

}  // namespace

// Raises the forms' shared-memory limits (a plan's creation calls it).
cudaError_t tcr_init()
{
    cudaError_t err = tcc_prepare(sllg_tcr_kernel<16, 16>, 3, Cfg<16, 16>::TOTAL);
    if (err == cudaSuccess) err = tcc_prepare(sllg_tcr_kernel<24, 16>, 3, Cfg<24, 16>::TOTAL);
    if (err == cudaSuccess) err = tcc_prepare(sllg_tcr_kernel<24, 24>, 3, Cfg<24, 24>::TOTAL);
    if (err == cudaSuccess) err = tcc_prepare(sllg_tcr_kernel<32, 32>, 3, Cfg<32, 32>::TOTAL);
    return err;
}

cudaError_t launch_tcr(const DevPlan &p, const __half *d, int nb, cudaStream_t stream)
{
    switch (nb) {
    case 32: return launch_form<16, 16>(p, d, stream);
    case 40: return launch_form<24, 16>(p, d, stream);
    case 48: return launch_form<24, 24>(p, d, stream);
    default: return launch_form<32, 32>(p, d, stream);
    }
}

}  // namespace magpy
