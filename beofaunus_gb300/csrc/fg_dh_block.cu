// Debye-Hueckel + Lennard-Jones sweeps in blocks of trials (all-pairs systems).
//
// Included by fg_api.cu after fg_kernels.cu (one translation unit).
//
// The Metropolis chain is sequential: trial t+1 sees the configuration that
// trial t left. For a pair potential that dependence is small and exact to
// undo: if trial a (particle i_a, old o_a -> new n_a) was accepted, the energy
// change of a later trial m (particle i_m != i_a, o_m -> n_m) differs from its
// value in the configuration before trial a by exactly
//     c(a, m) = [u(n_m, n_a) - u(o_m, n_a)] - [u(n_m, o_a) - u(o_m, o_a)].
// So a block of up to 32 trials is evaluated in parallel against the
// configuration at the start of the block (each warp sums two trials over all
// particles), the 32 x 32 corrections c(a, m) are evaluated in parallel, and
// one warp then walks the block in order: lane m keeps dU_m = base_m +
// sum of c(a, m) over accepted a < m, decides, and on acceptance every later
// lane adds its correction. A trial whose particle was already moved by an
// accepted trial of the block ends the block there; it is evaluated again at
// the start of the next one. Decisions, dU values and the acceptance sequence
// are those of the one-trial-at-a-time chain (Movebase::move, move.h:515-555).
//
// A system spreads one block over a thread-block cluster: CTA r sums the
// particles of slice r and stores its per-trial partial sums into every CTA's
// shared memory, and after one cluster barrier per block every CTA resolves
// the block identically (same numbers, same order) and applies the accepted
// moves to the shared master coordinates and its own slice.
//
// What bounds it: the base sums on large slices (issue rate, about 75 slots and
// 28 cycles of the SFU per 32 partners), a fixed part of about 0.3 us per
// trial (near pairs, corrections, barrier, resolution) on small ones. Base sums
// of 2001 particles on one CTA: 210 -> 120 cycles per warp of partners and SM
// quarter; per trial 2.24 -> 1.29 us on one CTA, 0.62 -> 0.38 us on 16.
namespace fg {

constexpr int kBlkTrials = 32;
constexpr int kBlkThreads = 512;

struct __align__(16) BlkView {   // one trial
    int hx, hy, hz;        // old high words
    float dx, dy, dz, d2;  // step (words), its square
    float wx, wy, wz;      // |d_o| beyond which the image may change
    float qc;              // q lB / (L / 2^32)
    int small;             // kappa |delta| < 1/4: expm1 by its Taylor series
    int far;               // a step longer than 4 sigma: blk_far_long
    int ti, i;             // type, particle
};
struct BlkConst {          // one system
    float kw, kl, near2, s2;   // kappa and -kappa log2(e) per word, 4 sigma^2 and sigma^2 in words^2 (uniform tables)
    float w2;                  // words^2 per Angstrom^2
    float step2;               // 16 sigma^2 of the smallest pair, words^2
};

struct BlkSmem {
    int4 *spos;      // slice: high words, .w = charge bits
    short4 *sext;    // slice: 16 more bits
    uint8_t *stype;  // slice: types
    Move *mv;        // [32] trials of the block
    BlkView *view;   // [32] what the base sums need of them
    float2 *thr;     // [32] threshold (df, already times kT)
    uint32_t *col;   // [32] earlier trials of the block on the same particle
    float2 *corr;    // [32][32] c(a, m) as df (cluster: two, by block parity)
    float2 *part;    // [32] this CTA's partial sums
    float2 *xpart;   // [2][C][32] every CTA's partial sums (by block parity)
    int *info;       // [4]: trials resolved in the block, decisions bitmask, queue length, some sum in fix[1], [2]
    uint32_t *queue; // near pairs (trial << 24 | slice index), evaluated densely after the sums
    unsigned long long *fix;  // [3][32] near-pair sums per trial (blk_fix_add)
};

constexpr int kBlkQueue = 1344;
// A correction beyond this (kT) belongs to a trial on top of where an accepted
// particle was: its dU would be the small rest of two large numbers. It is kept
// as a NaN, the block ends before a trial that took it, and the next block
// evaluates the trial (its first) as the configuration is.
constexpr float kBlkLargeCorr = 1.0e4f;

__host__ __device__ inline size_t blk_align(size_t x) { return (x + 15) & ~(size_t)15; }

__host__ __device__ inline size_t blk_smem_bytes(int ns, bool slice, int C) {
    size_t o = 0;
    if (slice) o += blk_align((size_t)ns * 16) + blk_align((size_t)ns * 8) + blk_align((size_t)ns);
    o += blk_align(sizeof(Move) * kBlkTrials) + blk_align(sizeof(BlkView) * kBlkTrials);
    o += blk_align(8 * kBlkTrials) + blk_align(4 * kBlkTrials);
    o += blk_align(8 * kBlkTrials * kBlkTrials) * (C > 1 ? 2 : 1) + blk_align(8 * kBlkTrials) + 16;
    o += blk_align((size_t)8 * 2 * C * kBlkTrials);
    o += blk_align(4 * kBlkQueue) + blk_align(3 * 8 * kBlkTrials);
    return o;
}

__device__ inline BlkSmem blk_carve(unsigned char *b, int ns, bool slice, int C) {
    BlkSmem s;
    size_t o = 0;
    if (slice) {
        s.spos = (int4 *)(b + o); o += blk_align((size_t)ns * 16);
        s.sext = (short4 *)(b + o); o += blk_align((size_t)ns * 8);
        s.stype = (uint8_t *)(b + o); o += blk_align((size_t)ns);
    } else {
        s.spos = nullptr; s.sext = nullptr; s.stype = nullptr;
    }
    s.mv = (Move *)(b + o); o += blk_align(sizeof(Move) * kBlkTrials);
    s.view = (BlkView *)(b + o); o += blk_align(sizeof(BlkView) * kBlkTrials);
    s.thr = (float2 *)(b + o); o += blk_align(8 * kBlkTrials);
    s.col = (uint32_t *)(b + o); o += blk_align(4 * kBlkTrials);
    s.corr = (float2 *)(b + o); o += blk_align(8 * kBlkTrials * kBlkTrials) * (C > 1 ? 2 : 1);
    s.part = (float2 *)(b + o); o += blk_align(8 * kBlkTrials);
    s.xpart = (float2 *)(b + o); o += blk_align((size_t)8 * 2 * C * kBlkTrials);
    s.info = (int *)(b + o); o += 16;
    s.queue = (uint32_t *)(b + o); o += blk_align(4 * kBlkQueue);
    s.fix = (unsigned long long *)(b + o);
    return s;
}

// Order-independent sums of near pairs in fixed point, by size so that no sum
// wraps: units of 2^-40 kT below 2^16 kT, 2^-24 below 2^32, 2^-4 for the overlaps
// beyond, held to 2^53 kT each (128 pairs of the largest size fit 63 bits).
__device__ __forceinline__ unsigned long long blk_to_fix(df v, float scale) {
    return (unsigned long long)(__float2ll_rn(v.hi * scale) + __float2ll_rn(v.lo * scale));
}
__device__ __noinline__ void blk_fix_add_large(unsigned long long *fix, df v) {
    const float x = fabsf(v.hi);
    if (x < 4294967296.0f) {
        atomicAdd(fix + kBlkTrials, blk_to_fix(v, 16777216.0f));
        return;
    }
    // (a NaN, of particles on top of each other, counts as the largest overlap)
    if (!(x < 9007199254740992.0f)) v = df{v.hi < 0.0f ? -9007199254740992.0f : 9007199254740992.0f, 0.0f};
    atomicAdd(fix + 2 * kBlkTrials, blk_to_fix(v, 16.0f));
}
__device__ __forceinline__ void blk_fix_add(const BlkSmem &s, int m, df v) {
    if (fabsf(v.hi) < 65536.0f) {
        atomicAdd(&s.fix[m], blk_to_fix(v, 1099511627776.0f));
    } else {
        s.info[3] = 1;
        blk_fix_add_large(&s.fix[m], v);
    }
}
__device__ __forceinline__ df blk_from_fix(unsigned long long u, float scale) {
    const long long v = (long long)u;
    const float h = i64_to_float(v);
    const long long r = v - __float2ll_rn(h);
    return fast_two_sum(h * scale, i64_to_float(r) * scale);
}
__device__ __forceinline__ df blk_fix_sum(const BlkSmem &s, int m) {
    df v = blk_from_fix(s.fix[m], 9.094947017729282e-13f);
    if (s.info[3]) {
        v = df_add(v, blk_from_fix(s.fix[kBlkTrials + m], 5.9604644775390625e-8f));
        v = df_add(v, blk_from_fix(s.fix[2 * kBlkTrials + m], 0.0625f));
    }
    return v;
}

__device__ __forceinline__ float blk_rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float blk_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The bulk of the all-pairs sum: partners beyond 2 sigma of both positions of a
// trial. Distances are kept in units of the high word (L / 2^32; the box is
// cubic), so that only the old position's differences are converted:
// r_n^2 - r_o^2 = |delta|^2 - 2 delta.d_o for the step delta, and per axis
// e (2 d_o + e) with e = -delta - 2^32 rint((d_o - delta) / 2^32) where the
// step may change the minimum image (a warp-uniform branch).
__device__ __forceinline__ BlkView blk_view(const Move &m, const SysDesc &d, float step2) {
    BlkView v;
    v.hx = m.ho[0]; v.hy = m.ho[1]; v.hz = m.ho[2];
    float w[3];
#pragma unroll
    for (int a = 0; a < 3; a++)
        w[a] = i64_to_float((long long)((uint64_t)m.xn[a] - (uint64_t)m.xo[a])) * 2.3283064365386963e-10f;
    v.dx = w[0]; v.dy = w[1]; v.dz = w[2];
    v.d2 = fmaf(w[0], w[0], fmaf(w[1], w[1], w[2] * w[2]));
    const float half = 2147483648.0f * 0.999999f;
    v.wx = half - fabsf(w[0]); v.wy = half - fabsf(w[1]); v.wz = half - fabsf(w[2]);
    v.qc = m.q * d.lB / d.s32[0];
    v.ti = m.ti;
    v.i = m.i;
    v.small = d.kappa * d.s32[0] * sqrtf(v.d2) < 0.25f;
    v.far = !(v.d2 <= step2);
    return v;
}
__device__ __forceinline__ float3 blk_diff(const BlkView &v, int4 p) {   // partner - old position, words
    return make_float3((float)(int)((uint32_t)p.x - (uint32_t)v.hx), (float)(int)((uint32_t)p.y - (uint32_t)v.hy),
                       (float)(int)((uint32_t)p.z - (uint32_t)v.hz));
}
__device__ __forceinline__ bool blk_wraps(const BlkView &v, float3 o) {
    return fabsf(o.x) > v.wx || fabsf(o.y) > v.wy || fabsf(o.z) > v.wz;
}
template <bool WRAP>
__device__ __forceinline__ float blk_dr2(const BlkView &v, float3 o) {   // r_n^2 - r_o^2, words^2
    if (!WRAP) return fmaf(-2.0f, fmaf(v.dx, o.x, fmaf(v.dy, o.y, v.dz * o.z)), v.d2);
    auto axis = [](float x, float dl) {
        const float k = __fadd_rn(__fmaf_rn(x - dl, 2.3283064365386963e-10f, 12582912.0f), -12582912.0f);
        const float e = fmaf(k, -4294967296.0f, -dl);
        return e * fmaf(2.0f, x, e);
    };
    return axis(o.x, v.dx) + axis(o.y, v.dy) + axis(o.z, v.dz);
}
__device__ __forceinline__ float blk_rsqrt(float x) {   // hardware estimate plus one Newton step, as rsqrt_nr
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y * fmaf(-0.5f * x * y, y, 1.5f);
}
// One partner: u(new) - u(old) of Debye-Hueckel in the difference form
// u_o (expm1(-kappa dr) - dr/r_o) / (1 + dr/r_o) = C e^{-kappa r_o}
// (expm1(-kappa dr) - dr/r_o) / r_n, whose rounding scales with the difference,
// and of LJ (at most 0.0125 kT each out here) as 4eps d3 (s3 - 1) with d3, s3
// the difference and sum of (sigma/r)^6. Reciprocal and exponential use the
// approximate SFU forms: their ~2 ulp enter only as relative errors of the
// (small) difference. UNI: sums d3 and d3 s3 go to l1, l2 (scaled at the end).
// Straight-line (selects, no branch), so that a warp's two trials interleave.
// Returns true (adding nothing) for a partner within 2 sigma; `skip` lanes add
// nothing either. For steps of up to 4 sigma only (of the smallest pair): r_n^2
// as r_o^2 + dR2 loses (r_o / r_n)^2 in relative accuracy, at most 9 there.
template <bool UNI, bool SMALL>
__device__ __forceinline__ bool blk_far(const BlkView &v, const BlkConst &c, const SysDesc &d, float3 o, float dR2,
                                        float qj, int tj, bool skip, float &acc, float &l1, float &l2) {
    const float r2o = fmaf(o.x, o.x, fmaf(o.y, o.y, o.z * o.z));
    const float r2n = r2o + dR2;
    float s2 = c.s2, near2 = c.near2, e4 = 0.0f;
    if (!UNI) {
        const int t = v.ti * d.n_types + tj;
        s2 = d.s2[t] * c.w2;
        near2 = 4.0f * s2;
        e4 = d.eps4[t];
    }
    const bool near = fminf(r2o, r2n) < near2;
    const bool none = near || skip;
    const float rio = blk_rsqrt(r2o), rin = blk_rsqrt(r2n);
    const float ro = r2o * rio;
    const float dr = dR2 * blk_rcp(fmaf(r2n, rin, ro));
    const float yy = -c.kw * dr;
    float em1;
    if (SMALL) {
        em1 = fmaf(yy, 1.0f / 5040.0f, 1.0f / 720.0f);
        em1 = fmaf(yy, em1, 1.0f / 120.0f);
        em1 = fmaf(yy, em1, 1.0f / 24.0f);
        em1 = fmaf(yy, em1, 1.0f / 6.0f);
        em1 = fmaf(yy, em1, 0.5f);
        em1 = fmaf(yy * yy, em1, yy);
    } else {
        em1 = expm1f(yy);
    }
    const float u = v.qc * qj * rin * blk_ex2(c.kl * ro) * fmaf(-dr, rio, em1);
    acc += none ? 0.0f : u;
    const float xo = s2 * (rio * rio), xn = s2 * (rin * rin);
    const float o3 = none ? 0.0f : xo * xo * xo, n3 = none ? 0.0f : xn * xn * xn;
    const float d3 = n3 - o3, s3 = n3 + o3;
    if (UNI) {
        l1 += d3;
        l2 = fmaf(d3, s3, l2);
    } else {
        acc = fmaf(e4 * d3, s3 - 1.0f, acc);
    }
    return near && !skip;
}

// The same for a longer step (qc: the trial's): both distances from their own
// exact differences and both energies by themselves, since far apart the
// difference form's error grows with r_o / r_n. rms error of a trial over the
// whole box, 16384 ions (L = 202 Angstrom): 6.4e-6 kT by blk_far, 3.7e-6 by the
// difference form on r_n of its own, 3.3e-6 so; steps of up to 40 Angstrom
// 7.4e-7, 7.4e-7, 6.7e-7. Time per trial as for short steps (0.39 us at 2001
// ions, 0.85 at 16384).
__device__ __forceinline__ bool blk_far_long(const Move &m, float qc, const BlkConst &c, int4 p, int tj, const SysDesc &d,
                                             float &acc) {
    auto r2_of = [&](const int h[3]) {
        const float x = (float)(int)((uint32_t)p.x - (uint32_t)h[0]), y = (float)(int)((uint32_t)p.y - (uint32_t)h[1]),
                    z = (float)(int)((uint32_t)p.z - (uint32_t)h[2]);
        return fmaf(x, x, fmaf(y, y, z * z));
    };
    const float r2n = r2_of(m.hn), r2o = r2_of(m.ho);
    const int t = d.uniform_types ? 0 : m.ti * d.n_types + tj;
    const float s2 = d.s2[t] * c.w2;
    if (fminf(r2n, r2o) < 4.0f * s2) return true;
    const float rin = blk_rsqrt(r2n), rio = blk_rsqrt(r2o);
    const float xn = s2 * (rin * rin), xo = s2 * (rio * rio), n3 = xn * xn * xn, o3 = xo * xo * xo;
    acc = fmaf(qc * __int_as_float(p.w), fmaf(rin, blk_ex2(c.kl * (r2n * rin)), -rio * blk_ex2(c.kl * (r2o * rio))), acc);
    acc = fmaf(d.eps4[t] * (n3 - o3), n3 + o3 - 1.0f, acc);
    return false;
}

// dU contribution of one partner (high words pj with charge bits, type tj,
// extension e) for trial m, as a df number.
__device__ __forceinline__ df blk_pair(const Move &m, int4 pj, int tj, const short4 *e, const SysDesc &d) {
    float a = 0.0f;
    df ad = {0.0f, 0.0f};
    pair_candidate<MODEL_DHLJ>(m, pj, tj, e, d, a, ad);
    return df_add_f(ad, a);
}

// Warp-aggregated append to the near-pair queue; true = the queue is full and
// the lane evaluates its pair in place.
__device__ __forceinline__ bool blk_enqueue(const BlkSmem &s, bool near, uint32_t code) {
    const unsigned active = __activemask();
    const unsigned m = __ballot_sync(active, near);
    if (!m) return false;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(m) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(&s.info[2], __popc(m));
    base = __shfl_sync(active, base, leader);
    if (!near) return false;
    const int slot = base + __popc(m & ((1u << lane) - 1u));
    if (slot < kBlkQueue) {
        s.queue[slot] = code;
        return false;
    }
    return true;
}

// A warp's sums of two trials in one tree: da's in lanes 0..15, db's in 16..31.
__device__ __forceinline__ df blk_two_sums(df da, df db) {
    const bool hi = (threadIdx.x & 31) >= 16;   // the half-warps exchange first
    const df give = hi ? da : db;
    df sum = hi ? db : da;
    sum = df_add(sum, df{__shfl_xor_sync(0xffffffffu, give.hi, 16), __shfl_xor_sync(0xffffffffu, give.lo, 16)});
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
        sum = df_add(sum, df{__shfl_xor_sync(0xffffffffu, sum.hi, o), __shfl_xor_sync(0xffffffffu, sum.lo, o)});
    return sum;
}

// blk_base for a warp with a step longer than 4 sigma.
template <bool SLICE>
__device__ __forceinline__ df blk_base_long(const BlkSmem &s, const SysDesc &d, const BlkConst &c, int ma, int mb, int j0,
                                            int ns) {
    const int lane = threadIdx.x & 31;
    df sum[2] = {{0.0f, 0.0f}, {0.0f, 0.0f}};
#pragma unroll 1
    for (int h = 0; h < 2; h++) {
        const int mm = h ? mb : ma;
        if (mm < 0) break;
        const Move &m = s.mv[mm];
        const int self = m.i - j0;
        const float qc = s.view[mm].qc;
        float f = 0.0f;
        df v = {0.0f, 0.0f};
        for (int jb = 0; jb < ns; jb += 32) {
            const int j = jb + lane, k = min(j, ns - 1);
            const int4 p = SLICE ? s.spos[k] : d.pos4[j0 + k];
            const int t = SLICE ? s.stype[k] : d.ptype[j0 + k];
            bool near = false;
            if (j < ns && j != self) near = blk_far_long(m, qc, c, p, t, d, f);
            if (__any_sync(0xffffffffu, near) && blk_enqueue(s, near, ((uint32_t)mm << 24) | (uint32_t)j))
                pair_candidate<MODEL_DHLJ>(m, p, t, SLICE ? &s.sext[k] : &d.pos_ext[j0 + k], d, f, v);
        }
        sum[h] = df_add_f(v, f);
    }
    return blk_two_sums(sum[0], sum[1]);
}

// Base sums of the trials ma and mb (mb < 0: none) over the CTA's slice by one
// warp, one partner per lane and turn for both (independent chains for the
// scheduler, one load of the partner); partners within 2 sigma go to the
// queue. The warp's sums are returned: ma's in lanes 0..15, mb's in 16..31.
template <bool SLICE, bool UNI>
__device__ __forceinline__ df blk_base(const BlkSmem &s, const SysDesc &d, const BlkConst &c, int ma, int mb, int j0,
                                       int ns) {
    const int lane = threadIdx.x & 31;
    const BlkView va = s.view[ma], vb = s.view[max(mb, 0)];
    const int sa = va.i - j0, sb = vb.i - j0;
    float fa = 0.0f, fb = 0.0f, a1 = 0.0f, a2 = 0.0f, b1 = 0.0f, b2 = 0.0f;
    df da = {0.0f, 0.0f}, db = {0.0f, 0.0f};
    const bool small = va.small && vb.small;   // warp-uniform
    for (int jb = 0; jb < ns; jb += 32) {
        const int j = jb + lane, k = min(j, ns - 1);
        const int4 p = SLICE ? s.spos[k] : d.pos4[j0 + k];
        const int t = UNI ? 0 : (SLICE ? s.stype[k] : d.ptype[j0 + k]);
        const float q = __int_as_float(p.w);
        const float3 oa = blk_diff(va, p), ob = blk_diff(vb, p);
        const bool ka = j >= ns || j == sa, kb = j >= ns || j == sb || mb < 0;
        float ra, rb;
        if (__any_sync(0xffffffffu, blk_wraps(va, oa) || blk_wraps(vb, ob))) {
            ra = blk_dr2<true>(va, oa);
            rb = blk_dr2<true>(vb, ob);
        } else {
            ra = blk_dr2<false>(va, oa);
            rb = blk_dr2<false>(vb, ob);
        }
        bool na, nb;
        if (small) {
            na = blk_far<UNI, true>(va, c, d, oa, ra, q, t, ka, fa, a1, a2);
            nb = blk_far<UNI, true>(vb, c, d, ob, rb, q, t, kb, fb, b1, b2);
        } else {
            na = blk_far<UNI, false>(va, c, d, oa, ra, q, t, ka, fa, a1, a2);
            nb = blk_far<UNI, false>(vb, c, d, ob, rb, q, t, kb, fb, b1, b2);
        }
        if (__any_sync(0xffffffffu, na || nb)) {
            const int tj = SLICE ? s.stype[k] : d.ptype[j0 + k];
            const short4 *e = SLICE ? &s.sext[k] : &d.pos_ext[j0 + k];
            if (blk_enqueue(s, na, ((uint32_t)ma << 24) | (uint32_t)j))
                pair_candidate<MODEL_DHLJ>(s.mv[ma], p, tj, e, d, fa, da);
            if (blk_enqueue(s, nb, ((uint32_t)max(mb, 0) << 24) | (uint32_t)j))
                pair_candidate<MODEL_DHLJ>(s.mv[max(mb, 0)], p, tj, e, d, fb, db);
        }
    }
    if (UNI) {
        fa = fmaf(d.eps4[0], a2 - a1, fa);
        fb = fmaf(d.eps4[0], b2 - b1, fb);
    }
    da = df_add_f(da, fa);
    db = df_add_f(db, fb);
    return blk_two_sums(da, db);
}

// One cluster of C CTAs per system; system members[blockIdx.x / C] of descs
// (members == nullptr: blockIdx.x / C). C == 1 runs without a cluster.
template <bool SLICE, bool CLUSTER>
__global__ void __launch_bounds__(kBlkThreads, 1) dh_block_kernel(const SysDesc *__restrict__ descs,
                                                                  const int *__restrict__ members, int C,
                                                                  int64_t end) {
    extern __shared__ __align__(16) unsigned char blk_smem_raw[];
    __shared__ __align__(16) SysDesc sd;
    const int sys = members ? members[blockIdx.x / C] : (int)(blockIdx.x / C);
    // launch-shape check: the partial sums are read from C CTAs of this
    // cluster; anything else records an error and touches no other CTA
    if (CLUSTER ? (int)blk_cluster_size() != C : C != 1) {
        if (threadIdx.x == 0) atomicOr(&descs[sys].sc->error, kErrLaunch);
        return;
    }
    const int rank = CLUSTER ? (int)blk_cluster_rank() : 0;
    load_desc(sd, descs + sys);
    const SysDesc &d = sd;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
    const int N = d.N;
    const int ns_full = (N + C - 1) / C;
    const int j0 = min(rank * ns_full, N), j1 = min(j0 + ns_full, N), ns = j1 - j0;
    BlkSmem s = blk_carve(blk_smem_raw, ns_full, SLICE, C);
    SysScalars *sc = d.sc;
    int64_t cur = sc->cursor;
    const int64_t stop = min(end, sc->n_trials);
    if (SLICE)
        for (int jj = tid; jj < ns; jj += blockDim.x) {
            s.spos[jj] = d.pos4[j0 + jj];
            s.sext[jj] = d.pos_ext[j0 + jj];
            s.stype[jj] = d.ptype[j0 + jj];
        }
    df U = {sc->u_hi, sc->u_lo};
    df Ut = {sc->utot_hi, sc->utot_lo};
    int64_t nacc = sc->n_accepted;
    int err = 0;
    if (CLUSTER) blk_cluster_barrier();
    else __syncthreads();
    int64_t nblock = 0;
    const bool uni = d.uniform_types != 0;
    float s2min = d.s2[0];
    for (int t = 1; t < d.n_types * d.n_types; t++) s2min = fminf(s2min, d.s2[t]);
    const BlkConst bc = {d.kappa * d.s32[0], -d.kappa * d.s32[0] * 1.4426950408889634f,
                         4.0f * d.s2[0] / (d.s32[0] * d.s32[0]), d.s2[0] / (d.s32[0] * d.s32[0]),
                         1.0f / (d.s32[0] * d.s32[0]), 16.0f * s2min / (d.s32[0] * d.s32[0])};
    // the trial records of the next block are loaded during this one (used if
    // this one resolves all its trials)
    Trial nx{};
    int64_t nx_at = -1;
    while (cur < stop) {
        const int kb = (int)((stop - cur) < (int64_t)kBlkTrials ? (stop - cur) : (int64_t)kBlkTrials);
        const int slot = (int)(nblock & 1);
        float2 *const xc = s.corr + (CLUSTER ? slot * kBlkTrials * kBlkTrials : 0);
        // ---- set up the block's trials (old coordinates: the block start)
        if (tid < kb) {
            const Trial tr = nx_at == cur ? nx : d.trials[cur + tid];
            int64_t xo[3], xn[3];
#pragma unroll
            for (int a = 0; a < 3; a++) {
                xo[a] = d.pos64[3 * tr.idx + a];
                xn[a] = (int64_t)((uint64_t)xo[a] + (uint64_t)tr.d[a]);
            }
            Move m;
            move_setup(m, tr.idx, xo, xn, __int_as_float(d.pos4[tr.idx].w), d.ptype[tr.idx], d);
            s.mv[tid] = m;
            s.view[tid] = blk_view(m, d, bc.step2);
            df thr = {tr.thr_hi, tr.thr_lo};
            if (d.kT != 1.0f) thr = dfm_f(thr, d.kT);
            s.thr[tid] = make_float2(thr.hi, thr.lo);
        }
        if (tid < 3 * kBlkTrials) s.fix[tid] = 0ull;
        if (tid == 0) s.info[2] = s.info[3] = 0;
        __syncthreads();
        if (tid < kb) {
            uint32_t c = 0;
            const int i = s.mv[tid].i;
            for (int a = 0; a < tid; a++)
                if (s.mv[a].i == i) c |= 1u << a;
            s.col[tid] = c;
        }
        nx_at = cur + kb;
        if (tid < kBlkTrials && nx_at + tid < stop) nx = d.trials[nx_at + tid];
        // ---- base sums: warp w takes trials w, w + nwarp, ... over this slice
        static_assert(kBlkTrials == 2 * (kBlkThreads / 32), "one turn of two trials per warp");
        if (warp < kb) {
            const int mb = warp + nwarp < kb ? warp + nwarp : -1;
            const bool far = s.view[warp].far || s.view[mb < 0 ? warp : mb].far;
            const df p = far   ? blk_base_long<SLICE>(s, d, bc, warp, mb, j0, ns)
                         : uni ? blk_base<SLICE, true>(s, d, bc, warp, mb, j0, ns)
                               : blk_base<SLICE, false>(s, d, bc, warp, mb, j0, ns);
            if (lane == 0) s.part[warp] = make_float2(p.hi, p.lo);
            if (lane == 16 && mb >= 0) s.part[mb] = make_float2(p.hi, p.lo);
        }
        __syncthreads();
        // ---- corrections c(a, m), a < m, and the queued near pairs, in one
        // pass over the threads: first this CTA's share of the kb (kb - 1) / 2 <=
        // 496 pairs of trials (into every CTA's table; two lanes per pair, one
        // for a's new and one for its old position), then its queue
        {
            const int np = 2 * ((kb * (kb - 1) / 2 + C - 1 - rank) / C), nq = min(s.info[2], kBlkQueue);
            for (int ub = warp * 32; ub < np + nq; ub += blockDim.x) {   // warp-uniform
                const int u = ub + lane;
                df v = {0.0f, 0.0f};
                int a = 0, m = 0;
                if (u < np) {
                    const int e = (u >> 1) * C + rank;
                    m = (int)((1.0f + sqrtf(8.0f * (float)e + 1.0f)) * 0.5f);
                    if (m * (m - 1) / 2 > e) m--;
                    if ((m + 1) * m / 2 <= e) m++;
                    a = e - m * (m - 1) / 2;
                }
                const bool live = u < np && s.mv[a].i != s.mv[m].i;
                if (live || (u >= np && u < np + nq)) {
                    int4 pj;
                    int tj;
                    short4 ext;
                    if (live) {
                        const Move &A = s.mv[a];
                        const bool old = u & 1;
                        tj = A.ti;
                        pj = make_int4(old ? A.ho[0] : A.hn[0], old ? A.ho[1] : A.hn[1], old ? A.ho[2] : A.hn[2],
                                       __float_as_int(A.q));
                        ext = make_short4((short)(old ? A.eo[0] : A.en[0]), (short)(old ? A.eo[1] : A.en[1]),
                                          (short)(old ? A.eo[2] : A.en[2]), 0);
                    } else {
                        const uint32_t q = s.queue[u - np];
                        const int jj = (int)(q & 0xFFFFFF), j = j0 + jj;
                        m = (int)(q >> 24);
                        tj = SLICE ? s.stype[jj] : d.ptype[j];
                        pj = SLICE ? s.spos[jj] : d.pos4[j];
                        ext = SLICE ? s.sext[jj] : d.pos_ext[j];
                    }
                    v = blk_pair(s.mv[m], pj, tj, &ext, d);
                    if (!live) blk_fix_add(s, m, v);
                }
                const df w = {__shfl_xor_sync(0xffffffffu, v.hi, 1), __shfl_xor_sync(0xffffffffu, v.lo, 1)};
                if (u < np) {
                    // lane pairs: new minus old; the two lanes share the stores
                    const df c = (u & 1) ? df_add(w, df_neg(v)) : df_add(v, df_neg(w));
                    const float2 out = make_float2(fabsf(c.hi) <= kBlkLargeCorr ? c.hi : __int_as_float(0x7FFFFFFF), c.lo);
                    if (CLUSTER) {
                        for (int r = u & 1; r < C; r += 2) blk_st_cluster(&xc[a * kBlkTrials + m], (unsigned)r, out);
                    } else if (!(u & 1)) {
                        xc[a * kBlkTrials + m] = out;
                    }
                }
            }
        }
        __syncthreads();
        // this CTA's sums, into every CTA of the cluster
        float2 *const xp = s.xpart + slot * C * kBlkTrials;
        if (tid < kBlkTrials * C) {
            const int m = tid & (kBlkTrials - 1), to = tid / kBlkTrials;
            if (m < kb) {
                const float2 p = s.part[m];
                const df v = df_add(df{p.x, p.y}, blk_fix_sum(s, m));
                if (CLUSTER) blk_st_cluster(&xp[rank * kBlkTrials + m], (unsigned)to, make_float2(v.hi, v.lo));
                else xp[m] = make_float2(v.hi, v.lo);
            }
        }
        if (CLUSTER) blk_cluster_barrier();
        else __syncthreads();
        // ---- resolve the block in order (warp 0; lane m = trial m)
        if (warp == 0) {
            df S = {0.0f, 0.0f};
            if (lane < kb)
                for (int r = 0; r < C; r++) {
                    const float2 p = xp[r * kBlkTrials + lane];
                    S = df_add(S, df{p.x, p.y});
                }
            const uint32_t colm = lane < kb ? s.col[lane] : 0u;
            const float2 th = lane < kb ? s.thr[lane] : make_float2(0.0f, 0.0f);
            uint32_t accm = 0;
            int done = kb;
            float2 cn = xc[min(lane, kBlkTrials - 1)];
            for (int a = 0; a < kb; a++) {
                // lane a decides: its S already holds the corrections of every
                // accepted trial before it in the block. Movebase::metropolis
                // (move.h:567-573): reject iff dU > kT (-ln u); a NaN dU
                // compares false there: accepted. Every lane forms its flags and
                // the sum it would go on with; lane a's flags select, so a step
                // costs one shuffle and no branch (250 -> 80 cycles)
                const float2 c = cn;
                cn = xc[min(a + 1, kBlkTrials - 1) * kBlkTrials + lane];
                const df Sc = df_add_quick(S, df{c.x, c.y});
                const int fl = ((colm & accm) != 0u ? 1 : 0) | (!df_gt(S, df{th.x, th.y}) ? 2 : 0);
                const int f = __shfl_sync(0xffffffffu, fl, a);
                if (f & 1) {   // its particle was moved by an accepted trial of this block
                    done = a;
                    break;
                }
                accm |= (uint32_t)(f >> 1) << a;
                const bool add = (f & 2) && lane > a;
                S.hi = add ? Sc.hi : S.hi;
                S.lo = add ? Sc.lo : S.lo;
            }
            // kBlkLargeCorr: the sums of the trials before do not depend on the later ones
            const uint32_t nan = __ballot_sync(0xffffffffu, lane < done && !(S.hi == S.hi));
            if (nan & ~1u) {
                done = __ffs(nan & ~1u) - 1;
                accm &= (1u << done) - 1u;
            }
            nacc += __popc(accm);
            if (nan & 1u) err |= kErrNonFinite;
            // lane m's S is trial m's dU as decided: log it, and add the
            // accepted ones to the running sums (a fixed-order warp sum)
            const bool take = lane < done && ((accm >> lane) & 1u);
            if (rank == 0 && d.log_trials && lane < done) {
                d.trial_du[cur + lane] = make_float2(S.hi, S.lo);
                d.trial_acc[cur + lane] = take ? 1 : 0;
            }
            const df sum = warp_sum_df(take ? S : df{0.0f, 0.0f});
            U = df_add(U, sum);
            Ut = df_add(Ut, sum);
            if (lane == 0) {
                s.info[0] = done;
                s.info[1] = (int)accm;
            }
        }
        __syncthreads();
        // ---- apply the accepted moves (at most one per particle per block)
        const int done = s.info[0];
        const uint32_t accm = (uint32_t)s.info[1];
        if (tid < done && (accm >> tid) & 1u) {
            const Move &m = s.mv[tid];
            const int4 rec = make_int4(m.hn[0], m.hn[1], m.hn[2], __float_as_int(m.q));
            const short4 ext = make_short4((short)m.en[0], (short)m.en[1], (short)m.en[2], 0);
            // every CTA writes the same values to the master arrays; each reads
            // them only after its own write
            d.pos64[3 * m.i + 0] = m.xn[0];
            d.pos64[3 * m.i + 1] = m.xn[1];
            d.pos64[3 * m.i + 2] = m.xn[2];
            d.pos4[m.i] = rec;
            d.pos_ext[m.i] = ext;
            if (SLICE && m.i >= j0 && m.i < j1) {
                s.spos[m.i - j0] = rec;
                s.sext[m.i - j0] = ext;
            }
        }
        cur += done;
        nblock++;
        __syncthreads();
    }
    if (rank == 0 && tid == 0) {
        sc->cursor = cur;
        sc->u_hi = U.hi;
        sc->u_lo = U.lo;
        sc->utot_hi = Ut.hi;
        sc->utot_lo = Ut.lo;
        sc->n_accepted = nacc;
        sc->error |= err;
    }
    if (CLUSTER) blk_cluster_barrier();   // no CTA leaves while another may read its shared memory
}

}  // namespace fg
