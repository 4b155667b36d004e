// Ewald + WCA sweeps in blocks of trials (one CTA per system).
//
// Included by fg_api.cu after fg_kernels.cu (one translation unit).
//
// Same idea as the Debye-Hueckel block kernel (fg_dh_block.cu): a block of up
// to 32 trials is evaluated against the configuration at the block start, and
// one warp resolves it in order with exact corrections for the trials it
// accepts. For Ewald the correction of trial m after an accepted trial a has
// three parts:
//   real space   [u(n_m,n_a) - u(o_m,n_a)] - [u(n_m,o_a) - u(o_m,o_a)]
//   surface      2 c dM_a . dM_m                 (E_surf = c |M|^2)
//   reciprocal   sum_k A'_k 2 Re(conj(D_a,k) D_m,k)
// with D_m,k = q (e^{ik.r_new} - e^{ik.r_old}) = 2 q sin(k.d / 2) i e^{ik.r_mid},
// r_mid the step's midpoint, the same increment the energy uses (its error is
// relative to |d|; a real sine times a phase takes 55 issue slots, the form
// q e^{ik.r_old}(e^{ik.d} - 1) took 65).
// The reciprocal parts of all pairs of the block form a 32 x 32 Gram matrix
// over k of the trials' increments; the warps accumulate it on the tensor cores
// (eb_gram_regs), each from the increments that it forms in registers.
// Q(k) itself stays the exact fixed-point sum: after the block each accepted
// trial's integer contributions are applied in order. A trial whose particle
// an accepted trial of the block already moved ends the block, and so does
// the accepted trial that makes a Q(k) rebuild due. In a batch that fills the
// GPU the CTA then rebuilds its system's Q(k) from scratch in place
// (eb_rebuild) and carries on, so one launch runs every system's whole
// stream; a system running alone exits instead and leaves the rebuild to the
// rebuild kernel, which spreads it over all SMs.
namespace fg {

constexpr int kEbTrials = 32;
constexpr int kEbThreads = 512;
constexpr int kEbKc = 128;   // scratch buffer rows (of 32 float2)
constexpr int kEbMaxCluster = 16;
// A correction beyond this (kT) belongs to a trial on top of where an accepted
// particle was: its dU would be the small rest of two large numbers. It is kept
// as a NaN, the block ends before a trial that took it, and the next block
// evaluates the trial (its first) as the configuration is.
constexpr float kEbLargeCorr = 1.0e4f;
constexpr int kEbGramN = 6 * 32 * 4;   // floats of one Gram accumulator set (eb_gram_regs' layout)

struct EbSmem {
    Smem b;          // sc_tab, qfix, kpack, cells as in the one-trial kernel; kvec here holds
                     // {A'_k, Q(k) as float (re, im), sqrt(A'_k)}: k itself comes from the integer n
    Move *mv;        // [32]
    float2 *thr;     // [32] threshold (df, times kT)
    uint32_t *col;   // [32] earlier trials on the same particle
    int *info;       // [8] resolved count, accepted mask, rebuild
    float2 *partR;   // [32] real-space base (df)
    float2 *kbase;   // [32] reciprocal base (df)
    float2 *corr;    // [32][32] real-space + surface corrections (df)
    float *G;        // [32][32] reciprocal cross terms
    float2 *delta;   // [kEbKc x 32] scratch: real-space queues and k-space trial records, then
                     // the Gram and reciprocal-base partials, then the commit's axis tables
    float2 *Mdf;     // [3] surface dipole M (df)
    // cluster only (written by the other CTAs into the leader's copy): per
    // rank its Gram sums [C][kEbGramN] and reciprocal bases [C][32], per trial
    // and part the real-space partial sums [32][parts]
    float *xgram;
    float2 *xkbase;
    float2 *xreal;
};

// Shared memory of one CTA holding Kl k-vectors, in a cluster of C CTAs.
__host__ __device__ inline size_t eb_layout(int N, int Kl, int ncell, bool cells, int C, size_t off[19]) {
    size_t b = 256 * 8 + 32 * 8;            // sc_tab, red
    off[0] = b; b += (size_t)Kl * 16;       // kvec
    off[1] = b; b += (size_t)Kl * 16;       // qfix
    off[2] = b; b = align16(b + (size_t)Kl * 4);           // kpack
    off[3] = b; if (cells) b = align16(b + (size_t)ncell * 4);   // ccount
    off[4] = b; if (cells) b = align16(b + (size_t)N * 4);       // pcs
    off[5] = b; b = align16(b + sizeof(Move) * kEbTrials);      // mv
    off[6] = b; b = align16(b + 8 * kEbTrials);                 // thr
    off[7] = b; b = align16(b + 4 * kEbTrials);                 // col
    off[8] = b; b = align16(b + 4 * 8);                         // info
    off[9] = b; b = align16(b + 8 * kEbTrials);                 // partR
    off[10] = b; b = align16(b + 8 * kEbTrials);                // kbase
    off[11] = b; b = align16(b + 8 * kEbTrials * kEbTrials);    // corr
    off[12] = b; b = align16(b + 4 * kEbTrials * kEbTrials);    // G
    off[13] = b; b = align16(b + 8 * kEbKc * kEbTrials);        // delta
    off[14] = b; b = align16(b + 8 * 3);                        // Mdf
    const int cx = C > 1 ? C : 0;
    off[15] = b; b = align16(b + (size_t)4 * kEbGramN * cx);    // xgram
    off[16] = b; b = align16(b + (size_t)8 * kEbTrials * cx);   // xkbase
    off[17] = b; b = align16(b + (size_t)8 * kEbTrials * (C > 1 ? (C + 1) / 2 : 0));   // xreal
    off[18] = b;
    return b;
}

__device__ inline EbSmem eb_carve(char *base, const SysDesc &d, bool cells) {
    size_t off[19];
    const int ncell = d.nc[0] * d.nc[1] * d.nc[2];
    eb_layout(d.N, d.eb_kmax, ncell, cells, d.eb_ctas, off);
    EbSmem s;
    s.b.sc_tab = (float2 *)base;
    s.b.red = (float2 *)(base + 256 * 8);
    s.b.kvec = (float4 *)(base + off[0]);
    s.b.qfix = (longlong2 *)(base + off[1]);
    s.b.qf = nullptr;
    s.b.ktab = nullptr;
    s.b.kpack = (uint32_t *)(base + off[2]);
    s.b.pos = nullptr;
    s.b.pos_ext = nullptr;
    s.b.ptype = nullptr;
    s.b.ccount = (int *)(base + off[3]);
    s.b.pcs = (uint32_t *)(base + off[4]);
    s.mv = (Move *)(base + off[5]);
    s.thr = (float2 *)(base + off[6]);
    s.col = (uint32_t *)(base + off[7]);
    s.info = (int *)(base + off[8]);
    s.partR = (float2 *)(base + off[9]);
    s.kbase = (float2 *)(base + off[10]);
    s.corr = (float2 *)(base + off[11]);
    s.G = (float *)(base + off[12]);
    s.delta = (float2 *)(base + off[13]);
    s.Mdf = (float2 *)(base + off[14]);
    s.xgram = (float *)(base + off[15]);
    s.xkbase = (float2 *)(base + off[16]);
    s.xreal = (float2 *)(base + off[17]);
    return s;
}

// One k-step of the Gram matrix on the tensor cores: components c = the real
// and imaginary parts of 4 consecutive k-vectors of X = sqrt(A') D. mma.sync
// m16n8k8 TF32 with the three-product split (hi hi + hi lo + lo hi, each
// operand split into a TF32 high part and the TF32 rounding of the rest)
// keeps FP32-level accuracy. Lane (gq = lane / 4, gt = lane % 4) holds the
// components gt and gt + 4 of trials gq + 8 r; these are the A fragments of
// the two 16-row tiles and, G being X X^T, the B fragments of the four
// 8-column tiles. Accumulated tiles (row tile, column tile): (0,0) (0,1)
// (0,2) (0,3) (1,2) (1,3), every pair a < m lies in one of them.
// x rounded to TF32 (to nearest, ties away: the bits of cvt.rna.tf32.f32 for
// finite x) with integer instructions: the conversion runs on the SFU, and 16
// of them per k-step and warp were 128 of the step's 480 cycles. (A NaN may
// lose itself here; the trial's reciprocal base, FP32 sums of the same
// amplitudes, keeps it.)
__device__ __forceinline__ uint32_t eb_tf32(float x) { return (__float_as_uint(x) + 0x1000u) & 0xFFFFE000u; }
__device__ __forceinline__ void eb_mma(float c[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void eb_gram_regs(const float xf[4][2], float gc[6][4]) {
    uint32_t hi[4][2], lo[4][2];
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            hi[r][h] = eb_tf32(xf[r][h]);
            lo[r][h] = eb_tf32(xf[r][h] - __uint_as_float(hi[r][h]));
        }
#pragma unroll
    for (int t = 0; t < 6; t++) {
        const int mi = t < 4 ? 0 : 1, nj = t < 4 ? t : t - 2;
        const uint32_t ah[4] = {hi[2 * mi][0], hi[2 * mi + 1][0], hi[2 * mi][1], hi[2 * mi + 1][1]};
        const uint32_t al[4] = {lo[2 * mi][0], lo[2 * mi + 1][0], lo[2 * mi][1], lo[2 * mi + 1][1]};
        eb_mma(gc[t], al, hi[nj][0], hi[nj][1]);
        eb_mma(gc[t], ah, lo[nj][0], lo[nj][1]);
        eb_mma(gc[t], ah, hi[nj][0], hi[nj][1]);
    }
}

// sin(x) with error relative to x for |x| <= 0.8 (next term < 3e-9 of it).
__device__ __forceinline__ float eb_sin(float x) {
    const float x2 = x * x;
    float s = fmaf(x2, 2.7557319223985893e-06f, -1.9841269841269841e-04f);
    s = fmaf(x2, s, 8.3333333333333333e-03f);
    s = fmaf(x2, s, -1.6666666666666667e-01f);
    return fmaf(x2 * x, s, x);
}

// Barrier 1 over the block's warps 1.. (nthreads = blockDim - 32 threads).
__device__ __forceinline__ void eb_qbar(int nthreads) {
    asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory");
}

// Stores into CTA `rank`'s copy of a shared-memory variable (the cluster's
// distributed shared memory).
__device__ __forceinline__ uint32_t eb_remote(const void *p, unsigned rank) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    uint32_t ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
    return ra;
}
__device__ __forceinline__ void eb_st_remote(float2 *p, unsigned rank, float2 v) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(eb_remote(p, rank)), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void eb_st_remote(float *p, unsigned rank, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(eb_remote(p, rank)), "f"(v) : "memory");
}
__device__ __forceinline__ void eb_st_remote(int *p, unsigned rank, int v) {
    asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(eb_remote(p, rank)), "r"(v) : "memory");
}

// Real-space base of one trial by one warp (or part `part` of `nparts`: the
// candidate batches part, part + nparts, ...). The phase is bound by issue
// slots, so each stage does as little as it can for as many as it must see:
// 1. Batches of 32 slots (of a stencil cell, or of all particles) are screened
//    by the distance to the step's midpoint against reach + |d|/2; all that is
//    kept of a batch is the ballot, in lane (batch mod 32). Skipped candidates
//    contribute exactly zero (every pair term is zero beyond reach2).
// 2. Every 32 batches the lanes write the slots of their set bits to a list.
// 3. The list is evaluated 32 at a time with all lanes busy.
// 4. Those within 1.5 sigma of either position (four a trial at 0.0037 ions per
//    cubic Angstrom) need erfcf, a correctly rounded root and divide or the
//    double-float core, some 2 k issue slots against 0.2 k: they wait in a
//    queue until both of the warp's trials are walked and are evaluated
//    together, two lanes per candidate (new and old position).
// One block of 32 trials on one CTA, cycles: 49 k -> 32 k at 800 ions without
// cells, 86 k -> 54 k at 16384 ions with cells, against queueing every screened
// pair with its position and a near pair in the batch where it was met.
constexpr int kEbNear = 16;      // entries of the near queue
constexpr int kEbList = 160;     // entries of the list
constexpr int kEbBatch = 64;     // cell batches listed at a time
constexpr int kEbQueueBytes = kEbNear * 24 + kEbList * 4 + kEbBatch * 8;   // of one warp
// s.delta before the sums are formed: the warps' queues, the trial records
// (2 x 16 bytes each), and from 28 KB the reciprocal-base partials
constexpr int kEbRecords = (kEbThreads / 32) * kEbQueueBytes;
static_assert(kEbRecords + 32 * kEbTrials <= 28672 && 28672 + 8 * kEbThreads <= 8 * kEbKc * kEbTrials, "eb scratch");
struct EbQueue {
    int4 *np;        // near queue: positions
    int2 *nm, *bat;  // near queue: slot, type + 256 x which of the warp's trials; batches: first slot, count
    int *list;       // slots within reach
    int nn;          // near queue length
};
__device__ __forceinline__ EbQueue eb_queue(void *base) {
    EbQueue q;
    q.np = reinterpret_cast<int4 *>(base);
    q.nm = reinterpret_cast<int2 *>(q.np + kEbNear);
    q.bat = q.nm + kEbNear;
    q.list = reinterpret_cast<int *>(q.bat + kEbBatch);
    q.nn = 0;
    return q;
}
// What a far pair needs of its trial, in registers.
struct EbFar {
    int ho[3], hn[3], hm[3];   // old, new position and their midpoint
    float q, qe;               // charge; qeqe of the single type
    float near2, rm2;          // squared distances: near pair, reach from the midpoint
    float sl[3];               // the axis factors (the descriptor lies in shared memory
                               // and would be read again after each warp barrier)
};
__device__ __forceinline__ float eb_r2(int4 a, const int h[3], const EbFar &m) {
    const float x = (float)(a.x - h[0]) * m.sl[0], y = (float)(a.y - h[1]) * m.sl[1], z = (float)(a.z - h[2]) * m.sl[2];
    return fmaf(x, x, fmaf(y, y, z * z));
}
// rsqrt_nr and erfc_nr for arguments that are neither subnormal nor huge:
// without the range checks of rsqrtf and __frcp_rn (a reciprocal after one
// Newton step).
__device__ __forceinline__ float eb_rsqrt(float r2) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(r2));
    return y * fmaf(-0.5f * r2 * y, y, 1.5f);
}
__device__ __forceinline__ float eb_erfc(float z) {
    const float x = fmaf(0.5f, z, 1.0f);
    float t;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(x));
    t = fmaf(t, fmaf(-x, t, 1.0f), t);
    return erfc_nr_at(t, z);
}
// u(new) - u(old) of a pair beyond 1.5 sigma of both positions: no WCA, no
// core; pair_ewald_wca<false>'s real-space term at both, without branches.
__device__ __forceinline__ float eb_far(const EbFar &m, float r2n, float r2o, float qj, int t, const SysDesc &d) {
    const float qq = m.q * qj * (d.uniform_types ? m.qe : d.qeqe[t]) * d.lB;
    float un, uo;
    if (d.kappa == 0.0f) {
        const float in = eb_rsqrt(r2n), io = eb_rsqrt(r2o);
        const float en = eb_erfc(d.alpha * (r2n * in)), eo = eb_erfc(d.alpha * (r2o * io));
        un = r2n <= d.rc2 ? qq * en * in : 0.0f;
        uo = r2o <= d.rc2 ? qq * eo * io : 0.0f;
    } else {
        un = pair_ewald_wca<false>(r2n, qq, 0.0f, 0.0f, 0.0f, d);
        uo = pair_ewald_wca<false>(r2o, qq, 0.0f, 0.0f, 0.0f, d);
    }
    return un - uo;
}
// The near queue's sum: lanes 2 e and 2 e + 1 take candidate e at the new and at
// the old position (with the opposite sign); which: the trial it belongs to.
__device__ __noinline__ df eb_near(const int4 *np, const int2 *nm, int n, const Move *m0, const Move *m1,
                                   const short4 *ext, const SysDesc &d, int &which) {
    const int lane = threadIdx.x & 31, e = lane >> 1;
    which = 0;
    if (e >= n) return df{0.0f, 0.0f};
    const int4 p = np[e];
    const int2 r = nm[e];
    which = r.y >> 8;
    const Move &m = which ? *m1 : *m0;
    const bool old = lane & 1;
    const int h0 = old ? m.ho[0] : m.hn[0], h1 = old ? m.ho[1] : m.hn[1], h2 = old ? m.ho[2] : m.hn[2];
    const float qj = __int_as_float(p.w), r2 = dist2(p, h0, h1, h2, d);
    const int t = d.uniform_types ? 0 : m.ti * d.n_types + (r.y & 255);
    df u;
    if (d.core_tab_n > 0 && r2 < d.s2[t]) {
        const short4 x = ext[r.x];
        u = pair_core_df<MODEL_EWALD>(p.x - h0, p.y - h1, p.z - h2, x.x - (old ? m.eo[0] : m.en[0]),
                                      x.y - (old ? m.eo[1] : m.en[1]), x.z - (old ? m.eo[2] : m.en[2]), m.q, qj, t, d);
    } else {
        u = df{pair_u<MODEL_EWALD, true>(r2, m.q, qj, t, d), 0.0f};
    }
    return old ? df_neg(u) : u;
}
// A warp's sums of its two trials; EbWalk::near empties the near queue into them.
struct EbWalk {
    const Move *m[2];
    float f;       // far pairs of the trial being walked
    df a0, a1;     // near pairs of either trial
};
template <bool CELLS>
__device__ __forceinline__ void eb_flush_near(EbQueue &q, EbWalk &w, const SysDesc &d) {
    if (!q.nn) return;   // warp-uniform
    __syncwarp();
    int which;
    const df v = eb_near(q.np, q.nm, q.nn, w.m[0], w.m[1], CELLS ? d.cell_ext : d.pos_ext, d, which);
    if (which) w.a1 = df_add(w.a1, v);
    else w.a0 = df_add(w.a0, v);
    __syncwarp();
    q.nn = 0;
}
// Evaluates n listed slots: far pairs at once, near ones into their queue.
template <bool CELLS>
__device__ __forceinline__ void eb_eval(int n, EbQueue &q, const EbFar &fm, int which, EbWalk &w, const SysDesc &d) {
    const int lane = threadIdx.x & 31;
    const Move &m = *w.m[which];
    __syncwarp();
    for (int e = 0; e < n; e += 32) {
        const bool in = e + lane < n;
        int idx = 0, t = 0;
        int4 p = make_int4(0, 0, 0, 0);
        bool nr = false;
        if (in) {
            idx = q.list[e + lane];
            p = (CELLS ? d.cell_pos : d.pos4)[idx];
            if (!d.uniform_types) t = CELLS ? d.cell_pid[idx] >> 24 : d.ptype[idx];
            const float r2n = eb_r2(p, fm.hn, fm), r2o = eb_r2(p, fm.ho, fm);
            nr = fminf(r2n, r2o) <= fm.near2;
            if (!nr) w.f += eb_far(fm, r2n, r2o, __int_as_float(p.w), m.ti * d.n_types + t, d);
            else nr = (CELLS ? d.cell_pid[idx] & 0xFFFFFF : idx) != m.i;   // itself is as near as can be
        }
        uint32_t nmask = __ballot_sync(0xffffffffu, nr);
        while (nmask) {   // warp-uniform
            if (q.nn == kEbNear) eb_flush_near<CELLS>(q, w, d);
            const int r = q.nn + __popc(nmask & ((1u << lane) - 1u));
            if (nr && r < kEbNear) {
                q.np[r] = p;
                q.nm[r] = make_int2(idx, t | which << 8);
                nr = false;
            }
            q.nn = min(q.nn + __popc(nmask), kEbNear);
            nmask = __ballot_sync(0xffffffffu, nr);
        }
    }
    __syncwarp();
}
// Up to 32 batches: batch b takes the slots from base + b step (N in all), or
// those of the cell batch q.bat[base + b].
template <bool CELLS>
__device__ __forceinline__ void eb_screen(int base, int step, int nb, EbQueue &q, const EbFar &fm, int which, EbWalk &w,
                                          const SysDesc &d) {
    constexpr int U = 4;   // batches a turn; the next turn's records are loaded meanwhile
    const int lane = threadIdx.x & 31, N = d.N;
    const int4 *const pos = (CELLS ? d.cell_pos : d.pos4) + lane;
    uint32_t mask = 0;
    int4 p[U];
    bool in[U];
    auto load = [&](int b) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            in[u] = false;
            if (b + u >= nb) continue;   // warp-uniform
            const int2 e = CELLS ? q.bat[base + b + u] : make_int2(base + (b + u) * step, N - (base + (b + u) * step));
            in[u] = lane < e.y;
            if (in[u]) p[u] = pos[e.x];
        }
    };
#pragma unroll
    for (int u = 0; u < U; u++) p[u] = make_int4(0, 0, 0, 0);
    load(0);
    for (int b = 0; b < nb; b += U) {   // warp-uniform
        bool f[U];
#pragma unroll
        for (int u = 0; u < U; u++) f[u] = in[u] && eb_r2(p[u], fm.hm, fm) <= fm.rm2;
        load(b + U);
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint32_t v = __ballot_sync(0xffffffffu, f[u]);
            if (lane == b + u) mask = v;
        }
    }
    const int first = lane >= nb ? 0 : CELLS ? q.bat[base + lane].x : base + lane * step;
    int inc = __popc(mask);
    const int own = inc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
    }
    const int total = __shfl_sync(0xffffffffu, inc, 31);
    int r = inc - own;
    for (int w0 = 0; w0 < total; w0 += kEbList) {   // warp-uniform
        while (mask && r < w0 + kEbList) {
            const int bit = 31 - __clz(mask);
            mask ^= 1u << bit;
            q.list[r - w0] = first + bit;
            r++;
        }
        eb_eval<CELLS>(min(total - w0, kEbList), q, fm, which, w, d);
    }
}

template <bool CELLS>
__device__ __forceinline__ void eb_pairs_warp(int which, EbWalk &w, const SysDesc &d, const Smem &s, EbQueue &q,
                                              float near2, int part, int nparts) {
    const Move &m = *w.m[which];
    const int lane = threadIdx.x & 31;
    // a partner within reach of the old or the new position lies within
    // reach + |d|/2 of the midpoint (a small margin covers the float rounding)
    const float reach2m = d.reach2 * 1.0001f + 1e-3f;
    const float hd = 0.5f * sqrtf(fmaf(m.dxf[0], m.dxf[0], fmaf(m.dxf[1], m.dxf[1], m.dxf[2] * m.dxf[2])));
    const float rm = sqrtf(reach2m) + hd + 1e-3f;
    EbFar fm;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        fm.ho[a] = m.ho[a];
        fm.hn[a] = m.hn[a];
        fm.hm[a] = m.ho[a] + ((int)(m.hn[a] - m.ho[a]) >> 1);
        fm.sl[a] = d.s32[a];
    }
    fm.q = m.q;
    fm.qe = d.qeqe[0];
    fm.near2 = near2;
    fm.rm2 = rm * rm;
    if (!CELLS) {
        const int N = d.N, step = 32 * nparts;
        for (int b = 32 * part; b < N; b += 32 * step) {
            const int left = nparts == 1 ? (N - b + 31) >> 5 : (N - b + step - 1) / step;
            eb_screen<CELLS>(b, step, min(left, 32), q, fm, which, w, d);
        }
        return;
    }
    // The stencil: the cells around the old cell, widened by one along each
    // axis where the particle changed cells (at most 4 x 4 x 4). Lane c (and
    // c + 32) takes stencil cell c: it drops the cell when no point of the
    // cell box lies within reach of the old or the new position, so that the
    // cell's particles cannot contribute; the remaining cells' batches are
    // listed by the warp's prefix sum over their numbers.
    int lo[3], len[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        // cell_of's coordinate
        const int co = (int)__umulhi((uint32_t)fm.ho[a] + 0x80000000u, (uint32_t)d.nc[a]);
        const int cn = (int)__umulhi((uint32_t)fm.hn[a] + 0x80000000u, (uint32_t)d.nc[a]);
        int delta = cn - co;
        if (delta > 1) delta -= d.nc[a];
        if (delta < -1) delta += d.nc[a];
        if ((delta > 1 || delta < -1) && lane == 0) atomicOr(&d.sc->error, kErrStencil);
        lo[a] = co + min(delta, 0) - 1;
        len[a] = 3 + (delta != 0 ? 1 : 0);
    }
    const int ncell = len[0] * len[1] * len[2];   // <= 64
    // reach of a cell box: squared distance (Angstrom^2) from the old and the
    // new position, on unwrapped coordinates u = h + 2^31 (the new one as the
    // old plus the minimum-image step, so that both lie on the stencil's side
    // of the box edge); a small margin covers the float rounding of the box
    // bounds (units of 2^32 / L carry ~2^8 units of rounding here)
    float uo[3], un[3], W[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        W[a] = 4294967296.0f / (float)d.nc[a];
        uo[a] = (float)((uint32_t)m.ho[a] + 0x80000000u);
        un[a] = uo[a] + (float)(int)(m.hn[a] - m.ho[a]);
    }
    int cidv[2], cntv[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int c = lane + 32 * h;
        cidv[h] = 0;
        cntv[h] = 0;
        if (c < ncell) {
            // by lengths of 3 or 4: c 171 >> 9 is c / 3 for c < 128
            const int c1 = len[0] == 4 ? c >> 2 : c * 171 >> 9, i0 = c - c1 * len[0];
            const int i2 = len[1] == 4 ? c1 >> 2 : c1 * 171 >> 9, i1 = c1 - i2 * len[1];
            const int cu[3] = {lo[0] + i0, lo[1] + i1, lo[2] + i2};
            float d2o = 0.0f, d2n = 0.0f;
            int cw[3];
#pragma unroll
            for (int a = 0; a < 3; a++) {
                const float A = (float)cu[a] * W[a], B = A + W[a];
                const float xo = fmaxf(fmaxf(A - uo[a], uo[a] - B), 0.0f) * d.s32[a];
                const float xn = fmaxf(fmaxf(A - un[a], un[a] - B), 0.0f) * d.s32[a];
                d2o = fmaf(xo, xo, d2o);
                d2n = fmaf(xn, xn, d2n);
                cw[a] = cu[a] + (cu[a] < 0 ? d.nc[a] : 0) - (cu[a] >= d.nc[a] ? d.nc[a] : 0);
            }
            cidv[h] = (cw[2] * d.nc[1] + cw[1]) * d.nc[0] + cw[0];
            if (fminf(d2o, d2n) <= reach2m) cntv[h] = s.ccount[cidv[h]];
        }
    }
    // inclusive prefix sums of the batches of the two halves
    const int nb0 = (cntv[0] + 31) >> 5, nb1 = (cntv[1] + 31) >> 5;
    int inc0 = nb0, inc1 = nb1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v0 = __shfl_up_sync(0xffffffffu, inc0, o), v1 = __shfl_up_sync(0xffffffffu, inc1, o);
        if (lane >= o) {
            inc0 += v0;
            inc1 += v1;
        }
    }
    const int tot0 = __shfl_sync(0xffffffffu, inc0, 31);
    const int total = tot0 + __shfl_sync(0xffffffffu, inc1, 31);
    // this part's: batches part, part + nparts, ...
    const int mine = nparts == 1 ? total : (total - part + nparts - 1) / nparts;
    const int st0 = inc0 - nb0 - part, st1 = tot0 + inc1 - nb1 - part;
    const int at0 = nparts == 1 ? st0 : (st0 + nparts - 1) / nparts, at1 = nparts == 1 ? st1 : (st1 + nparts - 1) / nparts;
    for (int w0 = 0; w0 < mine; w0 += kEbBatch) {   // warp-uniform
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; h++) {
            int at = (h ? at1 : at0) - w0;
            for (int x = (h ? at1 * nparts - st1 : at0 * nparts - st0); x < (h ? nb1 : nb0); x += nparts, at++)
                if (at >= 0 && at < kEbBatch) q.bat[at] = make_int2(cidv[h] * d.cap + 32 * x, cntv[h] - 32 * x);
        }
        __syncwarp();
        const int n = min(mine - w0, kEbBatch);
        for (int b = 0; b < n; b += 32) eb_screen<CELLS>(b, 0, min(n - b, 32), q, fm, which, w, d);
    }
}

// dU of trial m from one partner at high words p (charge bits in .w), type t,
// extension e, as a df number.
__device__ __forceinline__ df eb_pair(const Move &m, int4 p, int t, const short4 *e, const SysDesc &d) {
    float a = 0.0f;
    df ad = {0.0f, 0.0f};
    pair_candidate<MODEL_EWALD>(m, p, t, e, d, a, ad);
    return df_add_f(ad, a);
}

// updateAllComplexNumbers (ewald.h:388-415) inside the sweep, every
// update_frequency accepted trials (NonbondedEwald::update, ewald.h:633-640):
// Q(k) from scratch as the exact sum of every particle's integer
// contributions, compared with the running Q(k) in shared memory and adopted.
// The two agree bit for bit unless the device misbehaved (a contribution is a
// deterministic function of the fixed-point position), so the energy
// correction is zero; a difference is recorded (kErrQkMismatch where the
// system verifies) and its energy is added to the running sums, as the
// reference adds the drift it removes.
//   work split: thread t owns items t, t + blockDim, ... of the system's
//   rebuild list (rb_items: up to kRbLen values n of one (nx, ny) column, each
//   giving the k-vectors +n and -n). Per particle it forms w once (qk_w) and
//   per n the four rounded products a, r, b, c of w e_z(n) (qk_rint_bits),
//   whose sums give both contributions: (a - r, b + c) to +n and, e_z(-n)
//   being the conjugate and the rounding symmetric, (a + r, c - b) to -n;
//   term by term these are qk_term_bits' values. Particles pass through the
//   increment buffer in stages of 64 with their axis tables (8 threads build
//   one particle's table: e_x(0..kcc), e_y(-kcc..kcc), e_z(0..kcc)), stored
//   for pairs of particles so that one 16-byte load serves two; the four
//   sums run in 32 bits over a stage, then in int64 registers. The same items
//   carry the per-block Q(k) update (eb_commit_qk).
// All threads call it (block-uniform). Returns the energy correction
// (valid in thread 0) and whether any Q(k) differed.
constexpr int kRbLen = 4;
__host__ __device__ __forceinline__ int rb_tab_len(int kcc) { return 4 * kcc + 3; }
// entry t of the rebuild's axis tables: the e_x and e_y parts of qk_tab_len's
// layout, then e_z for n >= 0 only
__device__ __forceinline__ float2 rb_tab_entry(int t, int kcc, const int h[3], const float2 *__restrict__ tab) {
    return qk_tab_entry(t <= 3 * kcc + 1 ? t : t + kcc, kcc, h, tab);
}
// One stage of the rebuild for this thread's item: np particle pairs, whose
// axis tables sit as float4 {e_2p(t), e_2p+1(t)} at tab[p * T + t] (one
// 16-byte load gives an entry of both particles) and whose charges are
// q2[p]. The four sums carry 2 np kQkMagicBits (a padding particle has
// charge 0 and zero tables and adds exactly that).
template <int L>
__device__ __forceinline__ void rb_pass(const float4 *tab, int T, const float2 *q2, int np, int ix, int iy, int iz,
                                        unsigned sa[kRbLen], unsigned sr[kRbLen], unsigned sb[kRbLen],
                                        unsigned sc[kRbLen]) {
    for (int p = 0; p < np; p++) {
        const float4 *e = tab + p * T;
        const float2 q = q2[p];
        const float4 ex = e[ix], ey = e[iy];
        const float2 w0 = qk_w(q.x, make_float2(ex.x, ex.y), make_float2(ey.x, ey.y));
        const float2 w1 = qk_w(q.y, make_float2(ex.z, ex.w), make_float2(ey.z, ey.w));
#pragma unroll
        for (int u = 0; u < L; u++) {
            const float4 z = e[iz + u];
            sa[u] += qk_rint_bits(w0.x, z.x) + qk_rint_bits(w1.x, z.z);
            sr[u] += qk_rint_bits(w0.y, z.y) + qk_rint_bits(w1.y, z.w);
            sb[u] += qk_rint_bits(w0.x, z.y) + qk_rint_bits(w1.x, z.w);
            sc[u] += qk_rint_bits(w0.y, z.x) + qk_rint_bits(w1.y, z.z);
        }
    }
}
// Compare one rebuilt Q(k) (its total in the k-vector table's slot, see
// eb_rebuild) with the running value and adopt it; energy of the difference
// into e; the slot gets back its {A', Q as float, sqrt A'} from the k-vector
// array in global memory.
__device__ __forceinline__ void rb_adopt(const SysDesc &d, const EbSmem &s, int k, df &e, int &bad) {
    const longlong2 qn = reinterpret_cast<const longlong2 *>(s.b.kvec)[k];
    const longlong2 qo = s.b.qfix[k];
    const float A = d.kvec[k].w;
    const float2 fn = q_to_float(qn);
    if (qo.x != qn.x || qo.y != qn.y) {
        bad = 1;
        const float2 fo = q_to_float(qo);
        const float dre = fix28_to_float(qn.x - qo.x), dim = fix28_to_float(qn.y - qo.y);
        e = df_add_f(e, A * fmaf(dre, fo.x + fn.x, dim * (fo.y + fn.y)));
        s.b.qfix[k] = qn;
    }
    s.b.kvec[k] = make_float4(A, fn.x, fn.y, sqrtf(A));
}
__device__ __forceinline__ void rb_add(const EbSmem &s, int k, long long x, long long y) {
    longlong2 *t = reinterpret_cast<longlong2 *>(s.b.kvec) + k;
    longlong2 v = *t;
    v.x += x;
    v.y += y;
    *t = v;
}
// The int64 totals of the rebuilt Q(k) live in the k-vector table's own
// 16-byte slots (kvec[k], free while the rebuild runs: nothing else reads it
// until rb_adopt restores it), each owned by the thread of its item, so the
// thread's registers hold only the 32-bit sums of a stage.
__device__ __noinline__ bool eb_rebuild(const SysDesc &d, const EbSmem &s, df &corr) {
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31;
    const int kcc = d.kcc, T = rb_tab_len(kcc);
    // the increment buffer holds the stage's tables (pairs of particles) plus
    // kRbLen entries of headroom for the unused tail reads of rb_pass
    float4 *tab = reinterpret_cast<float4 *>(s.delta);
    const int npair = min(kEbThreads / 16, (kEbKc * kEbTrials / 2 - kRbLen) / T), stage = 2 * npair;
    float2 *q2 = reinterpret_cast<float2 *>(s.G);   // [npair], free between blocks
    const int shift = d.qk_shift;
    df e = {0.0f, 0.0f};
    int bad = 0;
    __syncthreads();   // every thread is past its last read of kvec
    for (int r0 = 0; r0 < d.n_rb_items; r0 += nt) {   // uniform over the block
        const int r = r0 + tid;
        int kp0 = 0, kn0 = 0, len = 0, n0 = 0, ix = 0, iy = 0, iz = 0;
        if (r < d.n_rb_items) {
            const int4 it = d.rb_items[r];
            kp0 = it.x & 0xFFFFFF;
            len = it.x >> 24;
            kn0 = it.y & 0xFFFFFF;
            n0 = it.y >> 24;
            ix = (int)(int8_t)(it.z & 0xFF);
            iy = 2 * kcc + 1 + (int)(int8_t)((it.z >> 8) & 0xFF);
            iz = 3 * kcc + 2 + n0;
        }
        const int wl = __reduce_max_sync(0xffffffffu, len);   // warp-uniform (items sorted by length)
        for (int u = 0; u < len; u++) {
            reinterpret_cast<longlong2 *>(s.b.kvec)[kp0 + u] = make_longlong2(0, 0);
            reinterpret_cast<longlong2 *>(s.b.kvec)[kn0 - u] = make_longlong2(0, 0);
        }
        // 8 threads per particle build its table (stage <= nt / 8); each
        // thread's particle record of the next stage is loaded during this
        // stage's sums
        const int jj = tid >> 3;
        int4 pn = make_int4(0, 0, 0, 0);
        int tn = 0;
        if (jj < min(stage, d.N)) {
            pn = d.pos4[jj];
            tn = d.ptype[jj];
        }
        for (int j0 = 0; j0 < d.N; j0 += stage) {
            const int nb = min(stage, d.N - j0), np = (nb + 1) >> 1;
            __syncthreads();   // the previous stage's tables are consumed
            float2 *tf = reinterpret_cast<float2 *>(tab);
            if (jj < 2 * np) {
                const bool live = jj < nb;
                const float qv = live ? qk_charge(__int_as_float(pn.w), d.eff[tn], d) : 0.0f;
                const int hp[3] = {pn.x, pn.y, pn.z};
                if ((tid & 7) == 0) reinterpret_cast<float *>(q2)[jj] = qv;
                for (int t = tid & 7; t < T; t += 8)
                    tf[((jj >> 1) * T + t) * 2 + (jj & 1)] =
                        live ? rb_tab_entry(t, kcc, hp, s.b.sc_tab) : make_float2(0.0f, 0.0f);
            }
            if (jj < stage && j0 + stage + jj < d.N) {
                pn = d.pos4[j0 + stage + jj];
                tn = d.ptype[j0 + stage + jj];
            }
            __syncthreads();
            if (wl > 0) {
                unsigned sa[kRbLen], sr[kRbLen], sb[kRbLen], sc[kRbLen];
#pragma unroll
                for (int u = 0; u < kRbLen; u++) sa[u] = sr[u] = sb[u] = sc[u] = 0u;
                switch (wl) {
                    case 1: rb_pass<1>(tab, T, q2, np, ix, iy, iz, sa, sr, sb, sc); break;
                    case 2: rb_pass<2>(tab, T, q2, np, ix, iy, iz, sa, sr, sb, sc); break;
                    case 3: rb_pass<3>(tab, T, q2, np, ix, iy, iz, sa, sr, sb, sc); break;
                    default: rb_pass<4>(tab, T, q2, np, ix, iy, iz, sa, sr, sb, sc); break;
                }
                // each of the four sums carries 2 np kQkMagicBits
                const unsigned off2 = 4u * (unsigned)np * kQkMagicBits;
#pragma unroll
                for (int u = 0; u < kRbLen; u++) {
                    if (u >= len) continue;
                    rb_add(s, kp0 + u, qk_widen((int)(sa[u] - sr[u]), shift),
                           qk_widen((int)(sb[u] + sc[u] - off2), shift));
                    if (n0 + u > 0)
                        rb_add(s, kn0 - u, qk_widen((int)(sa[u] + sr[u] - off2), shift),
                               qk_widen((int)(sc[u] - sb[u]), shift));
                }
            }
        }
        // compare with the running sums and adopt
        for (int u = 0; u < len; u++) {
            rb_adopt(d, s, kp0 + u, e, bad);
            if (n0 + u > 0) rb_adopt(d, s, kn0 - u, e, bad);
        }
    }
    // energy correction: warp sums, then warp 0 over the warps (fixed order)
    e = warp_sum_df(e);
    const int anybad = __syncthreads_or(bad);   // also: every thread is done with the buffers
    if (lane == 0) s.b.red[tid >> 5] = make_float2(e.hi, e.lo);
    __syncthreads();
    if (tid < 32) {
        df t = {0.0f, 0.0f};
        if (lane < (nt >> 5)) t = {s.b.red[lane].x, s.b.red[lane].y};
        corr = warp_sum_df(t);
    }
    __syncthreads();   // red is free again
    return anybad != 0;
}

// One item's differences over ng accepted trials (L values of n; the entries a
// shorter item reads past its own are dropped by the caller).
template <int L>
__device__ __forceinline__ void cq_pass(const float4 *tab, int T, const float *qg, int ng, int ix, int iy, int iz,
                                        unsigned da[kRbLen], unsigned dr[kRbLen], unsigned db[kRbLen],
                                        unsigned dc[kRbLen]) {
#pragma unroll 2
    for (int g = 0; g < ng; g++) {
        const float4 *e = tab + g * T;
        const float q2g = qg[g];
        const float4 ex = e[ix], ey = e[iy];
        const float2 wn = qk_w(q2g, make_float2(ex.x, ex.y), make_float2(ey.x, ey.y));
        const float2 wo = qk_w(q2g, make_float2(ex.z, ex.w), make_float2(ey.z, ey.w));
#pragma unroll
        for (int u = 0; u < L; u++) {
            const float4 z = e[iz + u];
            da[u] += qk_rint_bits(wn.x, z.x) - qk_rint_bits(wo.x, z.z);
            dr[u] += qk_rint_bits(wn.y, z.y) - qk_rint_bits(wo.y, z.w);
            db[u] += qk_rint_bits(wn.x, z.y) - qk_rint_bits(wo.x, z.w);
            dc[u] += qk_rint_bits(wn.y, z.x) - qk_rint_bits(wo.y, z.z);
        }
    }
}
// Adds an item's differences to its k-vectors' Q(k).
__device__ __forceinline__ void eb_commit_item(const EbSmem &s, int kp0, int kn0, int n0, int len, int shift,
                                               const unsigned da[kRbLen], const unsigned dr[kRbLen],
                                               const unsigned db[kRbLen], const unsigned dc[kRbLen]) {
#pragma unroll
    for (int u = 0; u < kRbLen; u++) {
        if (u >= len) continue;
        // +n: (a - r, b + c); -n: (a + r, c - b)
        longlong2 q = s.b.qfix[kp0 + u];
        q.x += qk_widen((int)(da[u] - dr[u]), shift);
        q.y += qk_widen((int)(db[u] + dc[u]), shift);
        s.b.qfix[kp0 + u] = q;
        float2 qf = q_to_float(q);
        s.b.kvec[kp0 + u].y = qf.x;
        s.b.kvec[kp0 + u].z = qf.y;
        if (n0 + u > 0) {
            q = s.b.qfix[kn0 - u];
            q.x += qk_widen((int)(da[u] + dr[u]), shift);
            q.y += qk_widen((int)(dc[u] - db[u]), shift);
            s.b.qfix[kn0 - u] = q;
            qf = q_to_float(q);
            s.b.kvec[kn0 - u].y = qf.x;
            s.b.kvec[kn0 - u].z = qf.y;
        }
    }
}
// Q(k) after a block: every accepted trial a adds c_k(new_a) - c_k(old_a)
// (ewald.h:665-705). Threads qt = 0..nq-1 (warps 1.. of the CTA, which
// synchronise among themselves on named barrier 1) own the rebuild's items
// (rb_items): per accepted trial they form w once for the new and the old
// position and, per n of the item, the four rounded products of each (the
// same integers the rebuild sums), accumulate the differences in 32 bits over
// the block's trials (at most 32 x 2^23) and add them to the exact int64 Q(k)
// of the item's (+n, -n) k-vectors at the end; integer sums, so the order of
// the trials does not matter. The axis tables of the accepted trials'
// new and old positions sit in the increment buffer as float4
// {new.re, new.im, old.re, old.im}, trial-major (tab[g * T + t]).
// On a cluster the CTA takes its own items [i0, i1), whose k-vectors it holds
// from k0 on (shared-memory index = k - k0).
__device__ __noinline__ void eb_commit_qk(const SysDesc &d, const EbSmem &s, uint32_t live, int qt, int nq, int i0,
                                          int i1, int k0) {
    int *alist = reinterpret_cast<int *>(s.corr);   // free after the resolution
    float *qg = s.G;                                // [32], free after the resolution
    if (qt < kEbTrials && ((live >> qt) & 1u)) {
        const int g = __popc(live & ((1u << qt) - 1u));
        alist[g] = qt;
        const Move &A = s.mv[qt];
        qg[g] = qk_charge(A.q, d.eff[A.ti], d);
    }
    const int na = __popc(live);
    const int kcc = d.kcc, T = rb_tab_len(kcc);
    float4 *tab = reinterpret_cast<float4 *>(s.delta);
    const int gmax = min(kEbTrials, (kEbKc * kEbTrials / 2 - kRbLen) / T);
    const int shift = d.qk_shift;
    for (int g0 = 0; g0 < na; g0 += gmax) {
        const int ng = min(gmax, na - g0);
        eb_qbar(nq);   // list written; the previous group's tables consumed
        for (int e = qt; e < ng * T; e += nq) {
            const int g = e / T, t = e - g * T;
            const Move &A = s.mv[alist[g0 + g]];
            const float2 en = rb_tab_entry(t, kcc, A.hn, s.b.sc_tab), eo = rb_tab_entry(t, kcc, A.ho, s.b.sc_tab);
            tab[e] = make_float4(en.x, en.y, eo.x, eo.y);
        }
        eb_qbar(nq);
        for (int r = i0 + qt; r < i1; r += nq) {
            const int4 it = d.rb_items[r];
            const int kp0 = (it.x & 0xFFFFFF) - k0, len = it.x >> 24, kn0 = (it.y & 0xFFFFFF) - k0, n0 = it.y >> 24;
            const int ix = (int)(int8_t)(it.z & 0xFF), iy = 2 * kcc + 1 + (int)(int8_t)((it.z >> 8) & 0xFF);
            const int iz = 3 * kcc + 2 + n0;
            unsigned da[kRbLen], dr[kRbLen], db[kRbLen], dc[kRbLen];
#pragma unroll
            for (int u = 0; u < kRbLen; u++) da[u] = dr[u] = db[u] = dc[u] = 0u;
            switch (__reduce_max_sync(__activemask(), len)) {   // items are sorted by length
                case 1: cq_pass<1>(tab, T, qg + g0, ng, ix, iy, iz, da, dr, db, dc); break;
                case 2: cq_pass<2>(tab, T, qg + g0, ng, ix, iy, iz, da, dr, db, dc); break;
                case 3: cq_pass<3>(tab, T, qg + g0, ng, ix, iy, iz, da, dr, db, dc); break;
                default: cq_pass<4>(tab, T, qg + g0, ng, ix, iy, iz, da, dr, db, dc); break;
            }
            eb_commit_item(s, kp0, kn0, n0, len, shift, da, dr, db, dc);
        }
    }
}

// Accepted trial: master and pair coordinates, and (in_cell: the particle
// stays in its cell) its record in the cell's slot array. Independent for
// distinct particles.
__device__ __forceinline__ void eb_commit_position(const Move &m, const SysDesc &d, const Smem &s, bool in_cell) {
    const int4 rec = make_int4(m.hn[0], m.hn[1], m.hn[2], __float_as_int(m.q));
    const short4 ext = make_short4((short)m.en[0], (short)m.en[1], (short)m.en[2], 0);
    d.pos64[3 * m.i + 0] = m.xn[0];
    d.pos64[3 * m.i + 1] = m.xn[1];
    d.pos64[3 * m.i + 2] = m.xn[2];
    d.pos4[m.i] = rec;
    d.pos_ext[m.i] = ext;
    if (d.use_cells && in_cell) {
        const int slot = (int)(s.pcs[m.i] & 0xFFFu);
        d.cell_pos[m.co * d.cap + slot] = rec;
        d.cell_ext[m.co * d.cap + slot] = ext;
    }
}
// A particle that changed cells: out of the old cell (the cell's last slot
// fills the hole) and into the next free slot of the new one, as
// commit_position does. One thread, accepted trials in order.
__device__ __forceinline__ void eb_cell_move(const Move &m, const SysDesc &d, const Smem &s) {
    const int4 rec = make_int4(m.hn[0], m.hn[1], m.hn[2], __float_as_int(m.q));
    const short4 ext = make_short4((short)m.en[0], (short)m.en[1], (short)m.en[2], 0);
    const int slot = (int)(s.pcs[m.i] & 0xFFFu);
    const int last = s.ccount[m.co] - 1;
    if (last != slot) {
        const int src = m.co * d.cap + last, dst = m.co * d.cap + slot;
        const int pid = d.cell_pid[src];
        d.cell_pos[dst] = d.cell_pos[src];
        d.cell_ext[dst] = d.cell_ext[src];
        d.cell_pid[dst] = pid;
        s.pcs[pid & 0xFFFFFF] = ((uint32_t)m.co << 12) | (uint32_t)slot;
    }
    s.ccount[m.co] = last;
    int ns = s.ccount[m.cn];
    if (ns >= d.cap) {
        d.sc->error |= kErrCellOverflow;
        ns = d.cap - 1;
    } else {
        s.ccount[m.cn] = ns + 1;
    }
    d.cell_pos[m.cn * d.cap + ns] = rec;
    d.cell_ext[m.cn * d.cap + ns] = ext;
    d.cell_pid[m.cn * d.cap + ns] = m.i | (m.ti << 24);
    s.pcs[m.i] = ((uint32_t)m.cn << 12) | (uint32_t)ns;
}

// The cell counts alone of eb_cell_move: the other CTAs of a cluster keep
// their own copy for their stencil walks.
__device__ __forceinline__ void eb_cell_count_move(const Move &m, const SysDesc &d, const Smem &s) {
    s.ccount[m.co] -= 1;
    const int ns = s.ccount[m.cn];
    if (ns < d.cap) s.ccount[m.cn] = ns + 1;
}

// Surface dipole change of a trial (Angstrom e), as surface_delta computes it.
__device__ __forceinline__ void eb_dM(const Move &m, const SysDesc &d, float dM[3]) {
    const float qe = m.q * d.eff[m.ti];
#pragma unroll
    for (int a = 0; a < 3; a++) dM[a] = qe * ((float)m.hn[a] * d.s32[a] - (float)m.ho[a] * d.s32[a]);
}

// CLUSTER: one system on a thread-block cluster of C = eb_ctas CTAs (a
// system alone, where one CTA would leave the other SMs idle). CTA r holds
// the k-vectors [k0, k1) and their Q(k) (eb_ranges[r]) and runs the k-steps of
// its own k-vectors, a 1/C share of the correction pairs and the real-space
// walks of its warps (trial m in C/2 parts over the cluster's 16 C warps);
// its partial sums go into CTA 0's shared memory (remote stores), and after a
// cluster barrier CTA 0 alone completes the sums and resolves the block, and
// hands the outcome to every CTA. Then CTA 0 writes the positions and cell
// lists to global memory, every CTA updates its own Q(k) and cell counts, and
// a cluster barrier makes the new positions visible to the whole cluster
// before the next block reads them. A rebuild ends the launch (the rebuild
// kernel takes it, as for any system alone). The sums run in another order
// than on one CTA, so the dU agree to rounding, not bit for bit.
template <bool CELLS, bool CLUSTER>
__global__ void __launch_bounds__(kEbThreads, 1) ewald_block_kernel(const SysDesc *__restrict__ descs, int64_t end,
                                                                    const float2 *__restrict__ sc_tab) {
    extern __shared__ __align__(16) char eb_smem_raw[];
    __shared__ __align__(16) SysDesc sd;
    const int C = CLUSTER ? (int)blk_cluster_size() : 1;
    const int rank = CLUSTER ? (int)blk_cluster_rank() : 0;
    load_desc(sd, descs + (CLUSTER ? blockIdx.x / C : blockIdx.x));
    const SysDesc &d = sd;
    EbSmem s = eb_carve(eb_smem_raw, d, CELLS);
    SysScalars *sc = d.sc;
    // the work split (16 threads per trial in the sums, two walks a warp) is
    // written for exactly kEbThreads threads; a cluster must match the
    // system's k-vector split (the same for every CTA of the cluster)
    if (blockDim.x != kEbThreads || (CLUSTER ? C != d.eb_ctas || C > kEbMaxCluster : d.eb_ctas != 1)) {
        if (threadIdx.x == 0) atomicOr(&sc->error, kErrLaunch);
        return;
    }
    if (sc->rebuild_pending || sc->cursor >= min(end, sc->n_trials)) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
    // this CTA's k-vectors [k0, k0 + K) and rebuild items [i0, i1)
    int k0 = 0, K = d.K, i0 = 0, i1 = d.n_rb_items;
    if (CLUSTER) {
        const int4 rg = d.eb_ranges[rank];
        k0 = rg.x;
        K = rg.y - rg.x;
        i0 = rg.z;
        i1 = rg.w;
    }
    // tables
    for (int t = tid; t < 256; t += blockDim.x) s.b.sc_tab[t] = sc_tab[t];
    for (int k = tid; k < K; k += blockDim.x) {
        const longlong2 q = d.qfix[k0 + k];
        const float2 qf = q_to_float(q);
        const float A = d.kvec[k0 + k].w;
        s.b.kvec[k] = make_float4(A, qf.x, qf.y, sqrtf(A));
        s.b.kpack[k] = d.kpack[k0 + k];
        s.b.qfix[k] = q;
    }
    // pi / L per axis: k.d / 2 = sum_a n_a (pi / L_a) d_a
    const float hpl[3] = {3.141592653589793f / d.L[0], 3.141592653589793f / d.L[1], 3.141592653589793f / d.L[2]};
    if (CELLS) {
        const int ncell = d.nc[0] * d.nc[1] * d.nc[2];
        for (int c = tid; c < ncell; c += blockDim.x) s.b.ccount[c] = d.cell_count[c];
        for (int j = tid; j < d.N; j += blockDim.x)
            s.b.pcs[j] = ((uint32_t)d.p_cell[j] << 12) | (uint32_t)d.p_slot[j];
    }
    // (1.5 sigma)^2 of the largest pair: pair_candidate's careful path (near)
    float near2 = d.s2[0];
    for (int t = 1; t < d.n_types * d.n_types; t++) near2 = fmaxf(near2, d.s2[t]);
    near2 *= 2.25f;
    if (tid < 3) s.Mdf[tid] = make_float2(sc->m[tid][0], sc->m[tid][1]);
    if (CLUSTER) blk_cluster_barrier();   // every CTA of the cluster runs before any remote store
    else __syncthreads();
    int64_t cur = sc->cursor;
    const int64_t stop = min(end, sc->n_trials);
    df U = {sc->u_hi, sc->u_lo};
    df Ut = {sc->utot_hi, sc->utot_lo};
    int cnt_acc = sc->cnt_accepted;
    int64_t nacc = sc->n_accepted;
    const int uf = d.update_frequency;
    bool rebuild = false;
    int err = 0;
    // k space: warp w takes the k-steps (4 k-vectors) w, w + 16, ...; lane
    // (gq, gt) holds the Gram fragments of trials gq + 8 r, components gt and
    // gt + 4 of the step (eb_gram_regs)
    const int gq = lane >> 2, gt = lane & 3, gh = gt & 1, gk = gt >> 1;
    // per-trial records of the k-space phase (in the increment buffer, past
    // the real-space queues): {d pi/L, 2 q eff}, {high words of the step's midpoint, fast}
    float4 *rA = reinterpret_cast<float4 *>(reinterpret_cast<char *>(s.delta) + kEbRecords);
    int4 *rB = reinterpret_cast<int4 *>(rA + kEbTrials);
    Trial next{};
    if (warp == 0 && cur + lane < stop) next = d.trials[cur + lane];
    while (cur < stop) {
        const int kb = (int)((stop - cur) < (int64_t)kEbTrials ? (stop - cur) : (int64_t)kEbTrials);
        // ---- trials of the block (old coordinates: the block start)
        if (warp == 0) {   // lane m: trial m
            float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            int4 b = make_int4(0, 0, 0, 1);
            int i = -1 - lane;
            if (lane < kb) {
                const Trial tr = next;   // loaded when the previous block was resolved
                int64_t xo[3], xn[3];
#pragma unroll
                for (int x = 0; x < 3; x++) {
                    xo[x] = d.pos64[3 * tr.idx + x];
                    xn[x] = (int64_t)((uint64_t)xo[x] + (uint64_t)tr.d[x]);
                }
                Move m;
                move_setup(m, tr.idx, xo, xn, __int_as_float(d.pos4[tr.idx].w), d.ptype[tr.idx], d);
                s.mv[lane] = m;
                i = m.i;
                df thr = {tr.thr_hi, tr.thr_lo};
                if (d.kT != 1.0f) thr = dfm_f(thr, d.kT);
                s.thr[lane] = make_float2(thr.hi, thr.lo);
                a = make_float4(m.dxf[0] * hpl[0], m.dxf[1] * hpl[1], m.dxf[2] * hpl[2], 2.0f * m.q * d.eff[m.ti]);
                // |k.d| / 2 <= kcc (|d_x| + |d_y| + |d_z|) pi/L: within the Taylor
                // range of eb_sin every k takes the branch-free path
                const bool fast = (float)d.kcc * (fabsf(a.x) + fabsf(a.y) + fabsf(a.z)) <= 0.8f;
                b = make_int4(m.ho[0] + ((int)(m.hn[0] - m.ho[0]) >> 1), m.ho[1] + ((int)(m.hn[1] - m.ho[1]) >> 1),
                              m.ho[2] + ((int)(m.hn[2] - m.ho[2]) >> 1), fast ? 1 : 0);
            }
            s.col[lane] = __match_any_sync(0xffffffffu, i) & ((1u << lane) - 1u);   // earlier trials on its particle
            rA[lane] = a;
            rB[lane] = b;
        }
        // the k-space records are the last shared input of the phases below:
        // from here each warp runs its corrections, its real-space walks and
        // its k-steps back to back, with no barrier between them (a warp
        // done walking early starts on k space)
        __syncthreads();
        // ---- real-space and surface corrections c(a, m), a < m: the
        // kb (kb - 1) / 2 pairs (cluster: a 1/C share per CTA, into CTA 0's
        // table), two lanes each, one for a's new and one for its old position
        {
            const int np = 2 * ((kb * (kb - 1) / 2 + C - 1 - rank) / C);
            for (int ub = warp * 32; ub < np; ub += blockDim.x) {   // warp-uniform
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
                const Move &A = s.mv[a];
                const Move &Mm = s.mv[m];
                if (u < np && A.i != Mm.i) {
                    const bool old = u & 1;
                    const int4 pj = make_int4(old ? A.ho[0] : A.hn[0], old ? A.ho[1] : A.hn[1], old ? A.ho[2] : A.hn[2],
                                              __float_as_int(A.q));
                    const short4 ext = make_short4((short)(old ? A.eo[0] : A.en[0]), (short)(old ? A.eo[1] : A.en[1]),
                                                   (short)(old ? A.eo[2] : A.en[2]), 0);
                    v = eb_pair(Mm, pj, A.ti, &ext, d);
                    if (!old && d.surf_c != 0.0f) {
                        float da[3], dm[3];
                        eb_dM(A, d, da);
                        eb_dM(Mm, d, dm);
                        v = df_add_f(v, 2.0f * d.surf_c * fmaf(da[0], dm[0], fmaf(da[1], dm[1], da[2] * dm[2])));
                    }
                }
                const df w = {__shfl_xor_sync(0xffffffffu, v.hi, 1), __shfl_xor_sync(0xffffffffu, v.lo, 1)};
                if (u < np && !(u & 1)) {
                    df c = df_add(v, df_neg(w));
                    if (!(fabsf(c.hi) <= kEbLargeCorr)) c.hi = __int_as_float(0x7FFFFFFF);
                    float2 *to = &s.corr[a * kEbTrials + m];
                    if (CLUSTER) eb_st_remote(to, 0, make_float2(c.hi, c.lo));
                    else *to = make_float2(c.hi, c.lo);
                }
            }
        }
        // ---- real-space base: warp w sums trials w, w + nwarp, ...; its
        // candidate queue lives in the (not yet used) increment buffer. On a
        // cluster warp g = 16 r + w of the cluster takes part g % P of trial
        // g / P (P = C / 2 parts per trial), into CTA 0's part table.
        {
            const int P = CLUSTER ? (C + 1) / 2 : 1;
            const int u0 = CLUSTER ? rank * nwarp + warp : warp, du = CLUSTER ? C * nwarp : nwarp;
            EbQueue q = eb_queue(reinterpret_cast<char *>(s.delta) + warp * kEbQueueBytes);
            EbWalk w{{s.mv + min(u0 / P, kb - 1), s.mv + min((u0 + du) / P, kb - 1)}, 0.0f, {0.0f, 0.0f}, {0.0f, 0.0f}};
            float f0 = 0.0f;   // at most two walks a warp: kb P <= 2 du
#pragma unroll 1
            for (int h = 0; h < 2; h++) {
                const int u = u0 + h * du;
                f0 = h ? w.f : 0.0f;
                w.f = 0.0f;
                if (u < kb * P) eb_pairs_warp<CELLS>(h, w, d, s.b, q, near2, u % P, P);
            }
            eb_flush_near<CELLS>(q, w, d);
            // both sums in one tree, the half-warps exchanging first
            const df p0 = df_add_f(w.a0, f0), p1 = df_add_f(w.a1, w.f);
            const bool hi = lane >= 16;
            df v = hi ? p1 : p0;
            const df o = hi ? p0 : p1;
            v = df_add(v, df{__shfl_xor_sync(0xffffffffu, o.hi, 16), __shfl_xor_sync(0xffffffffu, o.lo, 16)});
#pragma unroll
            for (int x = 8; x > 0; x >>= 1)
                v = df_add(v, df{__shfl_xor_sync(0xffffffffu, v.hi, x), __shfl_xor_sync(0xffffffffu, v.lo, x)});
            const int u = u0 + (lane >> 4) * du;
            if ((lane & 15) == 0 && u < kb * P) {
                const float2 p = make_float2(v.hi, v.lo);
                if (CLUSTER) eb_st_remote(&s.xreal[u], 0, p);
                else s.partR[u] = p;
            }
        }
        // ---- reciprocal base and Gram matrix. Lane (gq, gt) and its partner
        // lane ^ 1 need the same increments sqrt(A') D[trial][k] (trials
        // gq + 8 r, k-vectors 4 st + gk and 4 st + 2 + gk), one the real and
        // one the imaginary part: each computes half (r = 2 gh, 2 gh + 1) and
        // they swap the other part. No chunk buffer, no barriers in the loop.
        float kac[2] = {0.0f, 0.0f};   // reciprocal base of trials gq + 8 (2 gh + rr)
        float gc[6][4];
#pragma unroll
        for (int x = 0; x < 6; x++)
#pragma unroll
            for (int y = 0; y < 4; y++) gc[x][y] = 0.0f;
        for (int st = warp; 4 * st < K; st += kEbThreads / 32) {
            float xf[4][2];   // component gh of sqrt(A') D[gq + 8 r][k_j]
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const int kraw = 4 * st + 2 * j + gk;
                const int k = min(kraw, K - 1);
                int nx, ny, nz;
                unpack_n(s.b.kpack[k], nx, ny, nz);
                const float4 kv = s.b.kvec[k];   // {A', Re Q, Im Q, sqrt A'}
                const float fx = small_int_to_float(nx), fy = small_int_to_float(ny), fz = small_int_to_float(nz);
#pragma unroll
                for (int rr = 0; rr < 2; rr++) {
                    const int t = gq + 8 * (2 * gh + rr);
                    const float4 a = rA[t];
                    const int4 b = rB[t];
                    // D = q (e^{ik.r_new} - e^{ik.r_old}) = 2 q sin(k.d / 2) i e^{ik.r_mid}
                    const int hm[3] = {b.x, b.y, b.z};
                    float2 e = sincos_turns(phase(nx, ny, nz, hm), s.b.sc_tab);
                    const float half = fmaf(fx, a.x, fmaf(fy, a.y, fz * a.z));
                    float sn = eb_sin(half);
                    if (!b.w && fabsf(half) > 0.8f) {   // a long step: both angles from the exact phases
                        const Move &M = s.mv[t];
                        const uint32_t po = phase(nx, ny, nz, M.ho);
                        const int32_t hp = (int32_t)(phase(nx, ny, nz, M.hn) - po) >> 1;
                        e = sincos_turns(po + (uint32_t)hp, s.b.sc_tab);
                        sn = sincos_turns((uint32_t)hp, s.b.sc_tab).y;
                    }
                    const float amp = (kraw < K ? a.w : 0.0f) * sn;   // 0 past K and for idle trials
                    const float2 dd = make_float2(-amp * e.y, amp * e.x);
                    kac[rr] = fmaf(kv.x, fmaf(2.0f, fmaf(kv.y, dd.x, kv.z * dd.y), amp * amp), kac[rr]);
                    const float own = (gh ? dd.y : dd.x) * kv.w, other = (gh ? dd.x : dd.y) * kv.w;
                    const float recv = __shfl_xor_sync(0xffffffffu, other, 1);
                    xf[rr][j] = gh ? recv : own;
                    xf[2 + rr][j] = gh ? own : recv;
                }
            }
            eb_gram_regs(xf, gc);
        }
        // reciprocal base per trial: partials of (warp, lane, rr) summed in a
        // fixed order in df
        float *KP = reinterpret_cast<float *>(reinterpret_cast<char *>(s.delta) + 28672);   // [16][32][2]
        KP[(warp * 32 + lane) * 2] = kac[0];
        KP[(warp * 32 + lane) * 2 + 1] = kac[1];
        // Gram: the 16 warps' partial tiles meet in the (now free) increment
        // buffer in two rounds and are summed in a fixed order, so the result
        // does not depend on timing
        __syncthreads();
        float *P = reinterpret_cast<float *>(s.delta);   // [8 slots][6 tiles][32 lanes][4]
        {
            const int nw = kEbThreads / 32, slot = warp % (nw / 2);
            float *q = P + slot * (6 * 32 * 4) + lane * 4;
            if (warp < nw / 2) {
#pragma unroll
                for (int x = 0; x < 6; x++)
                    *reinterpret_cast<float4 *>(q + x * 128) = make_float4(gc[x][0], gc[x][1], gc[x][2], gc[x][3]);
            }
            {
                // warp w sums trials w and w + 16 over their 32 partials (16
                // warps, gk' = 0, 1) in one tree, the half-warps exchanging
                // first. Trial t = gq' + 8 r': lanes gq' * 4 + (r' >> 1) + 2 gk',
                // slot rr = r' & 1
                auto part = [&](int t) {
                    const int tq = t & 7, tr = t >> 3;
                    return KP[((lane >> 1) * 32 + tq * 4 + (tr >> 1) + 2 * (lane & 1)) * 2 + (tr & 1)];
                };
                const float p0 = part(warp), p1 = part(warp + 16);
                const bool hi = lane >= 16;
                df v = two_sum(hi ? p1 : p0, __shfl_xor_sync(0xffffffffu, hi ? p0 : p1, 16));
#pragma unroll
                for (int o = 8; o > 0; o >>= 1)
                    v = df_add(v, df{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)});
                if ((lane & 15) == 0) {
                    const int t = warp + lane;
                    if (CLUSTER) eb_st_remote(&s.xkbase[rank * kEbTrials + t], 0, make_float2(v.hi, v.lo));
                    else s.kbase[t] = make_float2(v.hi, v.lo);
                }
            }
            __syncthreads();
            if (warp >= nw / 2) {
#pragma unroll
                for (int x = 0; x < 6; x++) {
                    float4 v = *reinterpret_cast<float4 *>(q + x * 128);
                    v.x += gc[x][0];
                    v.y += gc[x][1];
                    v.z += gc[x][2];
                    v.w += gc[x][3];
                    *reinterpret_cast<float4 *>(q + x * 128) = v;
                }
            }
            __syncthreads();
            // element e = (tile, lane, j) of the accumulator layout
            for (int e = tid; e < kEbGramN; e += blockDim.x) {
                float v = 0.0f;
                for (int sl = 0; sl < nw / 2; sl++) v += P[sl * kEbGramN + e];
                if (CLUSTER) {   // CTA 0 adds the ranks' sums up below
                    eb_st_remote(&s.xgram[rank * kEbGramN + e], 0, v);
                    continue;
                }
                const int x = e >> 7, ln = (e >> 2) & 31, j = e & 3;
                const int mi = x < 4 ? 0 : 1, nj = x < 4 ? x : x - 2;
                const int row = 16 * mi + (ln >> 2) + ((j & 2) ? 8 : 0);
                const int col = 8 * nj + 2 * (ln & 3) + (j & 1);
                // one correction per pair (a, m): real space + surface + reciprocal
                const float2 c = s.corr[row * kEbTrials + col];
                const df cs = df_add_f(df{c.x, c.y}, 2.0f * v);
                s.corr[row * kEbTrials + col] = make_float2(cs.hi, cs.lo);
            }
        }
        if (CLUSTER) {
            // every CTA's partial sums are in CTA 0: it completes them in a
            // fixed order (ranks, parts)
            blk_cluster_barrier();
            if (rank == 0) {
                for (int e = tid; e < kEbGramN; e += blockDim.x) {
                    float v = 0.0f;
#pragma unroll
                    for (int r = 0; r < kEbMaxCluster; r++)   // all loads in flight at once
                        if (r < C) v += s.xgram[r * kEbGramN + e];
                    const int x = e >> 7, ln = (e >> 2) & 31, j = e & 3;
                    const int mi = x < 4 ? 0 : 1, nj = x < 4 ? x : x - 2;
                    const int row = 16 * mi + (ln >> 2) + ((j & 2) ? 8 : 0);
                    const int col = 8 * nj + 2 * (ln & 3) + (j & 1);
                    const float2 c = s.corr[row * kEbTrials + col];
                    const df cs = df_add_f(df{c.x, c.y}, 2.0f * v);
                    s.corr[row * kEbTrials + col] = make_float2(cs.hi, cs.lo);
                }
                // 16 threads per trial: one per rank and part, in one tree each
                const int t = tid >> 4, r = tid & 15, P = (C + 1) / 2;
                const float2 x = r < C ? s.xkbase[r * kEbTrials + t] : make_float2(0.0f, 0.0f);
                const float2 y = r < P && t < kb ? s.xreal[t * P + r] : make_float2(0.0f, 0.0f);
                df kv = {x.x, x.y}, rv = {y.x, y.y};
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) {
                    kv = df_add(kv, df{__shfl_xor_sync(0xffffffffu, kv.hi, o), __shfl_xor_sync(0xffffffffu, kv.lo, o)});
                    rv = df_add(rv, df{__shfl_xor_sync(0xffffffffu, rv.hi, o), __shfl_xor_sync(0xffffffffu, rv.lo, o)});
                }
                if (r == 0) {
                    s.kbase[t] = make_float2(kv.hi, kv.lo);
                    s.partR[t] = make_float2(rv.hi, rv.lo);
                }
            }
        }
        __syncthreads();
        // ---- resolve the block in order (warp 0 of CTA 0; lane m = trial m)
        if (warp == 0 && rank == 0) {
            df S = {0.0f, 0.0f};
            float dMl[3] = {0.0f, 0.0f, 0.0f};
            if (lane < kb) {
                const float2 r = s.partR[lane], kk = s.kbase[lane];
                S = df_add(df{r.x, r.y}, df{kk.x, kk.y});
                const df Mb[3] = {{s.Mdf[0].x, s.Mdf[0].y}, {s.Mdf[1].x, s.Mdf[1].y}, {s.Mdf[2].x, s.Mdf[2].y}};
                S = df_add(S, surface_delta(s.mv[lane], d, Mb, dMl));
            }
            const uint32_t colm = lane < kb ? s.col[lane] : 0u;
            const float2 th = lane < kb ? s.thr[lane] : make_float2(0.0f, 0.0f);
            uint32_t accm = 0;
            int done = kb;
            // NonbondedEwald::update (ewald.h:633): a rebuild after
            // update_frequency accepted trials ends the block there
            const int every = max(uf, 1), left = d.skip_rebuild ? 64 : max(every - cnt_acc, 1);
            // Lane a decides: its S already holds the corrections of every
            // accepted trial before it in the block. Movebase::metropolis
            // (move.h:567-573): reject iff dU > kT (-ln u); a NaN dU compares
            // false there: accepted. Every lane forms its flag and the sum it
            // would go on with; bit a of the flags' ballot selects. A step is
            // that chain alone, without a branch (180 -> 85 cycles): where the
            // block ends is found afterwards, the sums of the trials before that
            // not depending on the later ones.
            float2 cn = s.corr[lane];
#pragma unroll 4
            for (int a = 0; a < kb; a++) {
                const float2 c = cn;
                cn = s.corr[min(a + 1, kEbTrials - 1) * kEbTrials + lane];
                const df Sc = df_add_quick(S, df{c.x, c.y});
                const bool gt = S.hi > th.x || (S.hi == th.x && S.lo > th.y);
                const uint32_t ok = __ballot_sync(0xffffffffu, !gt) & (1u << a);
                accm |= ok;
                const bool add = ok && lane > a;
                S.hi = add ? Sc.hi : S.hi;
                S.lo = add ? Sc.lo : S.lo;
            }
            // a trial whose particle an accepted one moved ends the block, and so does kEbLargeCorr
            const bool nan = lane > 0 && lane < kb && !(S.hi == S.hi);
            const uint32_t again = __ballot_sync(0xffffffffu, (colm & accm) != 0u || nan);
            if (again) done = __ffs(again) - 1;
            if (done < 32) accm &= (1u << done) - 1u;
            if (__popc(accm) >= left) {   // and so does the accepted one that makes a rebuild due
                rebuild = true;
                done = (int)__fns(accm, 0, left) + 1;
                if (done < 32) accm &= (1u << done) - 1u;
            }
            nacc += __popc(accm);
            cnt_acc = rebuild ? 0 : (cnt_acc + __popc(accm)) % every;
            if (__any_sync(0xffffffffu, lane < done && !(S.hi == S.hi))) err |= kErrNonFinite;
            // lane m's S is trial m's dU as decided: log it, and add the
            // accepted ones to the running sums (a fixed-order warp sum)
            const bool take = lane < done && ((accm >> lane) & 1u);
            if (d.log_trials && lane < done) {
                d.trial_du[cur + lane] = make_float2(S.hi, S.lo);
                d.trial_acc[cur + lane] = take ? 1 : 0;
            }
            const df sum = warp_sum_df(take ? S : df{0.0f, 0.0f});
            U = df_add(U, sum);
            Ut = df_add(Ut, sum);
            if (lane == 0) {
                s.info[0] = done;
                s.info[1] = (int)accm;
                s.info[2] = rebuild ? 1 : 0;
                s.info[3] = cnt_acc;
            }
            if (CLUSTER && lane > 0 && lane < C) {   // the outcome, to the other CTAs
                eb_st_remote(&s.info[0], lane, done);
                eb_st_remote(&s.info[1], lane, (int)accm);
                eb_st_remote(&s.info[2], lane, rebuild ? 1 : 0);
                eb_st_remote(&s.info[3], lane, cnt_acc);
            }
        }
        if (CLUSTER) blk_cluster_barrier();
        else __syncthreads();
        const int done = s.info[0];
        const uint32_t accm = (uint32_t)s.info[1];
        rebuild = s.info[2] != 0;
        cnt_acc = s.info[3];
        if (warp == 0 && cur + done + lane < stop) next = d.trials[cur + done + lane];
        // ---- apply the accepted trials. Warp 0 commits the positions and
        // cell lists while warps 1.. update Q(k), synchronising among
        // themselves on named barrier 1; the block barrier below joins the two.
        const uint32_t live = accm & ((done >= 32) ? 0xffffffffu : ((1u << done) - 1u));
        if (warp == 0 && rank != 0) {
            // the other CTAs of a cluster: their cell counts alone
            if (CELLS && lane == 0)
                for (int a = 0; a < done; a++)
                    if (((accm >> a) & 1u) && s.mv[a].cn != s.mv[a].co) eb_cell_count_move(s.mv[a], d, s.b);
        } else if (warp == 0) {
            // positions (and, for a particle that stays in its
            // cell record) of the accepted trials, one lane each: the
            // particles are distinct; then lane 0 moves, in order, the
            // particles that changed cells
            const bool mine = (live >> lane) & 1u;
            bool mover = false;
            if (mine) {
                const Move &A = s.mv[lane];
                mover = CELLS && A.cn != A.co;
                eb_commit_position(A, d, s.b, !mover);
            }
            const uint32_t movers = __ballot_sync(0xffffffffu, mover);
            __syncwarp();   // the lanes' records are visible to lane 0
            if (lane == 0)
                for (uint32_t left = movers; left; left &= left - 1) eb_cell_move(s.mv[__ffs(left) - 1], d, s.b);
            // M: the accepted changes in one tree
            float dm[3] = {0.0f, 0.0f, 0.0f};
            if (mine) eb_dM(s.mv[lane], d, dm);
            df M[3];
#pragma unroll
            for (int x = 0; x < 3; x++) M[x] = warp_sum_df(df{dm[x], 0.0f});
            if (lane < 3) {
                const df v = lane == 0 ? M[0] : lane == 1 ? M[1] : M[2];
                const df t = df_add(df{s.Mdf[lane].x, s.Mdf[lane].y}, v);
                s.Mdf[lane] = make_float2(t.hi, t.lo);
            }
        } else if (tid >= 32 && live) {
            // Q(k) += sum over accepted trials of c_k(new) - c_k(old), over
            // the rebuild's items (eb_commit_qk): each thread owns items of
            // (+n, -n) k-vector pairs and adds every accepted trial's change
            eb_commit_qk(d, s, live, tid - 32, blockDim.x - 32, i0, i1, k0);
        }
        cur += done;
        if (CLUSTER) {
            // CTA 0's positions and cell lists are visible to the cluster
            blk_cluster_barrier();
            if (rebuild) break;   // the rebuild kernel takes it (rebuild_pending)
            continue;
        }
        __syncthreads();
        if (rebuild && !d.rebuild_in_kernel) break;   // the rebuild kernel takes it (rebuild_pending)
        if (rebuild) {
            df corr;
            const bool mism = eb_rebuild(d, s, corr);
            if (tid == 0) {
                U = df_add(U, corr);
                Ut = df_add(Ut, corr);
                sc->n_rebuilds++;
                if (mism && sc->verify_rebuild) err |= kErrQkMismatch;
            }
            rebuild = false;
        }
    }
    // write back Q(k), cells and the scalars (a cluster: every CTA its own
    // Q(k), CTA 0 the rest)
    if (CLUSTER) {
        for (int k = tid; k < K; k += blockDim.x) d.qfix[k0 + k] = s.b.qfix[k];
        if (rank == 0) store_back(d, s.b, false, CELLS);
    } else {
        store_back(d, s.b, true, CELLS);
    }
    if (tid == 0 && rank == 0) {
        sc->cursor = cur;
        sc->u_hi = U.hi;
        sc->u_lo = U.lo;
        sc->utot_hi = Ut.hi;
        sc->utot_lo = Ut.lo;
        sc->n_accepted = nacc;
        for (int a = 0; a < 3; a++) {
            sc->m[a][0] = s.Mdf[a].x;
            sc->m[a][1] = s.Mdf[a].y;
        }
        sc->cnt_accepted = cnt_acc;
        if (rebuild) sc->rebuild_pending = 1;
        sc->error |= err;
    }
}

}  // namespace fg
