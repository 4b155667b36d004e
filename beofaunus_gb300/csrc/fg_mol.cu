// Rigid dipolar molecules on the device: the TranslateRotate trial
// (move.h:1620-1705) and the whole-molecule energy change of
// NonbondedVector::g2All/g2g (energy.h:182-215, 1156-1196) over
//     CoulombGalore (multipole.h:569-598, the live operator: lB q q Q5(r/rc)/r)
//   + LennardJonesLB (potentials.h:2036-2040, no cutoff)
//   + IonDipole (multipole.h:993-996 -> q2mu 269-277, no cutoff)
//   + DipoleDipoleGalore reaction field (multipole.h:767-782, 910-920).
//
// Included by fg_api.cu (one translation unit).
//
// Work split. One system runs on a thread-block cluster of C CTAs (C <= 16,
// one per SM). CTA r owns the site slice [r N/C, (r+1) N/C) and the
// dipole-site slice [r D/C, (r+1) D/C), kept in its shared memory. Trials run in groups of up to
// kMolAhead, as the ion kernels run blocks (fg_dh_block.cu): every trial of the
// group is evaluated against the configuration at the group's start, one warp
// per trial and CTA, so that nothing but the warp's own sums happens per
// trial; if trial a was accepted, a later trial m of the group (another
// molecule) differs from that value by
//     c(a, m) = [u(n_m, n_a) - u(o_m, n_a)] - [u(n_m, o_a) - u(o_m, o_a)]
// over the two molecules' site pairs, which the cluster's warps evaluate for
// all a < m. The C partial sums and the c(a, m) meet in every CTA's shared
// memory (remote stores, one cluster barrier per group), every CTA resolves
// the group in order with the same numbers, and a trial whose molecule an
// accepted trial of the group moved ends the group (it is evaluated again in
// the next one): decisions are those of the one-trial-at-a-time chain. Each
// CTA keeps its own replica of the FP64-exact state (64-bit fixed-point
// positions, FP64 dipole vectors, mass centres) in global memory, so no CTA
// ever reads what another CTA wrote during the sweep.
//
// What bounds it: instruction issue in the pair loops (of 25 us per trial at
// 1000 x 20 sites on 4 CTAs the loop over far sites takes 9.5, image edges 1.8,
// near pairs 2.7, corrections 2, set-up 0.8). One trial at a time, six integer
// differences converted per pair and seven block barriers per trial took 50 us
// on 4 CTAs and 19 us on 16 (now 9).
//
// Precision. Positions are 64-bit fixed point (X = x/L 2^64). The rotation
// of a trial runs in FP64 on offsets from the rotation centre (20 sites per
// trial). Pair terms are FP32 except where that would exceed the 1e-6 kT
// budget:
//  * far pairs (both r_old, r_new >= rc): LJ and ion-dipole are small. Site j
//    is taken relative to the moved molecule's old mass centre (the 32-bit
//    minimum-image difference D_j, converted once per trial), site i as its
//    offset delta_i from that centre, so that a pair costs no conversion: D_j's
//    rounding is common to the old and the new position and its effect on
//    u_new - u_old cancels to first order;
//  * near pairs (r_old or r_new < rc) are queued and evaluated 32 at a time:
//    LJ and Coulomb as differences u(r_new) - u(r_old) whose
//    rounding error scales with the difference, from r_new^2 - r_old^2
//    computed from exact coordinate differences; terms with a dipole in FP32
//    (a few per trial);
//  * per-trial sums are double-float (df).
// The image convention is the reference's minimum image (Cuboid::vdist). For a
// site with |D| + max |delta| < L/2 on each axis D - delta is the minimum
// image of every pair; the others (19 % at 1000 molecules in 150 A) are
// collected and take min(|dx|, L - |dx|) for LJ and the exact integer
// difference for ion-dipole, which is odd in r.
#include "fg_mol_turns.h"

namespace fgm {

using fg::df;
using fg::df_add;
using fg::df_add_f;
using fg::df_gt;
using fg::hi32;
using fg::warp_sum_df;

constexpr int kMolThreads = 512;
constexpr int kMaxGroupSites = 31;   // lane gs of the setup warp computes the mass centre
constexpr int kMaxCluster = 16;
constexpr int kMolAhead = 16;   // trials of a group, one per warp
constexpr int kMolWarps = kMolThreads / 32;
constexpr int kMolPerLane = 4;  // sites per lane of the far loop
constexpr int kMolSiteQueue = 32 * (kMolPerLane + 1);   // a queue of less than 32 sites takes one more turn
constexpr int kMolPairQueue = 256;   // near pairs of a warp (about 110 at C = 16 and 425 at C = 4 for 1000 x 20
                                     // sites; what exceeds it the warp evaluates as it comes)
constexpr int kMolQueue = 2 * kMolSiteQueue + kMolPairQueue;   // words of a warp: two site queues, near pairs
// A correction beyond this (kT) belongs to a trial on top of where an accepted
// molecule was: its dU would be the small rest of two large numbers that a df
// holds to 2^-46 of their size. It is kept as a NaN, the group ends before a
// trial that took it, and the next group evaluates the trial (its first) against
// the configuration as it is.
constexpr float kMolLargeCorr = 1.0e4f;

// Error bits
constexpr int kMolErrNonFinite = 8;
constexpr int kMolErrLaunch = 64;   // launched with another cluster shape than requested

struct MolTrial {
    int32_t g;       // molecule index
    int32_t flags;   // 1 rotate, 2 translate, 4 explicit new coordinates (expl_*)
    int32_t center;  // rotation centre: 0 mass centre, 1 first site, 2 last site
    float thr_hi, thr_lo;  // -ln u as df: reject iff dU > threshold
    int32_t pad;
    double qw, qx, qy, qz;  // rotation quaternion (w, v)
    int64_t t[3];           // translation, fixed point
};

struct MolScalars {
    int64_t cursor;      // next trial
    int64_t n_trials;    // trials in the stream
    int64_t n_accepted;  // accepted so far (cumulative)
    int32_t error;
    int32_t pad;
    float u_hi, u_lo;        // sum of accepted dU of the current stream
    float utot_hi, utot_lo;  // running total energy
    int64_t acc0;        // n_accepted when the stream was staged
};

struct alignas(16) MolDesc {
    int32_t N, gs, M, D, nt, C, uniform_lj, cubic;
    float s32[3];       // L / 2^32 (one unit of the high word)
    float pad0[3];      // the later fields 8 bytes earlier cost the sweep 1.1 % (2.222 -> 2.245 ms, 256 trials of 1000 x 20)
    double s64d[3];     // L / 2^64
    double inv64d[3];   // 2^64 / L
    float lB, rc2, rc2near, rc1i, A5, B5, kT, rfB;
    float s32sq, pad2[3];  // (L / 2^32)^2 for cubic boxes
    double lBd, rcd, rfBd, pad3;
    long long rc2int;  // ceil(rc^2) in squared high-word units (cubic boxes)
    long long pad4;
    double s32sqd[3];
    float s2[256], eps4[256], lbqq[256];
    float qtype[16];
    double s2d[256], eps4d[256];  // FP64 copies for the total energy
    int64_t *rep_pos;  // C replicas x N x 3, fixed point
    double *rep_mu;    // C replicas x N x 3, dipole unit vectors
    int64_t *rep_cm;   // C replicas x M x 3, mass centres
    int4 *pos4;        // N: rounded high words (x, y, z), type
    int32_t *site_dip; // N: index in the dipole list, or -1
    int32_t *dip_site; // D: site of each dipole
    double *mus;       // N: dipole scalars (e Angstrom)
    float4 *dip4;      // D: mu-hat * mu (x, y, z), mu
    int4 *dip_pos4;    // D: positions of the dipole sites, .w = site << 8 | type
    const MolTrial *trials;
    float2 *log_du;
    uint8_t *log_acc;
    MolScalars *sc;
    const int64_t *expl_pos;  // gs x 3 new positions (explicit trials)
    const double *expl_mu;    // gs x 3 new dipole unit vectors
    const int64_t *expl_cm;   // 3, new mass centre
    double *eval_du;          // dU of an evaluated (not decided) trial
};

// ---------------------------------------------------------------- cluster PTX
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_size() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Store a float2 into the shared memory of CTA `rank` of this cluster.
__device__ __forceinline__ void st_cluster_f2(float2 *p, unsigned rank, float2 v) {
    unsigned a = (unsigned)__cvta_generic_to_shared(p), ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(ra), "f"(v.x), "f"(v.y) : "memory");
}

// ---------------------------------------------------------------- helpers
// a - b with two's-complement wrap (the minimum image of high words).
__device__ __forceinline__ int wsub(int a, int b) { return (int)((uint32_t)a - (uint32_t)b); }

struct D3 {
    double x, y, z;
};
__device__ __forceinline__ double dot3(const D3 &a, const D3 &b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ D3 cross3(const D3 &a, const D3 &b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
// Quaternion rotation as Eigen applies it: uv = v x p; uv += uv; p + w uv + v x uv.
__device__ __forceinline__ D3 qrot(double w, const D3 &v, const D3 &p) {
    D3 uv = cross3(v, p);
    uv = {uv.x + uv.x, uv.y + uv.y, uv.z + uv.z};
    D3 c = cross3(v, uv);
    return {p.x + w * uv.x + c.x, p.y + w * uv.y + c.y, p.z + w * uv.z + c.z};
}

// ---------------------------------------------------------------- shared memory
// Moved-molecule data of one trial of the group, set up by one warp (the
// rotations run in FP64, 1/64 of the FP32 rate: sixteen side by side take a
// quarter of what they take one after the other).
struct GroupBuf {
    int4 *go, *gn;    // old/new high words; .w = type | dipole flag (go) / site << 8 | type (gn)
    float4 *gfo;      // old dipole vector mu-hat * mu (x, y, z), mu (sites with a dipole)
    float4 *gfn;      // new dipole vector
    float4 *dlo;      // old offset from the reference point (Angstrom), .w = its square
    float4 *dln;      // new offset
    double *gmu;      // [gs][3] new unit dipole (FP64, for the replica)
    int64_t *gX;      // [gs][3] new fixed-point positions
    int64_t *gcm;     // [3] new mass centre
    float4 *lim;      // half box less the largest |offset| per axis; .w = squared distance from the
                      // reference point beyond which no pair of the molecule is near
    int4 *ref;        // reference point (high words of the old mass centre), .w = sites with a dipole
    uint32_t *qmask;  // sites with a charge
};

struct MolSmem {
    int4 *spos;     // site slice: high words, .w = type
    float4 *sdip;   // dipole slice: mu-hat * mu, mu (in global memory where it does not fit)
    int4 *sdpos;    // dipole slice positions, .w = site << 8 | type
    unsigned char *groups;   // `ahead` group buffers
    uint32_t *queue;   // [kMolWarps][kMolQueue]: a warp's sites that may change image, near sites, near pairs
    float2 *part;      // [2][kMaxCluster][kMolWarps] partial sums of the cluster's warps (by group parity)
    float2 *corr;      // [2][kMolAhead][kMolAhead] c(a, m)
    float *lbq;        // [16] lB q of each type
    int *info;         // [4] resolved, accepted, stop
    int *npair;        // [kMolWarps] near pairs queued by each warp
};

__host__ __device__ inline size_t mol_align16(size_t x) { return (x + 15) & ~(size_t)15; }

__host__ __device__ inline size_t mol_group_bytes(int gs) {
    return mol_align16((size_t)gs * 16 * 6) + mol_align16((size_t)gs * 3 * 8 * 2 + 3 * 8) + 48;
}

__host__ __device__ inline void mol_smem_layout(int ns, int nd, int gs, bool slice_smem, int ahead, size_t off[16]) {
    size_t o = 0;
    off[0] = o; o += mol_align16(slice_smem ? (size_t)ns * 16 : 0);   // spos
    off[1] = o; o += mol_align16((size_t)nd * 16);                    // sdip
    off[2] = o; o += mol_align16((size_t)nd * 16);                    // sdpos
    off[3] = o; o += ahead * mol_group_bytes(gs);                     // group buffers
    off[4] = o; o += (size_t)kMolWarps * kMolQueue * 4;               // queue
    off[5] = o; o += (size_t)2 * kMaxCluster * kMolWarps * 8;         // part
    off[6] = o; o += (size_t)2 * kMolAhead * kMolAhead * 8 + 64 + 16 + 4 * kMolWarps;   // corr, lbq, info, npair
    off[7] = o;
}

__device__ inline MolSmem mol_carve(unsigned char *base, int ns, int nd, int gs, bool slice_smem, int ahead) {
    size_t off[16];
    mol_smem_layout(ns, nd, gs, slice_smem, ahead, off);
    MolSmem s;
    s.spos = (int4 *)(base + off[0]);
    s.sdip = (float4 *)(base + off[1]);
    s.sdpos = (int4 *)(base + off[2]);
    s.groups = base + off[3];
    s.queue = (uint32_t *)(base + off[4]);
    s.part = (float2 *)(base + off[5]);
    s.corr = (float2 *)(base + off[6]);
    s.lbq = (float *)(s.corr + 2 * kMolAhead * kMolAhead);
    s.info = (int *)(s.lbq + 16);
    s.npair = s.info + 4;
    return s;
}
__device__ __forceinline__ GroupBuf mol_group(const MolSmem &s, int gs, int b) {
    unsigned char *g = s.groups + b * mol_group_bytes(gs);
    GroupBuf B;
    B.go = (int4 *)g;
    B.gn = B.go + gs;
    B.gfo = (float4 *)(B.gn + gs);
    B.gfn = B.gfo + gs;
    B.dlo = B.gfn + gs;
    B.dln = B.dlo + gs;
    g += mol_align16((size_t)gs * 16 * 6);
    B.gmu = (double *)g;
    B.gX = (int64_t *)(B.gmu + 3 * gs);
    B.gcm = B.gX + 3 * gs;
    g += mol_align16((size_t)gs * 3 * 8 * 2 + 3 * 8);
    B.lim = (float4 *)g;
    B.ref = (int4 *)(g + 16);
    B.qmask = (uint32_t *)(g + 32);
    return B;
}

// ---------------------------------------------------------------- pair terms
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Exact 32-bit difference vector a - b in Angstrom (FP32).
__device__ __forceinline__ float3 diff32(int4 a, int4 b, float3 s32) {
    return make_float3((float)wsub(a.x, b.x) * s32.x, (float)wsub(a.y, b.y) * s32.y, (float)wsub(a.z, b.z) * s32.z);
}
__device__ __forceinline__ float dot3f(float3 a, float3 b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, a.z * b.z)); }

// Coulomb part f(r) = Q5(r/rc) / r with Q5(q) = (q-1)^3 (A5 q^2 + B5 q - 1).
__device__ __forceinline__ float coul_f(float r, float rc1i, float A5, float B5) {
    const float q = r * rc1i;
    const float qm = q - 1.0f;
    return qm * qm * qm * fmaf(fmaf(A5, q, B5), q, -1.0f) / r;
}

// r_new^2 - r_old^2 (Angstrom^2) from exact integer arithmetic on the high
// words, each minimum image taken separately as Cuboid::vdist does.
__device__ __forceinline__ float dr2_exact(int4 pn, int4 po, int4 pj, const MolDesc &d) {
    const int hn[3] = {pn.x, pn.y, pn.z}, ho[3] = {po.x, po.y, po.z};
    if (d.cubic) return fg::dr2_words(pj, hn, ho) * d.s32sq;
    const int dn[3] = {wsub(pn.x, pj.x), wsub(pn.y, pj.y), wsub(pn.z, pj.z)};
    const int dO[3] = {wsub(po.x, pj.x), wsub(po.y, pj.y), wsub(po.z, pj.z)};
    double S = 0.0;
#pragma unroll
    for (int a = 0; a < 3; a++)
        S += (double)(((long long)dn[a] - dO[a]) * ((long long)dn[a] + dO[a])) * d.s32sqd[a];
    return (float)S;
}

// Near pair, kind A: moved site i (old po, new pn) against site j: LJ and
// Coulomb as differences whose rounding scales with the difference, and the
// ion-dipole term of i's dipole with j's charge (FP32, a few per trial).
__device__ __noinline__ float near_pair_a(int4 po, int4 pn, float4 fo, float4 fn, int4 pj, const MolDesc &d) {
    const float3 s32 = make_float3(d.s32[0], d.s32[1], d.s32[2]);
    const float3 ro = diff32(po, pj, s32), rn = diff32(pn, pj, s32);
    const float ro2 = dot3f(ro, ro), rn2 = dot3f(rn, rn);
    const float dR2 = dr2_exact(pn, po, pj, d);
    const int ti = po.w & 0xFF, tj = pj.w & 0xFF;
    const int t = ti * d.nt + tj;
    // LJ: 4eps x_o^3 (t^3 - 1)(x_o^3 (t^3 + 1) - 1), t^3 - 1 from tau = -dR2 / r_n^2
    const float xo = d.s2[t] / ro2;
    const float xo3 = xo * xo * xo;
    const float tau = -dR2 / rn2;
    const float t3m1 = tau * fmaf(tau, tau + 3.0f, 3.0f);
    float acc = d.eps4[t] * xo3 * t3m1 * fmaf(xo3, t3m1 + 2.0f, -1.0f);
    // Coulomb (CoulombGalore)
    const float A = d.lbqq[t];
    if (A != 0.0f) {
        const bool io = ro2 < d.rc2, in_ = rn2 < d.rc2;
        const float r_o = sqrtf(ro2), r_n = sqrtf(rn2);
        if (io && in_) {
            // f_n - f_o = [Q5(q_n) - Q5(q_o)] / r_n - Q5(q_o) dr / (r_n r_o)
            const float dr = dR2 / (r_n + r_o);
            const float qo = r_o * d.rc1i, qn = r_n * d.rc1i, dq = dr * d.rc1i;
            const float mo = qo - 1.0f, mn = qn - 1.0f;
            const float Po = fmaf(fmaf(d.A5, qo, d.B5), qo, -1.0f);
            const float Pn = fmaf(fmaf(d.A5, qn, d.B5), qn, -1.0f);
            const float dcube = dq * fmaf(mn, mn + mo, mo * mo);   // (q_n-1)^3 - (q_o-1)^3
            const float dP = dq * fmaf(d.A5, qn + qo, d.B5);       // P(q_n) - P(q_o)
            const float dQ = fmaf(dcube, Pn, mo * mo * mo * dP);
            acc += A * (dQ / r_n - mo * mo * mo * Po * dr / (r_n * r_o));
        } else if (io) {
            acc -= A * coul_f(r_o, d.rc1i, d.A5, d.B5);
        } else if (in_) {
            acc += A * coul_f(r_n, d.rc1i, d.A5, d.B5);
        }
    }
    if (po.w & 0x100) {
        // W2 of IonDipole(a = i, b = j): -lB q_j (mu_i . r) / r^3
        const float qj = d.qtype[tj];
        const float io = rsqrtf(ro2), in_ = rsqrtf(rn2);
        const float w = dot3f(make_float3(fn.x, fn.y, fn.z), rn) * in_ * in_ * in_ -
                        dot3f(make_float3(fo.x, fo.y, fo.z), ro) * io * io * io;
        acc -= d.lB * qj * w;
    }
    return acc;
}

// Near pair, kind B: moved site i against dipole k: ion-dipole with i's charge
// and, when i carries a dipole, dipole-dipole with the reaction field; the
// cutoff test is exact on the integer squared distance.
__device__ __noinline__ float near_pair_b(int4 po, int4 pn, float4 fo, float4 fn, int4 pk, float4 vk,
                                          const MolDesc &d) {
    const float3 s32 = make_float3(d.s32[0], d.s32[1], d.s32[2]);
    const float3 ro = diff32(po, pk, s32), rn = diff32(pn, pk, s32);
    const float ro2 = dot3f(ro, ro), rn2 = dot3f(rn, rn);
    const float io = rsqrtf(ro2), in_ = rsqrtf(rn2);
    const float3 v = make_float3(vk.x, vk.y, vk.z);
    const float qi = d.qtype[po.w & 0xFF];
    float acc = d.lB * qi * (dot3f(v, rn) * in_ * in_ * in_ - dot3f(v, ro) * io * io * io);
    if (po.w & 0x100) {
        auto dd = [&](float4 f, float3 r, float r2, float ri, int4 p) {
            // far pairs (a group's corrections pass them) first: the integer
            // squares of three half boxes would not fit 63 bits
            if (!(r2 < d.rc2near)) return 0.0f;
            const int dx = wsub(p.x, pk.x), dy = wsub(p.y, pk.y), dz = wsub(p.z, pk.z);
            bool inside;
            if (d.cubic) {
                // exact: |r|^2 < rc^2 on integers (rc2int = ceil(rc^2) in high-word units)
                inside = (long long)dx * dx + (long long)dy * dy + (long long)dz * dz < d.rc2int;
            } else {
                inside = (double)dx * dx * d.s32sqd[0] + (double)dy * dy * d.s32sqd[1] +
                             (double)dz * dz * d.s32sqd[2] < d.rcd * d.rcd;
            }
            if (!inside) return 0.0f;
            const float3 u = make_float3(f.x, f.y, f.z);
            const float r1 = r2 * ri;
            const float q = r1 * d.rc1i;
            const float dt = dot3f(u, v);
            // mu2mu with A = 1, B = rfB q^3: -(3 (u.r)(v.r)/r^2 - u.v + u.v B) / r^3
            const float T = fmaf(3.0f * dot3f(u, r), dot3f(v, r) * (ri * ri), -dt) + dt * (d.rfB * q * q * q);
            return -d.lB * T * ri * ri * ri;
        };
        acc += dd(fn, rn, rn2, in_, pn) - dd(fo, ro, ro2, io, po);
    }
    return acc;
}

// ---------------------------------------------------------------- trial setup
// New coordinates of the moved molecule: FP64 rotation of offsets from the
// centre, then translation. Items are spread over the warp's lanes: the gs
// sites, the mass centre, and the dipoles of the sites that carry one, so
// that positions and dipoles rotate in the same FP64 instructions. Old data
// come from this CTA's replica. Called by one warp.
__device__ __noinline__ void setup_trial(const MolTrial &tr, const MolDesc &d, const GroupBuf &B, int rank) {
    const int lane = threadIdx.x & 31;
    const int gs = d.gs, g = tr.g;
    const int64_t *P = d.rep_pos + (size_t)rank * d.N * 3;
    const double *MU = d.rep_mu + (size_t)rank * d.N * 3;
    const int64_t *CM = d.rep_cm + (size_t)rank * d.M * 3;
    const bool explicit_ = tr.flags & 4, rot = (tr.flags & 1) && !explicit_, trans = (tr.flags & 2) && !explicit_;
    const float3 s32 = make_float3(d.s32[0], d.s32[1], d.s32[2]);
    int64_t c[3] = {0, 0, 0};
    int rf[3];
    for (int a = 0; a < 3; a++) rf[a] = hi32(CM[3 * g + a]);
    if (rot) {
        if (tr.center == 0) {
            for (int a = 0; a < 3; a++) c[a] = CM[3 * g + a];
        } else {
            const int cs = g * gs + (tr.center == 1 ? 0 : gs - 1);
            for (int a = 0; a < 3; a++) c[a] = P[3 * cs + a];
        }
    }
    // this lane's site: type, dipole, charge
    const int my = g * gs + min(lane, gs - 1);
    int type = 0;
    bool has_mu = false, has_dip = false, has_q = false;
    if (lane < gs) {
        type = d.pos4[my].w & 0xFF;
        has_dip = d.site_dip[my] >= 0;
        has_q = d.qtype[type] != 0.0f;
        unsigned long long bits = 0;   // a nonzero dipole unit vector (compared as integers, off the FP64 pipe)
        for (int a = 0; a < 3; a++) bits |= (unsigned long long)__double_as_longlong(MU[3 * my + a]) << 1;
        if (explicit_ && d.expl_mu) bits = 1;
        has_mu = bits != 0;
        if (!has_mu) {
            for (int a = 0; a < 3; a++) B.gmu[3 * lane + a] = MU[3 * my + a];
            if (has_dip) B.gfo[lane] = B.gfn[lane] = make_float4(0.0f, 0.0f, 0.0f, (float)d.mus[my]);
        }
    }
    const uint32_t hm = __ballot_sync(0xffffffffu, has_mu), hd = __ballot_sync(0xffffffffu, has_dip);
    const uint32_t hq = __ballot_sync(0xffffffffu, has_q);
    const D3 qv = {tr.qx, tr.qy, tr.qz};
    const int nit = gs + 1 + __popc(hm);
    float4 dlo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), dln = dlo;   // the lane's site offsets (item = lane < gs)
    for (int b0 = 0; b0 < nit; b0 += 32) {
        const int it = b0 + lane;
        const bool dip = it > gs && it < nit, pos = it <= gs;
        int src = it;
        if (dip) {   // the (it - gs - 1)-th site with a dipole vector
            uint32_t m = hm;
            for (int k = it - gs - 1; k > 0; k--) m &= m - 1;
            src = __ffs(m) - 1;
        }
        const int site = g * gs + src;
        D3 v = {0.0, 0.0, 0.0};
        int64_t X[3] = {0, 0, 0};
        if (dip) {
            v = {MU[3 * site], MU[3 * site + 1], MU[3 * site + 2]};
        } else if (pos) {
            const int64_t *S = it < gs ? P + 3 * site : CM + 3 * g;
            for (int a = 0; a < 3; a++) X[a] = S[a];
            if (rot)
                v = {(double)(int64_t)((uint64_t)X[0] - (uint64_t)c[0]) * d.s64d[0],
                     (double)(int64_t)((uint64_t)X[1] - (uint64_t)c[1]) * d.s64d[1],
                     (double)(int64_t)((uint64_t)X[2] - (uint64_t)c[2]) * d.s64d[2]};
        }
        D3 w = v;
        if (rot) w = qrot(tr.qw, qv, v);   // positions, and DipoleParticle::rotate (point.h:672-679)
        if (dip) {
            if (explicit_ && d.expl_mu) w = {d.expl_mu[3 * src], d.expl_mu[3 * src + 1], d.expl_mu[3 * src + 2]};
            B.gmu[3 * src] = w.x;
            B.gmu[3 * src + 1] = w.y;
            B.gmu[3 * src + 2] = w.z;
            if ((hd >> src) & 1u) {
                const double m = d.mus[site];
                B.gfo[src] = make_float4((float)(v.x * m), (float)(v.y * m), (float)(v.z * m), (float)m);
                B.gfn[src] = make_float4((float)(w.x * m), (float)(w.y * m), (float)(w.z * m), (float)m);
            }
        } else if (pos) {
            int64_t Y[3] = {X[0], X[1], X[2]};
            if (rot) {
                Y[0] = (int64_t)((uint64_t)c[0] + (uint64_t)__double2ll_rn(w.x * d.inv64d[0]));
                Y[1] = (int64_t)((uint64_t)c[1] + (uint64_t)__double2ll_rn(w.y * d.inv64d[1]));
                Y[2] = (int64_t)((uint64_t)c[2] + (uint64_t)__double2ll_rn(w.z * d.inv64d[2]));
            }
            if (trans)
                for (int a = 0; a < 3; a++) Y[a] = (int64_t)((uint64_t)Y[a] + (uint64_t)tr.t[a]);
            if (it == gs) {
                if (explicit_ && d.expl_cm)
                    for (int a = 0; a < 3; a++) Y[a] = d.expl_cm[a];
                for (int a = 0; a < 3; a++) B.gcm[a] = Y[a];
            } else {
                if (explicit_)
                    for (int a = 0; a < 3; a++) Y[a] = d.expl_pos[3 * it + a];
                const int4 go = make_int4(hi32(X[0]), hi32(X[1]), hi32(X[2]), type | (has_dip ? 0x100 : 0));
                const int4 gn = make_int4(hi32(Y[0]), hi32(Y[1]), hi32(Y[2]), type | (site << 8));
                B.go[it] = go;
                B.gn[it] = gn;
                for (int a = 0; a < 3; a++) B.gX[3 * it + a] = Y[a];
                const float3 o = make_float3((float)wsub(go.x, rf[0]) * s32.x, (float)wsub(go.y, rf[1]) * s32.y,
                                             (float)wsub(go.z, rf[2]) * s32.z);
                const float3 n = make_float3((float)wsub(gn.x, rf[0]) * s32.x, (float)wsub(gn.y, rf[1]) * s32.y,
                                             (float)wsub(gn.z, rf[2]) * s32.z);
                dlo = make_float4(o.x, o.y, o.z, dot3f(o, o));
                dln = make_float4(n.x, n.y, n.z, dot3f(n, n));
                B.dlo[it] = dlo;
                B.dln[it] = dln;
            }
        }
    }
    // bounds of the offsets (non-negative floats order as their bit patterns)
    auto wmax = [](float x) { return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(x))); };
    const float mx = wmax(fmaxf(fabsf(dlo.x), fabsf(dln.x))), my_ = wmax(fmaxf(fabsf(dlo.y), fabsf(dln.y)));
    const float mz = wmax(fmaxf(fabsf(dlo.z), fabsf(dln.z))), mr = wmax(fmaxf(dlo.w, dln.w));
    if (lane == 0) {
        // the expanded r^2 loses (|D| / r)^2 in relative accuracy: a molecule
        // longer than the cutoff tests every pair with direct distances
        const float lim = (sqrtf(d.rc2near) + sqrtf(mr)) * 1.00001f;
        const float hb = 2147483648.0f * 0.999998f;   // half box in high-word units, with a margin for rounding
        *B.lim = make_float4(hb * s32.x - mx, hb * s32.y - my_, hb * s32.z - mz, mr <= d.rc2near ? lim * lim : 3.0e38f);
        *B.ref = make_int4(rf[0], rf[1], rf[2], (int)hd);
        *B.qmask = hq;
    }
}

// ---------------------------------------------------------------- energy change
// LJ of the moved sites against one site per lane at displacement D from the
// reference point, new minus old, any image (min(|dx|, L - |dx|)). With
// y = r^-6 and c = sigma^6, u = 4eps (c^2 y^2 - c y), so u_n - u_o =
// 4eps c dy (c (y_n + y_o) - 1), dy = y_n - y_o: uniform tables sum b1 = sum dy
// and b2 = sum dy (y_n + y_o) and scale at the end; else b1 sums the energies.
// Pairs within rc2near are left out and their bits returned.
struct MolView {   // the same in every thread of a warp
    float3 s32, L, half;   // Angstrom per high-word unit, box, half box less max |offset|
    int4 ref;
    float far2;            // sites beyond this squared distance from ref have no near pair
};
__device__ __forceinline__ MolView mol_view(const GroupBuf &B, float3 s32, float3 L) {
    const float4 lim = *B.lim;
    return MolView{s32, L, make_float3(lim.x, lim.y, lim.z), *B.ref, lim.w};
}
__device__ __forceinline__ float3 mol_disp(int4 p, const MolView &v) {
    return make_float3((float)wsub(p.x, v.ref.x) * v.s32.x, (float)wsub(p.y, v.ref.y) * v.s32.y,
                       (float)wsub(p.z, v.ref.z) * v.s32.z);
}
__device__ __forceinline__ int mol_outside(float3 D, const MolView &v) {   // axes on which some pair may change image
    return (fabsf(D.x) > v.half.x ? 1 : 0) + (fabsf(D.y) > v.half.y ? 1 : 0) + (fabsf(D.z) > v.half.z ? 1 : 0);
}
template <bool UNI>
__device__ __forceinline__ void mol_lj_add(const MolDesc &d, int ti, int tj, float yo, float yn, float &b1, float &b2) {
    const float dy = yn - yo, sy = yn + yo;
    if (UNI) {
        b1 += dy;
        b2 = fmaf(dy, sy, b2);
    } else {
        const int t = ti * d.nt + tj;
        const float s2 = d.s2[t], c = s2 * s2 * s2;
        b1 = fmaf(d.eps4[t] * c * dy, fmaf(c, sy, -1.0f), b1);
    }
}
template <bool UNI>
__device__ __forceinline__ uint32_t mol_lj_image(const MolDesc &d, const GroupBuf &B, const MolView &v, float3 D,
                                                 int tj, float &b1, float &b2) {
    uint32_t near = 0u;
    const int gs = d.gs;
    const float rc2near = d.rc2near;
    auto r2_of = [&](float4 o) {
        const float x = fabsf(D.x - o.x), y = fabsf(D.y - o.y), z = fabsf(D.z - o.z);
        const float mx = fminf(x, v.L.x - x), my = fminf(y, v.L.y - y), mz = fminf(z, v.L.z - z);
        return fmaf(mx, mx, fmaf(my, my, mz * mz));
    };
#pragma unroll 4
    for (int i = 0; i < gs; i++) {
        const float r2o = r2_of(B.dlo[i]), r2n = r2_of(B.dln[i]);
        const float io = rcp_approx(r2o), in_ = rcp_approx(r2n);
        const bool nr = fminf(r2o, r2n) < rc2near;
        near |= nr ? 1u << i : 0u;
        const float yo = nr ? 0.0f : io * io * io, yn = nr ? 0.0f : in_ * in_ * in_;
        mol_lj_add<UNI>(d, UNI ? 0 : B.go[i].w & 0xFF, tj, yo, yn, b1, b2);
    }
    return near;
}
// The same for kMolPerLane sites per lane that need no image: r^2 = |D|^2 +
// |delta|^2 - 2 D.delta from D2 = -2 D and A = |D|^2. A pair of distances takes
// 18 issue slots and two MUFU (against about 170 when every pair converted
// six integer differences); four sites share the two 16-byte loads of an
// offset pair, whose 512-byte broadcasts would otherwise fill the
// shared-memory port (8 of every 20 cycles per warp and SM quarter).
template <bool UNI>
__device__ __forceinline__ void mol_lj_far(const MolDesc &d, const GroupBuf &B, const float3 (&D2)[kMolPerLane],
                                           const float (&A)[kMolPerLane], const int (&tj)[kMolPerLane], float &b1,
                                           float &b2) {
    const int gs = d.gs;
#pragma unroll 2
    for (int i = 0; i < gs; i++) {
        const float4 o = B.dlo[i], n = B.dln[i];
        const int ti = UNI ? 0 : B.go[i].w & 0xFF;
#pragma unroll
        for (int u = 0; u < kMolPerLane; u++) {
            const float io = rcp_approx(fmaf(o.x, D2[u].x, fmaf(o.y, D2[u].y, fmaf(o.z, D2[u].z, A[u] + o.w))));
            const float in_ = rcp_approx(fmaf(n.x, D2[u].x, fmaf(n.y, D2[u].y, fmaf(n.z, D2[u].z, A[u] + n.w))));
            mol_lj_add<UNI>(d, ti, tj[u], io * io * io, in_ * in_ * in_, b1, b2);
        }
    }
}

// The same for one far site per lane whose image may change along one axis:
// the nearer of its two images along that axis, |D - delta|^2 and
// |D' - delta|^2 with D' = D -+ L, each expanded (28 issue slots per pair
// against 43 of the general form above).
template <bool UNI>
__device__ __forceinline__ void mol_lj_edge(const MolDesc &d, const GroupBuf &B, const MolView &v, float3 D, int tj,
                                            float &b1, float &b2) {
    float3 E = D;
    if (fabsf(D.x) > v.half.x) E.x = D.x - copysignf(v.L.x, D.x);
    else if (fabsf(D.y) > v.half.y) E.y = D.y - copysignf(v.L.y, D.y);
    else E.z = D.z - copysignf(v.L.z, D.z);
    const float A = dot3f(D, D), AE = dot3f(E, E);
    const float3 D2 = make_float3(-2.0f * D.x, -2.0f * D.y, -2.0f * D.z);
    const float3 E2 = make_float3(-2.0f * E.x, -2.0f * E.y, -2.0f * E.z);
    auto r2_of = [&](float4 o) {
        return fminf(fmaf(o.x, D2.x, fmaf(o.y, D2.y, fmaf(o.z, D2.z, A + o.w))),
                     fmaf(o.x, E2.x, fmaf(o.y, E2.y, fmaf(o.z, E2.z, AE + o.w))));
    };
    const int gs = d.gs;
#pragma unroll 4
    for (int i = 0; i < gs; i++) {
        const float io = rcp_approx(r2_of(B.dlo[i])), in_ = rcp_approx(r2_of(B.dln[i]));
        mol_lj_add<UNI>(d, UNI ? 0 : B.go[i].w & 0xFF, tj, io * io * io, in_ * in_ * in_, b1, b2);
    }
}

// W of IonDipole without its prefactor: (f_n . r_n) / r_n^3 - (f_o . r_o) / r_o^3.
__device__ __forceinline__ float ion_dipole_diff(float3 fo, float3 ro, float3 fn, float3 rn) {
    const float ro2 = dot3f(ro, ro), rn2 = dot3f(rn, rn);
    const float io = rsqrtf(ro2), in_ = rsqrtf(rn2);
    return dot3f(fn, rn) * in_ * in_ * in_ - dot3f(fo, ro) * io * io * io;
}
__device__ __forceinline__ float3 xyz(float4 v) { return make_float3(v.x, v.y, v.z); }
__device__ __forceinline__ float3 sub3(float4 a, float3 b) { return make_float3(a.x - b.x, a.y - b.y, a.z - b.z); }
// W2 of IonDipole(a = i, b = j) over the moved dipoles in mask m, with lbq =
// lB q_j: -lB q_j (mu_i . r) / r^3, r = r_i - r_j (exact image).
__device__ __forceinline__ float mol_w2_exact(const GroupBuf &B, uint32_t m, int4 pj, float lbq, float3 s32) {
    float w = 0.0f;
    for (; m; m &= m - 1) {
        const int i = __ffs(m) - 1;
        w -= lbq * ion_dipole_diff(xyz(B.gfo[i]), diff32(B.go[i], pj, s32), xyz(B.gfn[i]), diff32(B.gn[i], pj, s32));
    }
    return w;
}

// A queued near pair: moved site << 24 | dipole flag (0x800000) | slice index.
template <bool SLICE_SMEM>
__device__ __noinline__ float mol_near_pair(const MolDesc &d, const MolSmem &s, const GroupBuf &B, uint32_t c, int j0) {
    const int i = (int)((c >> 24) & 0x7F), idx = (int)(c & 0x7FFFFF);
    if (c & 0x800000u) return near_pair_b(B.go[i], B.gn[i], B.gfo[i], B.gfn[i], s.sdpos[idx], s.sdip[idx], d);
    return near_pair_a(B.go[i], B.gn[i], B.gfo[i], B.gfn[i], SLICE_SMEM ? s.spos[idx] : d.pos4[j0 + idx], d);
}
// The CTA's queued near pairs, 32 of one warp's queue at a time over all warps
// (chunk c of the queues laid end to end goes to warp c % kMolWarps); each
// result replaces its pair in the queue. Between block barriers.
template <bool SLICE_SMEM>
__device__ __forceinline__ void mol_near_pairs(const MolDesc &d, const MolSmem &s, int parts, int j0) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int mine = lane < kMolWarps ? s.npair[lane] : 0, nch = (mine + 31) >> 5;
    int end = nch;   // inclusive prefix sum of the chunks
#pragma unroll
    for (int o = 1; o < kMolWarps; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, end, o);
        if (lane >= o) end += x;
    }
    const int total = __shfl_sync(0xffffffffu, end, kMolWarps - 1);
    for (int c = warp; c < total; c += kMolWarps) {
        const int w = __popc(__ballot_sync(0xffffffffu, lane < kMolWarps && end <= c));   // the queue's warp
        const int k = (c - __shfl_sync(0xffffffffu, end - nch, w)) * 32 + lane;
        if (k < __shfl_sync(0xffffffffu, mine, w)) {
            uint32_t *q = s.queue + w * kMolQueue + 2 * kMolSiteQueue + k;
            *q = __float_as_uint(mol_near_pair<SLICE_SMEM>(d, s, mol_group(s, d.gs, w / parts), *q, j0));
        }
    }
}

// One warp's part of dU for trial m of the group (molecule g) over this CTA's
// slice (part `part` of `parts`): the site groups and dipole chunks part, part
// + parts, ... Sites beyond reach of the cutoff that need no image go through
// mol_lj_far as they come; those that may change image and those that may be
// near are collected in the warp's queues and taken 32 at a time. The near
// pairs stay in the warp's pair queue (their number to npair): all warps of the
// CTA share them out afterwards (mol_near_pairs), since a close molecule puts
// its 400 pairs on one warp. Everything is in a fixed order, and each kind of
// work has one place in the loop (the code stays within the instruction
// cache). All lanes call it; the lane's part of the sum is returned (df).
template <bool SLICE_SMEM, bool UNI>
__device__ __noinline__ df mol_base(const MolDesc &d, const MolSmem &sm, int m, int g, int j0, int ns, int nd,
                                    float3 s32, float3 L, int part, int parts) {
    const MolSmem s = sm;
    const int lane = threadIdx.x & 31, gs = d.gs;
    const uint32_t full = 0xffffffffu, below = (1u << lane) - 1u;
    const GroupBuf B = mol_group(s, gs, m);
    const MolView v = mol_view(B, s32, L);
    const int g_lo = g * gs, g_hi = g_lo + gs;
    const uint32_t dips = (uint32_t)v.ref.w;
    uint32_t *const bq = s.queue + (threadIdx.x >> 5) * kMolQueue, *const nq = bq + kMolSiteQueue,
             *const pq = nq + kMolSiteQueue;
    int nb = 0, nn = 0, np = 0;
    float b1 = 0.0f, b2 = 0.0f;
    df acc = {0.0f, 0.0f};
    auto site = [&](int jj) { return SLICE_SMEM ? s.spos[jj] : d.pos4[j0 + jj]; };
    auto push = [&](uint32_t *q, int &cnt, bool f, uint32_t val) {
        const uint32_t b = __ballot_sync(full, f);
        if (f) q[cnt + __popc(b & below)] = val;
        cnt += __popc(b);
    };
    auto drop = [&](uint32_t *q, int &cnt) {   // the first 32 entries are done: the rest moves up (a lane
        cnt = max(cnt - 32, 0);                 // writes only what it read itself)
        for (int e = lane; e < cnt; e += 32) q[e] = q[32 + e];
        __syncwarp();
    };
    const int gsites = 32 * kMolPerLane, nsg = (ns + gsites - 1) / gsites, ndg = (nd + 31) >> 5;
    for (int it = part; it < nsg + ndg; it += parts) {
        const bool last = it + parts >= nsg + ndg;   // this warp's last turn: the queues are emptied
        uint32_t near = 0u, code = 0u;
        if (it < nsg) {
            float3 D2[kMolPerLane];
            float A[kMolPerLane], lbq[kMolPerLane];
            int tj[kMolPerLane];
            bool any = false;
#pragma unroll
            for (int u = 0; u < kMolPerLane; u++) {
                const int jj = it * gsites + 32 * u + lane, j = j0 + jj;
                const bool in = jj < ns && !(j >= g_lo && j < g_hi);
                const int4 pj = site(min(jj, ns - 1));
                tj[u] = pj.w & 0xFF;
                const float3 D = mol_disp(pj, v);
                A[u] = dot3f(D, D);
                const int axes = mol_outside(D, v);
                const bool nr = in && (A[u] <= v.far2 || axes > 1);   // near, or a rare image along several axes
                const bool edge = in && !nr && axes == 1;
                const bool ok = in && !nr && !edge;
                if (__any_sync(full, nr || edge)) {
                    push(nq, nn, nr, (uint32_t)jj);
                    push(bq, nb, edge, (uint32_t)jj);
                }
                // a site taken elsewhere sits so far away that its terms vanish
                D2[u] = ok ? make_float3(-2.0f * D.x, -2.0f * D.y, -2.0f * D.z) : make_float3(-2.0e15f, 0.0f, 0.0f);
                A[u] = ok ? A[u] : 1.0e30f;
                lbq[u] = ok ? s.lbq[tj[u]] : 0.0f;
                any |= lbq[u] != 0.0f;
            }
            mol_lj_far<UNI>(d, B, D2, A, tj, b1, b2);
            if (dips != 0u && __any_sync(full, any)) {
                float w = 0.0f;
                for (uint32_t q = dips; q; q &= q - 1) {
                    const int i = __ffs(q) - 1;
                    const float4 o = B.dlo[i], n = B.dln[i];
                    const float3 fo = xyz(B.gfo[i]), fn = xyz(B.gfn[i]);
#pragma unroll
                    for (int u = 0; u < kMolPerLane; u++) {
                        const float3 D = make_float3(-0.5f * D2[u].x, -0.5f * D2[u].y, -0.5f * D2[u].z);
                        w = fmaf(-lbq[u], ion_dipole_diff(fo, sub3(o, D), fn, sub3(n, D)), w);
                    }
                }
                acc = df_add_f(acc, w);
            }
        } else {
            // dipoles of the slice against the moved charges: W1 of IonDipole(a = i,
            // b = k): lB q_i (mu_k . r) / r^3 (dipole-dipole is 0 beyond rc: near pairs)
            const int kk = (it - nsg) * 32 + lane, kc = min(kk, nd - 1);
            const int4 pk = s.sdpos[kc];
            const float3 f = xyz(s.sdip[kc]);
            const int ksite = pk.w >> 8;
            const bool in = kk < nd && !(ksite >= g_lo && ksite < g_hi);
            const float3 D = mol_disp(pk, v);
            float w = 0.0f;
            if (__any_sync(full, in && dot3f(D, D) <= v.far2)) {
                for (int i = 0; i < gs; i++) {
                    const float3 ro = diff32(B.go[i], pk, s32), rn = diff32(B.gn[i], pk, s32);
                    const bool nr = in && fminf(dot3f(ro, ro), dot3f(rn, rn)) < d.rc2near;
                    near |= nr ? 1u << i : 0u;
                    const float q = s.lbq[B.go[i].w & 0xFF];
                    if (!nr && q != 0.0f) w = fmaf(q, ion_dipole_diff(f, ro, f, rn), w);
                }
            } else {
                const bool image = __any_sync(full, in && mol_outside(D, v) != 0);
                for (uint32_t q = *B.qmask; q; q &= q - 1) {
                    const int i = __ffs(q) - 1;
                    const int4 po = B.go[i];
                    float3 ro = sub3(B.dlo[i], D), rn = sub3(B.dln[i], D);
                    if (image) {
                        ro = diff32(po, pk, s32);
                        rn = diff32(B.gn[i], pk, s32);
                    }
                    w = fmaf(s.lbq[po.w & 0xFF], ion_dipole_diff(f, ro, f, rn), w);
                }
            }
            if (in) acc = df_add_f(acc, w);
            code = 0x800000u | (uint32_t)kk;
        }
        __syncwarp();
        const int lim = last ? 1 : 32;
        while (true) {
            while (__any_sync(full, near != 0u)) {   // near pairs of this turn, one per lane at a time
                push(pq, np, near != 0u, ((uint32_t)(__ffs(near) - 1) << 24) | code);
                near &= near - 1;
                if (np > kMolPairQueue - 32) {   // no room for another turn: the last 32 now
                    __syncwarp();
                    np -= 32;
                    acc = df_add_f(acc, mol_near_pair<SLICE_SMEM>(d, s, B, pq[np + lane], j0));
                    __syncwarp();
                }
            }
            if (nn < lim && nb < lim) break;
            // up to 32 sites: near ones first (near stays 0 for the others)
            const bool nearq = nn >= lim;
            uint32_t *q = nearq ? nq : bq;
            const int cnt = nearq ? nn : nb;
            const int jj = (int)q[min(lane, cnt - 1)];
            const int4 pj = site(jj);
            float c1 = 0.0f, c2 = 0.0f;
            if (nearq) near = mol_lj_image<UNI>(d, B, v, mol_disp(pj, v), pj.w & 0xFF, c1, c2);
            else mol_lj_edge<UNI>(d, B, v, mol_disp(pj, v), pj.w & 0xFF, c1, c2);
            if (lane < cnt) {
                b1 += c1;
                b2 += c2;
                const float lbq = s.lbq[pj.w & 0xFF];
                if (lbq != 0.0f) acc = df_add_f(acc, mol_w2_exact(B, dips & ~near, pj, lbq, s32));
            } else {
                near = 0u;
            }
            code = (uint32_t)jj;
            __syncwarp();
            if (nearq) drop(nq, nn);
            else drop(bq, nb);
        }
    }
    if (lane == 0) s.npair[threadIdx.x >> 5] = np;
    if (UNI) {
        const float c = d.s2[0] * d.s2[0] * d.s2[0];
        return df_add_f(acc, d.eps4[0] * c * fmaf(c, b2, -b1));
    }
    return df_add_f(acc, b1);
}

// c(a, m): how much dU of trial m (buffer Bm) changes when trial a (buffer Ba,
// another molecule) is accepted: m's energy change against a's sites at their
// new positions minus that at their old ones. One warp; lanes over a's sites.
template <bool UNI>
__device__ __noinline__ df mol_correction(const MolDesc &d, const MolSmem &sm, int a, int m, float3 s32, float3 L) {
    const MolSmem s = sm;
    const int lane = threadIdx.x & 31, gs = d.gs;
    const GroupBuf Ba = mol_group(s, gs, a), Bm = mol_group(s, gs, m);
    const uint32_t full = 0xffffffffu;
    const MolView v = mol_view(Bm, s32, L);
    const bool in = lane < gs;
    const int4 pn = Ba.gn[min(lane, gs - 1)], po = Ba.go[min(lane, gs - 1)];
    const float3 Dn = mol_disp(pn, v), Do = mol_disp(po, v);
    const uint32_t dm = (uint32_t)v.ref.w, da = (uint32_t)Ba.ref->w, qm = *Bm.qmask;
    df acc = {0.0f, 0.0f};
    if (__any_sync(full, in && (dot3f(Dn, Dn) <= v.far2 || dot3f(Do, Do) <= v.far2))) {
        // close molecules: every site pair in the near form
        for (int e = lane; e < gs * gs; e += 32) {
            const int i = e / gs, j = e - i * gs;
            acc = df_add_f(acc, near_pair_a(Bm.go[i], Bm.gn[i], Bm.gfo[i], Bm.gfn[i], Ba.gn[j], d));
            acc = df_add_f(acc, -near_pair_a(Bm.go[i], Bm.gn[i], Bm.gfo[i], Bm.gfn[i], Ba.go[j], d));
            if ((da >> j) & 1u) {
                acc = df_add_f(acc, near_pair_b(Bm.go[i], Bm.gn[i], Bm.gfo[i], Bm.gfn[i], Ba.gn[j], Ba.gfn[j], d));
                acc = df_add_f(acc, -near_pair_b(Bm.go[i], Bm.gn[i], Bm.gfo[i], Bm.gfn[i], Ba.go[j], Ba.gfo[j], d));
            }
        }
        return warp_sum_df(acc);
    }
    const int tj = po.w & 0xFF;
    float n1 = 0.0f, n2 = 0.0f, o1 = 0.0f, o2 = 0.0f;
    auto y_of = [&](float3 D, float4 o) {   // r^-6, any image
        const float x = fabsf(D.x - o.x), y = fabsf(D.y - o.y), z = fabsf(D.z - o.z);
        const float mx = fminf(x, L.x - x), my = fminf(y, L.y - y), mz = fminf(z, L.z - z);
        const float i = rcp_approx(fmaf(mx, mx, fmaf(my, my, mz * mz)));
        return i * i * i;
    };
#pragma unroll 4
    for (int i = 0; i < gs; i++) {
        const float4 o = Bm.dlo[i], n = Bm.dln[i];
        const int ti = UNI ? 0 : Bm.go[i].w & 0xFF;
        mol_lj_add<UNI>(d, ti, tj, y_of(Dn, o), y_of(Dn, n), n1, n2);
        mol_lj_add<UNI>(d, ti, tj, y_of(Do, o), y_of(Do, n), o1, o2);
    }
    if (in) {
        if (UNI) {
            const float c = d.s2[0] * d.s2[0] * d.s2[0];
            acc = df_add_f(acc, d.eps4[0] * c * fmaf(c, n2 - o2, o1 - n1));
        } else {
            acc = df_add_f(acc, n1 - o1);
        }
        // m's dipoles with a's charges, a's dipoles with m's charges
        const float lbq = s.lbq[tj];
        if (lbq != 0.0f)
            acc = df_add_f(acc, mol_w2_exact(Bm, dm, pn, lbq, s32) - mol_w2_exact(Bm, dm, po, lbq, s32));
        if ((da >> lane) & 1u) {
            const float3 fn = xyz(Ba.gfn[lane]), fo = xyz(Ba.gfo[lane]);
            float w = 0.0f;
            for (uint32_t m = qm; m; m &= m - 1) {
                const int i = __ffs(m) - 1;
                w = fmaf(s.lbq[Bm.go[i].w & 0xFF],
                         ion_dipole_diff(fn, diff32(Bm.go[i], pn, s32), fn, diff32(Bm.gn[i], pn, s32)) -
                             ion_dipole_diff(fo, diff32(Bm.go[i], po, s32), fo, diff32(Bm.gn[i], po, s32)),
                         w);
            }
            acc = df_add_f(acc, w);
        }
    }
    return warp_sum_df(acc);
}

// ---------------------------------------------------------------- the sweep
// One cluster of C CTAs per system (blockIdx.x / C). EVAL: evaluate trial 0
// only, write its dU to eval_du, decide and commit nothing. Groups of up to
// `ahead` trials; a group of fewer trials than warps splits each trial's slice
// over several warps.
template <bool SLICE_SMEM, bool CLUSTER, bool EVAL>
__global__ void __launch_bounds__(kMolThreads, 1) mol_sweep_kernel(const MolDesc *__restrict__ descs, int ahead,
                                                                  int dips, int64_t quantum) {
    extern __shared__ __align__(16) unsigned char mol_smem_raw[];
    const int C = CLUSTER ? (int)descs[0].C : 1;
    const int sys = blockIdx.x / C;
    // launch-shape check: partial sums come from C CTAs of this cluster
    if (CLUSTER && (int)cluster_size() != C) {
        if (threadIdx.x == 0) atomicOr(&descs[sys].sc->error, kMolErrLaunch);
        return;
    }
    const int rank = CLUSTER ? (int)cluster_rank() : 0;
    const MolDesc &d = descs[sys];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ns_full = (d.N + C - 1) / C, nd_full = (d.D + C - 1) / C;
    const int j0 = min(rank * ns_full, d.N), j1 = min(j0 + ns_full, d.N), ns = j1 - j0;
    const int k0 = min(rank * nd_full, d.D), k1 = min(k0 + nd_full, d.D), nd = k1 - k0;
    const bool dip_smem = SLICE_SMEM || dips;
    MolSmem s = mol_carve(mol_smem_raw, ns_full, dip_smem ? nd_full : 0, d.gs, SLICE_SMEM, ahead);
    if (!dip_smem) {
        s.sdip = d.dip4 + k0;
        s.sdpos = d.dip_pos4 + k0;
    }
    if (SLICE_SMEM)
        for (int jj = tid; jj < ns; jj += blockDim.x) s.spos[jj] = d.pos4[j0 + jj];
    for (int kk = tid; dip_smem && kk < nd; kk += blockDim.x) {
        s.sdip[kk] = d.dip4[k0 + kk];
        s.sdpos[kk] = d.dip_pos4[k0 + kk];
    }
    if (tid < 16) s.lbq[tid] = tid < d.nt ? d.lB * d.qtype[tid] : 0.0f;
    int64_t cursor = EVAL ? 0 : d.sc->cursor;
    const int64_t n = EVAL ? 1 : min(d.sc->n_trials, cursor + quantum);   // at most quantum trials of the stream
    df usum = {d.sc->u_hi, d.sc->u_lo};
    df utot = {d.sc->utot_hi, d.sc->utot_lo};
    int64_t nacc = d.sc->n_accepted;
    const bool uni = d.uniform_lj != 0;
    const float3 s32 = make_float3(d.s32[0], d.s32[1], d.s32[2]);
    const float3 L = make_float3(s32.x * 4294967296.0f, s32.y * 4294967296.0f, s32.z * 4294967296.0f);
    int err = 0, buf = 0;
    if (CLUSTER) cluster_barrier();   // every CTA of the cluster runs before any remote store
    for (; cursor < n; buf ^= 1) {
        const int ng = (int)(n - cursor < (int64_t)ahead ? n - cursor : (int64_t)ahead);
        __syncthreads();   // the previous group's commits are in place
        for (int m = warp; m < ng; m += kMolWarps)
            setup_trial(d.trials[cursor + m], d, mol_group(s, d.gs, m), rank);
        __syncthreads();
        // ---- base sums: warp w takes part w % parts of trial w / parts
        const int parts = kMolWarps / ng, tm = warp / parts;
        float2 *const xpart = s.part + buf * kMaxCluster * kMolWarps, *const xcorr = s.corr + buf * kMolAhead * kMolAhead;
        df v = {0.0f, 0.0f};
        if (tm < ng) {
            const int g = d.trials[cursor + tm].g;
            v = uni ? mol_base<SLICE_SMEM, true>(d, s, tm, g, j0, ns, nd, s32, L, warp - tm * parts, parts)
                    : mol_base<SLICE_SMEM, false>(d, s, tm, g, j0, ns, nd, s32, L, warp - tm * parts, parts);
        } else if (lane == 0) {
            s.npair[warp] = 0;
        }
        __syncthreads();   // the near pairs are queued
        mol_near_pairs<SLICE_SMEM>(d, s, parts, j0);
        __syncthreads();
        if (tm < ng) {
            const float *res = reinterpret_cast<const float *>(s.queue + warp * kMolQueue + 2 * kMolSiteQueue);
            for (int k = lane; k < s.npair[warp]; k += 32) v = df_add_f(v, res[k]);
            v = warp_sum_df(v);
            v.hi = __shfl_sync(0xffffffffu, v.hi, 0);   // one value for every CTA: they must decide alike
            v.lo = __shfl_sync(0xffffffffu, v.lo, 0);
            if (CLUSTER) {
                if (lane < C) st_cluster_f2(&xpart[rank * kMolWarps + warp], (unsigned)lane, make_float2(v.hi, v.lo));
            } else if (lane == 0) {
                xpart[warp] = make_float2(v.hi, v.lo);
            }
        }
        // ---- corrections c(a, m), a < m, over the cluster's warps
        if (!EVAL)
            for (int e = rank * kMolWarps + warp, m = 1, lo = 0; e < ng * (ng - 1) / 2; e += C * kMolWarps) {
                while (e >= lo + m) lo += m++;   // pair e of the triangle: trial m, a = e - m (m - 1) / 2
                const int a = e - lo;
                if (d.trials[cursor + a].g == d.trials[cursor + m].g) continue;
                df c = uni ? mol_correction<true>(d, s, a, m, s32, L) : mol_correction<false>(d, s, a, m, s32, L);
                if (!(fabsf(c.hi) <= kMolLargeCorr)) c.hi = __int_as_float(0x7FFFFFFF);
                c.hi = __shfl_sync(0xffffffffu, c.hi, 0);
                c.lo = __shfl_sync(0xffffffffu, c.lo, 0);
                if (CLUSTER) {
                    if (lane < C) st_cluster_f2(&xcorr[a * kMolAhead + m], (unsigned)lane, make_float2(c.hi, c.lo));
                } else if (lane == 0) {
                    xcorr[a * kMolAhead + m] = make_float2(c.hi, c.lo);
                }
            }
        if (CLUSTER) cluster_barrier();
        else __syncthreads();
        // ---- resolve the group in order (warp 0 of every CTA, the same numbers; lane m = trial m)
        if (warp == 0) {
            df S = {0.0f, 0.0f};
            int lg = -1;
            float2 th = make_float2(0.0f, 0.0f);
            if (lane < ng) {
                for (int r = 0; r < C; r++)
                    for (int p = 0; p < parts; p++) {
                        const float2 x = xpart[r * kMolWarps + lane * parts + p];
                        S = df_add(S, df{x.x, x.y});
                    }
                const MolTrial &t = d.trials[cursor + lane];
                lg = t.g;
                th = make_float2(t.thr_hi, t.thr_lo);
            }
            if (EVAL && rank == 0 && lane == 0) *d.eval_du = (double)S.hi + (double)S.lo;
            uint32_t accm = 0;
            int done = EVAL ? 0 : ng, bad = 0;
            for (int a = 0; a < done; a++) {
                const float2 c = xcorr[a * kMolAhead + min(lane, kMolAhead - 1)];
                const int ga = __shfl_sync(0xffffffffu, lg, a);
                // every lane forms its own flags; lane a's are the ones used
                const int fl = (isfinite(S.hi) ? 0 : 2) | (df_gt(S, df{th.x, th.y}) ? 0 : 1);
                const int f = __shfl_sync(0xffffffffu, fl, a);
                if (__ballot_sync(0xffffffffu, lane < a && ((accm >> lane) & 1u) && lg == ga)) {
                    done = a;   // its molecule was moved by an accepted trial of this group
                    break;
                }
                if (f & 2) {   // after other trials: perhaps by kMolLargeCorr
                    bad = a == 0;
                    done = a;
                    break;
                }
                if (f & 1) {
                    accm |= 1u << a;
                    const df Sc = df_add(S, df{c.x, c.y});
                    const bool later = lane > a && lane < ng && lg != ga;
                    S.hi = later ? Sc.hi : S.hi;
                    S.lo = later ? Sc.lo : S.lo;
                }
            }
            // lane m's S is trial m's dU as decided
            const bool take = lane < done && ((accm >> lane) & 1u);
            if (rank == 0 && lane < done) {
                if (d.log_du) d.log_du[cursor + lane] = make_float2(S.hi, S.lo);
                if (d.log_acc) d.log_acc[cursor + lane] = take ? 1 : 0;
            }
            const df sum = warp_sum_df(take ? S : df{0.0f, 0.0f});
            usum = df_add(usum, sum);
            utot = df_add(utot, sum);
            if (lane == 0) {
                s.info[0] = done;
                s.info[1] = (int)accm;
                s.info[2] = bad;
            }
        }
        __syncthreads();
        if (EVAL) break;
        const int done = s.info[0];
        const uint32_t accm = (uint32_t)s.info[1];
        nacc += __popc(accm);
        // ---- apply the accepted trials (distinct molecules), one warp each
        for (int m = warp; m < done; m += kMolWarps) {
            if (!((accm >> m) & 1u)) continue;
            const GroupBuf B = mol_group(s, d.gs, m);
            const int g = d.trials[cursor + m].g, gs = d.gs;
            if (lane < gs) {
                const int site = g * gs + lane;
                int64_t *P = d.rep_pos + ((size_t)rank * d.N + site) * 3;
                double *MU = d.rep_mu + ((size_t)rank * d.N + site) * 3;
                for (int x = 0; x < 3; x++) {
                    P[x] = B.gX[3 * lane + x];
                    MU[x] = B.gmu[3 * lane + x];
                }
                const int4 pn = make_int4(B.gn[lane].x, B.gn[lane].y, B.gn[lane].z, B.go[lane].w & 0xFF);
                if (site >= j0 && site < j1) {
                    if (SLICE_SMEM) s.spos[site - j0] = pn;
                    else d.pos4[site] = pn;
                }
                const int k = d.site_dip[site];
                if (k >= k0 && k < k1) {
                    s.sdpos[k - k0] = make_int4(pn.x, pn.y, pn.z, (site << 8) | (pn.w & 0xFF));
                    s.sdip[k - k0] = B.gfn[lane];
                }
            } else if (lane == gs) {
                int64_t *CM = d.rep_cm + ((size_t)rank * d.M + g) * 3;
                for (int x = 0; x < 3; x++) CM[x] = B.gcm[x];
            }
        }
        cursor += done;
        if (s.info[2]) {
            err |= kMolErrNonFinite;
            break;
        }
    }
    __syncthreads();
    // write the slices back (each CTA its own range) and the scalars
    if (!EVAL) {
        if (SLICE_SMEM)
            for (int jj = tid; jj < ns; jj += blockDim.x) d.pos4[j0 + jj] = s.spos[jj];
        for (int kk = tid; dip_smem && kk < nd; kk += blockDim.x) {
            d.dip4[k0 + kk] = s.sdip[kk];
            d.dip_pos4[k0 + kk] = s.sdpos[kk];
        }
        if (rank == 0 && tid == 0) {
            MolScalars *sc = d.sc;
            sc->cursor = cursor;
            sc->n_accepted = nacc;
            sc->u_hi = usum.hi;
            sc->u_lo = usum.lo;
            sc->utot_hi = utot.hi;
            sc->utot_lo = utot.lo;
            sc->error |= err;
        }
    }
    if (CLUSTER) cluster_barrier();   // no CTA leaves while another may write its shared memory
}

// Apply an evaluated explicit trial (fg_mol_commit): new positions, dipoles
// and mass centre into every replica, the site/dipole records and the
// running energy. One block of >= gs + 1 threads.
__global__ void mol_commit_kernel(const MolDesc *__restrict__ descs, int g, int accepted, int nrep) {
    const MolDesc &d = descs[0];
    const int tid = threadIdx.x, gs = d.gs;
    if (!accepted) return;
    if (tid < gs) {
        const int site = g * gs + tid;
        int64_t X[3];
        for (int a = 0; a < 3; a++) X[a] = d.expl_pos[3 * tid + a];
        for (int r = 0; r < nrep; r++) {
            int64_t *P = d.rep_pos + ((size_t)r * d.N + site) * 3;
            double *MU = d.rep_mu + ((size_t)r * d.N + site) * 3;
            for (int a = 0; a < 3; a++) {
                P[a] = X[a];
                if (d.expl_mu) MU[a] = d.expl_mu[3 * tid + a];
            }
        }
        const int type = d.pos4[site].w & 0xFF;
        const int4 p4 = make_int4(hi32(X[0]), hi32(X[1]), hi32(X[2]), type);
        d.pos4[site] = p4;
        const int k = d.site_dip[site];
        if (k >= 0) {
            const double m = d.mus[site];
            const double *u = d.rep_mu + (size_t)site * 3;
            d.dip_pos4[k] = make_int4(p4.x, p4.y, p4.z, (site << 8) | type);
            d.dip4[k] = make_float4((float)(u[0] * m), (float)(u[1] * m), (float)(u[2] * m), (float)m);
        }
    } else if (tid == gs && d.expl_cm) {
        for (int r = 0; r < nrep; r++)
            for (int a = 0; a < 3; a++) d.rep_cm[((size_t)r * d.M + g) * 3 + a] = d.expl_cm[a];
    }
}

// IonDipole (q2mu, multipole.h:269-277) in FP64 with r = r_a - r_b:
// lB [qa mub (mub.r) - qb mua (mua.r)] / r^3, mu vectors already scaled.
__device__ __forceinline__ double ion_dipole64(double qa, const D3 &mua, double qb, const D3 &mub, const D3 &r,
                                               double lB) {
    const double r2i = 1.0 / dot3(r, r);
    const double r3i = sqrt(r2i) * r2i;
    return lB * (qa * dot3(mub, r) * r3i - qb * dot3(mua, r) * r3i);
}
// DipoleDipoleGalore with the reaction field (multipole.h:287-299, 767-782, 910-920).
__device__ __forceinline__ double dipole_dipole64(const D3 &ua, double ma, const D3 &ub, double mb, const D3 &r,
                                                  const MolDesc &d) {
    const double r2 = dot3(r, r);
    const double r1 = sqrt(r2);
    if (!(r1 < d.rcd)) return 0.0;
    const double q = r1 / d.rcd;
    const double bf = d.rfBd * q * q * q;
    const double r2i = 1.0 / r2;
    const double dt = dot3(ua, ub);
    const double T = (3.0 * dot3(ua, r) * dot3(ub, r) * r2i - dt) + dt * bf;
    return d.lBd * (-(ma * mb) * T * sqrt(r2i) * r2i);
}

// Total energy in FP64, as Energybase::systemEnergy sums it (energy.h:169-180):
// out[0] += intermolecular pairs, out[1] += intramolecular pairs
// (NonbondedVector::g_internal, energy.h:1207-1216). Grid: x over sites i
// (256 per block), y over chunks of j.
__global__ void mol_total_kernel(const MolDesc *__restrict__ descs, int chunk, double *out) {
    const MolDesc &d = descs[0];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int jb = blockIdx.y * chunk, je = min(jb + chunk, d.N);
    double inter = 0.0, intra = 0.0;
    if (i < d.N) {
        const int64_t *P = d.rep_pos;
        const int ti = d.pos4[i].w & 0xFF;
        const double qi = d.qtype[ti], mi = d.mus[i];
        const D3 ui = {d.rep_mu[3 * i], d.rep_mu[3 * i + 1], d.rep_mu[3 * i + 2]};
        const D3 vi = {ui.x * mi, ui.y * mi, ui.z * mi};
        for (int j = max(jb, i + 1); j < je; j++) {
            const int tj = d.pos4[j].w & 0xFF;
            const D3 r = {(double)(int64_t)((uint64_t)P[3 * i] - (uint64_t)P[3 * j]) * d.s64d[0],
                          (double)(int64_t)((uint64_t)P[3 * i + 1] - (uint64_t)P[3 * j + 1]) * d.s64d[1],
                          (double)(int64_t)((uint64_t)P[3 * i + 2] - (uint64_t)P[3 * j + 2]) * d.s64d[2]};
            const double r2 = dot3(r, r);
            double u = 0.0;
            // CoulombGalore (kappa = 0)
            const int t = ti * d.nt + tj;
            if (r2 < (double)d.rc2) {
                const double rr = sqrt(r2);
                const double q = rr / d.rcd, q2 = q * q;
                const double a2 = -66.0 * 1494.0 / 56916.0;
                const double Q = (q - 1.0) * (q - 1.0) * (q - 1.0) *
                                 (5.0 / 22.0 * q2 * a2 + 9.0 / 22.0 * q * a2 - 0.6 * q2 - 1.2 * q - 1.0);
                u += d.lBd * (double)d.qtype[ti] * (double)d.qtype[tj] / rr * Q;
            }
            // LennardJonesLB
            {
                double x = d.s2d[t] / r2;
                x = x * x * x;
                u += d.eps4d[t] * (x * x - x);
            }
            const double mj = d.mus[j];
            if (mi != 0.0 || mj != 0.0) {
                const D3 uj = {d.rep_mu[3 * j], d.rep_mu[3 * j + 1], d.rep_mu[3 * j + 2]};
                const D3 vj = {uj.x * mj, uj.y * mj, uj.z * mj};
                u += ion_dipole64(qi, vi, (double)d.qtype[tj], vj, r, d.lBd);
                if (mi != 0.0 && mj != 0.0) u += dipole_dipole64(ui, mi, uj, mj, r, d);
            }
            if (i / d.gs == j / d.gs) intra += u;
            else inter += u;
        }
    }
    // block sums, then one atomic per block
    __shared__ double red[2][32];
    for (int o = 16; o > 0; o >>= 1) {
        inter += __shfl_xor_sync(0xffffffffu, inter, o);
        intra += __shfl_xor_sync(0xffffffffu, intra, o);
    }
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = inter;
        red[1][threadIdx.x >> 5] = intra;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0, b = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
            a += red[0][w];
            b += red[1][w];
        }
        atomicAdd(&out[0], a);
        atomicAdd(&out[1], b);
    }
}

// A newly staged stream: cursor, per-stream sum and flags from zero.
__global__ void mol_begin_kernel(MolScalars *sc, int64_t n) {
    sc->cursor = 0;
    sc->n_trials = n;
    sc->acc0 = sc->n_accepted;
    sc->u_hi = sc->u_lo = 0.0f;
    sc->error = 0;
}
// The scalars of many systems into one array (one copy to the host).
__global__ void mol_gather_kernel(const MolDesc *descs, int n, MolScalars *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = *descs[i].sc;
}

}  // namespace fgm

// ==================================================================== host side
struct fg_molsys {
    fg_params P{};
    int N = 0, gs = 0, M = 0, D = 0;
    int device = 0;
    int C = 1;          // CTAs per system (thread-block cluster)
    int max_cluster = 1;
    cudaStream_t stream = nullptr;
    fgm::MolDesc desc{};
    fgm::MolDesc *d_desc = nullptr;
    int64_t *rep_pos = nullptr, *rep_cm = nullptr;
    double *rep_mu = nullptr, *mus = nullptr;
    int4 *pos4 = nullptr, *dip_pos4 = nullptr;
    int32_t *site_dip = nullptr, *dip_site = nullptr;
    float4 *dip4 = nullptr;
    fgm::MolTrial *trials = nullptr;
    int64_t trials_cap = 0;
    float2 *log_du = nullptr;
    uint8_t *log_acc = nullptr;
    int64_t log_cap = 0;
    fgm::MolScalars *sc = nullptr;
    int64_t *expl_pos = nullptr;
    double *expl_mu = nullptr, *eval_du = nullptr, *tot = nullptr;
    int64_t *expl_cm = nullptr;
    int pending = -1;   // molecule of an evaluated explicit trial awaiting fg_mol_commit
    double pending_du = 0.0;
    int64_t n_stream = 0;   // trials in the staged stream
    bool staged = false;    // a stream is staged and not yet run (it occupies the trial buffer)
    // mol_run's workspace of the system it launches from: 2 n descriptors, n scalars
    void *run_ws = nullptr;
    int run_cap = 0;
    fgm::MolDesc pushed{};  // what d_desc holds
    bool has_pushed = false;
    bool has_cm = false;
    bool state_set = false;
    std::vector<int32_t> types;
    std::vector<double> mus_h;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    size_t device_bytes = 0;
};

namespace {

int mol_dmalloc(fg_molsys *h, void **p, size_t bytes) {
    if (bytes == 0) bytes = 16;
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) return fail(FG_ERR_CUDA, "cudaMalloc of %zu bytes failed: %s", bytes, cudaGetErrorString(e));
    h->device_bytes += bytes;
    return FG_OK;
}
#define MOL_DMALLOC(ptr, bytes)                                        \
    do {                                                               \
        int rc_ = mol_dmalloc(h, (void **)&(ptr), (size_t)(bytes));    \
        if (rc_) return rc_;                                           \
    } while (0)

void mol_free(fg_molsys *h) {
    void *ptrs[] = {h->d_desc, h->rep_pos, h->rep_cm, h->rep_mu, h->mus, h->pos4, h->dip_pos4,
                    h->site_dip, h->dip_site, h->dip4, h->trials, h->log_du, h->log_acc, h->sc,
                    h->expl_pos, h->expl_mu, h->eval_du, h->tot, h->expl_cm, h->run_ws};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    if (h->ev0) cudaEventDestroy(h->ev0);
    if (h->ev1) cudaEventDestroy(h->ev1);
    if (h->stream) cudaStreamDestroy(h->stream);
}

// Geometry::anyCenter with equal masses (geometry.h:714-738) in fixed point:
// origin at the middle site, minimum-image offsets, mean, wrapped.
void mol_mass_center(const int64_t *X, int front, int gs, int64_t out[3]) {
    const int o = front + (int)((gs - 1) * 0.5);
    for (int a = 0; a < 3; a++) {
        long double s = 0;
        for (int i = front; i < front + gs; i++) s += (long double)(int64_t)((uint64_t)X[3 * i + a] - (uint64_t)X[3 * o + a]);
        out[a] = (int64_t)((uint64_t)X[3 * o + a] + (uint64_t)(int64_t)llroundl(s / gs));
    }
}

constexpr size_t kMolSmemMax = 220 * 1024;   // of the 227 KB a CTA may hold
// What a launch keeps in shared memory beside the queues.
struct MolFit {
    bool slice;   // the site slice
    bool dips;    // the dipole slice
    int ahead;    // trials per group
};
size_t mol_smem_bytes(const fg_molsys *h, int C, const MolFit &f) {
    size_t off[16];
    fgm::mol_smem_layout((h->N + C - 1) / C, f.dips ? (h->D + C - 1) / C : 0, h->gs, f.slice, f.ahead, off);
    return off[7];
}
// Trials per group: kMolAhead where their buffers fit beside the slices, fewer
// (at least four) where that keeps the site slice in shared memory; else it
// stays in global memory, and so does the dipole slice where it leaves no room
// for one trial (from some 5500 sites with a dipole in a CTA on).
MolFit mol_fit(const fg_molsys *h, int C) {
    for (int a = fgm::kMolAhead; a >= 4; a /= 2)
        if (mol_smem_bytes(h, C, {true, true, a}) <= kMolSmemMax) return {true, true, a};
    for (int a = fgm::kMolAhead; a >= 1; a /= 2)
        if (mol_smem_bytes(h, C, {false, true, a}) <= kMolSmemMax) return {false, true, a};
    return {false, false, fgm::kMolAhead};
}

struct MolLaunch {
    void (*fn)(const fgm::MolDesc *, int, int, int64_t);
    size_t smem;
    MolFit fit;
    bool cluster;
};

template <bool EVAL>
int mol_pick(const fg_molsys *h, MolLaunch &L) {
    L.fit = mol_fit(h, h->C);
    const bool cl = h->C > 1;
    L.smem = mol_smem_bytes(h, h->C, L.fit);
    L.cluster = cl;
    if (L.fit.slice) L.fn = cl ? fgm::mol_sweep_kernel<true, true, EVAL> : fgm::mol_sweep_kernel<true, false, EVAL>;
    else L.fn = cl ? fgm::mol_sweep_kernel<false, true, EVAL> : fgm::mol_sweep_kernel<false, false, EVAL>;
    cudaError_t e = cudaFuncSetAttribute((const void *)L.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem);
    if (e != cudaSuccess) return fail(FG_ERR_CUDA, "shared memory attribute: %s", cudaGetErrorString(e));
    if (cl) {
        e = cudaFuncSetAttribute((const void *)L.fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return fail(FG_ERR_CUDA, "cluster attribute: %s", cudaGetErrorString(e));
    }
    return FG_OK;
}

int mol_launch(const fg_molsys *h, const MolLaunch &L, const fgm::MolDesc *descs, int n_systems, cudaStream_t st,
               int64_t quantum = INT64_MAX / 2) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(n_systems * h->C));
    cfg.blockDim = dim3(fgm::kMolThreads);
    cfg.dynamicSmemBytes = L.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    if (L.cluster) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)h->C;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    cudaError_t e = cudaLaunchKernelEx(&cfg, L.fn, descs, L.fit.ahead, L.fit.dips ? 1 : 0, quantum);
    if (e != cudaSuccess) return fail(FG_ERR_CUDA, "molecule sweep launch: %s", cudaGetErrorString(e));
    return FG_OK;
}

// Clusters of this launch that the device runs at once (0: unknown).
int mol_slots(const fg_molsys *h, const MolLaunch &L) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)h->C);
    cfg.blockDim = dim3(fgm::kMolThreads);
    cfg.dynamicSmemBytes = L.smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)h->C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, (const void *)L.fn, &cfg) == cudaSuccess) return n;
    cudaGetLastError();
    return 0;
}

// Largest cluster the device runs for this kernel's shared memory (<= 16).
int mol_max_cluster(fg_molsys *h) {
    int best = 1;
    for (int c : {16, 8, 4, 2}) {
        const int saved = h->C;
        h->C = c;
        MolLaunch L;
        int rc = mol_pick<false>(h, L);
        h->C = saved;
        if (rc) continue;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)c);
        cfg.blockDim = dim3(fgm::kMolThreads);
        cfg.dynamicSmemBytes = L.smem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)c;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, (const void *)L.fn, &cfg) == cudaSuccess && n > 0) {
            best = c;
            break;
        }
        cudaGetLastError();
    }
    return best;
}

int mol_alloc_replicas(fg_molsys *h, int C) {
    if (h->rep_pos) cudaFree(h->rep_pos);
    if (h->rep_mu) cudaFree(h->rep_mu);
    if (h->rep_cm) cudaFree(h->rep_cm);
    h->rep_pos = nullptr;
    h->rep_mu = nullptr;
    h->rep_cm = nullptr;
    MOL_DMALLOC(h->rep_pos, (size_t)C * h->N * 3 * sizeof(int64_t));
    MOL_DMALLOC(h->rep_mu, (size_t)C * h->N * 3 * sizeof(double));
    MOL_DMALLOC(h->rep_cm, (size_t)C * h->M * 3 * sizeof(int64_t));
    h->desc.rep_pos = h->rep_pos;
    h->desc.rep_mu = h->rep_mu;
    h->desc.rep_cm = h->rep_cm;
    return FG_OK;
}

int mol_push_desc(fg_molsys *h) {
    h->desc.C = h->C;
    if (h->has_pushed && !std::memcmp(&h->pushed, &h->desc, sizeof(fgm::MolDesc))) return FG_OK;
    h->has_pushed = false;   // until the copy has gone out
    CK(cudaMemcpyAsync(h->d_desc, &h->desc, sizeof(fgm::MolDesc), cudaMemcpyHostToDevice, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    std::memcpy(&h->pushed, &h->desc, sizeof(fgm::MolDesc));
    h->has_pushed = true;
    return FG_OK;
}

int mol_ensure_trials(fg_molsys *h, int64_t n, bool log) {
    n = std::max<int64_t>(n, 1);
    if (n > h->trials_cap) {
        if (h->trials) cudaFree(h->trials);
        h->trials = nullptr;
        MOL_DMALLOC(h->trials, n * sizeof(fgm::MolTrial));
        h->trials_cap = n;
    }
    if (log && n > h->log_cap) {
        if (h->log_du) cudaFree(h->log_du);
        if (h->log_acc) cudaFree(h->log_acc);
        h->log_du = nullptr;
        h->log_acc = nullptr;
        MOL_DMALLOC(h->log_du, n * sizeof(float2));
        MOL_DMALLOC(h->log_acc, n);
        h->log_cap = n;
    }
    h->desc.trials = h->trials;
    return FG_OK;
}

int mol_read_scalars(fg_molsys *h, fgm::MolScalars &s) {
    CK(cudaMemcpyAsync(&s, h->sc, sizeof(s), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return FG_OK;
}
int mol_write_scalars(fg_molsys *h, const fgm::MolScalars &s) {
    CK(cudaMemcpyAsync(h->sc, &s, sizeof(s), cudaMemcpyHostToDevice, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return FG_OK;
}

// Copy replica 0 into replicas 1..C-1 (after the state changed through it).
int mol_sync_replicas(fg_molsys *h) {
    for (int r = 1; r < h->C; r++) {
        CK(cudaMemcpyAsync(h->rep_pos + (size_t)r * h->N * 3, h->rep_pos, (size_t)h->N * 3 * sizeof(int64_t),
                           cudaMemcpyDeviceToDevice, h->stream));
        CK(cudaMemcpyAsync(h->rep_mu + (size_t)r * h->N * 3, h->rep_mu, (size_t)h->N * 3 * sizeof(double),
                           cudaMemcpyDeviceToDevice, h->stream));
        CK(cudaMemcpyAsync(h->rep_cm + (size_t)r * h->M * 3, h->rep_cm, (size_t)h->M * 3 * sizeof(int64_t),
                           cudaMemcpyDeviceToDevice, h->stream));
    }
    CK(cudaStreamSynchronize(h->stream));
    return FG_OK;
}

int mol_total(fg_molsys *h, double out[2]) {
    CK(cudaMemsetAsync(h->tot, 0, 2 * sizeof(double), h->stream));
    const int chunk = 2048;
    dim3 grid((unsigned)((h->N + 255) / 256), (unsigned)((h->N + chunk - 1) / chunk));
    fgm::mol_total_kernel<<<grid, 256, 0, h->stream>>>(h->d_desc, chunk, h->tot);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(out, h->tot, 2 * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return FG_OK;
}

// MolTrial records from the reference's draws (or any explicit stream).
void mol_make_trials(const fg_molsys *h, int64_t n, const int32_t *mol, const double *axis, const double *angle,
                     const int32_t *center, const double *trans, const double *u, int rotate, int translate,
                     std::vector<fgm::MolTrial> &out) {
    out.resize(n);
    for (int64_t k = 0; k < n; k++) {
        fgm::MolTrial &t = out[k];
        t = fgm::MolTrial{};
        t.g = mol[k];
        t.flags = (rotate ? 1 : 0) | (translate ? 2 : 0);
        t.center = center ? center[k] : 0;
        t.qw = 1.0;
        if (rotate) {
            double ax = axis[3 * k], ay = axis[3 * k + 1], az = axis[3 * k + 2];
            const double nrm = std::sqrt(ax * ax + ay * ay + az * az);
            ax /= nrm; ay /= nrm; az /= nrm;
            const double ha = 0.5 * angle[k], sh = std::sin(ha);
            t.qw = std::cos(ha);
            t.qx = sh * ax; t.qy = sh * ay; t.qz = sh * az;
        }
        if (translate)
            for (int a = 0; a < 3; a++) t.t[a] = to_fix(trans[3 * k + a], h->P.box[a]);
        // Movebase::metropolis (move.h:567-573): reject iff u > exp(-dU)
        const double thr = -std::log(u[k]);
        const float2 f = split_df(thr);
        t.thr_hi = f.x;
        t.thr_lo = f.y;
        if (u[k] <= 0.0) { t.thr_hi = INFINITY; t.thr_lo = 0.0f; }
    }
}

// Stage a trial stream: validate, build MolTrial records, upload, reset the
// stream cursor and per-stream sums.
int mol_upload(fg_molsys *h, int64_t n, const int32_t *mol, const double *axis, const double *angle,
               const int32_t *center, const double *trans, const double *u, int rotate, int translate, bool log) {
    if (!h || n < 0 || (n > 0 && (!mol || !u))) return fail(FG_ERR_INVALID, "bad argument");
    if (rotate && n > 0 && (!axis || !angle)) return fail(FG_ERR_INVALID, "rotation needs axis and angle");
    if (translate && n > 0 && !trans) return fail(FG_ERR_INVALID, "translation needs trans");
    if (!h->state_set) return fail(FG_ERR_STATE, "fg_mol_set_state first");
    if (h->pending >= 0) return fail(FG_ERR_STATE, "a trial is pending: call fg_mol_commit");
    for (int64_t k = 0; k < n; k++) {
        if (mol[k] < 0 || mol[k] >= h->M) return fail(FG_ERR_INVALID, "molecule index out of range at %lld", (long long)k);
        if (center && (center[k] < 0 || center[k] > 2)) return fail(FG_ERR_INVALID, "bad centre kind");
    }
    int rc = mol_ensure_trials(h, n, log);
    if (rc) return rc;
    std::vector<fgm::MolTrial> tr;
    mol_make_trials(h, n, mol, axis, angle, center, trans, u, rotate, translate, tr);
    if (n > 0) CK(cudaMemcpyAsync(h->trials, tr.data(), n * sizeof(fgm::MolTrial), cudaMemcpyHostToDevice, h->stream));
    fgm::mol_begin_kernel<<<1, 1, 0, h->stream>>>(h->sc, n);
    CK(cudaGetLastError());
    h->n_stream = n;
    h->staged = true;
    h->desc.log_du = log ? h->log_du : nullptr;
    h->desc.log_acc = log ? h->log_acc : nullptr;
    h->desc.expl_pos = nullptr;
    h->desc.expl_mu = nullptr;
    h->desc.expl_cm = nullptr;
    return mol_push_desc(h);
}

// Run the staged streams of several systems in one launch per chunk (one
// cluster of C CTAs per system); launches hold at most kChunk trials each.
int mol_run(fg_molsys *const *sys, int n, fg_sweep_stats *per, fg_sweep_stats *total) {
    if (!sys || n < 1) return fail(FG_ERR_INVALID, "bad argument");
    fg_molsys *h0 = sys[0];
    MolFit fit{true, true, fgm::kMolAhead};   // what fits for every system
    int64_t maxn = 0;
    int fewest = INT32_MAX;   // molecules of the smallest system
    for (int i = 0; i < n; i++) {
        fg_molsys *h = sys[i];
        if (!h || !h->state_set) return fail(FG_ERR_STATE, "system %d has no state", i);
        if (h->C != h0->C) return fail(FG_ERR_INVALID, "systems must share the cluster size");
        if (h->device != h0->device) return fail(FG_ERR_INVALID, "systems must share the device");
        const MolFit f = mol_fit(h, h->C);
        fit = {fit.slice && f.slice, fit.dips && f.dips, std::min(fit.ahead, f.ahead)};
        maxn = std::max(maxn, h->n_stream);
        fewest = std::min(fewest, h->M);
        CK(cudaStreamSynchronize(h->stream));
    }
    MolLaunch L;
    L.cluster = h0->C > 1;
    L.fit = fit;
    L.smem = 0;
    for (int i = 0; i < n; i++) L.smem = std::max(L.smem, mol_smem_bytes(sys[i], sys[i]->C, fit));
    if (fit.slice) L.fn = L.cluster ? fgm::mol_sweep_kernel<true, true, false> : fgm::mol_sweep_kernel<true, false, false>;
    else L.fn = L.cluster ? fgm::mol_sweep_kernel<false, true, false> : fgm::mol_sweep_kernel<false, false, false>;
    CK(cudaFuncSetAttribute((const void *)L.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem));
    if (L.cluster) CK(cudaFuncSetAttribute((const void *)L.fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    const int64_t kChunk = 65536;   // most trials of one launch
    const fgm::MolTurns turns = fgm::mol_turns(maxn, n, mol_slots(h0, L), fgm::kMolAhead, fewest, kChunk);
    const int slots = turns.slots;
    const int64_t quantum = turns.quantum;
    cudaStream_t st = h0->stream;
    const fgm::MolDesc *descs = h0->d_desc;
    if (h0->run_cap < n) {
        const size_t each = 2 * sizeof(fgm::MolDesc) + sizeof(fgm::MolScalars);
        if (h0->run_ws) cudaFree(h0->run_ws);
        h0->run_ws = nullptr;
        h0->device_bytes -= (size_t)h0->run_cap * each;
        h0->run_cap = 0;
        int rc = mol_dmalloc(h0, &h0->run_ws, (size_t)n * each);
        if (rc) return rc;
        h0->run_cap = n;
    }
    fgm::MolScalars *const out =
        reinterpret_cast<fgm::MolScalars *>((char *)h0->run_ws + (size_t)h0->run_cap * 2 * sizeof(fgm::MolDesc));
    if (n > 1) {   // twice in a row, so that any rotation is one piece
        std::vector<fgm::MolDesc> v(2 * (size_t)n);
        for (int i = 0; i < n; i++) v[i] = v[n + i] = sys[i]->desc;
        CK(cudaMemcpyAsync(h0->run_ws, v.data(), v.size() * sizeof(fgm::MolDesc), cudaMemcpyHostToDevice, st));
        descs = reinterpret_cast<const fgm::MolDesc *>(h0->run_ws);
    }
    CK(cudaEventRecord(h0->ev0, st));
    int rc = FG_OK;
    int64_t nl = 0;
    if (slots >= n) {
        for (int64_t c = 0; c < maxn && !rc; c += kChunk, nl++) rc = mol_launch(h0, L, descs, n, st, kChunk);
    } else {
        // round r runs the systems (r slots + i) mod n, i < slots, for one quantum each
        const int64_t rounds = ((maxn + quantum - 1) / quantum * n + slots - 1) / slots;
        for (int64_t r = 0; r < rounds && !rc; r++, nl++)
            rc = mol_launch(h0, L, descs + r * slots % n, slots, st, quantum);
    }
    CK(cudaEventRecord(h0->ev1, st));
    for (int i = 0; i < n; i++) sys[i]->staged = false;
    if (rc) {
        cudaStreamSynchronize(st);
        return rc;
    }
    // the scalars of all systems in one copy
    fgm::mol_gather_kernel<<<(n + 127) / 128, 128, 0, st>>>(descs, n, out);
    CK(cudaGetLastError());
    std::vector<fgm::MolScalars> s1(n);
    CK(cudaMemcpyAsync(s1.data(), out, (size_t)n * sizeof(fgm::MolScalars), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    float ms = 0.0f;
    CK(cudaEventElapsedTime(&ms, h0->ev0, h0->ev1));
    fg_sweep_stats tot{};
    int errs = 0;
    for (int i = 0; i < n; i++) {
        fg_sweep_stats x{};
        x.trials = s1[i].cursor;
        x.accepted = s1[i].n_accepted - s1[i].acc0;
        x.energy_change = df_val(s1[i].u_hi, s1[i].u_lo);
        x.device_ms = ms;
        x.sweep_kernel_ms = ms;
        x.sweep_launches = (int32_t)nl;
        x.error_flags = s1[i].error;
        x.kernel_launches = nl;
        errs |= s1[i].error;
        if (per) per[i] = x;
        tot.trials += x.trials;
        tot.accepted += x.accepted;
        tot.energy_change += x.energy_change;
    }
    tot.device_ms = ms;
    tot.sweep_kernel_ms = ms;
    tot.sweep_launches = (int32_t)nl;
    tot.kernel_launches = nl;
    tot.error_flags = errs;
    if (total) *total = tot;
    if (errs) return fail(FG_ERR_DEVICE, "device error flags 0x%x", errs);
    return FG_OK;
}

}  // namespace

extern "C" {

int fg_mol_create(const fg_params *params, int32_t n_sites, int32_t sites_per_molecule, fg_molsys **out) {
    if (!params || !out) return fail(FG_ERR_INVALID, "null argument");
    *out = nullptr;
    const fg_params &P = *params;
    if (P.model != FG_MODEL_MULTIPOLE_RF) return fail(FG_ERR_INVALID, "fg_mol_create needs FG_MODEL_MULTIPOLE_RF");
    if (sites_per_molecule < 1 || sites_per_molecule > fgm::kMaxGroupSites)
        return fail(FG_ERR_INVALID, "sites per molecule must be 1..%d", fgm::kMaxGroupSites);
    if (n_sites < 2 * sites_per_molecule || n_sites % sites_per_molecule)
        return fail(FG_ERR_INVALID, "site count must be a multiple (>= 2) of the molecule size");
    if (n_sites >= (1 << 23)) return fail(FG_ERR_CAPACITY, "at most 2^23 sites");
    if (P.n_types < 1 || P.n_types > FG_MAX_TYPES) return fail(FG_ERR_INVALID, "bad type count");
    const double Lmin = std::min(P.box[0], std::min(P.box[1], P.box[2]));
    if (!(P.rf_cutoff > 0) || !(P.rf_cutoff < 0.5 * Lmin)) return fail(FG_ERR_INVALID, "cutoff must be in (0, L/2)");
    if (!(P.bjerrum > 0) || !(P.rf_eps_r > 0) || !(P.rf_eps_rf > 0)) return fail(FG_ERR_INVALID, "bad dielectric");
    fg_molsys *h = new fg_molsys();
    h->P = P;
    h->N = n_sites;
    h->gs = sites_per_molecule;
    h->M = n_sites / sites_per_molecule;
    auto bail = [&](int rc) {
        mol_free(h);
        delete h;
        return rc;
    };
    if (cudaGetDevice(&h->device) != cudaSuccess) return bail(fail(FG_ERR_CUDA, "no CUDA device"));
    if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess)
        return bail(fail(FG_ERR_CUDA, "stream"));
    cudaEventCreate(&h->ev0);
    cudaEventCreate(&h->ev1);
    fgm::MolDesc &d = h->desc;
    d.N = h->N;
    d.gs = h->gs;
    d.M = h->M;
    d.nt = P.n_types;
    bool uniform = true;
    for (int i = 0; i < P.n_types; i++)
        if (P.type_sigma[i] != P.type_sigma[0] || P.type_eps[i] != P.type_eps[0]) uniform = false;
    d.uniform_lj = uniform ? 1 : 0;
    for (int a = 0; a < 3; a++) {
        d.s32[a] = (float)(P.box[a] / 4294967296.0);
        d.s32sqd[a] = (P.box[a] / 4294967296.0) * (P.box[a] / 4294967296.0);
        d.s64d[a] = P.box[a] / TWO64;
        d.inv64d[a] = TWO64 / P.box[a];
    }
    const double rc = P.rf_cutoff;
    d.lB = (float)P.bjerrum;
    d.lBd = P.bjerrum;
    d.rc2 = (float)(rc * rc);
    d.rc2near = (float)((rc + 0.05) * (rc + 0.05));
    d.rc1i = (float)(1.0 / rc);
    d.rcd = rc;
    const double a2 = -66.0 * 1494.0 / 56916.0;   // CoulombGalore Q5 coefficient at kappa = 0
    d.A5 = (float)(5.0 / 22.0 * a2 - 0.6);
    d.B5 = (float)(9.0 / 22.0 * a2 - 1.2);
    d.rfBd = -(2 * (P.rf_eps_rf - P.rf_eps_r) / (2 * P.rf_eps_rf + P.rf_eps_r)) / P.rf_eps_r;
    d.rfB = (float)d.rfBd;
    d.cubic = (P.box[0] == P.box[1] && P.box[1] == P.box[2]) ? 1 : 0;
    d.s32sq = (float)((P.box[0] / 4294967296.0) * (P.box[0] / 4294967296.0));
    {
        const double u = rc / (P.box[0] / 4294967296.0);   // rc in high-word units
        d.rc2int = (long long)std::ceil(u * u);
    }
    d.kT = (float)(P.kT_scale > 0 ? P.kT_scale : 1.0);
    const int nt = P.n_types;
    for (int i = 0; i < nt; i++) {
        d.qtype[i] = (float)P.type_charge[i];
        for (int j = 0; j < nt; j++) {
            const double sig = 0.5 * (P.type_sigma[i] + P.type_sigma[j]);
            const double e4 = 4 * std::sqrt(P.type_eps[i] * P.type_eps[j]);
            d.s2[i * nt + j] = (float)(sig * sig);
            d.eps4[i * nt + j] = (float)e4;
            d.s2d[i * nt + j] = sig * sig;
            d.eps4d[i * nt + j] = e4;
            d.lbqq[i * nt + j] = (float)(P.bjerrum * P.type_charge[i] * P.type_charge[j]);
        }
    }
    if (uniform) {
        d.s2[0] = (float)(P.type_sigma[0] * P.type_sigma[0]);
        d.eps4[0] = (float)(4 * P.type_eps[0]);
    }
    int rc_;
#define TRY(x)                 \
    do {                       \
        rc_ = (x);             \
        if (rc_) return bail(rc_); \
    } while (0)
    TRY(mol_dmalloc(h, (void **)&h->d_desc, sizeof(fgm::MolDesc)));
    TRY(mol_dmalloc(h, (void **)&h->mus, (size_t)h->N * sizeof(double)));
    TRY(mol_dmalloc(h, (void **)&h->pos4, (size_t)h->N * sizeof(int4)));
    TRY(mol_dmalloc(h, (void **)&h->site_dip, (size_t)h->N * sizeof(int32_t)));
    TRY(mol_dmalloc(h, (void **)&h->sc, sizeof(fgm::MolScalars)));
    TRY(mol_dmalloc(h, (void **)&h->expl_pos, (size_t)h->gs * 3 * sizeof(int64_t)));
    TRY(mol_dmalloc(h, (void **)&h->expl_mu, (size_t)h->gs * 3 * sizeof(double)));
    TRY(mol_dmalloc(h, (void **)&h->expl_cm, 3 * sizeof(int64_t)));
    TRY(mol_dmalloc(h, (void **)&h->eval_du, sizeof(double)));
    TRY(mol_dmalloc(h, (void **)&h->tot, 2 * sizeof(double)));
    d.mus = h->mus;
    d.pos4 = h->pos4;
    d.site_dip = h->site_dip;
    d.sc = h->sc;
    d.eval_du = h->eval_du;
    h->max_cluster = mol_max_cluster(h);
    // default: enough CTAs that each owns <= ~1250 sites, within what the device runs
    int C = 1;
    while (C < h->max_cluster && (h->N + C - 1) / C > 1250) C *= 2;
    h->C = C;
    TRY(mol_alloc_replicas(h, C));
    TRY(mol_ensure_trials(h, 1, false));
    fgm::MolScalars s{};
    TRY(mol_write_scalars(h, s));
#undef TRY
    *out = h;
    return FG_OK;
}

int fg_mol_destroy(fg_molsys *h) {
    if (!h) return FG_OK;
    cudaStreamSynchronize(h->stream);
    mol_free(h);
    delete h;
    return FG_OK;
}

int fg_mol_set_state(fg_molsys *h, const double *xyz, const double *mu_unit, const double *mu_scalar,
                     const int32_t *type_ids, const double *mass_centers) {
    if (!h || !xyz || !type_ids) return fail(FG_ERR_INVALID, "null argument");
    const int N = h->N;
    std::vector<int64_t> X(3 * (size_t)N), CM(3 * (size_t)h->M);
    std::vector<double> MU(3 * (size_t)N, 0.0);
    std::vector<int4> p4(N);
    std::vector<int32_t> sd(N, -1), ds;
    h->types.assign(type_ids, type_ids + N);
    h->mus_h.assign(N, 0.0);
    for (int i = 0; i < N; i++) {
        if (type_ids[i] < 0 || type_ids[i] >= h->P.n_types) return fail(FG_ERR_INVALID, "bad type id at %d", i);
        for (int a = 0; a < 3; a++) {
            if (!std::isfinite(xyz[3 * i + a])) return fail(FG_ERR_INVALID, "non-finite position at %d", i);
            X[3 * i + a] = to_fix(xyz[3 * i + a], h->P.box[a]);
        }
        const double m = mu_scalar ? mu_scalar[i] : 0.0;
        if (m != 0.0) {
            if (!mu_unit) return fail(FG_ERR_INVALID, "dipole scalars need unit vectors");
            for (int a = 0; a < 3; a++) MU[3 * i + a] = mu_unit[3 * i + a];
            sd[i] = (int32_t)ds.size();
            ds.push_back(i);
        } else if (mu_unit) {
            for (int a = 0; a < 3; a++) MU[3 * i + a] = mu_unit[3 * i + a];
        }
        h->mus_h[i] = m;
        p4[i] = make_int4(hi32h(X[3 * i]), hi32h(X[3 * i + 1]), hi32h(X[3 * i + 2]), type_ids[i]);
    }
    for (int g = 0; g < h->M; g++) {
        if (mass_centers)
            for (int a = 0; a < 3; a++) CM[3 * g + a] = to_fix(mass_centers[3 * g + a], h->P.box[a]);
        else
            mol_mass_center(X.data(), g * h->gs, h->gs, &CM[3 * g]);
    }
    const int D = (int)ds.size();
    if (D != h->D || !h->dip4) {
        if (h->dip4) cudaFree(h->dip4);
        if (h->dip_pos4) cudaFree(h->dip_pos4);
        if (h->dip_site) cudaFree(h->dip_site);
        h->dip4 = nullptr;
        h->dip_pos4 = nullptr;
        h->dip_site = nullptr;
        MOL_DMALLOC(h->dip4, (size_t)std::max(D, 1) * sizeof(float4));
        MOL_DMALLOC(h->dip_pos4, (size_t)std::max(D, 1) * sizeof(int4));
        MOL_DMALLOC(h->dip_site, (size_t)std::max(D, 1) * sizeof(int32_t));
        h->D = D;
    }
    std::vector<float4> d4(std::max(D, 1));
    std::vector<int4> dp4(std::max(D, 1));
    for (int k = 0; k < D; k++) {
        const int i = ds[k];
        const double m = h->mus_h[i];
        d4[k] = make_float4((float)(MU[3 * i] * m), (float)(MU[3 * i + 1] * m), (float)(MU[3 * i + 2] * m), (float)m);
        dp4[k] = make_int4(p4[i].x, p4[i].y, p4[i].z, (i << 8) | type_ids[i]);
    }
    fgm::MolDesc &d = h->desc;
    d.D = D;
    d.dip4 = h->dip4;
    d.dip_pos4 = h->dip_pos4;
    d.dip_site = h->dip_site;
    cudaStream_t st = h->stream;
    for (int r = 0; r < h->C; r++) {
        CK(cudaMemcpyAsync(h->rep_pos + (size_t)r * N * 3, X.data(), X.size() * 8, cudaMemcpyHostToDevice, st));
        CK(cudaMemcpyAsync(h->rep_mu + (size_t)r * N * 3, MU.data(), MU.size() * 8, cudaMemcpyHostToDevice, st));
        CK(cudaMemcpyAsync(h->rep_cm + (size_t)r * h->M * 3, CM.data(), CM.size() * 8, cudaMemcpyHostToDevice, st));
    }
    CK(cudaMemcpyAsync(h->mus, h->mus_h.data(), (size_t)N * 8, cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(h->pos4, p4.data(), (size_t)N * sizeof(int4), cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(h->site_dip, sd.data(), (size_t)N * 4, cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(h->dip4, d4.data(), (size_t)std::max(D, 1) * sizeof(float4), cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(h->dip_pos4, dp4.data(), (size_t)std::max(D, 1) * sizeof(int4), cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(h->dip_site, ds.empty() ? sd.data() : ds.data(), (size_t)std::max(D, 1) * 4,
                       cudaMemcpyHostToDevice, st));
    int rc = mol_push_desc(h);
    if (rc) return rc;
    double tot[2];
    rc = mol_total(h, tot);
    if (rc) return rc;
    fgm::MolScalars s{};
    const float2 u = split_df(tot[0] + tot[1]);
    s.utot_hi = u.x;
    s.utot_lo = u.y;
    s.n_trials = h->n_stream;   // the stream that is staged runs on the new state, from its first trial
    rc = mol_write_scalars(h, s);
    if (rc) return rc;
    h->pending = -1;
    h->state_set = true;
    return FG_OK;
}

int fg_mol_get_state(fg_molsys *h, double *xyz, double *mu_unit, double *mass_centers) {
    if (!h || !h->state_set) return fail(FG_ERR_STATE, "no state");
    const int N = h->N;
    std::vector<int64_t> X(3 * (size_t)N), CM(3 * (size_t)h->M);
    std::vector<double> MU(3 * (size_t)N);
    CK(cudaMemcpyAsync(X.data(), h->rep_pos, X.size() * 8, cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(MU.data(), h->rep_mu, MU.size() * 8, cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(CM.data(), h->rep_cm, CM.size() * 8, cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    for (int i = 0; i < N; i++)
        for (int a = 0; a < 3; a++) {
            if (xyz) xyz[3 * i + a] = from_fix(X[3 * i + a], h->P.box[a]);
            if (mu_unit) mu_unit[3 * i + a] = MU[3 * i + a];
        }
    if (mass_centers)
        for (int g = 0; g < h->M; g++)
            for (int a = 0; a < 3; a++) mass_centers[3 * g + a] = from_fix(CM[3 * g + a], h->P.box[a]);
    return FG_OK;
}

int fg_mol_set_cluster(fg_molsys *h, int32_t ctas) {
    if (!h) return fail(FG_ERR_INVALID, "null handle");
    if (ctas < 1 || ctas > h->max_cluster || (ctas & (ctas - 1)))
        return fail(FG_ERR_INVALID, "cluster size must be a power of two in 1..%d", h->max_cluster);
    if (ctas == h->C) return FG_OK;
    std::vector<int64_t> X, CM;
    std::vector<double> MU;
    if (h->state_set) {
        X.resize(3 * (size_t)h->N);
        MU.resize(3 * (size_t)h->N);
        CM.resize(3 * (size_t)h->M);
        CK(cudaMemcpyAsync(X.data(), h->rep_pos, X.size() * 8, cudaMemcpyDeviceToHost, h->stream));
        CK(cudaMemcpyAsync(MU.data(), h->rep_mu, MU.size() * 8, cudaMemcpyDeviceToHost, h->stream));
        CK(cudaMemcpyAsync(CM.data(), h->rep_cm, CM.size() * 8, cudaMemcpyDeviceToHost, h->stream));
        CK(cudaStreamSynchronize(h->stream));
    }
    int rc = mol_alloc_replicas(h, ctas);
    if (rc) return rc;
    h->C = ctas;
    if (h->state_set) {
        for (int r = 0; r < ctas; r++) {
            CK(cudaMemcpyAsync(h->rep_pos + (size_t)r * h->N * 3, X.data(), X.size() * 8, cudaMemcpyHostToDevice,
                               h->stream));
            CK(cudaMemcpyAsync(h->rep_mu + (size_t)r * h->N * 3, MU.data(), MU.size() * 8, cudaMemcpyHostToDevice,
                               h->stream));
            CK(cudaMemcpyAsync(h->rep_cm + (size_t)r * h->M * 3, CM.data(), CM.size() * 8, cudaMemcpyHostToDevice,
                               h->stream));
        }
        CK(cudaStreamSynchronize(h->stream));
    }
    return mol_push_desc(h);
}

int fg_mol_get_cluster(fg_molsys *h, int32_t *ctas, int32_t *max_ctas) {
    if (!h) return fail(FG_ERR_INVALID, "null handle");
    if (ctas) *ctas = h->C;
    if (max_ctas) *max_ctas = h->max_cluster;
    return FG_OK;
}

int fg_mol_trial_du(fg_molsys *h, int32_t molecule, const double *new_xyz, const double *new_mu_unit,
                    const double *new_mass_center, double *du) {
    if (!h || !new_xyz || !du) return fail(FG_ERR_INVALID, "null argument");
    if (!h->state_set) return fail(FG_ERR_STATE, "fg_mol_set_state first");
    if (h->pending >= 0) return fail(FG_ERR_STATE, "a trial is pending: call fg_mol_commit");
    if (h->staged) return fail(FG_ERR_STATE, "a staged stream is waiting: run it first");
    if (molecule < 0 || molecule >= h->M) return fail(FG_ERR_INVALID, "molecule index out of range");
    std::vector<int64_t> X(3 * (size_t)h->gs);
    for (int s = 0; s < h->gs; s++)
        for (int a = 0; a < 3; a++) X[3 * s + a] = to_fix(new_xyz[3 * s + a], h->P.box[a]);
    CK(cudaMemcpyAsync(h->expl_pos, X.data(), X.size() * 8, cudaMemcpyHostToDevice, h->stream));
    if (new_mu_unit)
        CK(cudaMemcpyAsync(h->expl_mu, new_mu_unit, (size_t)h->gs * 3 * 8, cudaMemcpyHostToDevice, h->stream));
    int64_t cm[3];
    if (new_mass_center) {
        for (int a = 0; a < 3; a++) cm[a] = to_fix(new_mass_center[a], h->P.box[a]);
        CK(cudaMemcpyAsync(h->expl_cm, cm, sizeof(cm), cudaMemcpyHostToDevice, h->stream));
    }
    fgm::MolTrial t{};
    t.g = molecule;
    t.flags = 4;
    t.qw = 1.0;
    CK(cudaMemcpyAsync(h->trials, &t, sizeof(t), cudaMemcpyHostToDevice, h->stream));
    h->desc.expl_pos = h->expl_pos;
    h->desc.expl_mu = new_mu_unit ? h->expl_mu : nullptr;
    h->desc.expl_cm = new_mass_center ? h->expl_cm : nullptr;
    h->desc.trials = h->trials;
    int rc = mol_push_desc(h);
    if (rc) return rc;
    MolLaunch L;
    rc = mol_pick<true>(h, L);
    if (rc) return rc;
    rc = mol_launch(h, L, h->d_desc, 1, h->stream);
    if (rc) return rc;
    CK(cudaMemcpyAsync(du, h->eval_du, sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    h->pending = molecule;
    h->pending_du = *du;
    return FG_OK;
}

int fg_mol_commit(fg_molsys *h, int32_t accepted) {
    if (!h) return fail(FG_ERR_INVALID, "null handle");
    if (h->pending < 0) return fail(FG_ERR_STATE, "no pending trial");
    const int g = h->pending;
    h->pending = -1;
    if (!accepted) return FG_OK;
    fgm::mol_commit_kernel<<<1, 64, 0, h->stream>>>(h->d_desc, g, 1, h->C);
    CK(cudaGetLastError());
    fgm::MolScalars s;
    int rc = mol_read_scalars(h, s);
    if (rc) return rc;
    s.n_accepted++;
    const double ut = df_val(s.utot_hi, s.utot_lo) + h->pending_du;
    const float2 f = split_df(ut);
    s.utot_hi = f.x;
    s.utot_lo = f.y;
    return mol_write_scalars(h, s);
}

// Reference draws for n TranslateRotate trials on one molecule kind
// ("permol"), consuming the global slump as move.h:1624-1685 and 567-573 do.
int fg_mol_draw_stream(uint32_t seed, int32_t n_molecules, int64_t n, double dp, double dprot,
                       int32_t center_rotation, int32_t *mol, double *axis, int32_t *center, double *angle,
                       double *trans, double *u) {
    if (n_molecules < 1 || n < 0 || (n > 0 && (!mol || !u))) return fail(FG_ERR_INVALID, "bad argument");
    std::mt19937 eng(seed);
    std::uniform_real_distribution<double> U(0, 1);
    for (int64_t k = 0; k < n; k++) {
        std::uniform_int_distribution<int> pick(0, n_molecules - 1);
        mol[k] = pick(eng);                                     // slump.element(gvec)
        double v[3] = {0, 0, 0}, ang = 0.0, t[3] = {0, 0, 0};
        int c = 0;
        if (dprot > 1e-6) {
            double r2;
            do {                                                // Point::ranunit (point.h:74-88)
                for (int a = 0; a < 3; a++) v[a] = (2 * U(eng) - 1) * 1.0;
                r2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
            } while (r2 > 1);
            const double s = std::sqrt(r2);
            for (int a = 0; a < 3; a++) v[a] /= s;
            if (!center_rotation) c = (U(eng) < 0.5) ? 1 : 2;
            ang = dprot * (U(eng) - 0.5);                       // slump.half()
        }
        if (dp > 1e-6)
            for (int a = 0; a < 3; a++) t[a] = 1.0 * dp * (U(eng) - 0.5);
        const double um = U(eng);                               // Movebase::metropolis
        for (int a = 0; a < 3; a++) {
            if (axis) axis[3 * k + a] = v[a];
            if (trans) trans[3 * k + a] = t[a];
        }
        if (center) center[k] = c;
        if (angle) angle[k] = ang;
        u[k] = um;
    }
    return FG_OK;
}

// n TranslateRotate trials on the device. rotate/translate say whether the
// move has dprot/dp above 1e-6 (move.h:1642, 1671); the arrays are the draws
// (fg_mol_draw_stream). acc/du (may be NULL) receive per-trial results.
int fg_mol_stream_upload(fg_molsys *h, int64_t n, const int32_t *mol, const double *axis, const double *angle,
                         const int32_t *center, const double *trans, const double *u, int32_t rotate,
                         int32_t translate) {
    return mol_upload(h, n, mol, axis, angle, center, trans, u, rotate, translate, false);
}

int fg_mol_run_many(fg_molsys *const *systems, int32_t n_systems, fg_sweep_stats *per_system, fg_sweep_stats *total) {
    return mol_run(systems, n_systems, per_system, total);
}

int fg_mol_sweep(fg_molsys *h, int64_t n, const int32_t *mol, const double *axis, const double *angle,
                 const int32_t *center, const double *trans, const double *u, int32_t rotate, int32_t translate,
                 uint8_t *acc, double *du, fg_sweep_stats *stats) {
    const bool log = acc || du;
    int rc = mol_upload(h, n, mol, axis, angle, center, trans, u, rotate, translate, log);
    if (rc) return rc;
    fg_sweep_stats st{};
    rc = mol_run(&h, 1, nullptr, &st);
    if (stats) *stats = st;
    if (rc) return rc;
    if (log && n > 0) {
        std::vector<float2> l(n);
        std::vector<uint8_t> a(n);
        CK(cudaMemcpyAsync(l.data(), h->log_du, n * sizeof(float2), cudaMemcpyDeviceToHost, h->stream));
        CK(cudaMemcpyAsync(a.data(), h->log_acc, n, cudaMemcpyDeviceToHost, h->stream));
        CK(cudaStreamSynchronize(h->stream));
        for (int64_t k = 0; k < n; k++) {
            if (du) du[k] = df_val(l[k].x, l[k].y);
            if (acc) acc[k] = a[k];
        }
    }
    return FG_OK;
}

// comp = {intermolecular, intramolecular, total} in FP64 (systemEnergy).
int fg_mol_total_energy(fg_molsys *h, double *comp) {
    if (!h || !comp) return fail(FG_ERR_INVALID, "null argument");
    if (!h->state_set) return fail(FG_ERR_STATE, "no state");
    double t[2];
    int rc = mol_total(h, t);
    if (rc) return rc;
    comp[0] = t[0];
    comp[1] = t[1];
    comp[2] = t[1] + t[0];
    return FG_OK;
}

// Running total energy (initial total + accepted dU since fg_mol_set_state).
int fg_mol_running_energy(fg_molsys *h, double *u) {
    if (!h || !u) return fail(FG_ERR_INVALID, "null argument");
    fgm::MolScalars s;
    int rc = mol_read_scalars(h, s);
    if (rc) return rc;
    *u = df_val(s.utot_hi, s.utot_lo);
    return FG_OK;
}

int64_t fg_mol_device_bytes(fg_molsys *h) { return h ? (int64_t)h->device_bytes : 0; }

}  // extern "C"
