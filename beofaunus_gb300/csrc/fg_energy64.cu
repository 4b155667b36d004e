// FP64 system energy on the device (included by fg_api.cu): the reference's
// systemEnergy (energy.h:169-180) with every term in double precision, for
// moves whose dU is a difference of whole-system energies (the isobaric
// volume move) and for energy reports that need more than the FP32 pair
// path's ~1e-4 kT.
//
//   pairs: EwaldReal (ewald.h:97-110: the kappa-screened erfc form with the
//          effective charges' QeQe) + WeeksChandlerAndersen
//          (potentials.h:2186-2193), or DebyeHuckel (potentials.h:3314-3323)
//          + LennardJonesMixed (potentials.h:2036-2040), over all pairs i < j
//          with the minimum-image distance from the 64-bit fixed-point
//          difference;
//   Q(k):  sum_j q_j eff_j e^{i k.r_j} (ewald.h:388-415) with the phase
//          2 pi (n . X mod 2^64) / 2^64 taken exactly in integers, then sincos
//          in FP64; the reciprocal, self and surface terms are formed on the
//          host (ewald.h:259-311).
// Partial sums are formed and added in a fixed order, so the result does not
// depend on timing.
//
// GB300 issues FP64 at 1/64 of its FP32 rate (about 60 cycles per warp
// instruction and SM quarter), so FP64 is spent only on pairs that count.
// Ewald pairs: tiles of the pair triangle over all SMs; every pair is screened
// in FP32 on the 32-bit minimum image against the largest radius at which any
// term acts (reach), the few that pass (1.5 % at 8192 ions, rc 20 A) are
// queued per warp and evaluated in FP64 with all lanes busy, at each box's
// scale. Q(k): per-axis tables e^{i n x} in FP64 from the exact phases, one
// complex product per run of k-vectors and four FMAs per k-vector and
// particle instead of a sincos. 8192 ions, rc 20 A, kc 8 (1152 k-vectors):
// pairs 51 ms -> 0.29 ms per box (all pairs in FP64 on 32 blocks before), Q(k)
// 2.0 ms -> 0.16 ms. Bound: the FP64 pipe (erfc of the pairs inside the
// cutoff; the tables' sincos).
namespace fg {

constexpr int kE64Threads = 128;   // i particles of a tile, one per thread
constexpr int kE64Tile = 128;      // j particles of a tile
constexpr int kE64MaxBlocks = 2048;   // partial sums per box

struct E64Pair {       // per type pair (row-major nt x nt)
    double s2, eps4, qeqe, wca2;
};

// What one box needs: units of a coordinate (L / 2^64) and, for the FP32
// screen, of its high word (L / 2^32).
struct E64Box {
    double s3[3];
    float s32[3];
};

// Energy of one pair at the squared distance r2 (kT / e^2 units of the pair
// tables); 1/r from one FP64 rsqrt serves every term.
__device__ __forceinline__ double e64_pair(double r2, double qq, const E64Pair &P, double lB, double alpha,
                                           double kappa, double k2a, double rc2, int ewald) {
    const double ri = rsqrt(r2);
    double x = P.s2 * (ri * ri);
    x = x * x * x;
    if (!ewald) return lB * qq * exp(-kappa * (r2 * ri)) * ri + P.eps4 * (x * x - x);
    double u = 0.0;
    if (r2 <= rc2) {
        const double r = r2 * ri;
        if (k2a == 0.0) u = qq * P.qeqe * lB * erfc(alpha * r) * ri;
        else
            u = qq * P.qeqe * lB * 0.5 *
                (erfc(alpha * r + k2a) * exp(kappa * r) + erfc(alpha * r - k2a) * exp(-kappa * r)) * ri;
    }
    if (r2 <= P.wca2) u += P.eps4 * (x * x - x + 0.25);
    return u;
}

__device__ __forceinline__ double e64_r2(const long long *xi, const long long *xj, const E64Box &b) {
    double r2 = 0.0;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const double x = (double)(long long)((unsigned long long)xi[a] - (unsigned long long)xj[a]) * b.s3[a];
        r2 = fma(x, x, r2);
    }
    return r2;
}

// Pairs i < j of NBOX boxes (the same fixed-point positions at each box's
// scale). Block b takes the tiles b, b + gridDim.x, ... of the rectangle of
// (i tile, j tile), skipping those below the diagonal. reach2: no Ewald or
// WCA term acts beyond it, with the host's margin for the screen's rounding;
// part gets one sum per box and block.
template <int NBOX>
__global__ void __launch_bounds__(kE64Threads) energy64_pairs_kernel(const SysDesc *__restrict__ dsc,
                                                                   const double *__restrict__ q,
                                                                   const E64Pair *__restrict__ tp, int nt,
                                                                   E64Box b0, E64Box b1, double lB, double alpha,
                                                                   double kappa, double rc2, float reach2, int ewald,
                                                                   double *__restrict__ part) {
    constexpr int kWarps = kE64Threads / 32;
    __shared__ int4 hj[kE64Tile];
    __shared__ int queue[kWarps][32];   // i - i0 | (j - j0) << 16
    __shared__ double red[NBOX][kWarps];
    const SysDesc &d = *dsc;
    const int N = d.N, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nti = (N + kE64Threads - 1) / kE64Threads, ntj = (N + kE64Tile - 1) / kE64Tile;
    const double k2a = ewald && kappa > 0.0 ? kappa / (2.0 * alpha) : 0.0;
    double acc[NBOX];
#pragma unroll
    for (int b = 0; b < NBOX; b++) acc[b] = 0.0;
    auto add = [&](int i, int j) {
        const double qq = q[i] * q[j];
        const E64Pair P = tp[d.ptype[i] * nt + d.ptype[j]];
        long long xi[3], xj[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            xi[a] = d.pos64[3 * i + a];
            xj[a] = d.pos64[3 * j + a];
        }
#pragma unroll
        for (int b = 0; b < NBOX; b++)
            acc[b] += e64_pair(e64_r2(xi, xj, b ? b1 : b0), qq, P, lB, alpha, kappa, k2a, rc2, ewald);
    };
    for (long long t = blockIdx.x; t < (long long)nti * ntj; t += gridDim.x) {
        const int i0 = (int)(t / ntj) * kE64Threads, j0 = (int)(t % ntj) * kE64Tile;
        const int nj = min(kE64Tile, N - j0);
        if (j0 + nj - 1 <= i0) continue;   // nothing above the diagonal
        __syncthreads();
        for (int k = tid; k < nj; k += kE64Threads) hj[k] = d.pos4[j0 + k];
        __syncthreads();
        const int i = i0 + tid;
        if (!ewald) {   // no cutoff: every pair counts
            if (i < N)
                for (int k = max(0, i + 1 - j0); k < nj; k++) add(i, j0 + k);
            continue;
        }
        const int4 hi = i < N ? d.pos4[i] : make_int4(0, 0, 0, 0);
        int qn = 0;
        for (int k = 0; k < nj; k++) {
            const int4 p = hj[k];
            const float dx = (float)(int)((uint32_t)p.x - (uint32_t)hi.x);
            const float dy = (float)(int)((uint32_t)p.y - (uint32_t)hi.y);
            const float dz = (float)(int)((uint32_t)p.z - (uint32_t)hi.z);
            bool in = false;
#pragma unroll
            for (int b = 0; b < NBOX; b++) {
                const E64Box &B = b ? b1 : b0;
                const float x = dx * B.s32[0], y = dy * B.s32[1], z = dz * B.s32[2];
                in |= fmaf(x, x, fmaf(y, y, z * z)) <= reach2;
            }
            in = in && i < N && j0 + k > i;
            const uint32_t m = __ballot_sync(0xffffffffu, in);
            if (!m) continue;
            const int c = __popc(m);
            if (qn + c > 32) {
                __syncwarp();
                if (lane < qn) add(i0 + (queue[warp][lane] & 0xFFFF), j0 + (queue[warp][lane] >> 16));
                __syncwarp();
                qn = 0;
            }
            if (in) queue[warp][qn + __popc(m & ((1u << lane) - 1u))] = tid | (k << 16);
            qn += c;
        }
        __syncwarp();
        if (lane < qn) add(i0 + (queue[warp][lane] & 0xFFFF), j0 + (queue[warp][lane] >> 16));
        __syncwarp();
    }
#pragma unroll
    for (int b = 0; b < NBOX; b++) {
        double v = acc[b];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) red[b][warp] = v;
    }
    __syncthreads();
    if (tid < NBOX) {
        double s = 0.0;
        for (int w = 0; w < kWarps; w++) s += red[tid][w];
        part[(size_t)tid * gridDim.x + blockIdx.x] = s;
    }
}

// Partial Q(k) of the particles [blockIdx.x chunk, + chunk): one thread per run
// of k-vectors with the same (nx, ny) (kseg, at most kQkRun consecutive nz).
// The block builds the per-axis tables e^{i n 2 pi x_a / L_a}, n = 0..kcc, of
// kE64Stage particles at a time from the exact phases n X mod 2^64; a thread
// forms w = q eff e_x e_y once per particle and w e_z per k (e(-n) = conj).
// isotropic_pbc: the same with (cos, 0) tables, i.e. q eff cos cos cos.
constexpr int kE64Stage = 32;
constexpr int kE64QkThreads = 256;
__host__ __device__ inline size_t e64_qk_smem(int kcc) { return (size_t)kE64Stage * (3 * (kcc + 1) * 16 + 8); }
__global__ void __launch_bounds__(kE64QkThreads) energy64_qk_kernel(const SysDesc *__restrict__ dsc,
                                                                  const double *__restrict__ qe, int chunk,
                                                                  double2 *__restrict__ part) {
    extern __shared__ __align__(16) unsigned char e64_raw[];
    const SysDesc &d = *dsc;
    const int kcc = d.kcc, A = kcc + 1, T = 3 * A, tid = threadIdx.x;
    double2 *tab = reinterpret_cast<double2 *>(e64_raw);           // [stage][T]
    double *qs = reinterpret_cast<double *>(tab + kE64Stage * T);   // [stage]
    const int j0 = blockIdx.x * chunk, j1 = min(d.N, j0 + chunk);
    const int r = blockIdx.y * blockDim.x + tid;
    int k0 = 0, len = 0, nx = 0, ny = 0, nz = 0;
    if (r < d.nseg) {
        const int2 sg = d.kseg[r];
        k0 = sg.x & 0xFFFFFF;
        len = sg.x >> 24;
        nx = (int)(int8_t)(sg.y & 0xFF);
        ny = (int)(int8_t)((sg.y >> 8) & 0xFF);
        nz = (int)(int8_t)((sg.y >> 16) & 0xFF);
    }
    double re[kQkRun], im[kQkRun];
#pragma unroll
    for (int u = 0; u < kQkRun; u++) re[u] = im[u] = 0.0;
    for (int b = j0; b < j1; b += kE64Stage) {
        const int nb = min(kE64Stage, j1 - b);
        __syncthreads();
        for (int e = tid; e < nb * T; e += blockDim.x) {
            const int j = e / T, t = e - j * T, axis = t / A, n = t - axis * A;
            const unsigned long long ph = (unsigned long long)n * (unsigned long long)d.pos64[3 * (b + j) + axis];
            double s, c;
            // 2 pi / 2^64 times the signed turn fraction
            sincos((double)(long long)ph * 3.4061215800865545e-19, &s, &c);
            tab[e] = make_double2(c, d.iso ? 0.0 : s);
        }
        for (int j = tid; j < nb; j += blockDim.x) qs[j] = qe[b + j];
        __syncthreads();
        if (len == 0) continue;
        const int ay = ny < 0 ? -ny : ny;
        const double sy = ny < 0 ? -1.0 : 1.0;
        for (int j = 0; j < nb; j++) {
            const double2 *e = tab + j * T;
            const double2 ex = e[nx], ey = e[A + ay];
            const double ax = qs[j] * ex.x, ai = qs[j] * ex.y, eyi = sy * ey.y;
            const double wx = ax * ey.x - ai * eyi, wy = ax * eyi + ai * ey.x;
#pragma unroll
            for (int u = 0; u < kQkRun; u++)
                if (u < len) {
                    const int n = nz + u;
                    const double2 z = e[2 * A + (n < 0 ? -n : n)];
                    const double zi = n < 0 ? -z.y : z.y;
                    re[u] = fma(wx, z.x, fma(-wy, zi, re[u]));
                    im[u] = fma(wx, zi, fma(wy, z.x, im[u]));
                }
        }
    }
#pragma unroll
    for (int u = 0; u < kQkRun; u++)
        if (u < len) part[(size_t)blockIdx.x * d.K + k0 + u] = make_double2(re[u], im[u]);
}
// |Q(k)|^2 from the chunks' partial sums, one warp per k-vector: lane l adds
// the chunks l, l + 32, ..., then a shuffle tree (a fixed order).
__global__ void energy64_qk_sum_kernel(const double2 *__restrict__ part, int nchunk, int K, double *__restrict__ q2) {
    const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (k >= K) return;
    double re = 0.0, im = 0.0;
    for (int c = lane; c < nchunk; c += 32) {
        const double2 p = part[(size_t)c * K + k];
        re += p.x;
        im += p.y;
    }
    for (int o = 16; o > 0; o >>= 1) {
        re += __shfl_xor_sync(0xffffffffu, re, o);
        im += __shfl_xor_sync(0xffffffffu, im, o);
    }
    if (lane == 0) q2[k] = re * re + im * im;
}

}  // namespace fg

namespace {

// The FP64 energy's and the g(r) sampling's device workspace: grown when a call
// needs more, and kept with the system (freed with it) up to kWork64Keep: a
// batch may ask every member for its energy.
constexpr size_t kWork64Keep = (size_t)4 << 20;
constexpr size_t kWork64Qk = (size_t)3 << 20;   // Q(k) partial sums for which more chunks are taken
void drop_work64(fg_system *h) {   // after the call's last synchronisation
    if (h->work64_cap <= kWork64Keep) return;
    cudaFree(h->work64);
    h->work64 = nullptr;
    h->device_bytes -= h->work64_cap;
    h->work64_cap = 0;
}
int ensure_work64(fg_system *h, size_t bytes) {
    if (bytes <= h->work64_cap) return FG_OK;
    if (h->work64) {
        CK(cudaStreamSynchronize(h->stream));
        cudaFree(h->work64);
        h->work64 = nullptr;
        h->device_bytes -= h->work64_cap;
        h->work64_cap = 0;
    }
    int rc = dmalloc(h, &h->work64, bytes);
    if (rc) return rc;
    h->work64_cap = bytes;
    return FG_OK;
}

// {pairs, reciprocal, self, surface, total} in kT, FP64 throughout, of the
// current configuration in each of nbox boxes: boxes[b] (box b's lengths;
// the fixed-point positions X = x / L 2^64 stand for x = X L / 2^64 in any
// box, so scaling every position with the box is the same X). Q(k) comes
// from one pass (its exact phases depend on X only), the pair sum from one
// pass per box at that box's scale, and the k-vector weights, reciprocal
// prefactor and surface term are those of each box (ewald.h:330-378, 277-311).
int total_energy_fp64_boxes(fg_system *h, int nbox, const double (*boxes)[3], double (*c)[5]) {
    const int N = h->N, nt = h->P.n_types, K = h->K;
    const fg_params &P = h->P;
    const bool ewald = h->model == FG_MODEL_EWALD_WCA;
    if (nbox < 1 || nbox > 2) return fail(FG_ERR_INVALID, "one or two boxes");
    std::vector<fg::E64Pair> tp((size_t)nt * nt);
    std::vector<double> eff(nt, 1.0);
    const double kappa = ewald ? 1.0 / P.ewald_debye_length : 1.0 / P.dh_debye_length;
    for (int i = 0; i < nt; i++) {
        const double ri = 0.5 * P.type_sigma[i];
        if (ewald && P.type_charge[i] != 0.0 && std::fabs(kappa * ri) > 1e-9) eff[i] = std::sinh(ri * kappa) / ri / kappa;
    }
    double reach2 = P.ewald_cutoff * P.ewald_cutoff;
    for (int i = 0; i < nt; i++)
        for (int j = 0; j < nt; j++) {
            const double sig = 0.5 * (P.type_sigma[i] + P.type_sigma[j]);
            fg::E64Pair &e = tp[(size_t)i * nt + j];
            e.s2 = sig * sig;
            e.eps4 = 4 * std::sqrt(P.type_eps[i] * P.type_eps[j]);
            e.qeqe = eff[i] * eff[j];
            e.wca2 = e.s2 * std::pow(2, 2 / 6.);
            reach2 = std::max(reach2, e.wca2);
        }
    std::vector<double> qe(N);
    for (int j = 0; j < N; j++) qe[j] = h->charges[j] * eff[h->types[j]];
    // pair tiles over at most kE64MaxBlocks blocks; Q(k) chunks of at most 1024
    // particles, whole stages, and as many as their partial sums fit kWork64Qk
    // (8192 ions, K = 1152: 128 chunks of two stages)
    const long long nti = (N + fg::kE64Threads - 1) / fg::kE64Threads, ntj = (N + fg::kE64Tile - 1) / fg::kE64Tile;
    const int nb = (int)std::min<long long>(fg::kE64MaxBlocks, nti * ntj);
    const int most = std::max((N + 1023) / 1024, K > 0 ? (int)std::min<size_t>(512, kWork64Qk / ((size_t)K * sizeof(double2))) : 1);
    const int chunk = ((N + most - 1) / most + fg::kE64Stage - 1) / fg::kE64Stage * fg::kE64Stage;
    const int nchunk = K > 0 ? (N + chunk - 1) / chunk : 0;
    // one workspace, kept with the system and grown when needed: q, qe, pair
    // tables, partial sums, |Q(k)|^2, Q(k) partial sums
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    size_t off[7];
    off[0] = 0;
    off[1] = off[0] + up(N * sizeof(double));
    off[2] = off[1] + up(N * sizeof(double));
    off[3] = off[2] + up(tp.size() * sizeof(fg::E64Pair));
    off[4] = off[3] + up((size_t)nbox * nb * sizeof(double));
    off[5] = off[4] + up((size_t)K * sizeof(double));
    off[6] = off[5] + up((size_t)nchunk * K * sizeof(double2));
    int rc = ensure_work64(h, off[6]);
    if (rc) return rc;
    char *w = (char *)h->work64;
    double *d_q = (double *)(w + off[0]), *d_qe = (double *)(w + off[1]), *d_part = (double *)(w + off[3]);
    double *d_q2 = (double *)(w + off[4]);
    double2 *d_qk = (double2 *)(w + off[5]);
    fg::E64Pair *d_tp = (fg::E64Pair *)(w + off[2]);
    CK(cudaMemcpyAsync(d_q, h->charges.data(), N * sizeof(double), cudaMemcpyHostToDevice, h->stream));
    CK(cudaMemcpyAsync(d_qe, qe.data(), N * sizeof(double), cudaMemcpyHostToDevice, h->stream));
    CK(cudaMemcpyAsync(d_tp, tp.data(), tp.size() * sizeof(fg::E64Pair), cudaMemcpyHostToDevice, h->stream));
    fg::E64Box B[2];
    double unit = 0;   // a high-word difference is off by at most one unit per axis
    for (int b = 0; b < 2; b++)
        for (int a = 0; a < 3; a++) {
            const double L = boxes[std::min(b, nbox - 1)][a];
            B[b].s3[a] = std::ldexp(L, -64);
            B[b].s32[a] = (float)std::ldexp(L, -32);
            unit = std::max(unit, std::ldexp(L, -32));
        }
    const double screen2 = reach2 * 1.00001 + 8.0 * std::sqrt(reach2) * unit + 16.0 * unit * unit;
    auto pairs_fn = nbox == 2 ? fg::energy64_pairs_kernel<2> : fg::energy64_pairs_kernel<1>;
    pairs_fn<<<nb, fg::kE64Threads, 0, h->stream>>>(h->d_desc, d_q, d_tp, nt, B[0], B[1], P.bjerrum,
                                                    ewald ? P.ewald_alpha : 0.0, kappa,
                                                    ewald ? P.ewald_cutoff * P.ewald_cutoff : 0.0, (float)screen2,
                                                    ewald ? 1 : 0, d_part);
    CK(cudaGetLastError());
    if (K > 0) {
        const size_t smem = fg::e64_qk_smem(h->kc);
        rc = set_smem_attr((const void *)fg::energy64_qk_kernel, smem);
        if (rc) return rc;
        fg::energy64_qk_kernel<<<dim3(nchunk, (h->nseg + fg::kE64QkThreads - 1) / fg::kE64QkThreads), fg::kE64QkThreads,
                                 smem, h->stream>>>(h->d_desc, d_qe, chunk, d_qk);
        CK(cudaGetLastError());
        fg::energy64_qk_sum_kernel<<<(K + 3) / 4, 128, 0, h->stream>>>(d_qk, nchunk, K, d_q2);
        CK(cudaGetLastError());
    }
    std::vector<double> part((size_t)nbox * nb), q2(K);
    CK(cudaMemcpyAsync(part.data(), d_part, part.size() * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    if (K > 0) CK(cudaMemcpyAsync(q2.data(), d_q2, K * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    drop_work64(h);
    double M0[3] = {0, 0, 0};  // sum q eff x in the current box
    if (K > 0) {
        std::vector<double> xyz(3 * (size_t)N);
        rc = fg_get_state(h, xyz.data());
        if (rc) return rc;
        for (int j = 0; j < N; j++)
            for (int a = 0; a < 3; a++) M0[a] += qe[j] * xyz[3 * j + a];
    }
    for (int b = 0; b < nbox; b++) {
        double pairs = 0;
        for (int i = 0; i < nb; i++) pairs += part[(size_t)b * nb + i];
        double rec = 0, self = 0, surf = 0;
        if (K > 0) {
            fg_params Pb = P;
            for (int a = 0; a < 3; a++) Pb.box[a] = boxes[b][a];
            const double V = Pb.box[0] * Pb.box[1] * Pb.box[2];
            std::vector<int> n3;
            std::vector<double> ak, kv3;
            enumerate_k(Pb, n3, ak, kv3);
            if ((int)ak.size() != K) return fail(FG_ERR_INVALID, "the k-vector set changes with the box");
            for (int k = 0; k < K; k++) rec += ak[k] * q2[k];
            rec *= 2 * PI / V * P.bjerrum;
            self = h->self_energy;
            const double const_inf = (P.ewald_eps_surf < 1) ? 0.0 : 1.0;
            const double surf_c = const_inf * (2 * PI / ((2 * P.ewald_eps_surf + 1) * V)) * P.bjerrum;
            double M2 = 0;
            for (int a = 0; a < 3; a++) {
                const double m = M0[a] * (boxes[b][a] / P.box[a]);
                M2 += m * m;
            }
            surf = surf_c * M2;
        }
        c[b][0] = pairs;
        c[b][1] = rec;
        c[b][2] = self;
        c[b][3] = surf;
        c[b][4] = (surf + rec) + (self + pairs);
    }
    return FG_OK;
}

int total_energy_fp64(fg_system *h, double *c) {
    const double box[1][3] = {{h->P.box[0], h->P.box[1], h->P.box[2]}};
    double out[1][5];
    int rc = total_energy_fp64_boxes(h, 1, box, out);
    if (rc) return rc;
    for (int i = 0; i < 5; i++) c[i] = out[0][i];
    return FG_OK;
}

}  // namespace

extern "C" int fg_total_energy_fp64(fg_system *h, double *components5) {
    if (!h || !components5) return fail(FG_ERR_INVALID, "null argument");
    if (h->types.empty()) return fail(FG_ERR_STATE, "fg_set_state first");
    return total_energy_fp64(h, components5);
}
