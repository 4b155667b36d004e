// Pair distribution sampling on the device (included by fg_api.cu).
//
// Restates AtomRDF::update (analysis.h:2116-2134): every unordered pair
// i < j whose atom ids are {id1, id2} adds one count at the minimum-image
// distance r (Cuboid::sqdist, geometry.h:507-515, and dist = sqrt of it),
// binned as Table2D::round does (auxiliary.h:831): bin = int(r / dr + 0.5).
// The distance is formed in FP64 from the exact 64-bit fixed-point
// difference (its wrap is the minimum image), so a bin differs from the
// reference's only where r / dr + 0.5 lies within ~1e-15 of an integer.
//
// Tiles of 128 x 128 pairs over all SMs, a histogram per block in shared
// memory. FP64 runs at 1/64 of the FP32 rate here, so a pair is binned from
// its FP32 distance (32-bit minimum image) unless r / dr + 0.5 lies within
// the FP32 rounding bound of an integer; those few (about 1e-4 of the pairs)
// take the FP64 form, so every count is the FP64 one. 8192 ions: 6.0 ms -> 75 us
// per call (FP64 for every pair on 32 blocks before); bound by the pair loop's
// issue rate and the shared-memory atomics.
#include "fg_rdf_grid.h"

namespace fg {

constexpr int kRdfMaxBins = 8192;    // shared-memory histogram (uint32)

__global__ void __launch_bounds__(kRdfThreads) rdf_kernel(const SysDesc *__restrict__ dsc, int t1, int t2,
                                                        double3 sc, float3 s32, float slack, double inv_dr,
                                                        int n_bins, unsigned long long *__restrict__ hist,
                                                        unsigned long long *__restrict__ n_pairs) {
    extern __shared__ uint32_t h[];   // [n_bins]
    __shared__ int4 pj[kRdfTile];
    __shared__ uint8_t tj[kRdfTile];
    __shared__ unsigned long long cnt;
    const SysDesc &d = *dsc;
    const int N = d.N, tid = threadIdx.x;
    for (int b = tid; b < n_bins; b += blockDim.x) h[b] = 0u;
    if (tid == 0) cnt = 0ull;
    const int nti = (N + kRdfThreads - 1) / kRdfThreads, ntj = (N + kRdfTile - 1) / kRdfTile;
    const float idr = (float)fmin(inv_dr, 1e30);   // (finite: with smaller dr every pair takes the FP64 form)
    unsigned mine = 0;
    for (long long t = blockIdx.x; t < (long long)nti * ntj; t += gridDim.x) {
        const int i0 = (int)(t / ntj) * kRdfThreads, j0 = (int)(t % ntj) * kRdfTile;
        const int nj = min(kRdfTile, N - j0);
        if (j0 + nj - 1 <= i0) continue;   // pairs j > i only
        __syncthreads();
        for (int k = tid; k < nj; k += blockDim.x) {
            pj[k] = d.pos4[j0 + k];
            tj[k] = d.ptype[j0 + k];
        }
        __syncthreads();
        const int i = i0 + tid;
        if (i >= N) continue;
        const int ti = d.ptype[i];
        if (ti != t1 && ti != t2) continue;
        const int other = ti == t1 ? t2 : t1;
        const int4 pi = d.pos4[i];
        for (int k = max(0, i + 1 - j0); k < nj; k++) {
            if (tj[k] != other) continue;
            const int4 p = pj[k];
            const float dx = (float)(int)((uint32_t)pi.x - (uint32_t)p.x) * s32.x;
            const float dy = (float)(int)((uint32_t)pi.y - (uint32_t)p.y) * s32.y;
            const float dz = (float)(int)((uint32_t)pi.z - (uint32_t)p.z) * s32.z;
            const float f = fmaf(sqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz))), idr, 0.5f);
            // f is off by at most 6e-7 f + slack (conversions, units, square,
            // sum, root and scale each round once; slack: the high words'
            // own rounding)
            int bin = (int)fminf(f, 1e9f);
            if (fabsf(f - rintf(f)) <= fmaf(f, 6e-7f, slack)) {
                double r2 = 0.0;
                const double s3[3] = {sc.x, sc.y, sc.z};   // L / 2^64 per axis (FP64 box lengths)
#pragma unroll
                for (int a = 0; a < 3; a++) {
                    const double x = (double)(long long)((unsigned long long)d.pos64[3 * i + a] -
                                                         (unsigned long long)d.pos64[3 * (j0 + k) + a]) * s3[a];
                    r2 = fma(x, x, r2);
                }
                const double fb = sqrt(r2) * inv_dr + 0.5;   // >= 0.5: compared before the integer cast
                bin = fb < (double)n_bins ? (int)fb : n_bins;
            }
            mine++;
            if (bin < n_bins) atomicAdd(&h[bin], 1u);
        }
    }
    atomicAdd(&cnt, (unsigned long long)mine);
    __syncthreads();
    for (int b = tid; b < n_bins; b += blockDim.x)
        if (h[b]) atomicAdd(&hist[b], (unsigned long long)h[b]);
    if (tid == 0 && cnt) atomicAdd(n_pairs, cnt);
}

}  // namespace fg

extern "C" int fg_rdf_sample(fg_system *h, int32_t type1, int32_t type2, double dr, int32_t n_bins, int64_t *hist,
                             int64_t *n_pairs) {
    if (!h) return fail(FG_ERR_INVALID, "null handle");
    if (h->types.empty()) return fail(FG_ERR_STATE, "fg_set_state first");
    if (!(dr > 0.0) || n_bins < 1 || n_bins > fg::kRdfMaxBins || !hist)
        return fail(FG_ERR_INVALID, "need dr > 0, 1 <= n_bins <= %d and a histogram", fg::kRdfMaxBins);
    if (type1 < 0 || type2 < 0 || type1 >= h->P.n_types || type2 >= h->P.n_types)
        return fail(FG_ERR_INVALID, "type id out of range");
    const size_t bytes = ((size_t)n_bins + 1) * sizeof(unsigned long long);
    int rc = ensure_work64(h, bytes);
    if (rc) return rc;
    unsigned long long *d_buf = (unsigned long long *)h->work64;
    std::vector<unsigned long long> out((size_t)n_bins + 1);
    CK(cudaMemsetAsync(d_buf, 0, bytes, h->stream));
    double unit = 0;
    for (int a = 0; a < 3; a++) unit = std::max(unit, std::ldexp(h->P.box[a], -32));
    const int blocks = (int)fg::rdf_blocks(h->N, dh_sm_count());
    fg::rdf_kernel<<<blocks, fg::kRdfThreads, (size_t)n_bins * sizeof(uint32_t), h->stream>>>(
        h->d_desc, type1, type2,
        make_double3(std::ldexp(h->P.box[0], -64), std::ldexp(h->P.box[1], -64), std::ldexp(h->P.box[2], -64)),
        make_float3((float)std::ldexp(h->P.box[0], -32), (float)std::ldexp(h->P.box[1], -32),
                    (float)std::ldexp(h->P.box[2], -32)),
        (float)(2.0 * unit / dr + 1e-6), 1.0 / dr, n_bins, d_buf, d_buf + n_bins);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(out.data(), d_buf, bytes, cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    drop_work64(h);
    for (int b = 0; b < n_bins; b++) hist[b] += (int64_t)out[b];
    if (n_pairs) *n_pairs += (int64_t)out[n_bins];
    return FG_OK;
}
