// Field statistics of NSVE::do_stats as device reductions.
//
// * co-spectrum (kspace::cospectrum, bfps/cpp/kspace.cpp:521-598):
//   spec[int(|k|/dk)][i][j] += w * (Re a_i Re a_j + Im a_i Im a_j) over
//   k^2 <= kM^2, w = 1 on the kx = 0 plane and 2 elsewhere.  Summed in a
//   fixed order (per-warp shell arrays filled by segmented scans, warps
//   and block partials added in a fixed order): deterministic.
// * real-space moments and histograms (field::compute_rspace_stats,
//   bfps/cpp/field.cpp:661-889): min / <v^n>, n = 1..8 / max of the three
//   components and the magnitude, with the reference's initial values (0 for
//   the component extrema, max_estimate for the magnitude minimum).  Each
//   block writes its partials, which are reduced in a fixed order, so
//   the moments are deterministic.  Histogram counts are integer atomics.
#pragma once
#include "fft.cuh"
#include "passes.cuh"

namespace bfg {

// Blocks of the moments kernels: two 256-thread blocks on each of 148 SMs (128
// registers a thread), every one resident from the start.
constexpr int STATS_BLOCKS = 296;
constexpr int STATS_THREADS = 256;
constexpr int NQ = 40;  // 10 moments x 4 values
inline int stats_blocks(size_t npts) {
    const size_t b = (npts + STATS_THREADS - 1) / STATS_THREADS;
    return b < (size_t)STATS_BLOCKS ? (int)b : STATS_BLOCKS;
}

// Co-spectrum with a fixed order of summation (the result does not depend
// on scheduling: the same field gives the same bits, alone or beside other
// work).  A warp's unit is one (|ky|, |kz|): the up to four rows (+-ky, +-kz)
// hold the same |k| at the same kx, so each lane first adds the six distinct
// products of its kx over the rows and one scan serves all of them.  Along a
// row the shell index int(|k|/dk) does not decrease with kx, so the lanes of
// one shell form a contiguous run: a segmented inclusive scan (shuffles in a
// fixed pattern) sums each run, and the run's last lane adds it to its warp's
// own shell array in shared memory (no two lanes of a warp touch the same
// shell at once, and a warp's additions come in a fixed order).  Rows and row
// ends outside kM are not read.  The block then adds its warps' arrays in
// warp order into its partial, and spectrum_final adds the partials in a
// fixed order.
// Bound by the loads' latency and the scans' instructions: up to 16 warps per
// SM (as many as hold their shell arrays in shared memory), twelve loads in
// flight per lane.  256^3 FP32 (203 MB): 689 us with one scan of nine sums per
// row and four warps per SM, 58 us now.
constexpr int SPEC_BLOCKS = 148;
constexpr int SPEC_WARPS_MAX = 16;
constexpr int SPEC_NQ = 6;  // distinct products (i <= j)

template <typename T, int N>
__global__ void __launch_bounds__(SPEC_WARPS_MAX * 32)
spectrum_kernel(const KParams kp, const cpx<T>* __restrict__ f, int nshells, double dk,
                double* __restrict__ partial) {
    extern __shared__ double sh[];  // warps x nshells x SPEC_NQ
    const int nwarps = blockDim.x >> 5;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int nsq = nshells * SPEC_NQ;
    for (int i = threadIdx.x; i < nwarps * nsq; i += blockDim.x) sh[i] = 0.0;
    __syncthreads();
    double* mine = sh + (size_t)wid * nsq;
    const int nxv = kp.nxv;
    constexpr int H = N / 2 + 1;
    for (int item = blockIdx.x + gridDim.x * wid; item < H * H; item += gridDim.x * nwarps) {
        const int iy = item / H, iz = item - iy * H;
        const double ky = iy * kp.dky, kz = iz * kp.dkz;
        // (with a margin for the rounding of k^2: every mode is tested below)
        const double kout = kp.kM2 * (1.0 + 1e-12);
        if (ky * ky + kz * kz > kout) continue;
        // rows (+-ky, +-kz); the zero and Nyquist wavenumbers have no mirror
        const bool my = iy > 0 && iy < N / 2, mz = iz > 0 && iz < N / 2;
        const size_t rp = (size_t)kp.nxp * 3;
        const cpx<T>* r0 = f + ((size_t)iy * N + iz) * rp;
        const cpx<T>* r1 = f + ((size_t)iy * N + (N - iz)) * rp;
        const cpx<T>* r2 = f + ((size_t)(N - iy) * N + iz) * rp;
        const cpx<T>* r3 = f + ((size_t)(N - iy) * N + (N - iz)) * rp;
        for (int x0 = 0; x0 < nxv; x0 += 32) {
            const double kxl = x0 * kp.dkx;
            if ((kxl * kxl + ky * ky) + kz * kz > kout) break;  // |k| grows with kx
            const int ix = x0 + lane;
            int sidx = -1;
            double v[SPEC_NQ];
#pragma unroll
            for (int q = 0; q < SPEC_NQ; ++q) v[q] = 0.0;
            if (ix < nxv) {
                const double kx = ix * kp.dkx;
                const double k2 = (kx * kx + ky * ky) + kz * kz;
                if (k2 <= kp.kM2) {
                    sidx = (int)(sqrt(k2) / dk);
                    cpx<T> a[4][3];
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const cpx<T>* row = r == 0 ? r0 : (r == 1 ? r1 : (r == 2 ? r2 : r3));
                        const bool have = (r & 1 ? mz : true) && (r & 2 ? my : true);
#pragma unroll
                        for (int c = 0; c < 3; ++c)
                            a[r][c] = have ? row[ix * 3 + c] : mk<T>((T)0, (T)0);
                    }
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        double re[3], im[3];
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            re[c] = (double)a[r][c].x;
                            im[c] = (double)a[r][c].y;
                        }
                        int q = 0;
#pragma unroll
                        for (int i = 0; i < 3; ++i)
#pragma unroll
                            for (int j = i; j < 3; ++j, ++q) v[q] += re[i] * re[j] + im[i] * im[j];
                    }
                    const double w = ix == 0 ? 1.0 : 2.0;
#pragma unroll
                    for (int q = 0; q < SPEC_NQ; ++q) v[q] *= w;
                }
            }
            // segmented inclusive scan over runs of equal shell index
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int so = __shfl_up_sync(0xffffffffu, sidx, o);
                const bool take = lane >= o && so == sidx;
#pragma unroll
                for (int q = 0; q < SPEC_NQ; ++q) {
                    const double u = __shfl_up_sync(0xffffffffu, v[q], o);
                    if (take) v[q] += u;
                }
            }
            const int snext = __shfl_down_sync(0xffffffffu, sidx, 1);
            const bool tail = lane == 31 || snext != sidx;
            if (tail && sidx >= 0) {
#pragma unroll
                for (int q = 0; q < SPEC_NQ; ++q) mine[sidx * SPEC_NQ + q] += v[q];
            }
            __syncwarp();
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nsq; i += blockDim.x) {
        double acc = sh[i];
        for (int w = 1; w < nwarps; ++w) acc += sh[(size_t)w * nsq + i];
        partial[(size_t)blockIdx.x * nsq + i] = acc;
    }
}

// The block partials: eight groups of a block each add every eighth partial of
// 32 values in order, then the groups are added in order; the (3, 3) result
// is symmetric.
constexpr int SPEC_FINAL_GROUPS = 8;
__global__ void __launch_bounds__(32 * SPEC_FINAL_GROUPS)
spectrum_final(const double* __restrict__ partial, int nblocks, int nsq, double* __restrict__ spec) {
    __shared__ double red[SPEC_FINAL_GROUPS][32];
    const int o = threadIdx.x & 31, g = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + o;
    double acc = 0.0;
    if (i < nsq)
#pragma unroll 4
        for (int b = g; b < nblocks; b += SPEC_FINAL_GROUPS) acc += partial[(size_t)b * nsq + i];
    red[g][o] = acc;
    __syncthreads();
    if (g != 0 || i >= nsq) return;
    for (int k = 1; k < SPEC_FINAL_GROUPS; ++k) acc += red[k][o];
    const int s = i / SPEC_NQ, q = i - s * SPEC_NQ;
    const int r = q < 3 ? 0 : (q < 5 ? 1 : 2), c = q < 3 ? q : (q < 5 ? q - 2 : 2);
    spec[s * 9 + r * 3 + c] = acc;
    spec[s * 9 + c * 3 + r] = acc;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_min(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}

// Histogram ranges, computed on the host and read from the constant bank:
// estimates (components, magnitude), bin sizes, their reciprocals.
struct HistRange {
    double me[4], size[4], inv[4];
    int nbins;
    int safe;  // bin_of may use the reciprocals
};
inline HistRange hist_range(double me, double me_mag, int nbins) {
    HistRange h;
    h.nbins = nbins;
    h.safe = nbins < (1 << 16);
    for (int i = 0; i < 4; ++i) {
        h.me[i] = i < 3 ? me : me_mag;
        h.size[i] = 2 * h.me[i] / nbins;
        h.inv[i] = 1.0 / h.size[i];
        const double a = h.size[i] < 0 ? -h.size[i] : h.size[i];
        h.safe = h.safe && a > 1e-290 && a < 1e290;
    }
    return h;
}

// floor(x / size) for a histogram of nbins bins: the bin of the correctly
// rounded quotient.  The product with the reciprocal is within 2^-51 of it
// relative to its size, so where it lies further than that from an integer its
// floor is the quotient's; next to one (and for bin sizes whose reciprocal is
// not a normal number, safe = false) the division decides.  Values outside
// the histogram stay outside either way.
__device__ __forceinline__ int bin_of(double x, double size, double inv, int safe) {
    const double q = x * inv;
    int b = __double2int_rd(q);
    const double d = q - (double)b;
    if (!safe || d < 1e-10 || d > 1.0 - 1e-10) b = __double2int_rd(x / size);
    return b;
}

// Moments and histogram of npts points of 3 values, rows of nx points lying
// `pitch` points apart.  partial layout per block: [q], q = moment * 4 + value.
// Bound by the FP64 and conversion instructions (about 90 a point), not by
// memory, so: no division (bin_of) and no 64-bit index division per point, the
// power sums by fused products of v, v^2, v^3, v^4, the extrema of the
// components in T and of the magnitude on its square (sqrt is monotone), and
// the histogram of one value in consecutive words (all 32 banks; interleaved
// by value the four histograms met on eight).  256^3 FP32: 533 -> 219 us;
// 190 x 161 x 133 FP64: 168 -> 66 us.
template <typename T>
__global__ void __launch_bounds__(STATS_THREADS, 2)
moments_kernel(const T* __restrict__ r, int nx, int pitch, size_t npts, const HistRange h,
               double* __restrict__ partial, unsigned long long* __restrict__ hist) {
    const int nbins = h.nbins;
    extern __shared__ unsigned int shist[];  // 4 * nbins
    __shared__ double red[STATS_THREADS / 32][NQ];
    for (int i = threadIdx.x; i < nbins * 4; i += blockDim.x) shist[i] = 0;
    __syncthreads();
    T mn[3] = {(T)0, (T)0, (T)0}, mx[3] = {(T)0, (T)0, (T)0};
    double mn2 = INFINITY, mx2 = 0.0;  // of the squared magnitude
    double sm[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) sm[n][i] = 0.0;
    auto point = [&](const T* p) {
        double v[4];
        v[3] = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            mn[i] = p[i] < mn[i] ? p[i] : mn[i];
            mx[i] = p[i] > mx[i] ? p[i] : mx[i];
            v[i] = (double)p[i];
            v[3] += v[i] * v[i];
        }
        mn2 = v[3] < mn2 ? v[3] : mn2;
        mx2 = v[3] > mx2 ? v[3] : mx2;
        v[3] = sqrt(v[3]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int b = bin_of(i == 3 ? v[3] * 2 : v[i] + h.me[i], h.size[i], h.inv[i], h.safe);
            if (b >= 0 && b < nbins) atomicAdd(&shist[i * nbins + b], 1u);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const double v1 = v[i], v2 = v1 * v1, v3 = v2 * v1, v4 = v2 * v2;
            sm[0][i] += v1;
            sm[1][i] += v2;
            sm[2][i] += v3;
            sm[3][i] += v4;
            sm[4][i] = fma(v4, v1, sm[4][i]);
            sm[5][i] = fma(v4, v2, sm[5][i]);
            sm[6][i] = fma(v4, v3, sm[6][i]);
            sm[7][i] = fma(v4, v4, sm[7][i]);
        }
    };
    // points e, e + stride, ...; row and x advance without a division
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    size_t row = e / (size_t)nx;
    int x = (int)(e - row * (size_t)nx);
    const size_t drow = stride / (size_t)nx;
    const int dx = (int)(stride - drow * (size_t)nx);
    auto advance = [&] {
        row += drow;
        x += dx;
        if (x >= nx) {
            x -= nx;
            ++row;
        }
    };
    constexpr int U = 2;  // points whose loads are in flight together
    for (; e + (U - 1) * stride < npts; e += U * stride) {
        T p[U][3];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const T* src = r + (row * (size_t)pitch + x) * 3;
#pragma unroll
            for (int i = 0; i < 3; ++i) p[u][i] = src[i];
            advance();
        }
#pragma unroll
        for (int u = 0; u < U; ++u) point(p[u]);
    }
    for (; e < npts; e += stride) {
        T p[3];
        const T* src = r + (row * (size_t)pitch + x) * 3;
#pragma unroll
        for (int i = 0; i < 3; ++i) p[i] = src[i];
        advance();
        point(p);
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double a = warp_min(i == 3 ? fmin(h.me[3], sqrt(mn2)) : (double)mn[i < 3 ? i : 0]);
        const double b = warp_max(i == 3 ? sqrt(mx2) : (double)mx[i < 3 ? i : 0]);
        if (lane == 0) {
            red[wid][0 * 4 + i] = a;
            red[wid][9 * 4 + i] = b;
        }
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            const double t = warp_sum(sm[n][i]);
            if (lane == 0) red[wid][(n + 1) * 4 + i] = t;
        }
    }
    __syncthreads();
    if (threadIdx.x < NQ) {
        const int q = threadIdx.x;
        double acc = red[0][q];
        for (int w = 1; w < STATS_THREADS / 32; ++w) {
            const double v = red[w][q];
            if (q < 4) acc = fmin(acc, v);
            else if (q >= 36) acc = fmax(acc, v);
            else acc += v;
        }
        partial[(size_t)blockIdx.x * NQ + q] = acc;
    }
    for (int i = threadIdx.x; i < nbins * 4; i += blockDim.x)
        if (shist[i]) {
            const int v = i / nbins;
            atomicAdd(&hist[(i - v * nbins) * 4 + v], (unsigned long long)shist[i]);
        }
}

// One block per moment and value: every thread takes its partials in order,
// the warps' and lanes' results are combined in a fixed pattern.  One
// thread per quantity walking all partials took 450 us for 1184 of them; 296
// partials this way take 4.5 us.
constexpr int MOM_FINAL_THREADS = 128;
__global__ void __launch_bounds__(MOM_FINAL_THREADS)
moments_final(const double* __restrict__ partial, int nblocks, double inv_npts,
              double* __restrict__ out) {
    __shared__ double red[MOM_FINAL_THREADS / 32];
    const int q = blockIdx.x, t = threadIdx.x;
    const bool lo = q < 4, hi = q >= 36;
    auto both = [&](double a, double b) { return lo ? fmin(a, b) : (hi ? fmax(a, b) : a + b); };
    // block 0's partial is the neutral element of the extrema
    double acc = lo || hi ? partial[q] : 0.0;
    for (int b = t; b < nblocks; b += MOM_FINAL_THREADS) acc = both(acc, partial[(size_t)b * NQ + q]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc = both(acc, __shfl_down_sync(0xffffffffu, acc, o));
    if ((t & 31) == 0) red[t >> 5] = acc;
    __syncthreads();
    if (t != 0) return;
    for (int w = 1; w < MOM_FINAL_THREADS / 32; ++w) acc = both(acc, red[w]);
    out[q] = lo || hi ? acc : acc * inv_npts;
}

// count of non-finite values in a buffer (bfg_check_finite)
template <typename T>
__global__ void nonfinite_kernel(const T* __restrict__ a, size_t n,
                                 unsigned long long* __restrict__ count) {
    unsigned long long local = 0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        if (!isfinite(a[i])) ++local;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) local += __shfl_down_sync(0xffffffffu, local, o);
    if ((threadIdx.x & 31) == 0 && local) atomicAdd(count, local);
}

}  // namespace bfg
