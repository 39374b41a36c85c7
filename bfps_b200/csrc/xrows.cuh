// Warp-group C2R and R2C row passes, FP32, N = 64 .. 512: the transforms of a
// 3-vector field along x that stand alone (field::ift, field::dft, the
// statistics, the pressure), with the lane layouts of the nonlinear x pass
// (xpass.cuh): G lanes per row, Q = 32 / G rows per warp, eight values of a
// transform per lane, exchanges through the warp's own shared memory, rows in
// and out by TMA bulk copies completing on the warp's own mbarrier.
//
// Each warp has a buffer of complex rows and one of real rows.  The input
// buffer is read into registers (all three components), so the next block is
// requested before this one's transforms (R2C) or right after them (C2R) and
// arrives while they run and the output leaves.
//
// The real side may be the caller's array in the reference layout (rows of
// N + 2 points, the padding written as zero; PAD), which saves a copy of the
// field on each side of bfg_ift / bfg_dft.  Blocks of an even number of such
// rows (24 N + 48 bytes each pair) start on 16-byte boundaries; at N = 512 a
// block is one row, odd rows start 8 bytes past one: they are loaded from 8
// bytes earlier and stored with 8-byte stores.
//
// Memory-bound: 256^3, 403 MB per launch: 181 -> 77 us (C2R, 5.2 TB/s) and 193 -> 83 us
// (R2C, 4.9 TB/s) against the CTA-per-tile row_pass, which keeps FP64 and the other N.
#pragma once
#include "xpass.cuh"

namespace bfg {

namespace xr {

constexpr int NWARP = 12;  // warps per CTA, one CTA per SM

template <int N>
__host__ __device__ constexpr bool supported() { return N == 64 || N == 128 || N == 256 || N == 512; }

template <int N>
__host__ __device__ constexpr int lanes() { return N == 512 ? 32 : N / 16; }
template <int N>
__host__ __device__ constexpr int rows() { return 32 / lanes<N>(); }
template <int N>
__host__ __device__ constexpr int xblock() {
    if constexpr (N == 512) return xw::XBUF;
    else return xwg::Cfg<N>::XB;
}
// floats of a block of Q padded real rows, with room for the 8-byte shift
template <int N>
__host__ __device__ constexpr int real_floats() { return (rows<N>() * (N + 2) * 3 + 7) / 4 * 4; }

template <int N>
struct Smem {
    static constexpr int RL = (N / 2 + 4) * 3;
    cpx<float> cr[rows<N>() * RL];      // complex rows
    float rr[real_floats<N>()];         // real rows
    cpx<float> x[rows<N>() * xblock<N>()];
};
template <int N>
__host__ __device__ constexpr int table_len() {
    return N + (N == 512 ? 4 * xw::T2P : 0);
}
template <int N>
__host__ __device__ constexpr size_t smem_bytes() {
    return (size_t)NWARP * sizeof(Smem<N>) + (size_t)table_len<N>() * sizeof(cpx<float>) + NWARP * 8;
}

template <int N>
__device__ __forceinline__ void inverse(cpx<float> (&v)[8], cpx<float>* xb, const cpx<float> (&t1r)[8],
                                        const cpx<float>* t2, int l) {
    if constexpr (N == 512) xw::inv256(v, xb, t1r, t2, l);
    else xwg::inv_g<N>(v, xb, t1r, l);
}
template <int N>
__device__ __forceinline__ void forward(cpx<float> (&v)[8], cpx<float>* xb, const cpx<float> (&t1r)[8],
                                        const cpx<float>* t2, int l) {
    if constexpr (N == 512) xw::fwd256(v, xb, t1r, t2, l);
    else xwg::fwd_g<N>(v, xb, t1r, l);
}
// grid pair of register i of lane l
template <int N>
__device__ __forceinline__ int pair_of(int l, int i) {
    if constexpr (N == 512) return (l >> 2) + 8 * ((l & 3) + (i < 4 ? 0 : 4)) + 64 * (i & 3);
    else return xwg::grid_pair<N>(l, i);
}

// what a warp needs besides its buffers
template <int N>
struct Warp {
    int lane, grp, row, l;  // lane group, its row of the block, lane within it
    int odd;                // this lane takes odd x first (see the kernels)
    cpx<float>* xb;
    const cpx<float>*tw, *t2;
    cpx<float> t1r[8];      // W_M^{n1 l}
    unsigned long long* bar;
    int first, step, nblk;  // blocks of this warp
};

// tables, barriers and lane roles; ends with a block barrier
template <int N>
__device__ __forceinline__ Warp<N> setup(unsigned char* smem, const cpx<float>* __restrict__ tw_g,
                                         int nrows, Smem<N>** mine) {
    using C = cpx<float>;
    constexpr int G = lanes<N>();
    Smem<N>* ws = reinterpret_cast<Smem<N>*>(smem);
    C* tw = reinterpret_cast<C*>(ws + NWARP);
    C* t2 = tw + N;
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(tw + table_len<N>());
    const int tid = threadIdx.x, wid = tid >> 5;
    for (int i = tid; i < N; i += blockDim.x) tw[i] = tw_g[i];
    if constexpr (N == 512)
        if (tid < 32) t2[(tid >> 3) * xw::T2P + (tid & 7)] = tw_g[16 * ((tid >> 3) * (tid & 7))];
    if (tid < NWARP) mbar_init(&bars[tid], 1);
    fence_mbar_init();
    __syncthreads();
    pdl_wait();
    pdl_release();
    Warp<N> w;
    w.lane = tid & 31;
    w.grp = w.lane / G;
    w.row = G == 8 ? (w.grp & 1) * 2 + (w.grp >> 1) : w.grp;  // see row_nonlin_wg
    w.l = w.lane % G;
    // real rows are walked in words 6 n + c: lanes 16 pairs apart (N = 512),
    // or rows apart, share a bank; half of them start at the odd x, 3 words on
    w.odd = N == 512 ? (w.l >> 1) & 1 : w.row & 1;
    w.xb = ws[wid].x + w.grp * xblock<N>();
    w.tw = tw;
#pragma unroll
    for (int n1 = 0; n1 < 8; ++n1) w.t1r[n1] = tw_g[(2 * n1 * w.l) % N];
    w.t2 = t2;
    w.bar = &bars[wid];
    w.nblk = nrows / rows<N>();
    w.first = blockIdx.x * NWARP + wid;
    w.step = gridDim.x * NWARP;
    *mine = &ws[wid];
    return w;
}

}  // namespace xr

// complex rows (in0) -> real rows: rout, rows of N points, or with PAD the
// caller's array of rows of N + 2 points (one member)
template <int N, bool PAD>
__global__ void __launch_bounds__(xr::NWARP * 32, 1)
row_c2r_bulk(const Member<float>* __restrict__ mem, const Roles rl, float* __restrict__ user,
             const cpx<float>* __restrict__ tw_g, int rows_per, int nrows) {
    using namespace xr;
    using C = cpx<float>;
    constexpr int M = N / 2, G = lanes<N>(), Q = rows<N>(), RL = Smem<N>::RL;
    constexpr unsigned IN_BYTES = Q * RL * sizeof(C);
    constexpr int RP = PAD ? (N + 2) * 3 : N * 3;  // real row pitch (floats)
    constexpr unsigned OUT_BYTES = Q * RP * sizeof(float);
    constexpr bool BULK_OUT = OUT_BYTES % 16 == 0;
    static_assert(IN_BYTES % 16 == 0 && sizeof(Smem<N>) % 16 == 0, "bulk copies");
    static_assert(BULK_OUT || Q == 1, "odd rows are stored one by one");
    extern __shared__ __align__(128) unsigned char xr_smem[];
    Smem<N>* sp;
    const Warp<N> w = setup<N>(xr_smem, tw_g, nrows, &sp);
    Smem<N>& S = *sp;
    // kx columns that the rows of a member hold (passes.cuh, modes outside kM)
    int pm = -1, pc = M + 1;
    auto cols = [&](int m) {
        if constexpr (can_prune<float, N>()) {
            if (m != pm) {
                pm = m;
                pc = rl.prune & PRUNE_IN ? mem[m].kp.pcols : M + 1;
            }
        }
        return pc;
    };
    auto issue = [&](int blk) {
        bulk_wait_read();
        fence_proxy_async();
        __syncwarp();
        if (w.lane == 0) {
            const int m = blk * Q / rows_per;
            const size_t r = (size_t)(blk * Q - m * rows_per);
            const C* src = mbuf(mem[m], rl.in0) + r * RL;
            const int kc = cols(m);
            if (kc < M) {  // the rows' first kc columns, one copy per row
                const unsigned bytes = kc * 3 * (unsigned)sizeof(C);
                mbar_expect_tx(w.bar, Q * bytes);
                for (int q = 0; q < Q; ++q) bulk_load(S.cr + q * RL, src + q * RL, bytes, w.bar);
            } else {
                mbar_expect_tx(w.bar, IN_BYTES);
                bulk_load(S.cr, src, IN_BYTES, w.bar);
            }
        }
    };
    if (w.first < w.nblk) issue(w.first);
    unsigned par = 0;
    for (int blk = w.first; blk < w.nblk; blk += w.step) {
        if (!mbar_wait_bounded(w.bar, par)) break;
        par ^= 1u;
        const int m = blk * Q / rows_per;
        const size_t r0 = (size_t)(blk * Q - m * rows_per);
        C V[3][8];
        C* st = S.cr + w.row * RL;
        const int kin = cols(m);
        if (kin <= M) {  // columns from kin on are zero
            for (int e = 3 * kin + w.l; e < 3 * (M + 1); e += G) st[e] = zero_c<float>();
            __syncwarp();
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int k = w.l + G * q;
                const C a = st[3 * k + c];
                if (k == 0) {
                    const float x0 = a.x, xm = st[3 * M + c].x;
                    V[c][q] = mk<float>(x0 + xm, x0 - xm);
                } else {
                    V[c][q] = c2r_lo(a, st[3 * (M - k) + c], w.tw[k]);
                }
            }
            inverse<N>(V[c], w.xb, w.t1r, w.t2, w.l);
        }
        // the input rows are read and the previous output has left: next block
        if (blk + w.step < w.nblk) issue(blk + w.step);
        else bulk_wait_read();
        __syncwarp();
        float* rr = S.rr + w.row * RP;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int n = pair_of<N>(w.l, i);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                rr[(2 * n + w.odd) * 3 + c] = w.odd ? V[c][i].y : V[c][i].x;
                rr[(2 * n + 1 - w.odd) * 3 + c] = w.odd ? V[c][i].x : V[c][i].y;
            }
        }
        if constexpr (PAD)
            for (int e = w.l; e < 6; e += G) rr[N * 3 + e] = 0.f;
        float* dst = (PAD ? user : mreal(mem[m], rl.rout)) + r0 * RP;
        if constexpr (BULK_OUT) {
            fence_proxy_async();
            __syncwarp();
            if (w.lane == 0) {
                bulk_store(dst, S.rr, OUT_BYTES);
                bulk_commit();
            }
        } else {
            __syncwarp();
            for (int e = w.lane; e < RP / 2; e += 32)
                reinterpret_cast<float2*>(dst)[e] = reinterpret_cast<const float2*>(S.rr)[e];
            __syncwarp();
        }
    }
    bulk_wait_all();
}

// real rows (rin, rows of N points, or with PAD the caller's array of rows of
// N + 2 points) -> complex rows (out0).  PROD: 0 the values themselves, 1 the
// products u_c u_c, 2 u_c u_(c+1) of the three values of a point (the
// transforms of compute_pressure, vorticity_equation.cpp:452-492).
template <int N, bool PAD, int PROD>
__global__ void __launch_bounds__(xr::NWARP * 32, 1)
row_r2c_bulk(const Member<float>* __restrict__ mem, const Roles rl, const float* __restrict__ user,
             const cpx<float>* __restrict__ tw_g, int rows_per, int nrows) {
    using namespace xr;
    using C = cpx<float>;
    constexpr int M = N / 2, G = lanes<N>(), Q = rows<N>(), RL = Smem<N>::RL;
    constexpr int RP = PAD ? (N + 2) * 3 : N * 3;
    constexpr unsigned BLOCK_BYTES = Q * RP * sizeof(float);
    constexpr bool SHIFT = BLOCK_BYTES % 16 != 0;  // odd rows start 8 bytes past a boundary
    constexpr unsigned OUT_BYTES = Q * RL * sizeof(C);
    static_assert(!SHIFT || Q == 1, "one row per block");
    extern __shared__ __align__(128) unsigned char xr_smem[];
    Smem<N>* sp;
    const Warp<N> w = setup<N>(xr_smem, tw_g, nrows, &sp);
    Smem<N>& S = *sp;
    auto issue = [&](int blk) {
        bulk_wait_read();
        fence_proxy_async();
        __syncwarp();
        if (w.lane == 0) {
            const int m = blk * Q / rows_per;
            const size_t r = (size_t)(blk * Q - m * rows_per);
            const float* src = (PAD ? user : mreal(mem[m], rl.rin)) + r * RP;
            // a row's N * 12 bytes; the shifted ones from 8 bytes earlier
            const unsigned bytes = SHIFT ? N * 12 + ((r & 1) ? 16 : 0) : BLOCK_BYTES;
            mbar_expect_tx(w.bar, bytes);
            bulk_load(S.rr, src - ((SHIFT && (r & 1)) ? 2 : 0), bytes, w.bar);
        }
    };
    if (w.first < w.nblk) issue(w.first);
    unsigned par = 0;
    for (int blk = w.first; blk < w.nblk; blk += w.step) {
        if (!mbar_wait_bounded(w.bar, par)) break;
        par ^= 1u;
        const int m = blk * Q / rows_per;
        const size_t r0 = (size_t)(blk * Q - m * rows_per);
        C V[3][8];
        const float* rr = S.rr + w.row * RP + ((SHIFT && (r0 & 1)) ? 2 : 0);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int n = pair_of<N>(w.l, i);
            float f[3], g[3];  // first and second value read of the pair
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                f[c] = rr[(2 * n + w.odd) * 3 + c];
                g[c] = rr[(2 * n + 1 - w.odd) * 3 + c];
            }
            if constexpr (PROD > 0) {
                const float a[3] = {f[0], f[1], f[2]}, b[3] = {g[0], g[1], g[2]};
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const int d = PROD == 1 ? c : (c + 1) % 3;
                    f[c] = a[c] * a[d];
                    g[c] = b[c] * b[d];
                }
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) V[c][i] = w.odd ? mk<float>(g[c], f[c]) : mk<float>(f[c], g[c]);
        }
        // the real rows are in registers and the previous output has left
        if (blk + w.step < w.nblk) issue(blk + w.step);
        else bulk_wait_read();
        __syncwarp();
        C* so = S.cr + w.row * RL;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            forward<N>(V[c], w.xb, w.t1r, w.t2, w.l);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int k = w.l + G * q;
                const C zm = xw::mirror<G>(V[c], q, w.l);
                if (k == 0) {
                    const C z0 = V[c][0];
                    so[c] = mk<float>(z0.x + z0.y, 0.f);
                    so[3 * M + c] = mk<float>(z0.x - z0.y, 0.f);
                } else {
                    so[3 * k + c] = r2c_lo(V[c][q], zm, w.tw[k]);
                }
            }
        }
        // padding points of the output row carry zeros
        for (int e = w.l; e < RL - 3 * (M + 1); e += G) so[3 * (M + 1) + e] = zero_c<float>();
        fence_proxy_async();
        __syncwarp();
        if (w.lane == 0) {
            bulk_store(mbuf(mem[m], rl.out0) + r0 * RL, S.cr, OUT_BYTES);
            bulk_commit();
        }
    }
    bulk_wait_all();
}

}  // namespace bfg
