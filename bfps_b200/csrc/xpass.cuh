// Warp-per-row nonlinear x pass (the X pass of every RK stage), FP32, N = 512.
//
// Same result as row_nonlin (passes.cuh) -- per (z, y) row: C2R of the
// velocity and vorticity rows (half-length complex transforms with the
// C2R pre-processing), u x w / N^3 on the grid, R2C of the product -- but
// organised around the warp instead of the CTA:
//
//   * each warp owns whole rows: one TMA bulk copy per input row brings the
//     interleaved u and w rows (6240 bytes each) into the warp's own shared
//     memory, completing on one of the warp's two mbarriers; the next row's
//     u row is requested as soon as this row's u transforms are done, its w
//     row as soon as this row's output has left, so both arrive while the
//     warp still computes;
//   * a 256-point transform lives in registers, eight values per lane:
//     one radix-8 butterfly over registers, an exchange through the warp's
//     own shared buffer (radix-8 over 8-lane groups) and one by shuffles
//     (radix-4 over 4-lane groups), so no step of a row waits for another
//     warp (__syncwarp only, no block barrier);
//   * the product is formed in registers on the transformed values of all
//     six transforms (every transform leaves the grid points in the same
//     lane / register order);
//   * the output row (and, in stage 1, the real velocity row u(t) for the
//     tracers) leaves by TMA bulk stores.
//
// Lane layout of a 256-point transform (k frequency, n grid pair index,
// z[n] = (x[2n], x[2n+1])): the spectrum side holds Z[l + 32 q] in lane l,
// register q; the grid side holds z[n1 + 8 m1 + 64 m2] in lane 4 n1 + j,
// register (m1 == j ? 0 : 4) + m2, m1 in {j, j + 4}.  With n = n1 + 8 n2,
// k = l + 32 q: W_256^{nk} = W_256^{n1 l} W_8^{n1 q} W_32^{n2 l}, and the
// 32-point factor splits again with n2 = m1 + 8 m2, l = l1 + 4 l2.
//
// The exchange pitch keeps it free of bank conflicts for 8-byte accesses
// (half-warp wavefronts): [n1][l] rows of 36.
//
// Bound by the shared-memory data pipe (79 % of its wavefronts at 256^3 when
// both exchanges went through it and every transform read its twiddles there),
// not by DRAM: so the last exchange is made of shuffles of half the values (16
// wavefronts instead of 32 for radix 4, 8 for the radix 2 below), and the
// twiddles W_M^{n1 l}, the same for all nine transforms of a row, stay in
// registers; the forward transform applies them after its exchange, where they
// are the lane's own; the mirror values of the R2C post-processing come by
// shuffles too (16 wavefronts instead of 32).  256^3: 197 -> 173 us, 512^3: 1480 ->
// 1390 us per launch.
#pragma once
#include "bulk.cuh"
#include "passes.cuh"

namespace bfg {

namespace xw {

constexpr int NWARP = 12;              // warps per CTA, one CTA per SM
constexpr int XP1 = 36;                // exchange [n1][l] row pitch
constexpr int XBUF = 8 * XP1;          // 288 >= 256
constexpr int T2P = 9;                 // twiddle table [l1][m1] row pitch: the inverse
                                       // reads it with l1 over the lanes, which a
                                       // pitch of 8 puts on two banks for four rows

template <int N>
struct Smem {
    static constexpr int RL = (N / 2 + 4) * 3;  // padded interleaved row (complex)
    cpx<float> su[RL];                          // u row in, real u row out
    cpx<float> sw[RL];                          // w row in, output row out
    cpx<float> x[XBUF];                         // exchanges
};

__device__ __forceinline__ cpx<float> shfl_c(cpx<float> v, int m) {
    return mk<float>(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m));
}
__device__ __forceinline__ cpx<float> pick(bool c, cpx<float> a, cpx<float> b) {
    return mk<float>(c ? a.x : b.x, c ? a.y : b.y);
}
// Z[M - k] for k = l + G q of a spectrum Z[l + G q] in v[q] over G lanes: register
// 7 - q of lane G - l, or of lane 0 (l = 0) register 8 - q; the value for k = 0
// is not used
template <int G>
__device__ __forceinline__ cpx<float> mirror(const cpx<float> (&v)[8], int q, int l) {
    const int src = l == 0 ? 0 : G - l;
    const cpx<float> o = mk<float>(__shfl_sync(0xffffffffu, v[7 - q].x, src, G),
                                   __shfl_sync(0xffffffffu, v[7 - q].y, src, G));
    return pick(l == 0, v[(8 - q) & 7], o);
}
// 4 x 4 transpose over the four lanes j of a group: lane j's r[i] becomes lane
// i's r[j] (two exchanges of half the values, no shared memory)
__device__ __forceinline__ void transpose4(cpx<float>* r, int j) {
#pragma unroll
    for (int m = 1; m <= 2; m *= 2) {
        const bool up = (j & m) != 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i & m) continue;
            // the lower lane keeps r[i] and gives r[i + m], the upper the reverse
            const cpx<float> got = shfl_c(pick(up, r[i], r[i + m]), m);
            r[i] = pick(up, got, r[i]);
            r[i + m] = pick(up, r[i + m], got);
        }
    }
}

// 256-point inverse transform (sign +): Z[l + 32 q] in v[q] -> grid order;
// t1r[n1] = W_256^{n1 l} of this lane
__device__ __forceinline__ void inv256(cpx<float> (&v)[8], cpx<float>* xb,
                                       const cpx<float> (&t1r)[8],
                                       const cpx<float>* __restrict__ t2, int lane) {
    dft<float, true, 8>(v);  // over q -> n1
#pragma unroll
    for (int n1 = 1; n1 < 8; ++n1) v[n1] = cmulc(v[n1], t1r[n1]);  // W_256^{-n1 l}
    __syncwarp();
#pragma unroll
    for (int n1 = 0; n1 < 8; ++n1) xb[n1 * XP1 + lane] = v[n1];
    __syncwarp();
    const int n1 = lane >> 2, l1 = lane & 3;
#pragma unroll
    for (int l2 = 0; l2 < 8; ++l2) v[l2] = xb[n1 * XP1 + l1 + 4 * l2];
    dft<float, true, 8>(v);  // over l2 -> m1
#pragma unroll
    for (int m1 = 1; m1 < 8; ++m1) v[m1] = cmulc(v[m1], t2[l1 * T2P + m1]);  // W_32^{-l1 m1}
    // lane j of the group takes m1 = j and j + 4 of every l1
    transpose4(v, l1);
    transpose4(v + 4, l1);
    dft<float, true, 4>(v);  // over l1 -> m2
    dft<float, true, 4>(v + 4);
}

// 256-point forward transform (sign -): grid order in -> Z[l + 32 q] in v[q]
__device__ __forceinline__ void fwd256(cpx<float> (&v)[8], cpx<float>* xb,
                                       const cpx<float> (&t1r)[8],
                                       const cpx<float>* __restrict__ t2, int lane) {
    const int n1 = lane >> 2, j = lane & 3;
    dft<float, false, 4>(v);  // over m2 -> l1
    dft<float, false, 4>(v + 4);
#pragma unroll
    for (int l1 = 1; l1 < 4; ++l1) {
        v[l1] = cmul(v[l1], t2[l1 * T2P + j]);              // W_32^{m1 l1}, m1 = j
        v[4 + l1] = cmul(v[4 + l1], t2[l1 * T2P + j + 4]);  // m1 = j + 4
    }
    // lane l1 of the group takes every m1
    transpose4(v, j);
    transpose4(v + 4, j);
    const int l1 = j;
    dft<float, false, 8>(v);  // over m1 -> l2
    __syncwarp();
#pragma unroll
    for (int l2 = 0; l2 < 8; ++l2) xb[n1 * XP1 + l1 + 4 * l2] = v[l2];
    __syncwarp();
    v[0] = xb[lane];
#pragma unroll
    for (int i = 1; i < 8; ++i) v[i] = cmul(xb[i * XP1 + lane], t1r[i]);  // W_256^{n1 l}
    dft<float, false, 8>(v);  // over n1 -> q
}

}  // namespace xw

// Launch: one CTA of NWARP warps per SM (persistent), 208 KB of shared
// memory; warp w of CTA b takes rows b * NWARP + w, then strides by the
// number of warps in the grid.  Rows run over all members of the launch.
template <int N>
__host__ __device__ constexpr size_t xw_smem_bytes() {
    return (size_t)xw::NWARP * sizeof(xw::Smem<N>) +
           (size_t)(N + 4 * xw::T2P) * sizeof(cpx<float>) + xw::NWARP * 16;
}

template <int N, bool WRITE_RU>
__global__ void __launch_bounds__(xw::NWARP * 32, 1)
row_nonlin_warp(const Member<float>* __restrict__ mem, const Roles rl,
                const cpx<float>* __restrict__ tw_g, int rows_per, int nrows) {
    static_assert(N == 512, "warp x pass: 256-point half-length transforms");
    using namespace xw;
    using C = cpx<float>;
    constexpr int M = N / 2;
    constexpr int RL = Smem<N>::RL;
    constexpr unsigned ROW_BYTES = RL * sizeof(C);         // 6240
    constexpr unsigned RU_BYTES = N * 3 * sizeof(float);   // 6144
    static_assert(ROW_BYTES % 16 == 0 && RU_BYTES % 16 == 0, "bulk copy sizes");
    static_assert(sizeof(Smem<N>) % 16 == 0, "warp regions stay 16-byte aligned");

    extern __shared__ __align__(128) unsigned char xw_smem_raw[];
    Smem<N>* ws = reinterpret_cast<Smem<N>*>(xw_smem_raw);
    C* tw = reinterpret_cast<C*>(ws + NWARP);  // exp(-2 pi i m / N), m < N
    C* t2 = tw + N;                            // [l1][m1] = W_32^{l1 m1}, pitch T2P
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(t2 + 4 * T2P);

    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (int i = tid; i < N; i += blockDim.x) tw[i] = tw_g[i];
    C t1r[8];  // W_256^{n1 l} of this lane
#pragma unroll
    for (int n1 = 0; n1 < 8; ++n1) t1r[n1] = tw_g[(2 * n1 * lane) % N];
    if (tid < 32) t2[(tid >> 3) * T2P + (tid & 7)] = tw_g[16 * ((tid >> 3) * (tid & 7))];
    if (tid < 2 * NWARP) mbar_init(&bars[tid], 1);
    fence_mbar_init();
    __syncthreads();
    pdl_wait();
    pdl_release();

    Smem<N>& S = ws[wid];
    // bars[2 w]: the u row in su, bars[2 w + 1]: the w row in sw
    unsigned long long* bar_u = &bars[2 * wid];
    unsigned long long* bar_w = &bars[2 * wid + 1];
    unsigned par_u = 0, par_w = 0;
    const float inv_np = 1.0f / ((float)N * (float)N * (float)N);
    const int gw = blockIdx.x * NWARP + wid, nw = gridDim.x * NWARP;
    auto row_src = [&](int row, int b) -> const C* {
        const int m = row / rows_per;
        const size_t r = (size_t)(row - m * rows_per);
        return mbuf(mem[m], b ? rl.in1 : rl.in0) + r * RL;
    };
    // kx columns that the rows of a member hold on each side (read again only
    // where the member changes)
    int pm = -1, pc = M + 1;
    auto cols = [&](int row, int side) {
        const int m = row / rows_per;
        if (m != pm) {
            pm = m;
            pc = mem[m].kp.pcols;
        }
        return rl.prune & side ? pc : M + 1;
    };
    // loads are issued by lane 0 after every lane's earlier reads of the
    // destination (fence: ordered before the async proxy's writes) and after
    // the bulk stores that read it (wait_group.read)
    auto issue = [&](int row, int b) {
        bulk_wait_read();
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
            unsigned long long* bb = b ? bar_w : bar_u;
            const int kc = cols(row, PRUNE_IN);
            const unsigned bytes = kc < M ? kc * 3 * (unsigned)sizeof(C) : ROW_BYTES;
            mbar_expect_tx(bb, bytes);
            bulk_load(b ? S.sw : S.su, row_src(row, b), bytes, bb);
        }
    };
    if (gw < nrows) {
        issue(gw, 0);
        issue(gw, 1);
    }
    bool ok = true;
    // grid position of register i of the grid side: n = n1 + 8 m1 + 64 m2
    const int n1 = lane >> 2, j = lane & 3;

    for (int row = gw; row < nrows && ok; row += nw) {
        const int m = row / rows_per;
        const size_t r = (size_t)(row - m * rows_per);
        const int next = row + nw;
        const int kin = cols(row, PRUNE_IN), kout = cols(row, PRUNE_OUT);
        C U[3][8], Wv[3][8];
        // u: C2R pre-processing and inverse transforms (su -> U)
        ok = mbar_wait_bounded(bar_u, par_u);
        par_u ^= 1u;
        if (!ok) break;
        // columns from kin on are zero
        auto fill = [&](C* st) {
            if (kin > M) return;
            for (int e = 3 * kin + lane; e < 3 * (M + 1); e += 32) st[e] = zero_c<float>();
            __syncwarp();
        };
        fill(S.su);
#pragma unroll
        for (int f = 0; f < 6; ++f) {
            if (f == 3) {
                if constexpr (WRITE_RU) {
                    // u(t) in real space, [x][c] interleaved, through su.
                    // Lanes j and j + 2 hold grid pairs 16 apart (96 words,
                    // one bank): lanes j >= 2 store their odd x first, so
                    // that each store's 32 words fall on distinct banks
                    float* rr = reinterpret_cast<float*>(S.su);
                    const int hi = j >= 2 ? 1 : 0;
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int n = n1 + 8 * (i < 4 ? j : j + 4) + 64 * (i & 3);
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            rr[(2 * n + hi) * 3 + c] = hi ? U[c][i].y : U[c][i].x;
                            rr[(2 * n + 1 - hi) * 3 + c] = hi ? U[c][i].x : U[c][i].y;
                        }
                    }
                    fence_proxy_async();  // this lane's writes, visible to the bulk copy
                    __syncwarp();
                    if (lane == 0) {
                        bulk_store(mreal(mem[m], rl.rout) + r * (N * 3), rr, RU_BYTES);
                        bulk_commit();
                    }
                }
                // w: wait for its row
                ok = mbar_wait_bounded(bar_w, par_w);
                par_w ^= 1u;
                if (!ok) break;
                fill(S.sw);
            }
            const C* st = f < 3 ? S.su : S.sw;
            const int c = f % 3;
            C v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int k = lane + 32 * q;
                const C a = st[3 * k + c];
                if (k == 0) {
                    const float x0 = a.x, xm = st[3 * M + c].x;
                    v[q] = mk<float>(x0 + xm, x0 - xm);
                } else {
                    v[q] = c2r_lo(a, st[3 * (M - k) + c], tw[k]);
                }
            }
            xw::inv256(v, S.x, t1r, t2, lane);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (f < 3) U[c][i] = v[i];
                else Wv[c][i] = v[i];
            }
        }
        if (!ok) break;
        // su is free: the next row's u streams in during the rest of this row
        if (next < nrows) issue(next, 0);
        // u x w / N^3 at every grid point (two per complex word)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            C p[3];
#pragma unroll
            for (int cc = 0; cc < 3; ++cc) {
                const int c1 = (cc + 1) % 3, c2 = (cc + 2) % 3;
                const float tx = U[c1][i].x * Wv[c2][i].x - U[c2][i].x * Wv[c1][i].x;
                const float ty = U[c1][i].y * Wv[c2][i].y - U[c2][i].y * Wv[c1][i].y;
                p[cc] = mk<float>(tx * inv_np, ty * inv_np);
            }
#pragma unroll
            for (int cc = 0; cc < 3; ++cc) U[cc][i] = p[cc];
        }
        // forward transforms and R2C post-processing into sw (free since the
        // w transforms)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            C v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = U[c][i];
            xw::fwd256(v, S.x, t1r, t2, lane);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int k = lane + 32 * q;
                const C zm = xw::mirror<32>(v, q, lane);
                if (k == 0) {
                    const C z0 = v[0];
                    S.sw[c] = mk<float>(z0.x + z0.y, 0.f);
                    S.sw[3 * M + c] = mk<float>(z0.x - z0.y, 0.f);
                } else {
                    S.sw[3 * k + c] = r2c_lo(v[q], zm, tw[k]);
                }
            }
        }
        // padding points of the output row carry zeros
        if (lane < RL - 3 * (M + 1)) S.sw[3 * (M + 1) + lane] = zero_c<float>();
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
            bulk_store(mbuf(mem[m], rl.out0) + r * RL, S.sw,
                       kout < M ? kout * 3 * (unsigned)sizeof(C) : ROW_BYTES);
            bulk_commit();
        }
        // the next row's w once the store has read sw
        if (next < nrows) issue(next, 1);
    }
    bulk_wait_all();
}


// ---------------------------------------------------------------------------
// The same x pass for N = 64, 128 and 256 (FP32): G = N / 16 lanes per row
// and 32 / G rows per warp (8 rows at 64^3, 4 at 128^3, 2 at 256^3), so that
// every lane still keeps eight values of each transform.  A row's M = N / 2 = 8 G point
// transform is a radix-8 butterfly over the lane's registers (Z[l + G q],
// q = 0..7), a twiddle W_M^(n1 l), and a G-point transform over the row's
// lanes through the warp's exchange buffer:
//   G = 4:  one exchange [n1][l] (pitch 9), lane l then takes n1 = l and
//           l + 4: two radix-4 over l;
//   G = 8:  one exchange [n1][l] (pitch 9), radix 8 over l;
//   G = 16: l = l1 + 2 l2: exchange [n1][l] (pitch 18), radix 8 over l2,
//           twiddle W_16^(l1 m1), radix 2 over the lane pair l1 by shuffles.
// The pitches put the 16 lanes of every half-warp on distinct banks for the
// 8-byte accesses of each exchange (rows of a 128^3 warp are 72 apart, 8
// modulo 16, and of a 64^3 warp 68, 4 modulo 16, so the rows sharing a
// half-warp also fall apart).  The forward
// transform retraces the inverse's steps, so both keep the grid points in
// the same lane and register order:
//   G = 4:  lane l, register 4 e + i: n = l + 4 e + 8 i;
//   G = 8:  lane l of a row, register i: grid pair n = l + 8 i;
//   G = 16: lane 2 n1 + j, register i + 4 m2 (i < 4): n = n1 + 8 (j + 2 i) + 64 m2.
// The warp's rows are consecutive in HBM: one TMA bulk copy brings its u
// rows, one its w rows, one store takes the output rows (and in stage 1 one
// the real-velocity rows).
namespace xwg {

constexpr int NWARP = 12;  // warps per CTA, one CTA per SM

template <int N>
struct Cfg {
    static constexpr int M = N / 2;
    static constexpr int G = M / 8;                // lanes per row
    static constexpr int Q = 32 / G;               // rows per warp
    static constexpr int RL = (N / 2 + 4) * 3;     // padded interleaved row (complex)
    static constexpr int XB = G == 4 ? 68 : (G == 8 ? 72 : 144);  // exchange block per row
    static constexpr int P1 = G == 16 ? 18 : 9;                   // [n1][l] pitch
};

template <int N>
struct Smem {
    cpx<float> su[Cfg<N>::Q * Cfg<N>::RL];  // u rows in, real u rows out
    cpx<float> sw[Cfg<N>::Q * Cfg<N>::RL];  // w rows in, output rows out
    cpx<float> x[Cfg<N>::Q * Cfg<N>::XB];   // exchanges, one block per row
};

// inverse (sign +): Z[l + G q] in v[q] -> grid order (layout above)
template <int N>
__device__ __forceinline__ void inv_g(cpx<float> (&v)[8], cpx<float>* xb,
                                      const cpx<float> (&t1r)[8], int l) {
    constexpr int G = Cfg<N>::G, P1 = Cfg<N>::P1;
    dft<float, true, 8>(v);  // over q -> n1
#pragma unroll
    for (int n1 = 1; n1 < 8; ++n1) v[n1] = cmulc(v[n1], t1r[n1]);  // W_M^{-n1 l}
    __syncwarp();
#pragma unroll
    for (int n1 = 0; n1 < 8; ++n1) xb[n1 * P1 + l] = v[n1];
    __syncwarp();
    if constexpr (G == 4) {
        cpx<float> a[4], b[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            a[k] = xb[l * P1 + k];        // n1 = l
            b[k] = xb[(l + 4) * P1 + k];  // n1 = l + 4
        }
        dft<float, true, 4>(a);  // over l -> n2
        dft<float, true, 4>(b);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[i] = a[i];
            v[4 + i] = b[i];
        }
    } else if constexpr (G == 8) {
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = xb[l * P1 + k];  // lane l now takes n1 = l
        dft<float, true, 8>(v);                            // over l -> n2
    } else {
        const int n1 = l >> 1, l1 = l & 1;
#pragma unroll
        for (int l2 = 0; l2 < 8; ++l2) v[l2] = xb[n1 * P1 + l1 + 2 * l2];
        dft<float, true, 8>(v);  // over l2 -> m1
        if (l1) {
#pragma unroll
            for (int m1 = 1; m1 < 8; ++m1) v[m1] = mul_wr<float, true, 16>(v[m1], m1);  // W_16^{-m1}
        }
        // lane j of the pair takes m1 = j + 2 i of both l1
        cpx<float> own[4], got[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            own[i] = xw::pick(l1 != 0, v[2 * i + 1], v[2 * i]);
            got[i] = xw::shfl_c(xw::pick(l1 != 0, v[2 * i], v[2 * i + 1]), 1);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[i] = own[i] + got[i];  // m2 = 0
            v[i + 4] = l1 ? got[i] - own[i] : own[i] - got[i];  // m2 = 1
        }
    }
}

// forward (sign -): grid order in -> Z[l + G q] in v[q]
template <int N>
__device__ __forceinline__ void fwd_g(cpx<float> (&v)[8], cpx<float>* xb,
                                      const cpx<float> (&t1r)[8], int l) {
    constexpr int G = Cfg<N>::G, P1 = Cfg<N>::P1;
    if constexpr (G == 4) {
        cpx<float> a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            a[i] = v[i];      // n1 = l
            b[i] = v[4 + i];  // n1 = l + 4
        }
        dft<float, false, 4>(a);  // over n2 -> k
        dft<float, false, 4>(b);
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            xb[l * P1 + k] = a[k];
            xb[(l + 4) * P1 + k] = b[k];
        }
    } else if constexpr (G == 8) {
        dft<float, false, 8>(v);  // over n2 -> k (lane = n1)
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 8; ++k) xb[l * P1 + k] = v[k];
    } else {
        const int n1 = l >> 1, l1 = l & 1;
        // m1 = l1 + 2 i here; each lane of the pair takes its l1 of every m1
        cpx<float> own[4], got[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const cpx<float> sum = v[i] + v[i + 4], dif = v[i] - v[i + 4];
            const cpx<float> rot = xw::pick(l1 != 0, mul_wr<float, false, 16>(dif, 1 + 2 * i),
                                            mul_wr<float, false, 16>(dif, 2 * i));
            own[i] = xw::pick(l1 != 0, rot, sum);
            got[i] = xw::shfl_c(xw::pick(l1 != 0, sum, rot), 1);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[2 * i] = xw::pick(l1 != 0, got[i], own[i]);
            v[2 * i + 1] = xw::pick(l1 != 0, own[i], got[i]);
        }
        dft<float, false, 8>(v);  // over m1 -> l2
        __syncwarp();
#pragma unroll
        for (int l2 = 0; l2 < 8; ++l2) xb[n1 * P1 + l1 + 2 * l2] = v[l2];
    }
    __syncwarp();
    v[0] = xb[l];  // lane l takes spectrum column l
#pragma unroll
    for (int n1 = 1; n1 < 8; ++n1) v[n1] = cmul(xb[n1 * P1 + l], t1r[n1]);  // W_M^{n1 l}
    dft<float, false, 8>(v);  // over n1 -> q
}

// grid pair index of register i of lane l (layout above)
template <int N>
__device__ __forceinline__ int grid_pair(int l, int i) {
    if constexpr (Cfg<N>::G == 4) return l + 4 * (i >> 2) + 8 * (i & 3);
    else if constexpr (Cfg<N>::G == 8) return l + 8 * i;
    else return (l >> 1) + 8 * ((l & 1) + 2 * (i & 3)) + 64 * (i >> 2);
}

}  // namespace xwg

template <int N>
__host__ __device__ constexpr size_t xwg_smem_bytes() {
    return (size_t)xwg::NWARP * sizeof(xwg::Smem<N>) +
           (size_t)N * sizeof(cpx<float>) + xwg::NWARP * 16;
}

template <int N, bool WRITE_RU>
__global__ void __launch_bounds__(xwg::NWARP * 32, 1)
row_nonlin_wg(const Member<float>* __restrict__ mem, const Roles rl,
              const cpx<float>* __restrict__ tw_g, int rows_per, int nrows) {
    static_assert(N == 64 || N == 128 || N == 256, "warp-group x pass: 32- to 128-point half-length transforms");
    using namespace xwg;
    using C = cpx<float>;
    using CF = Cfg<N>;
    constexpr int M = CF::M, G = CF::G, Q = CF::Q, RL = CF::RL, XB = CF::XB;
    constexpr unsigned BLOCK_BYTES = Q * RL * sizeof(C);             // Q rows
    constexpr unsigned RU_BYTES = Q * N * 3 * sizeof(float);         // Q real rows
    static_assert(BLOCK_BYTES % 16 == 0 && RU_BYTES % 16 == 0, "bulk copy sizes");
    static_assert(sizeof(Smem<N>) % 16 == 0, "warp regions stay 16-byte aligned");
    static_assert(RU_BYTES <= BLOCK_BYTES, "real rows staged in su");

    extern __shared__ __align__(128) unsigned char xwg_smem_raw[];
    Smem<N>* ws = reinterpret_cast<Smem<N>*>(xwg_smem_raw);
    C* tw = reinterpret_cast<C*>(ws + NWARP);  // exp(-2 pi i m / N), m < N
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(tw + N);

    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (int i = tid; i < N; i += blockDim.x) tw[i] = tw_g[i];
    C t1r[8];  // W_M^{n1 l} of this lane
#pragma unroll
    for (int n1 = 0; n1 < 8; ++n1) t1r[n1] = tw_g[(2 * n1 * (lane % G)) % N];
    if (tid < 2 * NWARP) mbar_init(&bars[tid], 1);
    fence_mbar_init();
    __syncthreads();
    pdl_wait();
    pdl_release();

    Smem<N>& S = ws[wid];
    unsigned long long* bar_u = &bars[2 * wid];
    unsigned long long* bar_w = &bars[2 * wid + 1];
    unsigned par_u = 0, par_w = 0;
    const float inv_np = 1.0f / ((float)N * (float)N * (float)N);
    const int nblk = nrows / Q;  // Q divides N^2: blocks never straddle members
    const int gw = blockIdx.x * NWARP + wid, nw = gridDim.x * NWARP;
    // this lane's row in the block and its lane in the row; G = 8 puts rows
    // 0, 2 (and 1, 3) in one half-warp: 2 RL apart (8 modulo 16), so the
    // strided row accesses of the two rows (3 k + c) fall on distinct banks
    const int grp = lane / G;
    const int rr_ = G == 8 ? (grp & 1) * 2 + (grp >> 1) : grp;
    const int l = lane % G;
    C* xb = S.x + grp * XB;      // exchange block of this lane group
    auto block_src = [&](int blk, int b) -> const C* {
        const int row0 = blk * Q;
        const int m = row0 / rows_per;
        const size_t r = (size_t)(row0 - m * rows_per);
        return mbuf(mem[m], b ? rl.in1 : rl.in0) + r * RL;
    };
    // kx columns that the rows of a block's member hold on each side (a block
    // never straddles members; read again only where the member changes)
    int pm = -1, pc = M + 1;
    auto cols = [&](int blk, int side) {
        if constexpr (can_prune<float, N>()) {
            const int m = blk * Q / rows_per;
            if (m != pm) {
                pm = m;
                pc = mem[m].kp.pcols;
            }
            return rl.prune & side ? pc : M + 1;
        } else {
            return M + 1;
        }
    };
    auto issue = [&](int blk, int b) {
        bulk_wait_read();
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
            unsigned long long* bb = b ? bar_w : bar_u;
            const int kc = cols(blk, PRUNE_IN);
            if (kc < M) {  // the rows' first kc columns, one copy per row
                const unsigned bytes = kc * 3 * (unsigned)sizeof(C);
                mbar_expect_tx(bb, Q * bytes);
                for (int q = 0; q < Q; ++q)
                    bulk_load((b ? S.sw : S.su) + q * RL, block_src(blk, b) + q * RL, bytes, bb);
            } else {
                mbar_expect_tx(bb, BLOCK_BYTES);
                bulk_load(b ? S.sw : S.su, block_src(blk, b), BLOCK_BYTES, bb);
            }
        }
    };
    if (gw < nblk) {
        issue(gw, 0);
        issue(gw, 1);
    }
    bool ok = true;

    for (int blk = gw; blk < nblk && ok; blk += nw) {
        const int row0 = blk * Q;
        const int m = row0 / rows_per;
        const size_t r0 = (size_t)(row0 - m * rows_per);
        const int next = blk + nw;
        const int kin = cols(blk, PRUNE_IN), kout = cols(blk, PRUNE_OUT);
        C U[3][8], Wv[3][8];
        ok = mbar_wait_bounded(bar_u, par_u);
        par_u ^= 1u;
        if (!ok) break;
        // columns from kin on are zero
        auto fill = [&](C* st) {
            if (kin > M) return;
            for (int e = 3 * kin + l; e < 3 * (M + 1); e += G) st[rr_ * RL + e] = zero_c<float>();
            __syncwarp();
        };
        fill(S.su);
#pragma unroll
        for (int f = 0; f < 6; ++f) {
            if (f == 3) {
                if constexpr (WRITE_RU) {
                    // u(t) in real space, [x][c] interleaved, rows of N * 3
                    // floats one after the other, through su
                    float* rr = reinterpret_cast<float*>(S.su) + rr_ * (N * 3);
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int n = grid_pair<N>(l, i);
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            rr[(2 * n) * 3 + c] = U[c][i].x;
                            rr[(2 * n + 1) * 3 + c] = U[c][i].y;
                        }
                    }
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) {
                        bulk_store(mreal(mem[m], rl.rout) + r0 * (N * 3), S.su, RU_BYTES);
                        bulk_commit();
                    }
                }
                ok = mbar_wait_bounded(bar_w, par_w);
                par_w ^= 1u;
                if (!ok) break;
                fill(S.sw);
            }
            const C* st = (f < 3 ? S.su : S.sw) + rr_ * RL;
            const int c = f % 3;
            C v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int k = l + G * q;
                const C a = st[3 * k + c];
                if (k == 0) {
                    const float x0 = a.x, xm = st[3 * M + c].x;
                    v[q] = mk<float>(x0 + xm, x0 - xm);
                } else {
                    v[q] = c2r_lo(a, st[3 * (M - k) + c], tw[k]);
                }
            }
            inv_g<N>(v, xb, t1r, l);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (f < 3) U[c][i] = v[i];
                else Wv[c][i] = v[i];
            }
        }
        if (!ok) break;
        // su is free: the next block's u streams in during the rest of this one
        if (next < nblk) issue(next, 0);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            C p[3];
#pragma unroll
            for (int cc = 0; cc < 3; ++cc) {
                const int c1 = (cc + 1) % 3, c2 = (cc + 2) % 3;
                const float tx = U[c1][i].x * Wv[c2][i].x - U[c2][i].x * Wv[c1][i].x;
                const float ty = U[c1][i].y * Wv[c2][i].y - U[c2][i].y * Wv[c1][i].y;
                p[cc] = mk<float>(tx * inv_np, ty * inv_np);
            }
#pragma unroll
            for (int cc = 0; cc < 3; ++cc) U[cc][i] = p[cc];
        }
        C* so = S.sw + rr_ * RL;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            C v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = U[c][i];
            fwd_g<N>(v, xb, t1r, l);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int k = l + G * q;
                const C zm = xw::mirror<G>(v, q, l);
                if (k == 0) {
                    const C z0 = v[0];
                    so[c] = mk<float>(z0.x + z0.y, 0.f);
                    so[3 * M + c] = mk<float>(z0.x - z0.y, 0.f);
                } else {
                    so[3 * k + c] = r2c_lo(v[q], zm, tw[k]);
                }
            }
        }
        // padding points of the output rows carry zeros
        for (int e = l; e < RL - 3 * (M + 1); e += G) so[3 * (M + 1) + e] = zero_c<float>();
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
            C* dst = mbuf(mem[m], rl.out0) + r0 * RL;
            if (kout < M)
                for (int q = 0; q < Q; ++q)
                    bulk_store(dst + q * RL, S.sw + q * RL, kout * 3 * (unsigned)sizeof(C));
            else
                bulk_store(dst, S.sw, BLOCK_BYTES);
            bulk_commit();
        }
        if (next < nblk) issue(next, 1);
    }
    bulk_wait_all();
}

}  // namespace bfg
