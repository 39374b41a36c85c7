// Tracer step on sm_100a: tensor-product gather of the real velocity field at
// each tracer, fused with the Adams-Bashforth position update.
//
// Reference (single-rank semantics):
//   particles_field_computer::get_norm_pos_in_cell / pbc_field_layer /
//   apply_computation (bfps/cpp/particles/particles_field_computer.hpp:55-183)
//   particles_adams_bashforth::move_particles (particles_adams_bashforth.hpp:18-133)
//   particles_system::completeLoop (particles_system.hpp:210-217)
// The weights, positions and accumulation are double; the field is read in
// its storage precision and promoted, as in the reference.  The sum runs
// as (b_z b_y) b_x f over z, then y, with x innermost along the contiguous
// row (apply_computation runs z, x, y; the sums agree to rounding).
//
// The rhs history is a ring of nsteps slots: logical rhs[j] is slot
// (head + j) % nsteps.  The host rotates `head` after each loop
// (shift_rhs_vectors); logical rhs[0] is then known to be zero, so the
// kernel overwrites it instead of accumulating (accum = false).
#pragma once
#include <stdint.h>
#include <type_traits>
#include "interp_coeffs.h"

namespace bfg {

struct PParams {
    int64_t n;
    int N;            // grid points per axis
    double box[3];    // 2 pi / dk per axis
    double hstep[3];  // box / N
    int nsteps;
    int head;
    int order;        // AB order of this move
    int accum;        // rhs[0] += u(x) instead of =
    int move;         // 0: sample only (into out), 1: full loop
    int split;        // lane groups of one tracer that share its z planes (tracer_split)
    int many;         // the form for many tracers (tracer_many)
    double dt;
};

template <int NB, int MM>
__device__ __forceinline__ void beta_weights(double x, double* w) {
    using C = interp_coeffs<NB, MM>;
#pragma unroll
    for (int i = 0; i < C::npts; ++i) {
        double acc = C::c(i, C::ncoef - 1);
#pragma unroll
        for (int k = C::ncoef - 2; k >= 0; --k) acc = acc * x + C::c(i, k);
        w[i] = acc;
    }
}

// get_norm_pos_in_cell and pbc_field_layer for one axis
__device__ __forceinline__ void cell_of(double pos, double box, double h, int N, int* cell,
                                        double* frac) {
    const double nb = floor(pos / box);
    const double pib = pos - nb * box;
    const double ci = floor(pib / h);
    *frac = (pib - ci * h) / h;
    const int lvl = (int)floor(pos / h);
    *cell = ((lvl % N) + N) % N;
}

// periodic index of a stencil point: c in [-N, 2N) (stencils are narrower
// than the grid), so one conditional add or subtract replaces the modulo
__device__ __forceinline__ int wrap_once(int c, int N) {
    return c < 0 ? c + N : (c >= N ? c - N : c);
}

// 32-byte vector load (one L1 sector per lane), sm_100; p 32-byte aligned
__device__ __forceinline__ void ld_32b(const float* p, float* v) {
    asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]),
                   "=f"(v[6]), "=f"(v[7])
                 : "l"(p));
}
__device__ __forceinline__ void ld_32b(const double* p, double* v) {  // four doubles
    asm volatile("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];"
                 : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
                 : "l"(p));
}

constexpr int TRACER_THREADS = 128;

// Lanes that share one stencil row: two for FP32 fields, four for FP64 fields
// (n = 1: two).  A row is read as 32-byte sectors from its aligned-down start (up
// to four in FP32, nine in FP64 for n = 4).  With one lane per tracer the gather is
// bound by L1 wavefronts (about one per sector, as each lane's sector lies in
// another line); with the sectors of a row spread over the lanes of one load, a
// wavefront serves them all, and only the per-row address and FP64 work grows.
// Measured on B200, FP32 (4e6 tracers, n = 3, m = 2, 512^3): 3.26 ms with one
// lane, 2.70 ms with two, 4.47 ms with four (issue bound).  FP64 (50001
// tracers, n = 4, m = 1, 256^3): 490 us with one lane, 250 us with four (190 us
// with the loop shape below).  Narrow FP64 stencils have few sectors a row, so the
// lanes' own work weighs more: n = 1, 1e6 tracers, 128^3: 347 us with four lanes,
// 260 with two; n = 2: 300 tracers 9 us with four lanes, 11 with two, but 1e6
// in cell order 707 against 610.  So n = 2 takes two for many tracers.
template <typename T>
__host__ __device__ constexpr int tracer_lanes(int nb, bool many) {
    return sizeof(T) == 4 || nb == 1 || (nb == 2 && many) ? 2 : 4;
}
// Few tracers leave the chip waiting for one dependent row after another: then
// up to eight lane groups share a tracer, group g taking the z planes g, g +
// split, ..., as long as all groups together are no more than 256 threads on each
// of 148 SMs (the gather of more threads is bound by throughput, and every group
// repeats the cell and weight arithmetic).  Lanes and split depend on the number
// of tracers only, not on the device, so a system sums in the same order alone
// and in an ensemble, everywhere.  The FP32 n = 3 gather is not split at any
// count: the runtime plane stride spilled in its kernel, unrolled up to the
// register limit (4e6 tracers 2.47 -> 2.55 ms), and a second form of it for few
// tracers has not been tried.
// 1024 tracers, FP64, n = 2: 45 us with one lane per tracer, 14 us with
// four lanes a row and up to eight groups.
template <typename T>
__host__ __device__ constexpr bool tracer_splits(int nb) {
    return sizeof(T) == 8 || nb != 3;
}
template <typename T>
__host__ __device__ inline int tracer_split(int64_t n, int nb) {
    const int lanes = tracer_lanes<T>(nb, false), planes = 2 * nb + 2;
    int r = 1;
    if (!tracer_splits<T>(nb)) return r;
    while (r < 8 && 2 * r <= planes && 2 * r * lanes <= 32 && n * lanes * 2 * r <= 148 * 256) r *= 2;
    return r;
}
// Many tracers (PParams::many; never split): the two narrow gathers that lose by
// the runtime plane stride, or want fewer lanes, have a form of their own for them
// in the same kernel.  128^3, us for 1e5 / 2e5 / 1e6 tracers, common form against
// own form: FP32 n = 1 32 / 54 / 236 against 29 / 48 / 205; FP64 n = 2 79 / 147 / 701
// against 80 / 147 / 641.
constexpr int64_t TRACERS_MANY = 1 << 17;
template <typename T>
__host__ __device__ constexpr bool tracer_many_form(int nb) {
    return sizeof(T) == 4 ? nb == 1 : nb == 2;
}
template <typename T>
__host__ __device__ inline int tracer_many(int64_t n, int nb) {
    return tracer_many_form<T>(nb) && n > TRACERS_MANY ? 1 : 0;
}
// The gather waits for its rows (long scoreboard): rows of the y loop are
// unrolled so that several are in flight, and the kernels are given the
// registers for that (us or ms by rows and blocks per SM):
//   FP32, n = 3: eight rows, four blocks (4e6 tracers, 512^3: 2.43 ms; five blocks
//   2.47-2.52, four rows and six blocks 2.57); n = 2: three, four (1e5 tracers,
//   256^3: 75 us; one and six 100, two and five 94, six rows 76); n = 1: two, six
//   (1e6, 128^3: 205 us; three and four 234, two and eight 197, but 20000 tracers 17
//   against 15); n = 4: two, four (1e6, 128^3: 1.68 ms; three and four 1.77, one and
//   four 1.93); n = 5: three, four.
//   FP64: two rows, and three for n = 2 (1e6, 128^3: 641 us; two 659); four blocks,
//   n = 1 five (1e6, 128^3: 260 us; four 286).  n = 4, 50001 tracers, 256^3: 190 us;
//   one row 251, three rows and three blocks 263, four rows and two blocks 217.
template <typename T, int NB>
__host__ __device__ constexpr int tracer_row_unroll() {
    if (sizeof(T) == 8) return NB == 2 ? 3 : 2;
    return NB == 3 ? 2 * NB + 2 : (NB == 1 || NB == 4 ? 2 : 3);
}
template <typename T, int NB>
__host__ __device__ constexpr int tracer_min_blocks() {
    if (NB == 1) return sizeof(T) == 4 ? 6 : 5;
    return 4;
}
template <typename T>
__host__ __device__ inline int tracers_per_block(int split, int nb, bool many) {
    return TRACER_THREADS / (tracer_lanes<T>(nb, many) * split);
}

// sum of v over the L lanes of a tracer group, pairwise ((l0 + l1) + (l2 +
// l3) for four) on every lane (xor partners add the same two values, so all
// lanes agree)
template <int L>
__device__ __forceinline__ double group_sum(double v, unsigned gmask) {
#pragma unroll
    for (int m = 1; m < L; m *= 2) v += __shfl_xor_sync(gmask, v, m, L);
    return v;
}

#ifndef BFG_TRACER_ROWSUM_F64
#define BFG_TRACER_ROWSUM_F64 0
#endif
template <typename T>
using row_sum_t =
    typename std::conditional<sizeof(T) == 8 || BFG_TRACER_ROWSUM_F64 != 0, double, float>::type;

// The sum of row_gather from the stencil's points alone, with scalar loads: lane
// j takes the points ix = j, j + L, ... of each row (stencils across the periodic
// x boundary, and resum below).
template <typename T, int NB, int L, int U>
__device__ __forceinline__ void point_gather(const T* __restrict__ ru, int N, const int* g, int x0,
                                             const double* wx, const double* wy, const double* wz,
                                             int j, int z0, int zs, unsigned gmask, double& a0,
                                             double& a1, double& a2) {
    using SumT = row_sum_t<T>;
    constexpr int NP = 2 * NB + 2;
    constexpr int PPL = (NP + L - 1) / L;  // points per lane
    const size_t rowN = (size_t)N;
    SumT wj[PPL];
    int xj[PPL];
#pragma unroll
    for (int m = 0; m < PPL; ++m) {
        const int ix = j + L * m;
        SumT w = 0;
#pragma unroll
        for (int pt = 0; pt < NP; ++pt) w = ix == pt ? (SumT)wx[pt] : w;
        wj[m] = w;
        xj[m] = ix < NP ? wrap_once(x0 + ix, N) : -1;
    }
    double A[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
    for (int iz = z0; iz < NP; iz += zs) {
        const int z = wrap_once(g[2] - NB + iz, N);
        const double bz = wz[iz];
#pragma unroll(U)
        for (int iy = 0; iy < NP; ++iy) {
            const int y = wrap_once(g[1] - NB + iy, N);
            const T* row = ru + ((size_t)z * rowN + y) * rowN * 3;
            SumT s0 = 0, s1 = 0, s2 = 0;
#pragma unroll
            for (int m = 0; m < PPL; ++m) {
                if (xj[m] >= 0) {
                    s0 = fma((SumT)row[xj[m] * 3 + 0], wj[m], s0);
                    s1 = fma((SumT)row[xj[m] * 3 + 1], wj[m], s1);
                    s2 = fma((SumT)row[xj[m] * 3 + 2], wj[m], s2);
                }
            }
            const double bzy = bz * wy[iy];
            A[0] = fma(bzy, (double)s0, A[0]);
            A[1] = fma(bzy, (double)s1, A[1]);
            A[2] = fma(bzy, (double)s2, A[2]);
        }
    }
    a0 = group_sum<L>(A[0], gmask);
    a1 = group_sum<L>(A[1], gmask);
    a2 = group_sum<L>(A[2], gmask);
}

// Lane j (0..L-1) of a lane group reads vectors j, j + L, ... of each row of
// the group's z planes (iz = z0, z0 + zs, ...).  FP32 field (precision form):
// the x sums of the stencil rows run in FP32 with the x weights rounded to
// FP32, over the words a lane reads; the y/z weights, the accumulation of those
// sums over the rows, the sum over the lanes and everything after stay FP64.
// FP64 field: all of it in FP64.  Word i of the row segment read from the
// aligned-down start belongs to point (i - off) / 3, component
// (i - off) mod 3, so each lane's x weights are shifted once per tracer and its
// sums are kept per word phase i mod 3, mapped to components at the end.  Words
// of a vector beside the stencil enter with weight zero (see tracer_one).
template <typename T, int NB, int L>
__device__ __forceinline__ void row_gather(const T* __restrict__ ru, int N, const int* g, int x0,
                                           const double* wx, const double* wy, const double* wz,
                                           int j, int z0, int zs, unsigned gmask, double& a0,
                                           double& a1, double& a2) {
    using SumT = row_sum_t<T>;
    constexpr int NP = 2 * NB + 2;
    constexpr int VW = 32 / (int)sizeof(T);              // values per vector
    constexpr int NVMAX = (3 * NP + 2 * (VW - 1)) / VW;  // vectors covering any alignment
    constexpr int VPL = (NVMAX + L - 1) / L;             // vectors per lane
    const size_t rowN = (size_t)N;
    SumT wxf[NP];
#pragma unroll
    for (int ix = 0; ix < NP; ++ix) wxf[ix] = (SumT)wx[ix];
    if (x0 >= 0 && x0 + NP <= N) {
        const int e0 = x0 * 3;
        const int base = e0 & ~(VW - 1);
        const int off = e0 - base;
        // vectors holding stencil words, none past the end of the row
        const int nv = min((off + 3 * NP + VW - 1) / VW, (N * 3 - base) / VW);
        SumT wl[VPL][VW];
#pragma unroll
        for (int t = 0; t < VPL; ++t)
#pragma unroll
            for (int u = 0; u < VW; ++u) {
                const int k = VW * (j + L * t) + u - off;  // 3 * point + component
                SumT w = 0;
#pragma unroll
                for (int pt = 0; pt < NP; ++pt) w = (k >= 3 * pt && k < 3 * pt + 3) ? wxf[pt] : w;
                wl[t][u] = w;
            }
        // word u of vector v = j + L t has phase (VW v + u) mod 3: the sums are
        // kept per lane-relative phase (VW L t + u) mod 3 and rotated by VW j
        // at the end
        double ph[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
        for (int iz = z0; iz < NP; iz += zs) {
            const int z = wrap_once(g[2] - NB + iz, N);
            const double bz = wz[iz];
#pragma unroll(tracer_row_unroll<T, NB>())
            for (int iy = 0; iy < NP; ++iy) {
                const int y = wrap_once(g[1] - NB + iy, N);
                const T* row = ru + ((size_t)z * rowN + y) * rowN * 3 + base;
                const double bzy = bz * wy[iy];
                SumT sp[3] = {0, 0, 0};
#pragma unroll
                for (int t = 0; t < VPL; ++t) {
                    if (j + L * t < nv) {
                        T q[VW];
                        ld_32b(row + VW * (j + L * t), q);
#pragma unroll
                        for (int u = 0; u < VW; ++u)
                            sp[(VW * L * t + u) % 3] =
                                fma((SumT)q[u], wl[t][u], sp[(VW * L * t + u) % 3]);
                    }
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) ph[c] = fma(bzy, (double)sp[c], ph[c]);
            }
        }
        // lane-relative phase (k - VW j) mod 3 holds phase k
        const int r = (VW * j) % 3;
        double G[3];
#pragma unroll
        for (int k = 0; k < 3; ++k)
            G[k] = group_sum<L>(r == 0 ? ph[k] : (r == 1 ? ph[(k + 2) % 3] : ph[(k + 1) % 3]), gmask);
        // component c sits in phase (c + off) mod 3
        const int k0 = off % 3;
        a0 = k0 == 0 ? G[0] : (k0 == 1 ? G[1] : G[2]);
        a1 = k0 == 0 ? G[1] : (k0 == 1 ? G[2] : G[0]);
        a2 = k0 == 0 ? G[2] : (k0 == 1 ? G[0] : G[1]);
    } else {
        point_gather<T, NB, L, tracer_row_unroll<T, NB>()>(ru, N, g, x0, wx, wy, wz, j, z0, zs, gmask,
                                                           a0, a1, a2);
    }
}

// u at one tracer from the stencil's points alone; cell and weights are worked
// out again (the position read anew), so that none of them has to stay in
// registers during row_gather.
template <typename T, int NB, int MM, int L>
__device__ __forceinline__ void resum(const PParams& pp, const T* __restrict__ ru,
                                      const volatile double* pos, int sub, int z0, int zs,
                                      unsigned gmask, double* acc) {
    constexpr int NP = 2 * NB + 2;
    int g[3];
    double fr[3], wx[NP], wy[NP], wz[NP];
#pragma unroll
    for (int d = 0; d < 3; ++d) cell_of(pos[d], pp.box[d], pp.hstep[d], pp.N, &g[d], &fr[d]);
    beta_weights<NB, MM>(fr[0], wx);
    beta_weights<NB, MM>(fr[1], wy);
    beta_weights<NB, MM>(fr[2], wz);
    point_gather<T, NB, L, 1>(ru, pp.N, g, g[0] - NB, wx, wy, wz, sub % L, z0, zs, gmask, acc[0],
                              acc[1], acc[2]);
    for (int o = L; o < L * zs; o *= 2)
#pragma unroll
        for (int d = 0; d < 3; ++d) acc[d] += __shfl_xor_sync(gmask, acc[d], o);
}

// tracer i of one system, lane `sub` of its pp.split groups of L lanes (gmask: all
// of them; one group where not SPLIT): gather u(x_i), then (move) the
// Adams-Bashforth step, whose components the first lanes finish.
template <typename T, int NB, int MM, int L, bool SPLIT>
__device__ __forceinline__ void tracer_one(const PParams& pp, const T* __restrict__ ru,
                                           double* __restrict__ pos, double* __restrict__ hist,
                                           double* __restrict__ sample_out, int64_t i, int sub,
                                           unsigned gmask) {
    constexpr int NP = 2 * NB + 2;
    const int N = pp.N;
    double p[3];
    int g[3];
    double wx[NP], wy[NP], wz[NP];
#pragma unroll
    for (int d = 0; d < 3; ++d) p[d] = pos[i * 3 + d];
    double fr[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) cell_of(p[d], pp.box[d], pp.hstep[d], N, &g[d], &fr[d]);
    beta_weights<NB, MM>(fr[0], wx);
    beta_weights<NB, MM>(fr[1], wy);
    beta_weights<NB, MM>(fr[2], wz);

    // lane sub < L finishes components sub, sub + L, ...; only their coordinates
    // stay in registers during the gather
    constexpr int CPL = (3 + L - 1) / L;
    double xd[CPL];
#pragma unroll
    for (int m = 0; m < CPL; ++m) {
        const int d = sub + L * m;
        xd[m] = d == 0 ? p[0] : (d == 1 ? p[1] : p[2]);
    }

    double acc[3] = {0.0, 0.0, 0.0};
    const int z0 = SPLIT ? sub / L : 0, zs = SPLIT ? pp.split : 1;
    row_gather<T, NB, L>(ru, N, g, g[0] - NB, wx, wy, wz, sub % L, z0, zs, gmask, acc[0], acc[1],
                         acc[2]);
    // the groups' planes, pairwise; every lane of the tracer gets the sum
    for (int o = L; o < L * zs; o *= 2)
#pragma unroll
        for (int d = 0; d < 3; ++d) acc[d] += __shfl_xor_sync(gmask, acc[d], o);
    // Row vectors also hold words beside the stencil, which entered with weight
    // zero: an infinity or NaN among them makes the sum NaN.  So a sum that is not
    // finite is formed again from the stencil's points alone (the sums are the
    // same on all lanes of the tracer, so they all come here together).
    if (!(isfinite(acc[0]) && isfinite(acc[1]) && isfinite(acc[2])))
        resum<T, NB, MM, L>(pp, ru, pos + i * 3, sub, z0, zs, gmask, acc);
    if (sub >= L) return;
    const size_t slot = (size_t)pp.n * 3;
    const double dt = pp.dt;
    const int ns = pp.nsteps;
#pragma unroll
    for (int m = 0; m < CPL; ++m) {
        const int d = sub + L * m;
        if (d >= 3) continue;
        const double u = d == 0 ? acc[0] : (d == 1 ? acc[1] : acc[2]);
        if (!pp.move) {
            sample_out[i * 3 + d] = u;
            continue;
        }
        double* h0 = hist + (size_t)pp.head * slot + i * 3 + d;
        double r[6];
        r[0] = u;
        if (pp.accum) r[0] += *h0;
        *h0 = r[0];
#pragma unroll
        for (int k = 1; k < 6; ++k) {
            r[k] = 0.0;
            if (k < pp.order) {
                int sl = pp.head + k;
                sl = sl >= ns ? sl - ns : sl;
                r[k] = hist[(size_t)sl * slot + i * 3 + d];
            }
        }
        double x = xd[m];
        switch (pp.order) {
            case 1: x += dt * r[0]; break;
            case 2: x += dt * (3. * r[0] - r[1]) / 2.; break;
            case 3: x += dt * (23. * r[0] - 16. * r[1] + 5. * r[2]) / 12.; break;
            case 4:
                x += dt * (55. * r[0] - 59. * r[1] + 37. * r[2] - 9. * r[3]) / 24.;
                break;
            case 5:
                x += dt * (1901. * r[0] - 2774. * r[1] + 2616. * r[2] - 1274. * r[3] +
                           251. * r[4]) / 720.;
                break;
            case 6:
                x += dt * (4277. * r[0] - 7923. * r[1] + 9982. * r[2] - 7298. * r[3] +
                           2877. * r[4] - 475. * r[5]) / 1440.;
                break;
            default: break;
        }
        pos[i * 3 + d] = x;
    }
}

// thread t of a system's blocks: its tracer and lane, in the form that the system
// takes (LR lanes of one tracer, a power of two; all of them leave together)
template <typename T, int NB, int MM>
__device__ __forceinline__ void tracer_thread(const PParams& pp, const T* __restrict__ ru,
                                              double* __restrict__ pos, double* __restrict__ hist,
                                              double* __restrict__ sample_out, int64_t t) {
    auto form = [&](auto lanes, auto split) {
        constexpr int L = decltype(lanes)::value;
        constexpr bool SPLIT = decltype(split)::value;
        const int LR = SPLIT ? L * pp.split : L;
        const int64_t i = t >> (__ffs(LR) - 1);
        if (i >= pp.n) return;
        const int lane = threadIdx.x & 31;
        const unsigned gmask = (LR == 32 ? 0xffffffffu : (1u << LR) - 1u) << (lane & ~(LR - 1));
        tracer_one<T, NB, MM, L, SPLIT>(pp, ru, pos, hist, sample_out, i, (int)t & (LR - 1), gmask);
    };
    if constexpr (tracer_many_form<T>(NB)) {
        if (pp.many) {
            form(std::integral_constant<int, tracer_lanes<T>(NB, true)>(), std::false_type());
            return;
        }
    }
    form(std::integral_constant<int, tracer_lanes<T>(NB, false)>(),
         std::integral_constant<bool, tracer_splits<T>(NB)>());
}

template <typename T, int NB, int MM>
__global__ void __launch_bounds__(TRACER_THREADS, tracer_min_blocks<T, NB>())
tracer_kernel(const PParams pp, const T* __restrict__ ru, double* __restrict__ pos,
              double* __restrict__ hist, double* __restrict__ sample_out) {
    tracer_thread<T, NB, MM>(pp, ru, pos, hist, sample_out,
                             (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}

// the tracer systems of many ensemble members in one launch
struct TracerSet {
    PParams pp;     // head, order and accum advance on the device after each loop
    int step_idx;
    const void* ru;
    double* pos;
    double* hist;
};

// inc_step_idx + shift_rhs_vectors of every set (particles_system.hpp:191-208)
__global__ void tracer_sets_advance(TracerSet* __restrict__ sets, int nsets) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nsets) return;
    TracerSet& s = sets[k];
    s.step_idx += 1;
    s.pp.head = (s.pp.head - 1 + s.pp.nsteps) % s.pp.nsteps;
    s.pp.order = min(s.step_idx, s.pp.nsteps);
    s.pp.accum = 0;
}

// Each set owns whole blocks: block b belongs to the set k with
// bstart[k] <= b < bstart[k+1]; the set is found once per block and its
// descriptor copied to shared memory.
template <typename T, int NB, int MM>
__global__ void __launch_bounds__(TRACER_THREADS, tracer_min_blocks<T, NB>())
tracer_batch_kernel(const TracerSet* __restrict__ sets, const int64_t* __restrict__ bstart,
                    int nsets) {
    __shared__ TracerSet s;
    __shared__ int s_k;
    if (threadIdx.x == 0) {
        const int64_t b = blockIdx.x;
        int lo = 0, hi = nsets - 1;
        while (lo < hi) {  // last k with bstart[k] <= b
            const int mid = (lo + hi + 1) / 2;
            if (bstart[mid] <= b) lo = mid;
            else hi = mid - 1;
        }
        s_k = lo;
    }
    __syncthreads();
    {
        static_assert(sizeof(TracerSet) % 4 == 0, "descriptor copy");
        const int* src = reinterpret_cast<const int*>(&sets[s_k]);
        int* dst = reinterpret_cast<int*>(&s);
        for (int w = threadIdx.x; w < (int)(sizeof(TracerSet) / 4); w += blockDim.x) dst[w] = src[w];
    }
    __syncthreads();
    tracer_thread<T, NB, MM>(s.pp, (const T*)s.ru, s.pos, s.hist, nullptr,
                             ((int64_t)blockIdx.x - bstart[s_k]) * blockDim.x + threadIdx.x);
}

// ---------------------------------------------------------------------------
// Cell ordering of the tracers (counting sort on the (z, y) cell row).
// The single-rank reference reorders its arrays by z-layer in every
// redistribute (particles_distr_mpi.hpp:798-831); here the order only serves
// memory locality of the gather (every result is per tracer), so the arrays
// are re-sorted every few steps.  Order inside a bucket is not fixed.
__global__ void tracer_keys(const PParams pp, const double* __restrict__ pos,
                            unsigned* __restrict__ key, unsigned* __restrict__ rank,
                            unsigned* __restrict__ count) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= pp.n) return;
    const int N = pp.N;
    int gz, gy;
    double fr;
    cell_of(pos[i * 3 + 2], pp.box[2], pp.hstep[2], N, &gz, &fr);
    cell_of(pos[i * 3 + 1], pp.box[1], pp.hstep[1], N, &gy, &fr);
    const unsigned k = (unsigned)gz * (unsigned)N + (unsigned)gy;
    key[i] = k;
    rank[i] = atomicAdd(&count[k], 1u);
}

// Exclusive scan of the nb bucket counts in three launches: the sum of each
// 1024-bucket block, an exclusive scan of those sums (one CTA: nb <= 2^20,
// i.e. N <= 1024), then each block's own scan plus its block offset.
// Integer sums, so the offsets do not depend on the order of the additions.
// 1024 threads per CTA; returns v's exclusive prefix within the CTA and the
// CTA's total in *total.
__device__ __forceinline__ unsigned cta_scan_1024(unsigned v, unsigned* ws, unsigned* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    if (warp == 0) {
        unsigned w = ws[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        ws[lane] = w;  // inclusive over the warps
    }
    __syncthreads();
    *total = ws[31];
    return (warp == 0 ? 0u : ws[warp - 1]) + x - v;
}
__global__ void __launch_bounds__(1024) bucket_block_sums(const unsigned* __restrict__ count,
                                                          unsigned* __restrict__ bsum, int nb) {
    __shared__ unsigned ws[32];
    const int i = blockIdx.x * 1024 + threadIdx.x;
    unsigned total;
    cta_scan_1024(i < nb ? count[i] : 0u, ws, &total);
    if (threadIdx.x == 0) bsum[blockIdx.x] = total;
}
__global__ void __launch_bounds__(1024) bucket_scan_sums(unsigned* __restrict__ bsum, int nblk) {
    __shared__ unsigned ws[32];
    const int t = threadIdx.x;
    const unsigned v = t < nblk ? bsum[t] : 0u;
    unsigned total;
    const unsigned ex = cta_scan_1024(v, ws, &total);  // every read precedes the barriers
    if (t < nblk) bsum[t] = ex;
}
__global__ void __launch_bounds__(1024) bucket_scan_blocks(const unsigned* __restrict__ count,
                                                           const unsigned* __restrict__ bsum,
                                                           unsigned* __restrict__ offset, int nb) {
    __shared__ unsigned ws[32];
    const int i = blockIdx.x * 1024 + threadIdx.x;
    unsigned total;
    const unsigned ex = cta_scan_1024(i < nb ? count[i] : 0u, ws, &total);
    if (i < nb) offset[i] = bsum[blockIdx.x] + ex;
}

// The tracers in cell order.  tracer_perm records the source of every
// destination (src[offset[key] + rank] = i, one 4-byte store per tracer);
// tracer_gather then copies positions, rhs history and indexes with the
// writes in order and the reads at random (random partial-sector writes,
// as a direct scatter makes them, cost a read-modify-write each).
__global__ void tracer_perm(const PParams pp, const unsigned* __restrict__ key,
                            const unsigned* __restrict__ rank, const unsigned* __restrict__ offset,
                            unsigned* __restrict__ src) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= pp.n) return;
    src[offset[key[i]] + rank[i]] = (unsigned)i;
}

__global__ void tracer_gather(const PParams pp, const unsigned* __restrict__ src,
                              const double* __restrict__ pos, const double* __restrict__ hist,
                              const int64_t* __restrict__ idx, double* __restrict__ pos2,
                              double* __restrict__ hist2, int64_t* __restrict__ idx2) {
    const int64_t d = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= pp.n) return;
    const int64_t i = src[d];
    const size_t slot = (size_t)pp.n * 3;
#pragma unroll
    for (int c = 0; c < 3; ++c) pos2[d * 3 + c] = pos[i * 3 + c];
    for (int s = 0; s < pp.nsteps; ++s)
#pragma unroll
        for (int c = 0; c < 3; ++c) hist2[s * slot + d * 3 + c] = hist[s * slot + i * 3 + c];
    idx2[d] = idx[i];
}

}  // namespace bfg
