// Element tangents K_e = sum_q B_q^T (w_q D_q) B_q of P2 and P4 tetrahedra in fixed point (fixed.cuh), full or
// as the plastic correction of an elastic tangent: the sums of the reference's tangent kernels
// (cython/assemble_tangent_values_3d.c:13-214) scattered through the element -> CSR map.
//
// In FP64 these contractions run at that pipe's 1.6 multiply-adds per clock and SM (full P2 contraction of
// 19,200 elements 1,267 us, P4 correction of 2,150 plastic elements 1,362 us).  Here every product is three
// 32 x 32 -> 64-bit IMADs and every sum exact until it is converted once: 444 and 370 us, the IMADs 60 to 65 % of
// their pipe's time, then the conversions and the latency of the phases between barriers.  The moment form of the P2
// correction (assembly.cu) is faster from three points up.
//
// One CTA per element or part of its points (grid-stride), one node pair of K_e per thread: 3 x 3 entries in 18
// 64-bit accumulators, whose loads of a point (three gradients of node a, the H column of node b in nine 16-byte loads, conflict-free
// at its 144-byte stride) feed 81 IMADs.  Two nodes a per thread halve the loads but need 168 registers: 11
// warps an SM instead of 20, and a quarter more time on the P4 correction.  Symmetric tangents take the pairs on
// and above the diagonal (P2: 55, two warps; P4: 630, seven warps in rounds), others all.
//   1. gradients to 57 bits by their largest (P4: by the node's largest) and D (correction: w-less DS - D_el by 60-bit
//      subtraction) to 58 by the element's; w D rounded to 56
//   2. H[q][b][d][m] = sum_r D[m][row(d, r)] g_b,r for every point at once, kept as limbs
//   3. K[(a,c),(b,d)] = sum_q sum_r g_a,r H[q][b][d][row(c, r)]; 36 terms at most: limbs of 28 bits, the lower
//      one signed, so that the dropped products have no bias and both accumulators stay below 2^63
//   4. the sums, at 57 bits or so, become FP64 and are reduced into the CSR values
// Element matrices are nearer the exact sums than FP64's, in the norm (over distorted elements P2 0.8e-16 to
// 1.3e-16 against 1.6e-16 to 3.6e-16, P4 1.0e-16 to 1.1e-16 against 2.4e-16 to 3.0e-16).  P4's nodes differ by an
// order of magnitude in their gradients; with one exponent for all of an element's its tangent was at 4.0e-16.
// An element whose inputs are not all finite takes the same sums in FP64.
#include "fixed.cuh"
#include "ssp_internal.cuh"

namespace ssp {
namespace {

constexpr int kLimb = 28;
// Gradients of 57 bits, H of 56 by the element's or P4 node's largest: 36 terms of H times g stay below 2^63 in both
// accumulators.

struct Args {
    const double *d1, *d2, *d3, *DS, *w;
    const int32_t *emap;
    int n_elem;
    long long nnz;
    double *values;
    const int8_t *branch;
    const double *shear, *lame;
    double scale;
    const int32_t *elist, *elist_count;
};

// P4: 6.2 KB of shared memory a point of an element and 630 tiles.  A CTA of 12 points (half an element's) leaves room for
// three of 7 warps an SM, so that one's barriers and conversions hide behind another's products: 370 us for the
// correction of 2,150 elements against 399 of whole elements, a CTA of 20 warps an SM (two of 10: 379; thirds of
// 5 or 7 warps: 412, 391).
constexpr int kP4Threads = 224, kP4Parts = 2;

template <int NP, int NQ, bool SYM>
struct Shape {
    static constexpr int kTiles = SYM ? NP * (NP + 1) / 2 : NP * NP;
    // 20 or 21 warps an SM (96 registers); P4's tiles in several rounds
    static constexpr int kThreads = kTiles > 128 ? kP4Threads : (kTiles + 31) / 32 * 32;
    static constexpr int kMinCtas = 672 / kThreads;
    static constexpr int kParts = NQ > 12 ? kP4Parts : 1;  // an element's points, in parts
    static constexpr int kPoints = (NQ + kParts - 1) / kParts;
};

// NQ: the points of a part
template <int NP, int NQ>
struct Smem {
    int2 g[NQ][NP][3];
    alignas(16) int2 H[NQ][NP][18];  // [d][m] of node b
    alignas(16) int2 wD[NQ][36];     // column-major blocks: (m, k) at m + 6 k
    long long gl[NQ][2];      // shear, lame
    int2 wl[NQ];
    unsigned long long mags[32];
    int exps[3][32];
    int eg[NP], hb[NP];  // P4: a node's largest gradient exponent and bits of H
    int sq[NQ];
    int nq;
};

__device__ __forceinline__ double elastic_entry(int i, int j, double G, double L) {
    if (i < 3 && j < 3) return i == j ? 2.0 * G + L : L;
    return i == j ? G : 0.0;
}

template <int NP, int NQ, bool CORR>
__device__ __noinline__ void nonfinite_element(const Args &A, long long e, const int *sq, int nq) {
    constexpr int kNld = 3 * NP;
    const int32_t *em = A.emap + e * kNld * kNld;
    for (int idx = threadIdx.x; idx < kNld * kNld; idx += blockDim.x) {
        const int32_t p = em[idx];
        if (p < 0) continue;
        if (p >= A.nnz) {
            flag(SSP_DEV_BAD_INDEX);
            continue;
        }
        const int al = idx / kNld, be = idx - al * kNld, a = al / 3, c = al - 3 * a, b = be / 3, d = be - 3 * b;
        double acc = 0.0;
        for (int k = 0; k < nq; ++k) {
            const long long g = e * NQ + sq[k];
            const double ga[3] = {A.d1[g * NP + a], A.d2[g * NP + a], A.d3[g * NP + a]};
            const double gb[3] = {A.d1[g * NP + b], A.d2[g * NP + b], A.d3[g * NP + b]};
            double sum = 0.0;
            for (int x = 0; x < 3; ++x)
                for (int y = 0; y < 3; ++y) {
                    const int r = bt_row3(c, x), s = bt_row3(d, y);
                    double v = A.DS[36 * g + r + 6 * s];
                    if (CORR) v = A.scale * (v - elastic_entry(r, s, A.shear[g], A.lame[g]));
                    sum += ga[x] * v * gb[y];
                }
            acc += A.w[g] * sum;
        }
        red_add(A.values + p, acc);
    }
}

template <int NP, int NQ, bool SYM, bool CORR>
__global__ void __launch_bounds__(Shape<NP, NQ, SYM>::kThreads, Shape<NP, NQ, SYM>::kMinCtas)
    tangent_fixed_kernel(Args A) {
    using Sh = Shape<NP, NQ, SYM>;
    constexpr int kThreads = Sh::kThreads, kWarps = kThreads / 32, kNld = 3 * NP;
    constexpr int kPoints = Sh::kPoints, kBitsG = 57;
    static_assert(kPoints * 3 <= 36, "63 bits for the sums of a part");
    constexpr bool kByNode = NP > 10;
    constexpr int kGradRounds = (kPoints * NP + kThreads - 1) / kThreads, kDRounds = (kPoints * 36 + kThreads - 1) / kThreads;
    extern __shared__ __align__(16) unsigned char fx_raw[];
    Smem<NP, kPoints> &S = *reinterpret_cast<Smem<NP, kPoints> *>(fx_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    auto block_max = [&](int which, int v) {  // written before, read after a barrier
        v = __reduce_max_sync(0xffffffffu, v);
        if (lane == 0) S.exps[which][warp] = v;
    };
    auto block_or = [&](unsigned long long v) {
        const unsigned hi = __reduce_or_sync(0xffffffffu, static_cast<unsigned>(v >> 32)),
                       lo = __reduce_or_sync(0xffffffffu, static_cast<unsigned>(v));
        if (lane == 0) S.mags[warp] = static_cast<unsigned long long>(hi) << 32 | lo;
    };
    auto warps_or = [&]() {
        unsigned long long v = 0;
#pragma unroll
        for (int i = 0; i < kWarps; ++i) v |= S.mags[i];
        return v;
    };
    auto warps_max = [&](int which) {
        int v = 0;
#pragma unroll
        for (int i = 0; i < kWarps; ++i) v = max(v, S.exps[which][i]);
        return v;
    };

    const long long n_iter = A.elist ? static_cast<long long>(*A.elist_count) : static_cast<long long>(A.n_elem);
    for (long long item = blockIdx.x; item < Sh::kParts * n_iter; item += gridDim.x) {
        const int part = Sh::kParts > 1 ? static_cast<int>(item / n_iter) : 0;
        const long long it = item - part * n_iter, e = A.elist ? A.elist[it] : it;
        if (e < 0 || e >= A.n_elem) {  // uniform
            if (tid == 0) flag(SSP_DEV_BAD_INDEX);
            continue;
        }
        const long long g0 = e * NQ;
        const int32_t *em = A.emap + e * kNld * kNld;
        __syncthreads();  // the previous element is done with the shared buffers
        if (warp == 0) {
            const bool on = lane < NQ && (!CORR || A.branch[g0 + lane] != 0);
            const unsigned mask = __ballot_sync(0xffffffffu, on);
            // the element's points in equal parts, no more of them than needed
            const int all = __popc(mask), parts = (all + kPoints - 1) / kPoints, size = parts > 1 ? (all + parts - 1) / parts : all,
                      k = __popc(mask & ((1u << lane) - 1u)) - part * size;
            if (on && k >= 0 && k < size) S.sq[k] = lane;
            if (lane == 0) S.nq = max(0, min(size, all - part * size));
        }
        if (kByNode && tid < NP) S.eg[tid] = S.hb[tid] = 0;
        for (int i = tid; i * 32 < kNld * kNld; i += kThreads)  // the map, needed last
            asm volatile("prefetch.global.L2 [%0];" ::"l"(em + i * 32));
        __syncthreads();
        const int nq = S.nq;
        if (nq == 0) continue;  // uniform
        // inputs, and the largest exponents
        double gv[kGradRounds][3], dv[kDRounds];
        int ex_g = 0, ex_d = 0, ex_w = 0;
#pragma unroll
        for (int u = 0; u < kGradRounds; ++u) {
            const int i = tid + u * kThreads;
            gv[u][0] = gv[u][1] = gv[u][2] = 0.0;
            if (i < nq * NP) {
                const int k = i / NP;
                const long long src = (g0 + S.sq[k]) * NP + (i - k * NP);
                gv[u][0] = A.d1[src];
                gv[u][1] = A.d2[src];
                gv[u][2] = A.d3[src];
            }
        }
#pragma unroll
        for (int u = 0; u < kDRounds; ++u) {
            const int i = tid + u * kThreads;
            dv[u] = i < nq * 36 ? A.DS[(g0 + S.sq[i / 36]) * 36 + i % 36] : 0.0;
        }
        double g_pt = 0.0, l_pt = 0.0, w_pt = 0.0;
        if (tid < nq) {
            const long long g = g0 + S.sq[tid];
            w_pt = A.w[g];
            if (CORR) {
                w_pt *= A.scale;
                g_pt = A.shear[g];
                l_pt = A.lame[g];
            }
        }
#pragma unroll
        for (int u = 0; u < kGradRounds; ++u) {
            const int i = tid + u * kThreads, ex = max(fx_exponent(gv[u][0]), max(fx_exponent(gv[u][1]), fx_exponent(gv[u][2])));
            if (kByNode && i < nq * NP) atomicMax(&S.eg[i % NP], ex);
            ex_g = max(ex_g, ex);
        }
#pragma unroll
        for (int u = 0; u < kDRounds; ++u) ex_d = max(ex_d, fx_exponent(dv[u]));
        ex_d = max(ex_d, max(fx_exponent(g_pt), fx_exponent(l_pt)));
        ex_w = fx_exponent(w_pt);
        block_max(0, ex_g);
        block_max(1, ex_d);
        block_max(2, ex_w);
        __syncthreads();
        const int e_g = warps_max(0), e_d = warps_max(1), e_w = warps_max(2);
        if (max(e_g, max(e_d, e_w)) == 2047) {  // uniform
            nonfinite_element<NP, NQ, CORR>(A, e, S.sq, nq);
            continue;
        }
#pragma unroll
        for (int u = 0; u < kGradRounds; ++u) {
            const int i = tid + u * kThreads;
            if (i < nq * NP) {
                const int k = i / NP;
#pragma unroll
                for (int r = 0; r < 3; ++r) S.g[k][i - k * NP][r] = fx_split<kLimb>(fx_round<60 - kBitsG>(fx_from_f64(gv[u][r], kByNode ? S.eg[i - k * NP] : e_g, 60)));
            }
        }
        if (tid < nq) {
            S.wl[tid] = fx_split(fx_from_f64(w_pt, e_w, 58));
            S.gl[tid][0] = fx_from_f64(g_pt, e_d, 60);
            S.gl[tid][1] = fx_from_f64(l_pt, e_d, 60);
        }
        __syncthreads();
        long long dd[kDRounds];
        unsigned long long mag = 0;
#pragma unroll
        for (int u = 0; u < kDRounds; ++u) {
            const int i = tid + u * kThreads;
            dd[u] = 0;
            if (i < nq * 36) {
                dd[u] = fx_from_f64(dv[u], e_d, 60);
                if (CORR) {
                    const int k = i / 36, rr = (i - 36 * k) % 6, cc = (i - 36 * k) / 6;
                    if (rr < 3 && cc < 3) dd[u] -= S.gl[k][1];
                    if (rr == cc) dd[u] -= S.gl[k][0] << (rr < 3 ? 1 : 0);
                }
                mag |= fx_mag(dd[u]);
            }
        }
        block_or(mag);
        __syncthreads();
        const int room = fx_room(64 - __clzll(static_cast<long long>(warps_or())));
#pragma unroll
        for (int u = 0; u < kDRounds; ++u) {
            const int i = tid + u * kThreads;
            if (i < nq * 36) {
                const int k = i / 36;
                const long long v = FxSum(S.wl[k], fx_split_top<58>(fx_scale(dd[u], room))).value();
                S.wD[k][i - 36 * k] = fx_split<kLimb>(fx_round<2>(v));
            }
        }
        __syncthreads();
        // H of every point: item (point, beta), six strain components
        mag = 0;
        for (int i = tid; i < nq * kNld; i += kThreads) {
            const int k = i / kNld, be = i - k * kNld, n = be / 3, d = be - 3 * n;
            int2 gr[3];
            if (kByNode) mag = 0;
#pragma unroll
            for (int r = 0; r < 3; ++r) gr[r] = S.g[k][n][r];
            int4 *out = reinterpret_cast<int4 *>(&S.H[k][n][6 * d]);
            const int4 *c0 = reinterpret_cast<const int4 *>(&S.wD[k][6 * bt_row3(d, 0)]),
                       *c1 = reinterpret_cast<const int4 *>(&S.wD[k][6 * bt_row3(d, 1)]),
                       *c2 = reinterpret_cast<const int4 *>(&S.wD[k][6 * bt_row3(d, 2)]);
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const int4 x0 = c0[m], x1 = c1[m], x2 = c2[m];
                FxSum s(gr[0], {x0.x, x0.y}), t(gr[0], {x0.z, x0.w});
                s.add_prod(gr[1], {x1.x, x1.y});
                t.add_prod(gr[1], {x1.z, x1.w});
                s.add_prod(gr[2], {x2.x, x2.y});
                t.add_prod(gr[2], {x2.z, x2.w});
                const long long hs = s.value<kLimb>(), ht = t.value<kLimb>();
                mag |= fx_mag(hs) | fx_mag(ht);  // 64-bit for now
                out[m] = make_int4(static_cast<int>(hs), static_cast<int>(hs >> 32), static_cast<int>(ht),
                                   static_cast<int>(ht >> 32));
            }
            if (kByNode) atomicMax(&S.hb[n], 64 - __clzll(static_cast<long long>(mag)));
        }
        if (!kByNode) block_or(mag);
        __syncthreads();
        const int h_bits = kByNode ? 0 : 64 - __clzll(static_cast<long long>(warps_or()));
        for (int i = tid; i < nq * NP * 9; i += kThreads) {
            int4 *p = reinterpret_cast<int4 *>(&S.H[0][0][0]) + i;
            const int room_h = fx_room(kByNode ? S.hb[i / 9 % NP] : h_bits);
            const int4 x = *p;
            const long long hs = static_cast<long long>(static_cast<unsigned long long>(static_cast<unsigned>(x.y)) << 32 |
                                                        static_cast<unsigned>(x.x)),
                            ht = static_cast<long long>(static_cast<unsigned long long>(static_cast<unsigned>(x.w)) << 32 |
                                                        static_cast<unsigned>(x.z));
            const int2 hl = fx_round_split<kLimb, 6>(fx_scale(hs, room_h)), tl = fx_round_split<kLimb, 6>(fx_scale(ht, room_h));
            *p = make_int4(hl.x, hl.y, tl.x, tl.y);
        }
        __syncthreads();
        // total = hh 2^56 + mid 2^28
        const int unit_wd = fx_unit(e_w, 58) + fx_unit(e_d, 60) + fx_top_unit<58>(room) + kFxDrop + 2;
        const int unit_e = unit_wd + 4 * kLimb + (kByNode ? 0 : 2 * fx_unit(e_g, kBitsG) + fx_top_unit<56>(fx_room(h_bits)));
        const unsigned nnz32 = static_cast<unsigned>(A.nnz < 0x7FFFFFFFll ? A.nnz : 0x7FFFFFFFll);
        auto emit = [&](int32_t p, double v) {
            if (static_cast<unsigned>(p) < nnz32) red_add(A.values + p, v);
            else if (p >= 0) flag(SSP_DEV_BAD_INDEX);
        };
#pragma unroll 1
        for (int tile = tid; tile < Sh::kTiles; tile += kThreads) {
            int a, b;  // the tile: rows of node a, columns of node b
            if (SYM) {
                // row a of the upper triangle starts at tile a (2 NP + 1 - a) / 2
                a = static_cast<int>(((2 * NP + 1) - sqrtf(static_cast<float>((2 * NP + 1) * (2 * NP + 1) - 8 * tile))) * 0.5f);
                a -= a * (2 * NP + 1 - a) / 2 > tile;
                a += (a + 1) * (2 * NP - a) / 2 <= tile;
                b = a + tile - a * (2 * NP + 1 - a) / 2;
            } else {
                a = tile / NP;
                b = tile - a * NP;
            }
            FxSum acc[3][3];
            const int2 *gp = &S.g[0][a][0];
            const int4 *hp = reinterpret_cast<const int4 *>(&S.H[0][b][0]);
#pragma unroll 1
            for (int k = 0; k < nq; ++k, gp += 3 * NP, hp += 9 * NP) {
                const int2 ga[3] = {gp[0], gp[1], gp[2]};
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const int4 h0 = hp[3 * d], h1 = hp[3 * d + 1], h2 = hp[3 * d + 2];
                    const int2 h[6] = {{h0.x, h0.y}, {h0.z, h0.w}, {h1.x, h1.y}, {h1.z, h1.w}, {h2.x, h2.y}, {h2.z, h2.w}};
                    constexpr int kRow[3][3] = {{0, 3, 5}, {3, 1, 4}, {5, 4, 2}};
#pragma unroll
                    for (int c = 0; c < 3; ++c)
#pragma unroll
                        for (int r = 0; r < 3; ++r) acc[c][d].add_prod(ga[r], h[kRow[c][r]]);
                }
            }
            const int unit_k = kByNode ? unit_e + fx_unit(S.eg[a], kBitsG) + fx_unit(S.eg[b], kBitsG) + fx_top_unit<56>(fx_room(S.hb[b])) : unit_e;
            // the tile's positions first (and its mirror's): behind a reduction each load would wait by itself
            const int32_t *up = em + 3 * a * kNld + 3 * b, *low = em + 3 * b * kNld + 3 * a;
            int32_t pu[9], pl[9];
#pragma unroll
            for (int i = 0; i < 9; ++i) {
                pu[i] = up[i / 3 * kNld + i % 3];
                pl[i] = SYM && a != b ? low[i % 3 * kNld + i / 3] : -1;
            }
            if (SYM && a == b) {  // the upper triangle of a diagonal tile counts twice
                pl[1] = pu[3], pl[2] = pu[6], pl[5] = pu[7];
                pu[3] = pu[6] = pu[7] = -1;
            }
#pragma unroll
            for (int i = 0; i < 9; ++i) {
                const double v = fx_to_f64(acc[i / 3][i % 3].template value<kLimb>(), unit_k);
                emit(pu[i], v);
                if (SYM) emit(pl[i], v);
            }
        }
    }
}

template <int NP, int NQ, bool SYM, bool CORR>
int launch(const Args &a, cudaStream_t st) {
    using Sh = Shape<NP, NQ, SYM>;
    auto kernel = tangent_fixed_kernel<NP, NQ, SYM, CORR>;
    constexpr int smem = static_cast<int>(sizeof(Smem<NP, Sh::kPoints>));
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return SSP_ERR_CUDA;
    int dev = 0, sms = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, Sh::kThreads, smem);
    if (per_sm < 1) per_sm = 1;
    // More CTAs than fit, so that the device hands them out as others end.  P4 corrections: 1 to 24 points an element
    // (in one go 442 us for 2,150 elements, 8 times 399, 16 times 408); full tangents: no last wave (P2: 477 us in
    // one go, 8 times 448, 16 times 444).  P2 corrections here have few points and a long list's empty CTAs cost
    // more: 88 us in one go, 8 times 92.
    long long grid = (long long)sms * per_sm * (a.elist ? (NP > 10 ? 8 : 1) : 16);
    if (grid > Sh::kParts * (long long)a.n_elem) grid = Sh::kParts * (long long)a.n_elem;
    kernel<<<static_cast<unsigned>(grid), Sh::kThreads, smem, st>>>(a);
    return launch_status();
}

}  // namespace

int tangent_fixed(int n_p, bool sym, bool corr, const double *d1, const double *d2, const double *d3, const double *DS,
                  const double *w, const int32_t *emap, int n_elem, long long nnz, double *values, const int8_t *branch,
                  const double *shear, const double *lame, double scale, const int32_t *elist,
                  const int32_t *elist_count, cudaStream_t st) {
    const Args a{d1, d2, d3, DS, w, emap, n_elem, nnz, values, branch, shear, lame, scale, elist, elist_count};
    if (n_p == 10) {
        if (corr) return launch<10, 11, true, true>(a, st);
        return sym ? launch<10, 11, true, false>(a, st) : launch<10, 11, false, false>(a, st);
    }
    if (corr) return launch<35, 24, true, true>(a, st);
    return sym ? launch<35, 24, true, false>(a, st) : launch<35, 24, false, false>(a, st);
}

}  // namespace ssp
