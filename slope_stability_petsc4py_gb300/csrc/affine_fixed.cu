// Strain and internal force of straight-sided P4 tetrahedra in fixed point (fixed.cuh): the sums of
// strain3_affine_kernel and force3_affine_kernel (assembly.cu), whose FP64 form took 197 and 160 us on 10,374
// elements at that pipe's rate (now 66 and 81).  Each is a product with the reference element's gradient table, the same for
// every element (strain: 34 nodes x 9 products a point, force: 24 points x 9 a node), so a block converts the
// table once, keeps it in shared memory and strides over groups of elements.  Products of values of 55 bits
// (strain: 56) in limbs of 28, the lower one signed: up to 120 terms without bias or overflow; a total's
// hh 2^56 + mid 2^28 is kept from 2^54 up where it has the room.  One exponent per element for each input.
// An element whose inputs are not all finite takes the FP64 sums.
#include "fixed.cuh"
#include "ssp_internal.cuh"

namespace ssp {
namespace {

constexpr int kStrainThreads = 192, kForceThreads = 352;  // P4: 8 elements of 24 points, 10 of 35 nodes
constexpr int kBits = 55, kStrainBits = 56;

// the table's exponent (every thread of the block), its limbs into s_ghat; syncs
template <int BITS>
__device__ __forceinline__ int load_table(const double *ghat, int n, int2 *s_ghat, int *s_exp) {
    if (threadIdx.x == 0) *s_exp = 0;
    __syncthreads();
    int e = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) e = max(e, fx_exponent(ghat[i]));
    e = __reduce_max_sync(0xffffffffu, e);
    if ((threadIdx.x & 31) == 0) atomicMax(s_exp, e);
    __syncthreads();
    e = *s_exp;
    if (e < 2047)
        for (int i = threadIdx.x; i < n; i += blockDim.x) s_ghat[i] = fx_split<28>(fx_round<60 - BITS>(fx_from_f64(ghat[i], e, 60)));
    return e;
}

struct ElementUnits {
    int unit, finite;
};

__global__ void __launch_bounds__(kStrainThreads, 3) strain3_affine_fixed_kernel(
    const double *__restrict__ jinv, const double *__restrict__ ghat, const double *__restrict__ u,
    const int32_t *__restrict__ dof, long long n_u, int n_elem, int n_p, int n_q, int group, double *__restrict__ E) {
    extern __shared__ __align__(16) unsigned char raw[];
    const int nld = 3 * n_p, n_table = n_q * nld;
    int2 *s_ghat = reinterpret_cast<int2 *>(raw);         // [n_q][n_p][3]
    int2 *s_d = s_ghat + n_table;                         // [group][n_p][3]: u_a - u_0
    int2 *s_j = s_d + group * nld;                        // [group][9]
    ElementUnits *s_e = reinterpret_cast<ElementUnits *>(s_j + group * 9);
    int *s_exp = reinterpret_cast<int *>(s_e + group);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int e_t = load_table<kStrainBits>(ghat, n_table, s_ghat, s_exp);
    const int n_groups = (n_elem + group - 1) / group;
    for (int gi = blockIdx.x; gi < n_groups; gi += gridDim.x) {
        const long long e0 = (long long)gi * group;
        const int here = static_cast<int>(n_elem - e0 < group ? n_elem - e0 : group);
        __syncthreads();  // table written; the previous group is read
        // a warp per element: displacement differences to its first node, brought to 55 bits
        for (int k = warp; k < here; k += kStrainThreads / 32) {
            const int32_t *dl = dof + (e0 + k) * nld;
            int e_u = 0;
            bool bad = false;
            auto value = [&](int i) {
                const int32_t lid = dl[i];
                if (lid < 0 || lid >= n_u) {
                    bad = true;
                    return 0.0;
                }
                return u[lid];
            };
            for (int i = lane; i < nld; i += 32) {
                const double v = value(i);
                e_u = max(e_u, fx_exponent(v));
                s_d[k * nld + i] = make_int2(__double2loint(v), __double2hiint(v));
            }
            if (bad) flag(SSP_DEV_BAD_INDEX);
            const double jv = lane < 9 ? jinv[(e0 + k) * 9 + lane] : 0.0;
            e_u = __reduce_max_sync(0xffffffffu, e_u);
            const int e_j = __reduce_max_sync(0xffffffffu, fx_exponent(jv));
            const bool finite = e_u < 2047 && e_j < 2047 && e_t < 2047;
            __syncwarp();
            if (finite) {
                long long u0[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) u0[c] = fx_from_f64(__hiloint2double(s_d[k * nld + c].y, s_d[k * nld + c].x), e_u, 60);
                __syncwarp();
                unsigned long long mag = 0;
                for (int i = lane; i < nld; i += 32) {
                    const int c = i % 3;
                    const long long d = fx_from_f64(__hiloint2double(s_d[k * nld + i].y, s_d[k * nld + i].x), e_u, 60) -
                                        (c == 0 ? u0[0] : (c == 1 ? u0[1] : u0[2]));
                    mag |= fx_mag(d);
                    s_d[k * nld + i] = make_int2(static_cast<int>(d), static_cast<int>(d >> 32));
                }
                const int room = fx_room(fx_warp_bits(mag));
                for (int i = lane; i < nld; i += 32) {
                    const int2 x = s_d[k * nld + i];
                    const long long d = static_cast<long long>(static_cast<unsigned long long>(static_cast<unsigned>(x.y)) << 32 |
                                                               static_cast<unsigned>(x.x));
                    s_d[k * nld + i] = fx_round_split<28, 62 - kStrainBits>(fx_scale(d, room));
                }
                if (lane < 9) s_j[k * 9 + lane] = fx_split(fx_from_f64(jv, e_j, 58));
                if (lane == 0)
                    s_e[k] = {fx_unit(e_u, 60) + fx_top_unit<kStrainBits>(room) + fx_unit(e_t, kStrainBits) + 56 + fx_unit(e_j, 58) + kFxDrop, 1};
            } else if (lane == 0) {
                s_e[k] = {0, 0};
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < here * n_q; i += kStrainThreads) {
            const int k = i / n_q, q = i - k * n_q;
            double s[6];
            if (s_e[k].finite) {
                FxSum G[3][3];  // G_ik = sum_{a >= 1} (u_a - u_0)_i ghat_a,k(q)
                const int2 *dp = s_d + k * nld + 3, *gp = s_ghat + q * nld + 3;
#pragma unroll 2
                for (int a = 1; a < n_p; ++a, dp += 3, gp += 3) {
                    const int2 d[3] = {dp[0], dp[1], dp[2]}, g[3] = {gp[0], gp[1], gp[2]};
#pragma unroll
                    for (int x = 0; x < 3; ++x)
#pragma unroll
                        for (int y = 0; y < 3; ++y) G[x][y].add_prod(d[x], g[y]);
                }
                long long v[9];
                unsigned long long mag = 0;
#pragma unroll
                for (int x = 0; x < 9; ++x) mag |= fx_mag(G[x / 3][x % 3].hh);
                const bool small = __clzll(static_cast<long long>(mag)) >= 4;  // two bits to spare
                mag = 0;
#pragma unroll
                for (int x = 0; x < 9; ++x) {
                    const FxSum &g = G[x / 3][x % 3];
                    v[x] = small ? g.value_up<28, 2>() : g.value<28>();
                    mag |= fx_mag(v[x]);
                }
                const int lz = min(__clzll(static_cast<long long>(mag)), 63) - 6;  // to 58 bits
                const int up = max(lz, 0), down = max(-lz, 0);
                int2 Gl[3][3], J[3][3];
#pragma unroll
                for (int x = 0; x < 9; ++x) {
                    Gl[x / 3][x % 3] = fx_split((v[x] << up) >> down);
                    J[x / 3][x % 3] = s_j[k * 9 + x];
                }
                const int unit = s_e[k].unit - (small ? 2 : 0) - up + down;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    FxSum n(Gl[c][0], J[0][c]);  // (G J^{-1})_cc
                    n.add_prod(Gl[c][1], J[1][c]);
                    n.add_prod(Gl[c][2], J[2][c]);
                    s[c] = fx_to_f64(n.value(), unit);
                    const int x = c == 2 ? 0 : c, y = c == 0 ? 1 : 2;  // (0,1), (1,2), (0,2)
                    FxSum t(Gl[x][0], J[0][y]);
                    t.add_prod(Gl[y][0], J[0][x]);
#pragma unroll
                    for (int m = 1; m < 3; ++m) {
                        t.add_prod(Gl[x][m], J[m][y]);
                        t.add_prod(Gl[y][m], J[m][x]);
                    }
                    s[3 + c] = fx_to_f64(t.value(), unit);
                }
            } else {
                double G[3][3] = {};
                const int32_t *dl = dof + (e0 + k) * nld;
                const double *je = jinv + (e0 + k) * 9;
#pragma unroll 1
                for (int a = 0; a < n_p; ++a)
                    for (int x = 0; x < 3; ++x) {
                        const int32_t lid = dl[3 * a + x];
                        const double v = lid < 0 || lid >= n_u ? 0.0 : u[lid];
                        for (int y = 0; y < 3; ++y) G[x][y] += v * ghat[(q * n_p + a) * 3 + y];
                    }
                for (int c = 0; c < 3; ++c) {
                    const int x = c == 2 ? 0 : c, y = c == 0 ? 1 : 2;
                    s[c] = s[3 + c] = 0.0;
                    for (int m = 0; m < 3; ++m) {
                        s[c] += G[c][m] * je[3 * m + c];
                        s[3 + c] += G[x][m] * je[3 * m + y] + G[y][m] * je[3 * m + x];
                    }
                }
            }
            double2 *o = reinterpret_cast<double2 *>(E + 6 * (e0 * n_q + i));
            o[0] = make_double2(s[0], s[1]);
            o[1] = make_double2(s[2], s[3]);
            o[2] = make_double2(s[4], s[5]);
        }
    }
}

__global__ void __launch_bounds__(kForceThreads, 2) force3_affine_fixed_kernel(
    const double *__restrict__ jinv, const double *__restrict__ ghat, const double *__restrict__ w,
    const double *__restrict__ S, const int32_t *__restrict__ elem_row, int n_rows, int n_elem, int n_p, int n_q, int group,
    double *__restrict__ F) {
    extern __shared__ __align__(16) unsigned char raw[];
    const int n_table = n_q * n_p * 3;
    int2 *s_ghat = reinterpret_cast<int2 *>(raw);                          // [n_q][n_p][3]
    int2 *s_T = s_ghat + n_table;                                          // [group][n_q][9]
    unsigned long long *s_mag = reinterpret_cast<unsigned long long *>(s_T + group * n_q * 9);
    int *s_ex = reinterpret_cast<int *>(s_mag + group);                    // [group][3]: stress, weight, J^{-1}
    int *s_exp = s_ex + group * 3;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int e_t = load_table<kBits>(ghat, n_table, s_ghat, s_exp);
    const int n_groups = (n_elem + group - 1) / group;
    for (int gi = blockIdx.x; gi < n_groups; gi += gridDim.x) {
        const long long e0 = (long long)gi * group;
        const int here = static_cast<int>(n_elem - e0 < group ? n_elem - e0 : group);
        __syncthreads();  // table written; the previous group is read
        for (int k = warp; k < here; k += kForceThreads / 32) {
            const double *Se = S + 6 * (e0 + k) * n_q, *we = w + (e0 + k) * n_q;
            int e_s = 0, e_w = 0;
            for (int i = lane; i < 6 * n_q; i += 32) e_s = max(e_s, fx_exponent(Se[i]));
            for (int i = lane; i < n_q; i += 32) e_w = max(e_w, fx_exponent(we[i]));
            const int e_j = lane < 9 ? fx_exponent(jinv[(e0 + k) * 9 + lane]) : 0;
            e_s = __reduce_max_sync(0xffffffffu, e_s);
            e_w = __reduce_max_sync(0xffffffffu, e_w);
            const int e_jm = __reduce_max_sync(0xffffffffu, e_j);
            if (lane == 0) {
                s_ex[3 * k] = e_s;
                s_ex[3 * k + 1] = e_w;
                s_ex[3 * k + 2] = e_jm;
                s_mag[k] = 0;
            }
        }
        __syncthreads();
        auto finite = [&](int k) { return max(max(s_ex[3 * k], s_ex[3 * k + 1]), max(s_ex[3 * k + 2], e_t)) < 2047; };
        // T = w sigma J^{-T} of the group's points: 64-bit first, the elements' magnitudes gathered
        for (int i = threadIdx.x; i < here * n_q; i += kForceThreads) {
            const int k = i / n_q;
            if (!finite(k)) continue;
            const long long g = e0 * n_q + i;
            const int2 wl = fx_split(fx_from_f64(w[g], s_ex[3 * k + 1], 58));
            const double2 *s2 = reinterpret_cast<const double2 *>(S + 6 * g);
            int2 ws[6];
#pragma unroll
            for (int h = 0; h < 3; ++h) {
                const double2 v = s2[h];
                ws[2 * h] = fx_split(FxSum(wl, fx_split(fx_from_f64(v.x, s_ex[3 * k], 58))).value());
                ws[2 * h + 1] = fx_split(FxSum(wl, fx_split(fx_from_f64(v.y, s_ex[3 * k], 58))).value());
            }
            const double *je = jinv + (e0 + k) * 9;
            constexpr int kRow[3][3] = {{0, 3, 5}, {3, 1, 4}, {5, 4, 2}};
            unsigned long long mag = 0;
            long long *T = reinterpret_cast<long long *>(s_T) + 9 * i;
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                int2 jl[3];
#pragma unroll
                for (int z = 0; z < 3; ++z) jl[z] = fx_split(fx_from_f64(je[3 * m + z], s_ex[3 * k + 2], 58));
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    FxSum t(ws[kRow[a][0]], jl[0]);
                    t.add_prod(ws[kRow[a][1]], jl[1]);
                    t.add_prod(ws[kRow[a][2]], jl[2]);
                    const long long v = t.value();
                    mag |= fx_mag(v);
                    T[3 * a + m] = v;
                }
            }
            atomicOr(&s_mag[k], mag);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < here * n_q * 9; i += kForceThreads) {
            const int k = i / (9 * n_q);
            if (!finite(k)) continue;
            const int room = fx_room(64 - __clzll(static_cast<long long>(s_mag[k])));
            s_T[i] = fx_round_split<28, 62 - kBits>(fx_scale(reinterpret_cast<long long *>(s_T)[i], room));
        }
        __syncthreads();
        for (int i = threadIdx.x; i < here * n_p; i += kForceThreads) {
            const int k = i / n_p, node = i - k * n_p;
            const int32_t *er = elem_row + (e0 * n_p + i) * 3;
            const int row[3] = {er[0], er[1], er[2]};
            if (row[0] < 0 && row[1] < 0 && row[2] < 0) continue;
            if (row[0] >= n_rows || row[1] >= n_rows || row[2] >= n_rows) {
                flag(SSP_DEV_BAD_INDEX);
                continue;
            }
            double f[3];
            if (finite(k)) {
                FxSum acc[3];
                const int2 *T = s_T + k * n_q * 9, *gp = s_ghat + 3 * node;
#pragma unroll 2
                for (int q = 0; q < n_q; ++q, T += 9, gp += 3 * n_p) {
                    const int2 g[3] = {gp[0], gp[1], gp[2]};
#pragma unroll
                    for (int a = 0; a < 3; ++a)
#pragma unroll
                        for (int z = 0; z < 3; ++z) acc[a].add_prod(T[3 * a + z], g[z]);
                }
                const int room = fx_room(64 - __clzll(static_cast<long long>(s_mag[k])));
                const int unit = fx_unit(s_ex[3 * k], 58) + fx_unit(s_ex[3 * k + 1], 58) + kFxDrop + fx_unit(s_ex[3 * k + 2], 58) +
                                 kFxDrop + fx_top_unit<kBits>(room) + fx_unit(e_t, kBits) + 54;
#pragma unroll
                for (int a = 0; a < 3; ++a) f[a] = fx_to_f64((acc[a].hh << 2) + fx_round<26>(acc[a].mid), unit);
            } else {
                f[0] = f[1] = f[2] = 0.0;
                const double *je = jinv + (e0 + k) * 9;
#pragma unroll 1
                for (int q = 0; q < n_q; ++q) {
                    const long long g = (e0 + k) * n_q + q;
                    const double *s = S + 6 * g, *gh = ghat + (q * n_p + node) * 3;
                    double d[3];
                    for (int z = 0; z < 3; ++z) d[z] = w[g] * (je[z] * gh[0] + je[3 + z] * gh[1] + je[6 + z] * gh[2]);
                    f[0] += s[0] * d[0] + s[3] * d[1] + s[5] * d[2];
                    f[1] += s[3] * d[0] + s[1] * d[1] + s[4] * d[2];
                    f[2] += s[5] * d[0] + s[4] * d[1] + s[2] * d[2];
                }
            }
#pragma unroll
            for (int a = 0; a < 3; ++a)
                if (row[a] >= 0) red_add(F + row[a], f[a]);
        }
    }
}

template <typename Kernel, typename... A>
int launch(Kernel kernel, int threads, size_t smem, int n_groups, cudaStream_t st, A... args) {
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) != cudaSuccess)
        return SSP_ERR_CUDA;
    int dev = 0, sms = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
    if (per_sm < 1) per_sm = 1;
    const long long full = (long long)sms * per_sm;
    kernel<<<static_cast<unsigned>(n_groups < full ? n_groups : full), threads, smem, st>>>(args...);
    return launch_status();
}

}  // namespace

int strain3_affine_fixed(const double *jinv, const double *ghat, const double *u, const int32_t *dof, int n_u, int n_elem,
                         int n_p, int n_q, double *E, cudaStream_t st) {
    const int group = n_q < kStrainThreads ? kStrainThreads / n_q : 1;
    const size_t smem = 8 * (3 * (size_t)n_p * n_q + 3 * (size_t)n_p * group + 9 * (size_t)group) + sizeof(ElementUnits) * group + 16;
    return launch(strain3_affine_fixed_kernel, kStrainThreads, smem, (n_elem + group - 1) / group, st, jinv, ghat, u, dof,
                  (long long)n_u, n_elem, n_p, n_q, group, E);
}

int force3_affine_fixed(const double *jinv, const double *ghat, const double *w, const double *S, const int32_t *elem_row,
                        int n_rows, int n_elem, int n_p, int n_q, double *F, cudaStream_t st) {
    const int group = n_p < kForceThreads ? kForceThreads / n_p : 1;
    const size_t smem = 8 * (3 * (size_t)n_p * n_q + 9 * (size_t)n_q * group + (size_t)group) + 4 * (3 * (size_t)group + 1) + 16;
    return launch(force3_affine_fixed_kernel, kForceThreads, smem, (n_elem + group - 1) / group, st, jinv, ghat, w, S,
                  elem_row, n_rows, n_elem, n_p, n_q, group, F);
}

}  // namespace ssp
