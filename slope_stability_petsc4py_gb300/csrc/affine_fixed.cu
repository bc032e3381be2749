// Strain and internal force of straight-sided P4 tetrahedra in fixed point (fixed.cuh): the sums of
// strain3_affine_kernel and force3_affine_kernel (assembly.cu), whose FP64 form took 197 and 160 us on 10,374
// elements at that pipe's rate (now 70 and 84).  Each is a product with the reference element's gradient table, the same for
// every element (strain: 34 nodes x 9 products a point, force: 24 points x 9 a node), so a block converts the
// table once, keeps it in shared memory and strides over groups of elements.  Products of values of 56 bits in limbs of
// 28, the lower one signed: every sum exact.  What a thread does once a point, the products with
// J^{-1}, stays in FP64, whose pipe is idle here.
//
// An element has an exponent for each displacement component (strain) and for each entry of w sigma J^{-T} (force,
// three sums a force component): a component that is small beside the others, or an element that is thin
// or a needle, keeps the bits that it has in FP64.  An element whose inputs are not all finite takes the FP64 sums.
#include "fixed.cuh"
#include "ssp_internal.cuh"

namespace ssp {
namespace {

constexpr int kStrainThreads = 192, kForceThreads = 352;  // P4: 8 elements of 24 points, 10 of 35 nodes
constexpr int kBits = 56;
// the strain's sums in units of 2^56, the force's of 2^55
static_assert(kAffineMaxNodes <= 127 && kAffineMaxPoints <= 63, "sums below 2^63");

// the table's exponent (every thread of the block), its limbs into s_ghat; syncs
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
        for (int i = threadIdx.x; i < n; i += blockDim.x) s_ghat[i] = fx_split<28>(fx_round<60 - kBits>(fx_from_f64(ghat[i], e, 60)));
    return e;
}

struct ElementUnits {
    int unit[3], finite;
};

__global__ void __launch_bounds__(kStrainThreads, 4) strain3_affine_fixed_kernel(
    const double *__restrict__ jinv, const double *__restrict__ ghat, const double *__restrict__ u,
    const int32_t *__restrict__ dof, long long n_u, int n_elem, int n_p, int n_q, int group, double *__restrict__ E) {
    extern __shared__ __align__(16) unsigned char raw[];
    const int nld = 3 * n_p, n_table = n_q * nld;
    int2 *s_ghat = reinterpret_cast<int2 *>(raw);         // [n_q][n_p][3]
    int2 *s_d = s_ghat + n_table;                         // [group][n_p][3]: u_a - u_0
    double *s_j = reinterpret_cast<double *>(s_d + group * nld);  // [group][9]
    ElementUnits *s_e = reinterpret_cast<ElementUnits *>(s_j + group * 9);
    int *s_exp = reinterpret_cast<int *>(s_e + group);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int e_t = load_table(ghat, n_table, s_ghat, s_exp);
    const int n_groups = (n_elem + group - 1) / group;
    for (int gi = blockIdx.x; gi < n_groups; gi += gridDim.x) {
        const long long e0 = (long long)gi * group;
        const int here = static_cast<int>(n_elem - e0 < group ? n_elem - e0 : group);
        __syncthreads();  // table written; the previous group is read
        // a warp per element: displacement differences to its first node, each component brought to 56 bits
        for (int k = warp; k < here; k += kStrainThreads / 32) {
            const int32_t *dl = dof + (e0 + k) * nld;
            int e_u[3] = {0, 0, 0};
            bool bad = false;
            for (int i = lane; i < nld; i += 32) {
                const int32_t lid = dl[i];
                const bool in = lid >= 0 && lid < n_u;
                const double v = in ? u[lid] : 0.0;
                bad |= !in;
                const int c = i % 3, ex = fx_exponent(v);
#pragma unroll
                for (int x = 0; x < 3; ++x) e_u[x] = max(e_u[x], x == c ? ex : 0);
                s_d[k * nld + i] = make_int2(__double2loint(v), __double2hiint(v));
            }
            if (bad) flag(SSP_DEV_BAD_INDEX);
            if (lane < 9) s_j[k * 9 + lane] = jinv[(e0 + k) * 9 + lane];
#pragma unroll
            for (int x = 0; x < 3; ++x) e_u[x] = __reduce_max_sync(0xffffffffu, e_u[x]);
            const bool finite = max(max(e_u[0], e_u[1]), max(e_u[2], e_t)) < 2047;
            __syncwarp();
            if (finite) {
                long long u0[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) u0[c] = fx_from_f64(__hiloint2double(s_d[k * nld + c].y, s_d[k * nld + c].x), e_u[c], 60);
                __syncwarp();
                unsigned long long mag[3] = {0, 0, 0};
                for (int i = lane; i < nld; i += 32) {
                    const int c = i % 3;
                    const long long d = fx_from_f64(__hiloint2double(s_d[k * nld + i].y, s_d[k * nld + i].x),
                                                    c == 0 ? e_u[0] : (c == 1 ? e_u[1] : e_u[2]), 60) -
                                        (c == 0 ? u0[0] : (c == 1 ? u0[1] : u0[2]));
#pragma unroll
                    for (int x = 0; x < 3; ++x) mag[x] |= x == c ? fx_mag(d) : 0ull;
                    s_d[k * nld + i] = make_int2(static_cast<int>(d), static_cast<int>(d >> 32));
                }
                int room[3];
#pragma unroll
                for (int x = 0; x < 3; ++x) room[x] = fx_room(fx_warp_bits(mag[x]));
                for (int i = lane; i < nld; i += 32) {
                    const int2 x = s_d[k * nld + i];
                    const int c = i % 3;
                    const long long d = static_cast<long long>(static_cast<unsigned long long>(static_cast<unsigned>(x.y)) << 32 |
                                                               static_cast<unsigned>(x.x));
                    s_d[k * nld + i] = fx_round_split<28, 62 - kBits>(fx_scale(d, c == 0 ? room[0] : (c == 1 ? room[1] : room[2])));
                }
                if (lane == 0) {
                    const int unit_t = fx_unit(e_t, kBits) + 56;
                    s_e[k] = {{fx_unit(e_u[0], 60) + fx_top_unit<kBits>(room[0]) + unit_t,
                               fx_unit(e_u[1], 60) + fx_top_unit<kBits>(room[1]) + unit_t,
                               fx_unit(e_u[2], 60) + fx_top_unit<kBits>(room[2]) + unit_t}, 1};
                }
            } else if (lane == 0) {
                s_e[k] = {{0, 0, 0}, 0};
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < here * n_q; i += kStrainThreads) {
            const int k = i / n_q, q = i - k * n_q;
            double Gd[3][3];
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
                unsigned long long mag = 0;
#pragma unroll
                for (int x = 0; x < 9; ++x) mag |= fx_mag(G[x / 3][x % 3].hh);
                const bool small = __clzll(static_cast<long long>(mag)) >= 4;  // two bits to spare
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    const int unit = s_e[k].unit[x] - (small ? 2 : 0);
#pragma unroll
                    for (int y = 0; y < 3; ++y)
                        Gd[x][y] = fx_to_f64(small ? G[x][y].value_up<28, 2>() : G[x][y].value<28>(), unit);
                }
            } else {
                const int32_t *dl = dof + (e0 + k) * nld;
                auto value = [&](int j) {
                    const int32_t lid = dl[j];
                    return lid < 0 || lid >= n_u ? 0.0 : u[lid];
                };
                const double u0[3] = {value(0), value(1), value(2)};
                for (int x = 0; x < 9; ++x) Gd[x / 3][x % 3] = 0.0;
#pragma unroll 1
                for (int a = 1; a < n_p; ++a)
                    for (int x = 0; x < 3; ++x) {
                        const double du = value(3 * a + x) - u0[x];
                        for (int y = 0; y < 3; ++y) Gd[x][y] = fma(du, ghat[(q * n_p + a) * 3 + y], Gd[x][y]);
                    }
            }
            const double *je = s_j + k * 9;
            double s[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const double j0 = je[3 * m], j1 = je[3 * m + 1], j2 = je[3 * m + 2];
                s[0] = fma(Gd[0][m], j0, s[0]);
                s[1] = fma(Gd[1][m], j1, s[1]);
                s[2] = fma(Gd[2][m], j2, s[2]);
                s[3] = fma(Gd[0][m], j1, fma(Gd[1][m], j0, s[3]));
                s[4] = fma(Gd[1][m], j2, fma(Gd[2][m], j1, s[4]));
                s[5] = fma(Gd[0][m], j2, fma(Gd[2][m], j0, s[5]));
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
    int *s_ex = reinterpret_cast<int *>(s_T + group * n_q * 9);            // [group][9]: exponents of T's entries
    int *s_exp = s_ex + group * 9;
    const int e_t = load_table(ghat, n_table, s_ghat, s_exp);
    const int n_groups = (n_elem + group - 1) / group;
    for (int gi = blockIdx.x; gi < n_groups; gi += gridDim.x) {
        const long long e0 = (long long)gi * group;
        const int here = static_cast<int>(n_elem - e0 < group ? n_elem - e0 : group);
        __syncthreads();  // table written; the previous group is read
        // T = w sigma J^{-T} of the group's points in FP64, then its entries' largest exponents
        double *Td = reinterpret_cast<double *>(s_T);
        for (int i = threadIdx.x; i < here * n_q; i += kForceThreads) {
            const int k = i / n_q;
            const long long g = e0 * n_q + i;
            const double wq = w[g];
            const double2 *s2 = reinterpret_cast<const double2 *>(S + 6 * g);
            const double2 a = s2[0], b = s2[1], c = s2[2];
            const double s0 = wq * a.x, s1 = wq * a.y, s2_ = wq * b.x, s3 = wq * b.y, s4 = wq * c.x, s5 = wq * c.y;
            const double ws[3][3] = {{s0, s3, s5}, {s3, s1, s4}, {s5, s4, s2_}};
            const double *je = jinv + (e0 + k) * 9;
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const double j0 = je[3 * m], j1 = je[3 * m + 1], j2 = je[3 * m + 2];
#pragma unroll
                for (int x = 0; x < 3; ++x)
                    Td[9 * i + 3 * x + m] = fma(ws[x][0], j0, fma(ws[x][1], j1, ws[x][2] * j2));
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < here * 9; i += kForceThreads) {
            const double *t = Td + (i / 9) * (9 * n_q) + i % 9;
            int e = 0;
#pragma unroll 8
            for (int q = 0; q < n_q; ++q) e = max(e, fx_exponent(t[9 * q]));
            s_ex[i] = e;
        }
        __syncthreads();
        auto finite = [&](int k) {
            int e = e_t;
#pragma unroll
            for (int j = 0; j < 9; ++j) e = max(e, s_ex[9 * k + j]);
            return e < 2047;
        };
        for (int i = threadIdx.x; i < here * n_q * 9; i += kForceThreads) {
            const int k = i / (9 * n_q), e = s_ex[9 * k + i % 9];
            if (e < 2047) s_T[i] = fx_split<28>(fx_round<60 - kBits>(fx_from_f64(Td[i], e, 60)));
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
                FxSum acc[3][3];
                const int2 *T = s_T + k * n_q * 9, *gp = s_ghat + 3 * node;
#pragma unroll 2
                for (int q = 0; q < n_q; ++q, T += 9, gp += 3 * n_p) {
                    const int2 g[3] = {gp[0], gp[1], gp[2]};
#pragma unroll
                    for (int a = 0; a < 3; ++a)
#pragma unroll
                        for (int z = 0; z < 3; ++z) acc[a][z].add_prod(T[3 * a + z], g[z]);
                }
                const int unit = fx_unit(e_t, kBits) + 55;
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    double v[3];
#pragma unroll
                    for (int z = 0; z < 3; ++z)
                        v[z] = fx_to_f64(acc[a][z].value_up<28, 1>(), unit + fx_unit(s_ex[9 * k + 3 * a + z], kBits));
                    f[a] = v[0] + (v[1] + v[2]);
                }
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
    const size_t smem = 8 * (3 * (size_t)n_p * n_q + 9 * (size_t)n_q * group) + 4 * (9 * (size_t)group + 1) + 16;
    return launch(force3_affine_fixed_kernel, kForceThreads, smem, (n_elem + group - 1) / group, st, jinv, ghat, w, S,
                  elem_row, n_rows, n_elem, n_p, n_q, group, F);
}

}  // namespace ssp
