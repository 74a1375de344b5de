// Coarse-to-fine (chebtransform, coarseToFine and the fine chebtransform,
// ifgfoperator.hpp:1087-1124, 1539-1637) with compile-time orders.
#include <type_traits>

#include "mult.hpp"

namespace ifgf
{

// Coarse-to-fine with compile-time orders and refinement factor F (the same
// in every dimension), for the common order triples.  T is the working
// precision (double, or float in the mixed pipeline); the three matrices are
// staged in shared memory in T.
template <typename T> struct Vec2;
template <> struct Vec2<double>
{
    using type = double2;
};
template <> struct Vec2<float>
{
    using type = float2;
};

// The three per-dimension matrices as a kernel parameter: with every loop
// unrolled, each entry is a compile-time offset into the parameter bank and
// enters its FMA as a constant operand, so the contraction reads only the
// data operand from shared memory.
template <int H0, int H1, int H2, int L0, int L1, int L2, int F, typename T>
struct C2FMats
{
    T a0[F * L0 * H0];
    T a1[F * L1 * H1];
    T a2[F * L2 * H2];
};

// Row stride of the second intermediate: F0 F1 rounded up so that the rows
// of consecutive m2 start F0 banks apart (conflict-free stage-2 stores).
template <int F0, int F1>
__host__ __device__ constexpr int c2f_row_stride()
{
    int s = F0 * F1;
    while (s % 16 != F0 % 16)
        s++;
    return s;
}

// stage 2 of the fixed coarse-to-fine kernel: threads per fine column
// block j0 (its L0 x H2 row vectors, whole warps, so that a warp works for
// one j0 only)
template <int H2, int L0> __host__ __device__ constexpr int c2f_stage2_group()
{
    return (L0 * H2 + 31) / 32 * 32;
}

// one thread per row vector of the widest of the three stages
template <int H0, int H1, int H2, int L0, int L1, int L2, int F>
constexpr int c2f_fixed_threads()
{
    constexpr int s1 = H1 * H2, s2 = F * c2f_stage2_group<H2, L0>(), s3 = F * L0 * F * L1;
    constexpr int m = s1 > s2 ? (s1 > s3 ? s1 : s3) : (s2 > s3 ? s2 : s3);
    return (m + 31) / 32 * 32;
}

// Coarse-to-fine with compile-time orders and refinement factor F (the same
// in every dimension), one coarse cone per block, register-tiled: every
// thread loads one input vector of a mode product into registers once and
// produces all output rows that use it.
//   stage 1 (thread = (m1, m2)):  Y1[i0][m1][m2] = sum_m A0[i0][m] X[m][m1][m2]
//   stage 2 (thread = (i0, m2)):  Y2[m2][i0 + F0 i1] = sum_m A1[i1][m] Y1[i0][m][m2]
//   stage 3 (thread = i0 + F0 i1): C[j2 L2 + i2] = sum_m A2[j2 L2 + i2][m] Y2[m][.]
// Stage 3 writes the coefficients of every active sub-cone straight to
// global memory.  Warps follow the sub-cones: a stage-2 warp works for one
// fine column block j0 and skips the row blocks j1 whose sub-cones (j0, j1,
// j2) are all inactive; stage-3 threads go sub-cone by sub-cone (L0 L1 each),
// so that a warp spans about two sub-cones, skips the j2 where they are
// inactive and writes each active one's rows as contiguous runs.  NPL
// planes per CTA (blockIdx.y: planes NPL y ...): each matrix constant, index
// and barrier then serves NPL row vectors (2 for FP32 batches: 3.15 -> 3.03
// ms per batched matvec at N = 1e6).  T is the working precision (double,
// or float in the mixed pipeline).
template <int H0, int H1, int H2, int L0, int L1, int L2, int F, typename T, int NPL>
__global__ void __launch_bounds__(c2f_fixed_threads<H0, H1, H2, L0, L1, L2, F>())
    coarse_to_fine_fixed_kernel(C2FArgs a, const C2FMats<H0, H1, H2, L0, L1, L2, F, T> M)
{
    using V = typename Vec2<T>::type;
    constexpr int F0 = F * L0, F1 = F * L1;
    constexpr int P_HI = H0 * H1 * H2, P_LO = L0 * L1 * L2;
    constexpr int S2 = c2f_row_stride<F0, F1>();
    constexpr int Y1N = F0 * H1 * H2, YN = Y1N + S2 * H2; // elements per plane
    extern __shared__ __align__(16) unsigned char c2f_raw[];
    // plane p: Y1 at p YN ([m2][m1][i0], i0 fastest), Y2 at p YN + Y1N ([m2][S2])
    V* Y = reinterpret_cast<V*>(c2f_raw);
    __shared__ int gsub[F * F * F];
    const int c = a.idx ? a.idx[blockIdx.x] : (int)blockIdx.x;
    const int t = threadIdx.x;
    const int box = a.cc_box[c], el = a.cc_el[c];
    const int p0 = blockIdx.y * NPL; // first plane of the CTA
    if (t < F * F * F)
    {
        const int nc0 = a.G.nc[0], nc1 = a.G.nc[1];
        const int hid0 = el % nc0, hid1 = (el / nc0) % nc1, hid2 = el / (nc0 * nc1);
        const int nf0 = a.G.nf[0], nf1 = a.G.nf[1];
        const long long nft = (long long)nf0 * nf1 * a.G.nf[2];
        const int* fm = a.fmap + a.G.fmap_off + (long long)(box - a.G.box_off) * nft;
        const int j0 = t % F, j1 = (t / F) % F, j2 = t / (F * F);
        gsub[t] = fm[((hid2 * F + j2) * nf1 + (hid1 * F + j1)) * nf0 + (hid0 * F + j0)];
    }
    if (t < H1 * H2)
    {
        V x[NPL][H0];
#pragma unroll
        for (int p = 0; p < NPL; p++)
        {
            const V* src = reinterpret_cast<const V*>(a.cvals) + (p0 + p) * a.cv_plane +
                           (size_t)c * P_HI + H0 * t;
#pragma unroll
            for (int m = 0; m < H0; m++)
                x[p][m] = src[m];
        }
#pragma unroll
        for (int i0 = 0; i0 < F0; i0++)
        {
#pragma unroll
            for (int p = 0; p < NPL; p++)
            {
                T re = 0, im = 0;
#pragma unroll
                for (int m = 0; m < H0; m++)
                {
                    re = fma(M.a0[i0 * H0 + m], x[p][m].x, re);
                    im = fma(M.a0[i0 * H0 + m], x[p][m].y, im);
                }
                Y[p * YN + i0 + F0 * t] = V{re, im};
            }
        }
    }
    __syncthreads();
    constexpr int G2 = c2f_stage2_group<H2, L0>();
    if (t < F * G2 && t % G2 < L0 * H2)
    {
        const int j0 = t / G2, u = t % G2;
        const int i0 = j0 * L0 + u % L0, m2 = u / L0;
        V x[NPL][H1];
#pragma unroll
        for (int p = 0; p < NPL; p++)
#pragma unroll
            for (int m = 0; m < H1; m++)
                x[p][m] = Y[p * YN + i0 + F0 * (m + H1 * m2)];
#pragma unroll
        for (int j1 = 0; j1 < F; j1++)
        {
            bool used = false;
#pragma unroll
            for (int j2 = 0; j2 < F; j2++)
                used |= gsub[j0 + F * (j1 + F * j2)] >= 0;
            if (!used)
                continue; // no active sub-cone reads these rows
#pragma unroll
            for (int i1 = j1 * L1; i1 < (j1 + 1) * L1; i1++)
            {
#pragma unroll
                for (int p = 0; p < NPL; p++)
                {
                    T re = 0, im = 0;
#pragma unroll
                    for (int m = 0; m < H1; m++)
                    {
                        re = fma(M.a1[i1 * H1 + m], x[p][m].x, re);
                        im = fma(M.a1[i1 * H1 + m], x[p][m].y, im);
                    }
                    Y[p * YN + Y1N + i0 + F0 * i1 + S2 * m2] = V{re, im};
                }
            }
        }
    }
    __syncthreads();
    if (t < F0 * F1)
    {
        const int q = t % (L0 * L1), sc = t / (L0 * L1);
        const int i0 = q % L0, i1 = q / L0, j0 = sc % F, j1 = sc / F;
        const int i0f = j0 * L0 + i0, i1f = j1 * L1 + i1;
        V x[NPL][H2];
#pragma unroll
        for (int p = 0; p < NPL; p++)
#pragma unroll
            for (int m = 0; m < H2; m++)
                x[p][m] = Y[p * YN + Y1N + i0f + F0 * i1f + S2 * m];
#pragma unroll
        for (int j2 = 0; j2 < F; j2++)
        {
            const int gf = gsub[j0 + F * (j1 + F * j2)];
            if (gf < 0)
                continue;
#pragma unroll
            for (int i2 = 0; i2 < L2; i2++)
            {
#pragma unroll
                for (int p = 0; p < NPL; p++)
                {
                    T re = 0, im = 0;
#pragma unroll
                    for (int m = 0; m < H2; m++)
                    {
                        re = fma(M.a2[(j2 * L2 + i2) * H2 + m], x[p][m].x, re);
                        im = fma(M.a2[(j2 * L2 + i2) * H2 + m], x[p][m].y, im);
                    }
                    V* fco = reinterpret_cast<V*>(a.fcoef) + (p0 + p) * a.fc_plane;
                    fco[(size_t)gf * P_LO + i0 + L0 * i1 + L0 * L1 * i2] = V{re, im};
                }
            }
        }
    }
}

template <int H0, int H1, int H2, int L0, int L1, int L2, int F, typename T>
constexpr size_t c2f_fixed_smem(int npl = 1)
{
    constexpr int F0 = F * L0, F1 = F * L1;
    return (size_t)npl * (F0 * H1 * H2 + c2f_row_stride<F0, F1>() * H2) * 2 * sizeof(T);
}

// Launches the fixed-size coarse-to-fine kernel when (hi, lo, f) is one of the
// instantiated shapes; returns false otherwise.
template <typename T>
static bool launch_c2f_fixed(const C2FArgs& fa, const double* A_host, unsigned grid,
                             cudaStream_t st, unsigned planes = 1)
{
    const int* h = fa.hi;
    const int* l = fa.lo;
    const int f = fa.f[0];
    if (fa.f[1] != f || fa.f[2] != f || (f != 3 && f != 1) || A_host == nullptr)
        return false;
    // refinement factor 3 (fine grid 3x the coarse one) or 1 (the modified
    // Helmholtz kernel: fine = coarse grid)
#define IFGF_C2F_CASE_F(A, B, C, D, E, G, F)                                                  \
    {                                                                                          \
        C2FMats<A, B, C, D, E, G, F, T> mats;                                                  \
        T* dst = mats.a0;                                                                      \
        constexpr int NA = F * (D * A + E * B + G * C);                                        \
        static_assert(sizeof(mats) == NA * sizeof(T), "matrix block layout");                  \
        for (int i = 0; i < NA; i++)                                                           \
            dst[i] = (T)A_host[i];                                                             \
        /* FP32: two planes per CTA share every matrix constant and index */                  \
        constexpr int NPL = std::is_same<T, float>::value ? 2 : 1;                             \
        const int npl = planes % NPL == 0 ? NPL : 1;                                           \
        const size_t sm = c2f_fixed_smem<A, B, C, D, E, G, F, T>(npl);                         \
        auto kern = npl == 2 ? coarse_to_fine_fixed_kernel<A, B, C, D, E, G, F, T, NPL>        \
                             : coarse_to_fine_fixed_kernel<A, B, C, D, E, G, F, T, 1>;         \
        if (sm > 48 * 1024)                                                                    \
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);  \
        kern<<<dim3(grid, planes / npl), c2f_fixed_threads<A, B, C, D, E, G, F>(), sm, st>>>(  \
            fa, mats);                                                                         \
        return true;                                                                           \
    }
#define IFGF_C2F_CASE(A, B, C, D, E, G)                                                       \
    if (h[0] == A && h[1] == B && h[2] == C && l[0] == D && l[1] == E && l[2] == G)            \
    {                                                                                          \
        if (f == 3)                                                                            \
            IFGF_C2F_CASE_F(A, B, C, D, E, G, 3)                                               \
        else                                                                                   \
            IFGF_C2F_CASE_F(A, B, C, D, E, G, 1)                                               \
    }
    IFGF_C2F_CASE(5, 8, 8, 2, 5, 5)
    IFGF_C2F_CASE(6, 9, 9, 3, 6, 6)
    IFGF_C2F_CASE(7, 10, 10, 4, 7, 7)
    // p = 11 and 12: one CTA of up to 512 threads per SM by its shared memory
    // (137 KB at p = 12), yet at N = 3e4, p = 12 1.0 ms per FP64 matvec where
    // the runtime-order kernel takes 7.7
    IFGF_C2F_CASE(8, 11, 11, 5, 8, 8)
    IFGF_C2F_CASE(9, 12, 12, 6, 9, 9)
#undef IFGF_C2F_CASE
#undef IFGF_C2F_CASE_F
    return false;
}

bool launch_c2f_fixed_f32(const C2FArgs& fa, const double* A_host, unsigned grid, cudaStream_t st,
                          unsigned planes)
{
    return launch_c2f_fixed<float>(fa, A_host, grid, st, planes);
}

bool launch_c2f_fixed_f64(const C2FArgs& fa, const double* A_host, unsigned grid, cudaStream_t st)
{
    return launch_c2f_fixed<double>(fa, A_host, grid, st);
}

} // namespace ifgf
