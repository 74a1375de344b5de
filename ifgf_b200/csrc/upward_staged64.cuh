// FP64 upward transfer (transferInterp, ifgfoperator.hpp:1639-1705) with the
// children's coefficient blocks staged in shared memory.  Included by
// mult_kernels.cuh inside namespace ifgf.
#pragma once

// Chebyshev sums of R points in one FP64 coefficient block in shared memory:
// each coefficient (one 16-byte load) feeds 2 R FMAs (R for REAL blocks,
// whose imaginary parts are zero).  The basis along the outermost dimension
// is advanced by its recurrence instead of kept, and blocks of more than 128
// coefficients loop over that dimension (code size).
template <int N0, int N1, int N2, int R, bool REAL>
__device__ __forceinline__ void cheb_staged64(const double2* __restrict__ c, const double (&x)[R][3],
                                              double (&ore)[R], double (&oim)[R])
{
    double t0[R][N0], t1[R][N1], ta[R], tb[R];
#pragma unroll
    for (int r = 0; r < R; r++)
    {
        cheb_basis<double, N0>(x[r][0], t0[r]);
        cheb_basis<double, N1>(x[r][1], t1[r]);
        ta[r] = 1.0;     // T_k of the current slab
        tb[r] = x[r][2]; // T_{k-1}, as T_{-1} = T_1 before the first slab
        ore[r] = oim[r] = 0.0;
    }
    auto slab = [&](int k) {
        const double2* ck = c + N0 * N1 * k;
        double br[R], bi[R];
#pragma unroll
        for (int j = 0; j < N1; j++)
        {
            double cr[R], ci[R];
#pragma unroll
            for (int i = 0; i < N0; i++)
            {
                const double2 v = ck[i + N0 * j];
#pragma unroll
                for (int r = 0; r < R; r++)
                {
                    cr[r] = i == 0 ? v.x : fma(v.x, t0[r][i], cr[r]);
                    if (!REAL)
                        ci[r] = i == 0 ? v.y : fma(v.y, t0[r][i], ci[r]);
                }
            }
#pragma unroll
            for (int r = 0; r < R; r++)
            {
                br[r] = j == 0 ? cr[r] : fma(cr[r], t1[r][j], br[r]);
                if (!REAL)
                    bi[r] = j == 0 ? ci[r] : fma(ci[r], t1[r][j], bi[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < R; r++)
        {
            ore[r] = fma(br[r], ta[r], ore[r]);
            if (!REAL)
                oim[r] = fma(bi[r], ta[r], oim[r]);
            const double tn = fma(2.0 * x[r][2], ta[r], -tb[r]);
            tb[r] = ta[r];
            ta[r] = tn;
        }
    };
    if constexpr (N0 * N1 * N2 <= 128)
    {
#pragma unroll
        for (int k = 0; k < N2; k++)
            slab(k);
    }
    else
    {
#pragma unroll 1
        for (int k = 0; k < N2; k++)
            slab(k);
    }
}

// Out of line: it runs for the few nodes whose tabulated element is inactive.
template <int KIND>
__device__ __noinline__ bool ups64_fallback(const UpArgs& a, int box, int el, int n, int cb,
                                            const int* fm, cplx<double>& v)
{
    return upward_fallback64<KIND>(a, box, el, n, cb, fm, v);
}

// Threads: blocks of more than 200 coefficients leave room for fewer CTAs per
// SM, so these take twice as many.
__host__ __device__ constexpr int ups64_threads(int p_lo) { return p_lo > 200 ? 128 : 64; }

// Stride (in double2) of a staged block: odd, so that the blocks of eight
// consecutive runs start in eight different 16-byte bank groups.
__host__ __device__ constexpr int ups64_stride(int p_lo) { return p_lo | 1; }

// Runs staged at a time: about 16 KB of blocks, at least four runs (rows
// average a handful; a run has about ten groups of entries at p = 8 and some
// twenty-five at p = 12).
template <int N0, int N1, int N2> int ups64_rch(int fe_pad, int threads)
{
    constexpr int per = ups64_stride(N0 * N1 * N2) * (int)sizeof(double2);
    const int fit = std::max(4, (threads > 128 ? 48 : 16) * 1024 / per);
    return fe_pad < fit ? fe_pad : fit;
}
template <int N0, int N1, int N2> size_t ups64_smem(int P_hi, int rch, int fe_pad)
{
    return ((size_t)P_hi + (size_t)rch * ups64_stride(N0 * N1 * N2)) * sizeof(double2) +
           ((size_t)16 * (fe_pad + 1) + 16) * sizeof(int);
}

// Levels of few cones, which leave SMs idle or short of warps, take 256 threads
// per cone and stage three times the runs, where those CTAs (two per SM) all
// reside at once: measured (ms) 264 cones 0.029 instead of 0.056, 192 cones
// 0.031 instead of 0.068, but 663 cones 0.069 and 0.067, 917 cones 0.060 and
// 0.051.
constexpr int UPS64_FEW = 2 * 148;

// Entries evaluated together per thread (sharing every coefficient load);
// CTAs per SM give every thread 128 registers.
constexpr int UPS64_R = 2;

// One CTA per parent cone (CTAs ordered by cone element, so that consecutive
// ones share their geometry-table rows in L2).  When it starts it resolves
// the fine cone and the first group of every run of all eight children in one
// pass of independent loads; then, child by child, the coefficient blocks of
// up to rch runs are copied into shared memory (cp.async, one warp per
// block) and the runs' groups of UPGEO_RUN entries are evaluated from there.
// Each node is updated once per child, so the per-node sums need no atomics.
// Bound by the shared loads (a 16-byte load takes about three wavefronts for
// the few blocks a warp reads and feeds 2 R FMAs) and the latency of the
// chunks' copies.  The kernel it replaces gathered every coefficient from
// global memory: at N = 1e6, p = 9 the transfer took 57.4 ms per matvec and
// takes 28.0; at N = 2e5, p = 8 4.1 and 2.5.  Measured at N = 1e6 for entries
// per thread / threads / KB of blocks / CTAs per SM: 2 / 64 / 16 / 8 28.3 ms,
// 2 / 64 / 16 / 10 29.7, 2 / 96 / 24 / 6 32.9, 4 / 64 / 24 / 6 30.1,
// 4 / 64 / 16 / 4 35.6, 4 / 32 / 8 / 12 35.5: warps in flight are worth more
// than fewer loads.
template <int KIND, int N0, int N1, int N2, int THREADS>
__global__ void __launch_bounds__(THREADS, 512 / THREADS)
    upward_staged64_kernel(const __grid_constant__ UpArgs a)
{
    constexpr int R = UPS64_R;
    constexpr int P_LO = N0 * N1 * N2;
    constexpr int BS = ups64_stride(P_LO);
    constexpr int SUB = UPGEO_RUN / R; // work items per table group
    constexpr bool REAL = KIND == K_LAPLACE;
    extern __shared__ __align__(16) double2 up_sh64[];
    double2* acc = up_sh64;
    double2* blk = up_sh64 + a.P_hi;
    const int FL = a.fe_pad + 1;
    int* run_gf = reinterpret_cast<int*>(blk + (size_t)a.rch * BS); // [8][FL] child fine cone
    int* run_g = run_gf + 8 * FL;                                   // [8][FL] first group
    int* row_n = run_g + 8 * FL; // [8] runs of the row, [8] groups of the row
    const int c = a.idx[blockIdx.x];
    const int slot = a.slot[blockIdx.x];
    const int box = a.cc_box[c], el = a.cc_el[c];
    const int warp = threadIdx.x >> 5;
    const int ngroups = a.P_pad / UPGEO_RUN;
    for (int n = threadIdx.x; n < a.P_hi; n += THREADS)
        acc[n] = make_double2(0.0, 0.0);
    if (threadIdx.x < 8)
    {
        row_n[threadIdx.x] = a.fe_pad;
        row_n[8 + threadIdx.x] = ngroups;
    }
    __syncthreads();
    const LevelGeom& C = a.GC;
    const long long nf = (long long)C.nf[0] * C.nf[1] * C.nf[2];
    for (int i = threadIdx.x; i < 8 * FL; i += THREADS)
    {
        const int o = i / FL, r = i - o * FL;
        const int cb = a.T.box_child[8 * box + o];
        const int2 f = a.fe_list[((size_t)slot * 8 + o) * FL + r];
        run_gf[i] = cb >= 0 && f.x >= 0 ? a.fmap[C.fmap_off + (long long)(cb - C.box_off) * nf + f.x]
                                        : -1;
        run_g[i] = f.y;
        if (f.x < 0 && f.y >= 0)
        {
            // the sentinel after the row's last run: (-1, groups of the row)
            row_n[o] = r;
            row_n[8 + o] = f.y;
        }
    }
    __syncthreads();
    for (int o = 0; o < 8; o++)
    {
        const int cb = a.T.box_child[8 * box + o];
        if (cb < 0)
            continue;
        const int* rgf = run_gf + o * FL;
        const int* rg = run_g + o * FL;
        const UpGeo64* row = a.geo64 + ((size_t)slot * 8 + o) * a.P_pad;
        const int nrun = row_n[o];
        for (int r0 = 0; r0 < nrun; r0 += a.rch)
        {
            const int r1 = min(r0 + a.rch, nrun);
            const int g_beg = rg[r0];
            // the next run's first group, or the row's end
            const int g_end = r1 < nrun ? rg[r1] : row_n[8 + o];
            __syncthreads(); // the previous runs' blocks are no longer read
            for (int r = r0 + warp; r < r1; r += THREADS / 32)
            {
                const int gf = rgf[r];
                if (gf < 0)
                    continue;
                const double2* src = a.fcoef + (size_t)gf * P_LO;
                double2* dst = blk + (size_t)(r - r0) * BS;
                for (int i = threadIdx.x & 31; i < P_LO; i += 32)
                    cp_async16(dst + i, src + i);
            }
            cp_async_wait_all();
            __syncthreads();
            for (int it = threadIdx.x; it < (g_end - g_beg) * SUB; it += THREADS)
            {
                const int h = it % SUB, g = g_beg + it / SUB;
                int rl = 0; // the group's run, relative to r0
                while (r0 + rl + 1 < r1 && rg[r0 + rl + 1] <= g)
                    rl++;
                const UpGeo64* ent = row + (size_t)(h * R) * ngroups + g;
                if (rgf[r0 + rl] < 0)
                {
                    // tabulated element inactive in this child: absolute coordinates
                    const int* fm = a.fmap + C.fmap_off + (long long)(cb - C.box_off) * nf;
                    for (int r = 0; r < R; r++)
                    {
                        const int n = ent[(size_t)r * ngroups].node;
                        cplx<double> v;
                        if (n >= 0 && ups64_fallback<KIND>(a, box, el, n, cb, fm, v))
                        {
                            acc[n].x += v.re;
                            acc[n].y += v.im;
                        }
                    }
                    continue;
                }
                double x[R][3], vr[R], vi[R];
#pragma unroll
                for (int r = 0; r < R; r++)
#pragma unroll
                    for (int d = 0; d < 3; d++)
                        x[r][d] = ent[(size_t)r * ngroups].loc[d];
                cheb_staged64<N0, N1, N2, R, REAL>(blk + (size_t)rl * BS, x, vr, vi);
#pragma unroll
                for (int r = 0; r < R; r++)
                {
                    const UpGeo64& e = ent[(size_t)r * ngroups];
                    const int n = e.node;
                    if (n < 0)
                        continue;
                    const double2 s = acc[n];
                    acc[n] = REAL ? make_double2(fma(vr[r], e.tr, s.x), 0.0)
                                  : make_double2(s.x + (vr[r] * e.tr - vi[r] * e.ti),
                                                 s.y + (vr[r] * e.ti + vi[r] * e.tr));
                }
            }
        }
    }
    __syncthreads();
    for (int n = threadIdx.x; n < a.P_hi; n += THREADS)
        a.cvals[(size_t)c * a.P_hi + n] = acc[n];
}
