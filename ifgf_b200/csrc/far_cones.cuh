// Far field of the FP64 matvec, cone by cone (included by mult_kernels.cuh
// inside namespace ifgf).  The far-cone plan (far_cones.cu) lists, for every
// fine cone, the targets that evaluate it, in tiles of eight places, so a
// cone's coefficient block goes straight from memory into matrix fragments
// for all of its targets and the Chebyshev sums of eight targets at a time
// run on the FP64 tensor cores.  The values go to one array in cone order;
// far_gather_kernel adds every target's values in the order of its far list
// (the same order in every call).
#pragma once

// How the sums of order (N0, N1, N2) map to m8n8k4 products: the columns are
// the dimension ND of the block (times real and imaginary part, or real
// blocks alone), the inner dimension runs over the other two, P and Q.  The
// four lanes of a row take the four parity classes of (i_P, i_Q): each lane
// then advances its own basis values by the step-two recurrence
// T_{m+2} = 2 T_2 T_m - T_{m-2} and never selects by index.
template <int N0, int N1, int N2, bool REAL> struct ConeShape
{
    static constexpr int steps(int nd)
    {
        const int np = nd == 0 ? N1 : N0, nq = nd == 0 ? N2 : N1;
        return ((np + 1) / 2) * ((nq + 1) / 2);
    }
    static constexpr int cols(int nd) { return (REAL ? 1 : 2) * (nd == 0 ? N0 : N2); }
    static constexpr int cost(int nd) { return steps(nd) * ((cols(nd) + 7) / 8); }
    // fewer products; with as many, fewer steps
    static constexpr int ND =
        cost(0) < cost(2) || (cost(0) == cost(2) && steps(0) < steps(2)) ? 0 : 2;
    static constexpr int NN = ND == 0 ? N0 : N2;
    static constexpr int NP = ND == 0 ? N1 : N0, NQ = ND == 0 ? N2 : N1;
    static constexpr int KP = (NP + 1) / 2, KQ = (NQ + 1) / 2, KS = KP * KQ;
    static constexpr int NT = (cols(ND) + 7) / 8;
    // offset of coefficient (p, q, n) in a block
    __device__ static int at(int p, int q, int n)
    {
        return ND == 0 ? n + N0 * (p + N1 * q) : p + N0 * (q + N1 * n);
    }
};

__device__ __forceinline__ void dmma884(double (&c)[2], double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}

// T_par, T_{par+2}, ... at x
template <int K> __device__ __forceinline__ void cheb_parity(double x, bool odd, double (&t)[K])
{
    const double x2 = fma(2.0 * x, x, -1.0);
    t[0] = odd ? x : 1.0;
    double prev = odd ? x : x2; // T_{par-2}
#pragma unroll
    for (int m = 1; m < K; m++)
    {
        const double next = fma(2.0 * x2, t[m - 1], -prev);
        prev = t[m - 1];
        t[m] = next;
    }
}

// asin(v) for |v| <= sin(0.2628): v + v z P(z), z = v^2, P through Chebyshev
// points of (asin(v) / v - 1) / z (3e-18)
__device__ __forceinline__ double asin_small(double v)
{
    constexpr double c[8] = {0.16666666666665989, 0.07500000000267835,  0.044642856736902034,
                             0.030381975200200743, 0.02237085433704478, 0.017385107934204745,
                             0.013502348595571055, 0.015027759225438878};
    const double z = v * v;
    double p = c[7];
#pragma unroll
    for (int i = 6; i >= 0; i--)
        p = fma(p, z, c[i]);
    return fma(v * z, p, v);
}

struct FarConeArgs
{
    FarConePtrs fc;
    const LevelGeom* __restrict__ lv;
    TreeArgs T;
    const double* __restrict__ tx;
    const double* __restrict__ ty;
    const double* __restrict__ tz;
    const double2* __restrict__ fcoef;
    KParams kp;
};

constexpr int FAR_CONE_THREADS = 128;

// One warp per 32 consecutive places of the plan, four tiles of eight: lane =
// place for the local coordinates and the centred factor, row lane / 4 of the
// products for the sums; both views meet in the warp's shared memory.
// At N = 1e6, p = 9 (3.8e8 pairs) the far field of a matvec takes 17.0 ms with
// the gather; the kernel that looks up every pair and reads its coefficients
// lane by lane took 43.3.  At N = 2e5, p = 8 1.6 and 3.45 ms, N = 2e4 Laplace
// 0.13 and 0.72, 4000 points 0.031 and 0.135.  The FP64 and
// matrix pipes together are about 57 % busy at p = 8, issue slots 65 %.  A
// first form gave a warp up to 64 places of one cone: its second batch of 32
// lanes was mostly empty (22.9 ms).
template <int KIND, int N0, int N1, int N2>
__global__ void __launch_bounds__(FAR_CONE_THREADS)
    far_cone_kernel(const __grid_constant__ FarConeArgs a)
{
    constexpr bool REAL = KIND == K_LAPLACE;
    constexpr int P_LO = N0 * N1 * N2;
    using S = ConeShape<N0, N1, N2, REAL>;
    __shared__ double xs[FAR_CONE_THREADS / 32][3][32];
    __shared__ double2 vs[FAR_CONE_THREADS / 32][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long group = blockIdx.x * (long long)(FAR_CONE_THREADS / 32) + warp;
    if (group >= a.fc.n_groups)
        return;
    const int cone = a.fc.tile_cone[4 * group + (lane >> 3)]; // -1 past the last tile
    const long long place = 32 * group + lane;
    const int t = a.fc.tgt[place]; // -1: padding
    // the tiles' coefficient blocks on their way to L1
    for (int q = 0; q < 4; q++)
    {
        const int c = __shfl_sync(~0u, cone, 8 * q);
        if (c >= 0 && (q == 0 || c != __shfl_sync(~0u, cone, 8 * q - 8)))
            for (int o = 128 * lane; o < P_LO * (int)sizeof(double2); o += 32 * 128)
                asm volatile("prefetch.global.L1 [%0];" ::"l"(
                    reinterpret_cast<const char*>(a.fcoef + (size_t)c * P_LO) + o));
    }
    DistInv D{1.0, 1.0};
    if (t >= 0)
    {
        const int2 be = a.fc.meta[cone];
        const int box = be.x, lev = a.T.box_level[box];
        const LevelGeom& G = a.lv[lev];
        const double H = a.T.box_H[box];
        const int2 ct = a.fc.level[lev]; // (trig table offset, narrow cones)
        const double p[3] = {a.tx[t] - a.T.box_c[3 * box], a.ty[t] - a.T.box_c[3 * box + 1],
                             a.tz[t] - a.T.box_c[3 * box + 2]};
        const double r2 = fma(p[0], p[0], p[1] * p[1]), d2 = fma(p[2], p[2], r2);
        double x[3];
        if (ct.y && !odd_square(r2) && d2 < INF64)
        {
            // angles relative to the cone's centre line, from the sines of
            // their differences
            const int i0 = be.y % G.nf[0], i12 = be.y / G.nf[0];
            const int i1 = i12 % G.nf[1], i2 = i12 / G.nf[1];
            const double2 th = a.fc.trig[ct.x + i1], ph = a.fc.trig[ct.x + G.nf[1] + i2];
            const double b0 = G.dmin[0] + ((double)i0 + 0.5) * G.hf[0];
            const DistInv R = dist_inv<true>(r2);
            D = dist_inv<true>(d2);
            x[0] = fma(H, D.id, -b0) * (2.0 * G.hfi[0]);
            x[1] = asin_small(fma(R.d, th.y, -(p[2] * th.x)) * D.id) * (2.0 * G.hfi[1]);
            x[2] = asin_small(fma(p[1], ph.y, -(p[0] * ph.x)) * R.id) * (2.0 * G.hfi[2]);
        }
        else
        {
            double s[3];
            cart_to_interp(p[0], p[1], p[2], H, s);
            to_local(be.y, s, G.dmin, G.hf, G.hfi, G.nf, x);
            D = dist_inv<false>(d2);
        }
#pragma unroll
        for (int d = 0; d < 3; d++)
            xs[warp][d][lane] = x[d];
    }
    else
#pragma unroll
        for (int d = 0; d < 3; d++)
            xs[warp][d][lane] = 0.0;
    __syncwarp();
    // the lane's parity class and its part of the tile's coefficient block
    const bool op = lane & 1, oq = lane & 2;
    const int row = lane >> 2, r = lane & 3;
    double b[S::KS][S::NT];
    int have = -1;
#pragma unroll 1
    for (int q = 0; q < 4; q++)
    {
        const int c = __shfl_sync(~0u, cone, 8 * q);
        if (c < 0)
            break;
        if (c != have)
        {
            const double2* blk = a.fcoef + (size_t)c * P_LO;
#pragma unroll
            for (int s = 0; s < S::KS; s++)
#pragma unroll
                for (int nt = 0; nt < S::NT; nt++)
                {
                    const int ip = 2 * (s / S::KQ) + (op ? 1 : 0),
                              iq = 2 * (s % S::KQ) + (oq ? 1 : 0);
                    const int col = 8 * nt + row, n = REAL ? col : col >> 1;
                    b[s][nt] = 0.0;
                    if (ip < S::NP && iq < S::NQ && n < S::NN)
                    {
                        const double2* v = blk + S::at(ip, iq, n);
                        b[s][nt] = !REAL && (col & 1) ? v->y : v->x;
                    }
                }
            have = c;
        }
        const double y0 = xs[warp][0][8 * q + row], y1 = xs[warp][1][8 * q + row],
                     y2 = xs[warp][2][8 * q + row];
        double tp[S::KP], tq[S::KQ], acc[S::NT][2];
        cheb_parity<S::KP>(S::ND == 0 ? y1 : y0, op, tp);
        cheb_parity<S::KQ>(S::ND == 0 ? y2 : y1, oq, tq);
#pragma unroll
        for (int nt = 0; nt < S::NT; nt++)
            acc[nt][0] = acc[nt][1] = 0.0;
#pragma unroll
        for (int s = 0; s < S::KS; s++)
        {
            const double w = tp[s / S::KQ] * tq[s % S::KQ];
#pragma unroll
            for (int nt = 0; nt < S::NT; nt++)
                dmma884(acc[nt], w, b[s][nt]);
        }
        // columns 2 r and 2 r + 1 of every product, times T_n of their n
        const double xn = S::ND == 0 ? y0 : y2;
        double sr = 0.0, si = 0.0;
        if constexpr (REAL)
        {
            // n = 8 nt + 2 r + e: steps of eight by T_8
            double u[9];
            u[0] = 1.0;
            u[1] = xn;
#pragma unroll
            for (int m = 2; m < 9; m++)
                u[m] = fma(2.0 * xn, u[m - 1], -u[m - 2]);
            double e0 = r == 0 ? u[0] : r == 1 ? u[2] : r == 2 ? u[4] : u[6];
            double e1 = r == 0 ? u[1] : r == 1 ? u[3] : r == 2 ? u[5] : u[7];
            double p0 = r == 0 ? u[8] : r == 1 ? u[6] : r == 2 ? u[4] : u[2];
            double p1 = r == 0 ? u[7] : r == 1 ? u[5] : r == 2 ? u[3] : u[1];
#pragma unroll
            for (int nt = 0; nt < S::NT; nt++)
            {
                sr = fma(acc[nt][0], e0, fma(acc[nt][1], e1, sr));
                if (nt + 1 < S::NT)
                {
                    const double n0 = fma(2.0 * u[8], e0, -p0), n1 = fma(2.0 * u[8], e1, -p1);
                    p0 = e0, p1 = e1, e0 = n0, e1 = n1;
                }
            }
            sr += __shfl_xor_sync(~0u, sr, 1);
            sr += __shfl_xor_sync(~0u, sr, 2);
            if (r == 0)
                vs[warp][8 * q + row].x = sr;
        }
        else
        {
            // n = 4 nt + r: steps of four by T_4
            const double u2 = fma(2.0 * xn, xn, -1.0), u3 = fma(2.0 * xn, u2, -xn),
                         u4 = fma(2.0 * u2, u2, -1.0);
            double e = r == 0 ? 1.0 : r == 1 ? xn : r == 2 ? u2 : u3;
            double p = r == 0 ? u4 : r == 1 ? u3 : r == 2 ? u2 : xn; // T_{4-r}
#pragma unroll
            for (int nt = 0; nt < S::NT; nt++)
            {
                sr = fma(acc[nt][0], e, sr);
                si = fma(acc[nt][1], e, si);
                if (nt + 1 < S::NT)
                {
                    const double next = fma(2.0 * u4, e, -p);
                    p = e;
                    e = next;
                }
            }
            // even lanes collect the real parts, odd ones the imaginary parts
            const double give = op ? sr : si;
            double keep = (op ? si : sr) + __shfl_xor_sync(~0u, give, 1);
            keep += __shfl_xor_sync(~0u, keep, 2);
            if (r < 2)
                reinterpret_cast<double*>(&vs[warp][8 * q + row])[r] = keep;
        }
    }
    __syncwarp();
    if (t >= 0)
    {
        const cplx<double> f = Plugin<KIND>::cf(D, a.kp);
        const double2 v = vs[warp][lane];
        static_cast<double2*>(a.fc.val)[place] =
            REAL ? make_double2(v.x * f.re, 0.0)
                 : make_double2(v.x * f.re - v.y * f.im, v.x * f.im + v.y * f.re);
    }
}

// The same for the mixed pipeline, one thread per two places of a tile: the
// FP32 lookup's local coordinates, FP32 coefficients and sums; every coefficient
// load serves both places, and the lanes of a tile read one block.  At N = 1e6,
// p = 9 11.1 ms per matvec with the gather; looking every pair up and
// reading each lane's block took 17.0, one place per thread 14.5 (L1 73 % busy).
constexpr int FAR_CONE_PER = 2;
template <int KIND, int N0, int N1, int N2>
__global__ void __launch_bounds__(FAR_CONE_THREADS)
    far_cone_mixed_kernel(const __grid_constant__ FarConeArgs a)
{
    constexpr int P_LO = N0 * N1 * N2, R = FAR_CONE_PER;
    const long long place = (blockIdx.x * (long long)FAR_CONE_THREADS + threadIdx.x) * R;
    if (place >= 32 * a.fc.n_groups)
        return;
    const int cone = a.fc.tile_cone[place / FAR_TILE]; // -1 past the last tile
    int t[R];
#pragma unroll
    for (int r = 0; r < R; r++)
        t[r] = a.fc.tgt[place + r]; // -1: padding
    const float2* blk = reinterpret_cast<const float2*>(a.fcoef) + (size_t)max(cone, 0) * P_LO;
    if (cone >= 0) // the block's lines on their way to L1
        for (int o = 128 * (threadIdx.x % (FAR_TILE / R)); o < P_LO * (int)sizeof(float2);
             o += 128 * (FAR_TILE / R))
            asm volatile("prefetch.global.L1 [%0];" ::"l"(reinterpret_cast<const char*>(blk) + o));
    bool any = false;
#pragma unroll
    for (int r = 0; r < R; r++)
        any |= t[r] >= 0;
    if (!any)
        return;
    const int2 be = a.fc.meta[cone];
    const int box = be.x, lev = a.T.box_level[box];
    const double H = a.T.box_H[box];
    const double xc[3] = {a.T.box_c[3 * box], a.T.box_c[3 * box + 1], a.T.box_c[3 * box + 2]};
    float loc[R][3], vr[R], vi[R];
    double d2[R];
#pragma unroll
    for (int r = 0; r < R; r++)
    {
        const int tr = t[r] >= 0 ? t[r] : 0;
        const double p[3] = {a.tx[tr] - xc[0], a.ty[tr] - xc[1], a.tz[tr] - xc[2]};
        d2[r] = p[0] * p[0] + p[1] * p[1] + p[2] * p[2];
        if (lookup_f(a.fc.lookup[lev], p, H, loc[r]) != be.y && t[r] >= 0)
        {
            // a pair that the FP64 lookup placed
            const LevelGeom& G = a.lv[lev];
            double s[3], ld[3];
            cart_to_interp(p[0], p[1], p[2], H, s);
            to_local(be.y, s, G.dmin, G.hf, G.hfi, G.nf, ld);
            loc[r][0] = (float)ld[0];
            loc[r][1] = (float)ld[1];
            loc[r][2] = (float)ld[2];
        }
    }
    ChebMulti<float, N0, N1, N2, R>::eval(blk, loc, nullptr, vr, vi);
#pragma unroll
    for (int r = 0; r < R; r++)
        if (t[r] >= 0)
        {
            const cplx<float> f = cf_mixed<KIND>(d2[r], a.kp);
            reinterpret_cast<float2*>(a.fc.val)[place + r] =
                make_float2(vr[r] * f.re - vi[r] * f.im, vr[r] * f.im + vi[r] * f.re);
        }
}
