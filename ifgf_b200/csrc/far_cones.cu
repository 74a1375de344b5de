// Builds the far-cone plan and sums its values per target.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cub/cub.cuh>

#include "far_cones.hpp"

namespace ifgf
{

void FarConePlan::release()
{
    mem.release();
    p = FarConePtrs();
    pairs = places = 0;
    ready = refused = captured = false;
    wait = 0;
}

namespace
{

constexpr int THREADS = 256;

// One CTA per target leaf, one thread per (far box, target) pair: the pair's
// fine cone (the FP64 lookup that marked the active cones,
// ifgfoperator.hpp:1736-1891; mixed: the FP32 lookup of the mixed far
// kernels), its index in pos, and the pairs of every cone counted, lanes of
// one cone together.
template <bool MIXED>
__global__ void __launch_bounds__(THREADS)
    count_kernel(const LevelGeom* __restrict__ lv, TreeArgs T, const double* __restrict__ tx,
                 const double* __restrict__ ty, const double* __restrict__ tz,
                 const int* __restrict__ fmap, const int* __restrict__ tl_first,
                 const int* __restrict__ tl_last, const long long* __restrict__ far_off,
                 const int* __restrict__ far_src, const long long* __restrict__ leaf_off, int* pos,
                 int* count, unsigned long long* err, int L)
{
    __shared__ LookupF lfs[MIXED ? MAX_LEVELS : 1];
    if (MIXED)
    {
        for (int l = threadIdx.x; l < L; l += blockDim.x)
            make_lookupf(lv[l], lfs[l]);
        __syncthreads();
    }
    const int tl = blockIdx.x;
    const int t0 = tl_first[tl], cnt = tl_last[tl] - t0;
    const long long f0 = far_off[tl], n = (far_off[tl + 1] - f0) * cnt, o = leaf_off[tl];
    for (long long base = 0; base < n; base += THREADS)
    {
        const long long q = base + threadIdx.x;
        int gf = -1;
        if (q < n)
        {
            const int sb = far_src[f0 + q / cnt], t = t0 + (int)(q % cnt);
            const int lev = T.box_level[sb];
            const LevelGeom& G = lv[lev];
            const double p[3] = {tx[t] - T.box_c[3 * sb], ty[t] - T.box_c[3 * sb + 1],
                                 tz[t] - T.box_c[3 * sb + 2]};
            const long long nft = (long long)G.nf[0] * G.nf[1] * G.nf[2];
            const int* fm = fmap + G.fmap_off + (long long)(sb - G.box_off) * nft;
            if (MIXED)
            {
                float loc[3];
                gf = fine_lookup_fast(lfs[lev], G, fm, p, T.box_H[sb], loc, err);
            }
            else
            {
                double s[3];
                cart_to_interp(p[0], p[1], p[2], T.box_H[sb], s);
                const int fe = element_for_point(s, G.dmin, G.dmax, G.hfi, G.nf);
                if (fe >= 0)
                {
                    gf = fm[fe];
                    if (gf < 0)
                        atomicAdd(err, 1ull);
                }
            }
            pos[o + q] = gf;
        }
        const unsigned same = __match_any_sync(~0u, gf);
        if (gf >= 0 && (threadIdx.x & 31) == __ffs(same) - 1)
            atomicAdd(count + gf, __popc(same));
    }
}

// Places every pair in its cone's list (cursor: next free entry of each
// cone): its target in tgt, its place in pos.  Targets of one warp that
// share a cone stay in order and adjacent.
__global__ void __launch_bounds__(THREADS)
    place_kernel(const int* __restrict__ tl_first, const int* __restrict__ tl_last,
                 const long long* __restrict__ far_off, const long long* __restrict__ leaf_off,
                 int* pos, int* cursor, int* tgt)
{
    const int tl = blockIdx.x, lane = threadIdx.x & 31;
    const int t0 = tl_first[tl], cnt = tl_last[tl] - t0;
    const long long n = (far_off[tl + 1] - far_off[tl]) * cnt, o = leaf_off[tl];
    for (long long base = 0; base < n; base += THREADS)
    {
        const long long q = base + threadIdx.x;
        const int gf = q < n ? pos[o + q] : -1;
        const unsigned same = __match_any_sync(~0u, gf);
        const int lead = __ffs(same) - 1;
        int at = 0;
        if (gf >= 0 && lane == lead)
            at = atomicAdd(cursor + gf, __popc(same));
        at = __shfl_sync(~0u, at, lead) + __popc(same & ((1u << lane) - 1));
        if (gf >= 0)
        {
            pos[o + q] = at;
            tgt[at] = t0 + (int)(q % cnt);
        }
    }
}

// counts rounded up to whole tiles
__global__ void pad_kernel(int* count, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        count[i] = (count[i] + FAR_TILE - 1) / FAR_TILE * FAR_TILE;
}

__global__ void tile_kernel(const int* __restrict__ off, int n, int* tile_cone)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        for (int k = off[i] / FAR_TILE; k < off[i + 1] / FAR_TILE; k++)
            tile_cone[k] = i;
}

__global__ void lookup_kernel(const LevelGeom* __restrict__ lv, int L, LookupF* out)
{
    for (int l = threadIdx.x; l < L; l += blockDim.x)
        make_lookupf(lv[l], out[l]);
}

__global__ void meta_kernel(const int* __restrict__ box, const int* __restrict__ el, int n,
                            int2* meta)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        meta[i] = make_int2(box[i], el[i]);
}

unsigned blocks_for(long long n)
{
    return (unsigned)std::max<long long>(1, std::min<long long>((n + 255) / 256, 148 * 32));
}

} // namespace

namespace
{

// Places of a plan's arrays in its one allocation; the build's scratch shares
// the values' place.
struct Layout
{
    long long n_fine = 0, pairs = 0, most = 0;
    size_t bytes = 0, scan_b = 0, count_b = 0;
    size_t val, pos, tgt, tile, meta, lookup, host, leaf, trig, lev;
    bool fits = false; // there are pairs, and fewer than 2^31 places
    explicit Layout(const FarConeBuild& b)
    {
        size_t n_trig = 0;
        for (const LevelGeom& G : *b.lv)
        {
            n_fine += G.n_fine;
            n_trig += (size_t)(G.nf[1] + G.nf[2]);
        }
        pairs = b.leaf_off->back();
        // places at most: every cone with pairs wastes less than a tile
        most = (pairs + (FAR_TILE - 1) * std::min(n_fine, pairs) + 31) / 32 * 32;
        fits = pairs > 0 && n_fine > 0 && most < (1ll << 31) - 1 && n_fine < (1ll << 31) - 2;
        if (!fits)
            return;
        cub::DeviceScan::ExclusiveSum(nullptr, scan_b, (int*)nullptr, (int*)nullptr,
                                      (int)n_fine + 1);
        auto place = [&](size_t n) {
            const size_t at = bytes;
            bytes += (n + 255) / 256 * 256;
            return at;
        };
        count_b = ((size_t)(n_fine + 1) * sizeof(int) + 255) / 256 * 256;
        const size_t value_b = b.mixed ? sizeof(float2) : sizeof(double2);
        val = place(std::max((size_t)most * value_b, 2 * count_b + scan_b));
        pos = place((size_t)pairs * sizeof(int));
        tgt = place((size_t)most * sizeof(int));
        tile = place((size_t)most / FAR_TILE * sizeof(int));
        meta = place((size_t)n_fine * sizeof(int2));
        lookup = place(b.lv->size() * sizeof(LookupF));
        host = bytes; // from here on filled on the host
        leaf = place(b.leaf_off->size() * sizeof(long long));
        trig = place(n_trig * sizeof(double2));
        lev = place(b.lv->size() * sizeof(int2));
    }
};

} // namespace

void reserve_far_cones(const FarConeBuild& b, FarConePlan& plan)
{
    const Layout at(b);
    if (!at.fits || at.bytes > FAR_CONES_RESERVE)
        return;
    // an operator that just fits the device does without; the build tries again
    (void)plan.mem.try_alloc(at.bytes);
}

void build_far_cones(const FarConeBuild& b, FarConePlan& plan)
{
    const auto start = std::chrono::steady_clock::now();
    const std::vector<LevelGeom>& lv = *b.lv;
    const int L = (int)lv.size(), nl = b.n_tleaf;
    const Layout at(b);
    const long long n_fine = at.n_fine;
    if (plan.mem.n < at.bytes)
        plan.mem.release();
    if (!at.fits)
    {
        plan.refused = true;
        return;
    }
    // host tables: leaf offsets; sines and cosines of the centre angles of
    // every level's fine cones
    std::vector<double2> trig;
    std::vector<int2> level(L);
    for (int l = 0; l < L; l++)
    {
        const LevelGeom& G = lv[l];
        // narrow: half widths within the range of asin_small
        level[l] = make_int2((int)trig.size(), std::max(G.hf[1], G.hf[2]) <= 0.525 ? 1 : 0);
        for (int d = 1; d < 3; d++)
            for (int i = 0; i < G.nf[d]; i++)
            {
                const double c = G.dmin[d] + ((double)i + 0.5) * G.hf[d];
                trig.push_back(make_double2(std::sin(c), std::cos(c)));
            }
    }
    if (!plan.mem.p && at.bytes > (size_t(256) << 20))
    {
        size_t free_b = 0, total_b = 0;
        IFGF_CUDA(cudaMemGetInfo(&free_b, &total_b));
        if (at.bytes > free_b / 4)
        {
            plan.wait = FAR_CONES_RETRY;
            return;
        }
    }
    if (!plan.mem.p && plan.mem.try_alloc(at.bytes) != cudaSuccess)
    {
        plan.wait = FAR_CONES_RETRY;
        return;
    }
    unsigned char* m = plan.mem.p;
    std::vector<unsigned char> host(at.bytes - at.host);
    std::copy_n((const unsigned char*)b.leaf_off->data(), b.leaf_off->size() * sizeof(long long),
                host.data() + (at.leaf - at.host));
    std::copy_n((const unsigned char*)trig.data(), trig.size() * sizeof(double2),
                host.data() + (at.trig - at.host));
    std::copy_n((const unsigned char*)level.data(), level.size() * sizeof(int2),
                host.data() + (at.lev - at.host));
    const cudaStream_t st = b.stream;
    IFGF_CUDA(cudaMemcpyAsync(m + at.host, host.data(), host.size(), cudaMemcpyHostToDevice, st));
    int* pos = (int*)(m + at.pos);
    int* tgt = (int*)(m + at.tgt);
    int* tile = (int*)(m + at.tile);
    int2* meta = (int2*)(m + at.meta);
    const long long* leaf_off = (const long long*)(m + at.leaf);
    int* count = (int*)(m + at.val);
    int* off = (int*)(m + at.val + at.count_b);
    size_t scan_b = at.scan_b;
    IFGF_CUDA(cudaMemsetAsync(count, 0, (n_fine + 1) * sizeof(int), st));
    IFGF_CUDA(cudaMemsetAsync(tgt, 0xff, at.meta - at.tgt, st)); // and the tiles
    lookup_kernel<<<1, 32, 0, st>>>(b.lv_dev, L, (LookupF*)(m + at.lookup));
    for (int l = 0; l < L; l++)
        if (lv[l].n_fine > 0)
            meta_kernel<<<blocks_for(lv[l].n_fine), 256, 0, st>>>(b.cone_box[l], b.cone_el[l],
                                                                  (int)lv[l].n_fine,
                                                                  meta + lv[l].fine_off);
    const auto count_pairs = b.mixed ? count_kernel<true> : count_kernel<false>;
    count_pairs<<<nl, THREADS, 0, st>>>(b.lv_dev, b.T, b.tx, b.ty, b.tz, b.fmap, b.tl_first,
                                        b.tl_last, b.far_off, b.far_src, leaf_off, pos, count,
                                        b.err, L);
    pad_kernel<<<blocks_for(n_fine), 256, 0, st>>>(count, (int)n_fine);
    IFGF_CUDA(cub::DeviceScan::ExclusiveSum(m + at.val + 2 * at.count_b, scan_b, count, off,
                                            (int)n_fine + 1, st));
    tile_kernel<<<blocks_for(n_fine), 256, 0, st>>>(off, (int)n_fine, tile);
    // every cone's entry of off becomes its cursor; the last one stays
    place_kernel<<<nl, THREADS, 0, st>>>(b.tl_first, b.tl_last, b.far_off, leaf_off, pos, off,
                                         tgt);
    IFGF_CUDA(cudaGetLastError());
    int used = 0;
    IFGF_CUDA(cudaMemcpyAsync(&used, off + n_fine, sizeof(int), cudaMemcpyDeviceToHost, st));
    IFGF_CUDA(cudaStreamSynchronize(st));
    if (used == 0) // every pair outside its box's domain
    {
        plan.release();
        plan.refused = true;
        return;
    }
    plan.pairs = at.pairs;
    plan.places = ((long long)used + 31) / 32 * 32;
    plan.p = FarConePtrs{tile,
                         plan.places / 32,
                         tgt,
                         meta,
                         (const int2*)(m + at.lev),
                         (const double2*)(m + at.trig),
                         pos,
                         leaf_off,
                         m + at.val,
                         (const LookupF*)(m + at.lookup)};
    plan.ready = true;
    plan.ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - start)
                  .count();
}

// One CTA per target leaf: thread (ti, si) adds the values of target ti over
// far boxes si, si + S, ... (S = threads / targets); the S sums and the near
// sum are added in a fixed order and written in the caller's order.  Bound
// by memory (20 bytes a pair, mixed 12); with one value in flight per thread
// the FP64 far field at N = 1e6 took 17.9 ms, with eight 17.3.
template <typename V>
__global__ void __launch_bounds__(THREADS)
    far_gather_kernel(FarConePtrs fc, const int* __restrict__ tl_first,
                      const int* __restrict__ tl_last, const long long* __restrict__ far_off,
                      const double2* __restrict__ unear, const long long* __restrict__ tgt_perm,
                      double* out, int real_out)
{
    __shared__ double2 part[THREADS];
    const int tl = blockIdx.x;
    const int t0 = tl_first[tl], all = tl_last[tl] - t0;
    const int nbox = (int)(far_off[tl + 1] - far_off[tl]);
    for (int base = 0; base < all; base += THREADS)
    {
        const int cnt = min(THREADS, all - base);
        const int S = THREADS / cnt;
        const int ti = threadIdx.x % cnt, si = threadIdx.x / cnt;
        double2 acc = make_double2(0.0, 0.0);
        if (si < S)
        {
            const int* pos = fc.pos + fc.leaf_off[tl] + base + ti;
            // eight places, then their values, in flight together
            constexpr int U = 8;
            for (int e = si; e < nbox; e += U * S)
            {
                int at[U];
                V v[U];
#pragma unroll
                for (int k = 0; k < U; k++)
                    at[k] = e + k * S < nbox ? pos[(long long)(e + k * S) * all] : -1;
#pragma unroll
                for (int k = 0; k < U; k++)
                    v[k] = at[k] >= 0 ? static_cast<const V*>(fc.val)[at[k]] : V{0, 0};
#pragma unroll
                for (int k = 0; k < U; k++)
                {
                    acc.x += (double)v[k].x;
                    acc.y += (double)v[k].y;
                }
            }
        }
        __syncthreads(); // the previous chunk's sums are no longer read
        part[threadIdx.x] = acc;
        __syncthreads();
        if (si == 0)
        {
            for (int s = 1; s < S; s++)
            {
                acc.x += part[ti + s * cnt].x;
                acc.y += part[ti + s * cnt].y;
            }
            const double2 nr = unear[t0 + base + ti];
            acc.x += nr.x;
            acc.y += nr.y;
            const long long o = tgt_perm[t0 + base + ti];
            if (real_out)
                out[o] = acc.x;
            else
                reinterpret_cast<double2*>(out)[o] = acc;
        }
    }
}

void launch_far_gather(const MultPtrs& m, const FarConePtrs& fc, void* d_u, bool real,
                       cudaStream_t st)
{
    const auto kern = m.mixed ? far_gather_kernel<float2> : far_gather_kernel<double2>;
    kern<<<m.n_tleaf, THREADS, 0, st>>>(fc, m.tl_first, m.tl_last, m.tl_far_off, m.unear,
                                        m.tgt_perm, (double*)d_u, real ? 1 : 0);
}

} // namespace ifgf
