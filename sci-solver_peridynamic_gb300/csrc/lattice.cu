// lattice.cu -- the system product A w for bodies filled on a lattice
// (mixed precision).
//
// The reference fills every body on a simple-cubic lattice of spacing 2 r
// (src/examples/scene.cpp:33-135) and bonds each particle to the others within
// the horizon (src/core/kdtree.h:304-353); its product computeAx
// (src/core/cg_solver.cuh:343-383) then gathers one 3x3 block and one vector
// entry per bond.  Here, when every particle sits within 0.3 spacings of a
// distinct lattice site, each bond joins two sites whose offset lies in a
// small stencil (80 offsets for a horizon of 2.5 spacings).  The slots are
// renumbered brick by brick (bricks of 16 x 8 x 4 sites, x fastest), and the
// product runs one brick per block iteration: the halo of the brick's sites
// (each particle's entry of w and its deviation from its site) arrives in shared
// memory by two asynchronous copies, then each thread walks the stencil columns
// of two z-adjacent rows, so that a neighbour read from shared memory serves
// both rows whose stencil it is in.  Threads take x-consecutive pairs, so the
// neighbours at one stencil entry are x-consecutive shared-memory words, and the
// only per-bond stream is 1/d0 per (row, stencil entry), 0 where there is no
// live bond (stored scaled by 2^100, see kLatScale).
//
// The per-bond arithmetic is the gather product's (step_rows.cuh,
// mixed_bond_chunk): the Jacobian applied to w_p - w_q is
//   c [ (1/d0 - 1/d) (w_p - w_q) + (xi . (w_p - w_q)) xi / d^3 ],
// with the bond vector xi = d_q - (d_p - h v_k) from the stencil offset v_k
// and the two deviations d from the lattice sites (per step, FP64 rounded
// once to FP32 within half a supercell), in pairs of FP32 lanes (f32x2).
#include <algorithm>
#include <climits>
#include <cmath>
#include <vector>

#include "step_rows.cuh"

namespace pdgb {

namespace {

#define LT_TRY(x)                              \
    do {                                       \
        cudaError_t e_ = (x);                  \
        if (e_ != cudaSuccess) return e_;      \
    } while (0)

// Bricks of 16 x 8 x 4 sites (8 x 8 x 4 for a reach of 3 sites), a thread per
// pair of z-adjacent rows, a warp per chunk of 32 pairs.  Runs of 8 pairs in x
// keep every 8 lanes of a 16-byte shared-memory access consecutive.
constexpr int kLatBY = 8;
constexpr int kLatBZ = 4;
constexpr int kLatRZ = 2;             // rows of a thread
__host__ __device__ constexpr int lat_bx(int R) { return R <= 2 ? 16 : 8; }
constexpr int kLatMaxPairs = 16 * kLatBY * (kLatBZ / kLatRZ);   // of a brick
__host__ __device__ constexpr int lat_warps(int R) { return lat_bx(R) * kLatBY * (kLatBZ / kLatRZ) / 32; }
// the table of a chunk comes in slabs of whole stencil columns: so many of each
// reach, at most kLatSlab entries (of 256 bytes)
constexpr int kLatSlab = 12;
__host__ __device__ constexpr int lat_slab_columns(int RC) { return RC >= 2 ? kLatSlab / (2 * RC + 1) : 4; }
// The table holds 2^100 / d0: then min(1/d, entry) is 1/d for a live bond (its
// entry is near 1e31 or more) and 0 for "no bond" (entry 0), one instruction,
// and 1/d0 - 1/d = fma(entry, 2^-100, -1/d) is exact scaling by a power of two.
constexpr float kLatScale = 1.2676506002282294e30f;     // 2^100
constexpr float kLatUnscale = 7.888609052210118e-31f;   // 2^-100
__host__ __device__ constexpr int lat_halo_sites(int R)
{
    return (lat_bx(R) + 2 * R) * (kLatBY + 2 * R) * (kLatBZ + 2 * R);
}
// shared memory: barriers, the halo (a box of the direction, float4 per site,
// then the deviations as they lie in the image: x, y pairs, then z), and two
// slabs of the table per warp
__host__ __device__ constexpr int lat_image_bytes(int R) { return 12 * lat_halo_sites(R); }
__host__ __device__ constexpr int lat_halo_bytes(int R) { return (28 * lat_halo_sites(R) + 127) / 128 * 128; }
constexpr int kLatBarrierBytes = 256;
constexpr int kLatSlabBytes = kLatSlab * 32 * (int)sizeof(float2);
__host__ __device__ constexpr int lat_smem(int R)
{
    return kLatBarrierBytes + lat_halo_bytes(R) + 2 * lat_warps(R) * kLatSlabBytes;
}

// 1/sqrt(x) by the hardware approximation without a denormal path: a live
// bond's d^2 is far above the FP32 denormal range, and an empty or padding
// entry (d^2 = 0 -> +inf) is masked to 0 by its caller.  The file is built
// without flush-to-zero: the CG dot products of small right-hand sides
// (1e-20 entries, products near 1e-40) must keep their denormal terms.
__device__ __forceinline__ float rsqrt_ftz(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

int blocks_for(long long n) { return (int)std::max<long long>(1, std::min<long long>((n + kBlock - 1) / kBlock, 8192)); }

// ---- detection ------------------------------------------------------------------------
// site = rint((X - anchor) / h) per axis; ext[0..2] = min, ext[3..5] = max,
// ext[6] != 0 when some coordinate lies more than 0.3 h from its site
__global__ void __launch_bounds__(kBlock) k_lat_sites(const dbl4* __restrict__ x, int n, double ax, double ay,
                                                      double az, double inv_h, int4* __restrict__ site,
                                                      int* __restrict__ ext)
{
    int mn[3] = {INT_MAX, INT_MAX, INT_MAX}, mx[3] = {INT_MIN, INT_MIN, INT_MIN};
    int fail = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const dbl4 p = x[i];
        const double f[3] = {(p.x - ax) * inv_h, (p.y - ay) * inv_h, (p.z - az) * inv_h};
        int s[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double r = rint(f[k]);
            if (!(fabs(f[k] - r) <= 0.3) || !(fabs(r) < 1.0e8)) {
                fail = 1;
                s[k] = 0;
            } else {
                s[k] = (int)r;
            }
            mn[k] = min(mn[k], s[k]);
            mx[k] = max(mx[k], s[k]);
        }
        site[i] = make_int4(s[0], s[1], s[2], 0);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        mn[k] = __reduce_min_sync(0xffffffffu, mn[k]);
        mx[k] = __reduce_max_sync(0xffffffffu, mx[k]);
    }
    fail = __reduce_or_sync(0xffffffffu, fail);
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            atomicMin(&ext[k], mn[k]);
            atomicMax(&ext[3 + k], mx[k]);
        }
        if (fail) atomicOr(&ext[6], 1);
    }
}

// every live bond's site offset marked in the kLatTab^3 table (fail[0] set
// when an offset exceeds kLatRmax on some axis)
__global__ void __launch_bounds__(kBlock) k_lat_offsets(int n, const int4* __restrict__ site,
                                                        const int* __restrict__ row_ptr, const int* __restrict__ cnt,
                                                        const int* __restrict__ col, int* __restrict__ tab,
                                                        int* __restrict__ fail)
{
    __shared__ int stab[kLatTab * kLatTab * kLatTab];
    for (int i = threadIdx.x; i < kLatTab * kLatTab * kLatTab; i += blockDim.x) stab[i] = 0;
    __syncthreads();
    int bad = 0;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const int4 sp = site[p];
        const int rs = row_ptr[p], cn = cnt[p];
        for (int j = 0; j < cn; ++j) {
            const int4 sq = site[col[rs + j]];
            const int dx = sq.x - sp.x, dy = sq.y - sp.y, dz = sq.z - sp.z;
            if (abs(dx) > kLatRmax || abs(dy) > kLatRmax || abs(dz) > kLatRmax) {
                bad = 1;
                continue;
            }
            stab[((dz + kLatRmax) * kLatTab + (dy + kLatRmax)) * kLatTab + (dx + kLatRmax)] = 1;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kLatTab * kLatTab * kLatTab; i += blockDim.x)
        if (stab[i]) atomicOr(&tab[i], 1);
    if (bad) atomicOr(fail, 1);
}

// *fail set when a bond of a row, live or restorable (cnt_bk), is no entry of the stencil
__global__ void __launch_bounds__(kBlock) k_lat_holds(DeviceState S, const __grid_constant__ LatticeParams lp,
                                                      int* __restrict__ fail)
{
    int bad = 0;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < S.n; p += gridDim.x * blockDim.x) {
        const int4 sp = lp.site[p];
        const int rs = S.row_ptr[p], cn = max(S.cnt[p], S.cnt_bk[p]);
        for (int j = 0; j < cn; ++j) {
            const int4 sq = lp.site[S.col[rs + j]];
            const int dx = sq.x - sp.x, dy = sq.y - sp.y, dz = sq.z - sp.z;
            if (abs(dx) > kLatRmax || abs(dy) > kLatRmax || abs(dz) > kLatRmax ||
                lp.offk[((dz + kLatRmax) * kLatTab + (dy + kLatRmax)) * kLatTab + (dx + kLatRmax)] < 0)
                bad = 1;
        }
    }
    if (bad) atomicOr(fail, 1);
}

// shifted sites and the brick-major sort key of every slot
__global__ void __launch_bounds__(kBlock) k_lat_keys(int n, int4* __restrict__ site, int3 lo, int bx, int3 nb,
                                                     unsigned* __restrict__ key, int* __restrict__ val)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int4 s = site[i];
        s.x -= lo.x;
        s.y -= lo.y;
        s.z -= lo.z;
        site[i] = s;
        const unsigned brick = ((unsigned)(s.z / kLatBZ) * (unsigned)nb.y + (unsigned)(s.y / kLatBY)) * (unsigned)nb.x +
                               (unsigned)(s.x / bx);
        const unsigned local = ((unsigned)(s.z % kLatBZ) * kLatBY + (unsigned)(s.y % kLatBY)) * (unsigned)bx +
                               (unsigned)(s.x % bx);
        key[i] = brick * (unsigned)(bx * kLatBY * kLatBZ) + local;
        val[i] = i;
    }
}

__global__ void k_lat_dups(const unsigned* __restrict__ key, int n, int* __restrict__ fail)
{
    for (int i = 1 + blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (key[i] == key[i - 1]) atomicOr(fail, 1);
}

// ---- renumbering (new slot i holds old slot n2o[i]) -------------------------------------
template <typename T>
__global__ void k_lat_gather(const T* __restrict__ in, const int* __restrict__ n2o, T* __restrict__ out, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = in[n2o[i]];
}

__global__ void k_lat_inverse(const int* __restrict__ n2o, int* __restrict__ o2n, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) o2n[n2o[i]] = i;
}

__global__ void k_lat_lengths(const int* __restrict__ row_ptr, const int* __restrict__ n2o, unsigned* __restrict__ len,
                              int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int o = n2o[i];
        len[i] = (unsigned)(row_ptr[o + 1] - row_ptr[o]);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) len[n] = 0u;
}

__global__ void k_lat_remap_col(const int* __restrict__ row_ptr_old, const int* __restrict__ col_old,
                                const unsigned* __restrict__ row_ptr_new, const int* __restrict__ n2o,
                                const int* __restrict__ o2n, int* __restrict__ col_new, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int o = n2o[i];
        const int a = row_ptr_old[o], len = row_ptr_old[o + 1] - a;
        const int b = (int)row_ptr_new[i];
        for (int j = 0; j < len; ++j) col_new[b + j] = o2n[col_old[a + j]];
    }
}

__global__ void __launch_bounds__(kBlock) k_lat_dense(const int4* __restrict__ site, int n, int R, int mx, int my,
                                                      int* __restrict__ dense)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int4 s = site[i];
        dense[i] = (int)(((long long)(s.z + R) * my + (s.y + R)) * mx + (s.x + R));
    }
}

// ---- 1/d0 table ------------------------------------------------------------------------
// [chunk][entry][32 pairs] words of a pair's two rows.
__global__ void __launch_bounds__(kBlock) k_lat_ell(DeviceState S, const __grid_constant__ LatticeParams lp, int force)
{
    if (!force && ((volatile int*)S.flags)[1] == 0) return;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < S.n; p += gridDim.x * blockDim.x) {
        const int rp = lp.row_pair[p];   // 64 chunk + 2 lane + row
        float* e = lp.ell + (size_t)(rp >> 6) * lp.K * 64 + (rp & 63);
        for (int k = 0; k < lp.K; ++k) e[k * 64] = 0.f;
        const int4 sp = lp.site[p];
        const int rs = S.row_ptr[p], cn = S.cnt[p];
        for (int j = 0; j < cn; ++j) {
            const int4 sq = lp.site[S.col[rs + j]];
            const int t = ((sq.z - sp.z + kLatRmax) * kLatTab + (sq.y - sp.y + kLatRmax)) * kLatTab +
                          (sq.x - sp.x + kLatRmax);
            e[lp.offk[t] * 64] = S.inv_d0[rs + j] * kLatScale;
        }
    }
}

// ---- deviations from the lattice sites ------------------------------------------------
// grid_d[site of i] = (d, n): x - (org + h site) = d + sup n per axis with n =
// rint(. / sup) (FP64, exact: sup is a power of two), d rounded once to FP32;
// n packed in 10 bits per axis (+512).  |n| stays below 512 for displacements
// below 500 supercells; larger ones are clamped (the deviation then loses
// digits).  (Sites without a particle keep 0: their table entries are 0, so any
// finite deviation does.)
__global__ void __launch_bounds__(kBlock) k_lat_delta(const dbl4* __restrict__ x64, int n,
                                                      const __grid_constant__ LatticeParams lp, double sup)
{
    const double inv_sup = 1.0 / sup;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const dbl4 x = x64[i];
        const int4 s = lp.site[i];
        const double dev[3] = {x.x - (lp.org[0] + lp.h * s.x), x.y - (lp.org[1] + lp.h * s.y),
                               x.z - (lp.org[2] + lp.h * s.z)};
        float d[3];
        int packed = 0;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double m = fmin(fmax(rint(dev[k] * inv_sup), -511.0), 511.0);
            d[k] = (float)(dev[k] - m * sup);
            packed |= ((int)m + 512) << (10 * k);
        }
        lp.grid_d[lp.dense[i]] = make_float4(d[0], d[1], d[2], __int_as_float(packed));
    }
}

// The deviations of every brick's halo as the product copies them into shared
// memory, once per step (every product of a solve reads them): re-referenced
// to the brick, d + sup (n - n_brick) with n_brick the wrap counts of the
// brick's first slot (within a brick's halo they differ by at most one for any
// strain a bond survives, so |d| stays within 1.5 sup).  12 bytes per halo site
// in two runs cost the product less than a box of grid_d (16 bytes per site in
// shared memory and its reads): 134 against 143 us at 1M particles.
__device__ __forceinline__ float wrap_delta(int nq, int nb, int shift, float sup)
{
    return sup * small_int_to_float(((nq >> shift) & 1023) - ((nb >> shift) & 1023));
}

template <int R>
__global__ void __launch_bounds__(kBlock) k_lat_image(const __grid_constant__ LatticeParams lp, float sup)
{
    constexpr int HX = lat_bx(R) + 2 * R, HY = kLatBY + 2 * R, HXY = HX * HY, H = lat_halo_sites(R);
    const int mx = lp.map_dim[0], mxy = lp.map_dim[0] * lp.map_dim[1];
    for (int b = blockIdx.x; b < lp.n_bricks; b += gridDim.x) {
        const int corner = lp.brick_corner[b];
        const int nb = __float_as_int(lp.grid_d[lp.dense[lp.brick_start[b]]].w);
        float2* xy = (float2*)(lp.image + (size_t)b * 3 * H);
        float* z = (float*)(xy + H);
        for (int h = threadIdx.x; h < H; h += kBlock) {
            const int iz = h / HXY;
            const int r2 = h - iz * HXY;
            const int iy = r2 / HX;
            const float4 d = lp.grid_d[corner + iz * mxy + iy * mx + (r2 - iy * HX)];
            const int nq = __float_as_int(d.w);
            xy[h] = make_float2(d.x + wrap_delta(nq, nb, 0, sup), d.y + wrap_delta(nq, nb, 10, sup));
            z[h] = d.z + wrap_delta(nq, nb, 20, sup);
        }
    }
}

// ---- the direction on the dense grid of sites --------------------------------------------
// The product reads its vector from a dense grid of the map's extent (lp.grid_w,
// zero where there is no particle), so that a brick's halo is one box.
__global__ void __launch_bounds__(kBlock) k_lat_scatter(int n, const int* __restrict__ dense, float4* __restrict__ grid_w,
                                                        const float4* __restrict__ in)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 v = in[i];
        grid_w[dense[i]] = make_float4(v.x, v.y, v.z, 0.f);
    }
}

// p = r + beta p (xpby_elem), in slot order and on the grid
__global__ void __launch_bounds__(kBlock) k_lat_xpby(int n, const int* __restrict__ dense, float4* __restrict__ grid_w,
                                                     const CgScalars* sc, const float4* __restrict__ r,
                                                     float4* __restrict__ p)
{
    if (((volatile const CgScalars*)sc)->done) return;
    const float beta = (float)sc->beta;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 ri = r[i], pi = p[i];
        const float4 q = make_float4(ri.x + beta * pi.x, ri.y + beta * pi.y, ri.z + beta * pi.z, 0.f);
        p[i] = q;
        grid_w[dense[i]] = q;
    }
}

// ---- the product -----------------------------------------------------------------------
// Blocks take bricks from a counter (lp.sched[0]) in brick order, a warp per
// chunk of 32 row pairs.  Everything the computation reads comes by bulk
// copies: the halo of a brick (a box of the direction's grid, the deviations as
// one run of the image) once the block is done with the brick before, and each
// warp's table in slabs, two ahead and across bricks, so that some 70 KB per SM are
// in flight at any time -- at a DRAM latency of 1 us (2.5 us under a full stream)
// loads into registers cannot hold that many: with one stencil column (40 bytes a
// thread) loaded ahead the product took 150 us at 1M particles however few
// instructions it had, 105 us without the table.
// Entry k's bond vector is xi = d_q - (d_p - h v_k), formed in FP32 with the
// differences of w; h v_k is exact.  The order of the columns, farthest first, is
// that of their terms' size, smallest first: a row's sums stay small for longer,
// and so do their roundings, which are most of the product's error (80 entries:
// 2.96e-8 of the largest value, root mean square; 3.10e-8 in the order z, y, x of
// the offsets, 3.26e-8 with the largest columns first).
// Every wait is bounded (lp.wait_ns, a second): on expiry the block records the
// error in the handle's scalars and ends the solve there, waits once more for every
// copy of its own still in flight (a second at most, whatever the limit) and
// returns; later products of the handle take no bricks.

__device__ __forceinline__ unsigned long long lat_now_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity)
{
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}
// A lane's own answer: lanes of a warp may differ, so none of them leaves its
// path for it (a vote of the warp per wait: 123 against 115 us at 1M particles).
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, unsigned long long limit)
{
    if (bar_try(bar, parity)) return true;
    const unsigned long long t0 = lat_now_ns();
    while (!bar_try(bar, parity))
        if (lat_now_ns() - t0 > limit) return false;
    return true;
}

// The rows of a thread: their sites' words and the sums of a1 (w_q - w_p) + g xi
// with g = xi . (w_q - w_p) / d^3 (the row's term with the sign of w_q - w_p,
// negated at the end).
struct LatRows {
    float2 d[kLatRZ], w[kLatRZ];   // (d.x, d.y), (w.x, w.y)
    float dz[kLatRZ], wz[kLatRZ];
    float2 sxy[kLatRZ];
    float sz[kLatRZ];
};
struct LatHalo {
    const float4* w;
    const float2* xy;
    const float* z;
};

// The stencil's column (dx, dy) of reach RC: entries dz = -RC .. RC of the
// thread's rows, e[dz + RC] one word each.  Every site of the column is read
// once and serves the rows it is a neighbour of.
// q: shared-memory index of the site (dx, dy) from the thread's lowest row.
template <int R, int RC>
__device__ __forceinline__ void lat_column(const LatHalo& halo, int q, const float2 (&e)[2 * RC + 1], float2 cxy,
                                           const float (&cz)[kLatTab], LatRows& row)
{
    constexpr int HXY = (lat_bx(R) + 2 * R) * (kLatBY + 2 * R);
    const float2 m1 = make_float2(-1.f, -1.f);
    float2 pxy[kLatRZ];
#pragma unroll
    for (int i = 0; i < kLatRZ; ++i) pxy[i] = __ffma2_rn(cxy, m1, row.d[i]);   // d_p - h v
#pragma unroll
    for (int j = -RC; j < kLatRZ + RC; ++j) {
        const float4 qw4 = halo.w[q + j * HXY];
        const float2 qd = halo.xy[q + j * HXY];
        const float qz = halo.z[q + j * HXY];
        const float2 qw = make_float2(qw4.x, qw4.y);
#pragma unroll
        for (int i = 0; i < kLatRZ; ++i) {
            const int dz = j - i;
            if (dz < -RC || dz > RC) continue;
            const float s = i == 0 ? e[dz + RC].x : e[dz + RC].y;
            const float2 xy = __ffma2_rn(pxy[i], m1, qd);      // d_q - (d_p - h v)
            const float2 wxy = __ffma2_rn(row.w[i], m1, qw);   // w_q - w_p
            const float zs = qz - (row.dz[i] - cz[dz + kLatRmax]);
            const float wz = qw4.z - row.wz[i];
            float inv_d = rsqrt_ftz(fmaf(xy.x, xy.x, fmaf(xy.y, xy.y, zs * zs)));
            inv_d = fminf(inv_d, s);   // no live bond (s = 0): the term vanishes
            const float a1 = fmaf(s, kLatUnscale, -inv_d);
            const float g = fmaf(xy.x, wxy.x, fmaf(xy.y, wxy.y, zs * wz)) * (inv_d * inv_d * inv_d);
            row.sxy[i] = __ffma2_rn(make_float2(a1, a1), wxy, __ffma2_rn(make_float2(g, g), xy, row.sxy[i]));
            row.sz[i] = fmaf(a1, wz, fmaf(g, zs, row.sz[i]));
        }
    }
}

// bulk copy of `bytes` from global memory to shared memory, completing on `bar`,
// with the table's lines first to leave L2
__device__ __forceinline__ void copy_slab(uint32_t dst, const void* src, int bytes, uint32_t bar, uint64_t policy)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(dst),
        "l"((uint64_t)src), "r"(bytes), "r"(bar), "l"(policy)
        : "memory");
}

// One warp's stream of slabs: the chunk's, in the order of lp.slab_entry, then
// those of the chunk it will take from the next brick.
struct LatStream {
    uint32_t ring, bars;    // the warp's two slabs and their barriers (shared-memory addresses)
    uint64_t policy;
    int issued = 0, used = 0;
};
__device__ __forceinline__ void lat_issue(LatStream& s, const LatticeParams& lp, int chunk, int slab)
{
    const int slot = s.issued & 1;
    const int e0 = lp.slab_entry[slab], e1 = lp.slab_entry[slab + 1];
    copy_slab(s.ring + slot * kLatSlabBytes, (const float2*)lp.ell + ((size_t)chunk * lp.K + e0) * 32, (e1 - e0) * 256,
              s.bars + 8 * slot, s.policy);
    ++s.issued;
}

// The stencil's columns of reach RC, the first one c, slab by slab; after a slab
// the one two further on is asked for, of the next chunk at the end.  Once a wait
// has run out (ok) a lane asks for nothing more; the waits that it still makes until
// the block's vote, one per slab, are bounded like the first.
template <int R, int RC>
__device__ __forceinline__ void lat_columns(const LatticeParams& lp, const LatHalo& halo, int base, const float2* ring,
                                            LatStream& s, int chunk, int next, int& slab, int& c, int count,
                                            const float (&cz)[kLatTab], LatRows& row, bool& ok)
{
    constexpr int N = 2 * RC + 1, M = lat_slab_columns(RC);
    const int lane = threadIdx.x & 31;
    for (; count > 0; count -= M) {
        const int slot = s.used & 1;
        ok &= bar_wait(s.bars + 8 * slot, (s.used >> 1) & 1, lp.wait_ns);
        ++s.used;
        const float2* e2 = ring + slot * (kLatSlabBytes / (int)sizeof(float2)) + lane;
#pragma unroll 1
        for (int m = 0; m < min(M, count); ++m, ++c, e2 += N * 32) {
            float2 e[N];
#pragma unroll
            for (int k = 0; k < N; ++k) e[k] = e2[k * 32];
            lat_column<R, RC>(halo, base + lp.coff[c], e, make_float2(lp.ccx[c], lp.ccy[c]), cz, row);
        }
        __syncwarp();   // every lane is done with the slab
        const int ahead = ++slab + 1;
        if (lane == 0 && ok) {
            if (ahead < lp.slabs) lat_issue(s, lp, chunk, ahead);
            else if (next >= 0) lat_issue(s, lp, next, ahead - lp.slabs);
        }
    }
}

// At most 112 registers, which leaves an SM room for a 256-thread block of a vector
// kernel beside two of these: with 115, three bodies of 1M particles that each make
// four products on a stream of their own took 480 us a body, 461 with 109.
template <int R, bool DOT>
__global__ void __maxnreg__(R <= 2 ? 112 : 128)
    k_spmv_lattice(StepParams P, DeviceState S, const __grid_constant__ LatticeParams lp, float4* __restrict__ out,
                   ReduceSlot slot, CgScalars* cg, double* dot_out)
{
    if (DOT && cg && ((volatile CgScalars*)cg)->done) return;
    constexpr int HX = lat_bx(R) + 2 * R, HY = kLatBY + 2 * R, HXY = HX * HY, H = lat_halo_sites(R);
    extern __shared__ __align__(128) unsigned char lat_smem_raw[];
    __shared__ int s_ahead;
    const uint32_t bars = (uint32_t)__cvta_generic_to_shared(lat_smem_raw);   // the halo's, then two per warp
    const unsigned char* stage = lat_smem_raw + kLatBarrierBytes;
    const LatHalo halo{(const float4*)stage, (const float2*)(stage + 16 * H), (const float*)(stage + 24 * H)};
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned char* ring = stage + lat_halo_bytes(R) + warp * 2 * kLatSlabBytes;
    LatStream s;
    s.ring = (uint32_t)__cvta_generic_to_shared(ring);
    s.bars = bars + 8 + 16 * warp;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(s.policy));
    const auto load_halo = [&](int b) {   // thread 0
        const int corner = lp.brick_corner[b];
        const int mx = lp.map_dim[0], my = lp.map_dim[1];
        const int cx = corner % mx, cy = corner / mx % my, cz = corner / mx / my;
        const uint32_t dst = bars + kLatBarrierBytes;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bars), "r"(28 * H) : "memory");
        asm volatile(
            "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
            "[%6];" ::"r"(dst),
            "l"((uint64_t)&lp.box_w), "r"(0), "r"(cx), "r"(cy), "r"(cz), "r"(bars)
            : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst + 16 * H),
                     "l"((uint64_t)(lp.image + (size_t)b * 3 * H)), "r"(lat_image_bytes(R)), "r"(bars)
                     : "memory");
    };
    // this warp's chunk of a brick, or -1
    const auto chunk_of = [&](int b) {
        if (b >= lp.n_bricks) return -1;
        const int c = __ldg(lp.chunk_start + b) + warp;
        return c < __ldg(lp.chunk_start + b + 1) ? c : -1;
    };
    int b = 0;
    if (threadIdx.x == 0) {
        for (int k = 0; k < 1 + 2 * lat_warps(R); ++k) bar_init(bars + 8 * k, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        b = (int)atomicAdd(&lp.sched[0], 1u);
        // (no bricks once a wait of the handle has run out; in a solve `done` says so)
        if (!(DOT && cg) && ((volatile CgScalars*)S.sc)->wait_error) b = lp.n_bricks;
        s_ahead = b;
    }
    __syncthreads();
    b = s_ahead;
    __syncthreads();
    if (threadIdx.x == 0 && b < lp.n_bricks) {
        s_ahead = (int)atomicAdd(&lp.sched[0], 1u);
        load_halo(b);
    }
    int chunk = chunk_of(b);
    if (lane == 0 && chunk >= 0)
        for (int k = 0; k < min(2, lp.slabs); ++k) lat_issue(s, lp, chunk, k);
    // the chunk's row pair of this lane, read a brick ahead: the halo index of
    // the lower site and the slots (139 -> 134 us at 1M particles)
    int base_n = 0;
    int2 slots_n = make_int2(-1, -1);
    if (chunk >= 0) {
        base_n = __ldg(lp.pair_base + chunk * 32 + lane);
        slots_n = __ldg((const int2*)lp.pair_slot + chunk * 32 + lane);
    }
    DotAcc32 acc;
    bool ok = true;
    const float c0 = (float)P.bond_coeff, t2 = (float)P.t2, m = (float)P.mass;
    float cz[kLatTab];
#pragma unroll
    for (int k = 0; k < kLatTab; ++k) cz[k] = lp.cz[k];
    int it = 0;   // bricks taken
    ok = lp.wait_ns != 0 || b >= lp.n_bricks;
    while (ok && b < lp.n_bricks) {
        ok = bar_wait(bars, it & 1, lp.wait_ns);
        const int ahead = *(volatile int*)&s_ahead;   // the next brick
        const int next = chunk_of(ahead);
        if (chunk >= 0) {
            const int base = base_n;
            const int2 slots = slots_n;
            const uint8_t ab2[2] = {slots.x >= 0 ? S.act[slots.x] : (uint8_t)0, slots.y >= 0 ? S.act[slots.y] : (uint8_t)0};
            if (next >= 0) {
                base_n = __ldg(lp.pair_base + next * 32 + lane);
                slots_n = __ldg((const int2*)lp.pair_slot + next * 32 + lane);
            }
            LatRows row;
#pragma unroll
            for (int i = 0; i < kLatRZ; ++i) {
                const float4 w = halo.w[base + i * HXY];
                row.d[i] = halo.xy[base + i * HXY];
                row.dz[i] = halo.z[base + i * HXY];
                row.w[i] = make_float2(w.x, w.y);
                row.wz[i] = w.z;
                row.sxy[i] = make_float2(0.f, 0.f);
                row.sz[i] = 0.f;
            }
            const float2* ring2 = (const float2*)ring;
            int c = 0, slab = 0;
            lat_columns<R, 0>(lp, halo, base, ring2, s, chunk, next, slab, c, lp.ncol[0], cz, row, ok);
            lat_columns<R, 1>(lp, halo, base, ring2, s, chunk, next, slab, c, lp.ncol[1], cz, row, ok);
            if constexpr (R >= 2) lat_columns<R, 2>(lp, halo, base, ring2, s, chunk, next, slab, c, lp.ncol[2], cz, row, ok);
            if constexpr (R >= 3) lat_columns<R, 3>(lp, halo, base, ring2, s, chunk, next, slab, c, lp.ncol[3], cz, row, ok);
#pragma unroll
            for (int i = 0; i < kLatRZ; ++i) {
                const int p = i == 0 ? slots.x : slots.y;
                if (p < 0) continue;
                const uint8_t ab = ab2[i];
                if (is_dirichlet(ab & kActMask))
                    out[p] = make_float4(0.f, 0.f, 0.f, 0.f);
                else
                    mixed_row_result<DOT>(P, S, p, ab, c0, t2, m, make_float4(row.w[i].x, row.w[i].y, row.wz[i], 0.f),
                                          -row.sxy[i].x, -row.sxy[i].y, -row.sz[i], out, acc);
            }
        } else if (next >= 0) {
            if (lane == 0 && ok)
                for (int k = 0; k < min(2, lp.slabs); ++k) lat_issue(s, lp, next, k);
            base_n = __ldg(lp.pair_base + next * 32 + lane);
            slots_n = __ldg((const int2*)lp.pair_slot + next * 32 + lane);
        }
        if (__syncthreads_or(ok ? 0 : 1)) {   // the block is done with the halo, or gave up
            ok = false;
            break;
        }
        b = ahead;
        chunk = next;
        ++it;
        if (threadIdx.x == 0 && b < lp.n_bricks) {
            s_ahead = (int)atomicAdd(&lp.sched[0], 1u);
            load_halo(b);
        }
    }
    if (!ok) {   // record it, end the solve, and wait once more for the copies in flight
        ((volatile CgScalars*)S.sc)->wait_error = 1;
        ((volatile CgScalars*)S.sc)->done = 1;
        bar_wait(bars, it & 1, kWaitLatticeNs);   // the halo's (its phase is over where another wait ran out)
        for (int k = max(0, s.issued - 2); k < s.issued; ++k)   // (lane 0's: the latest of each of its two slots)
            bar_wait(s.bars + 8 * (k & 1), (k >> 1) & 1, kWaitLatticeNs);
    }
    __syncthreads();
    // every block has taken its last brick index: the last to arrive resets the counter
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&lp.sched[1], 1u) == gridDim.x - 1) {
            lp.sched[0] = 0u;
            lp.sched[1] = 0u;
        }
    }
    if (DOT) {
        block_reduce_finish(acc, slot, [cg, dot_out](double pAp) {
            if (cg) cg_fin_alpha(cg, pAp);
            if (dot_out) *dot_out = pAp;
        });
    }
}

}  // namespace

cudaError_t lattice_holds(const DeviceState& S, const LatticeParams& lp, int* ok, cudaStream_t st)
{
    int *d = nullptr, fail = 0;
    LT_TRY(cudaMalloc(&d, sizeof(int)));
    cudaError_t e = cudaMemsetAsync(d, 0, sizeof(int), st);
    if (e == cudaSuccess) {
        k_lat_holds<<<blocks_for(S.n), kBlock, 0, st>>>(S, lp, d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&fail, d, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d);
    *ok = fail == 0;
    return e;
}

size_t lattice_smem_bytes(const LatticeParams& lp)
{
    return (size_t)lat_smem(lp.R);
}

void launch_lattice_delta(const DeviceState& S, const LatticeParams& lp, double sup, cudaStream_t st)
{
    if (S.n <= 0 || !lp.grid_d) return;
    k_lat_delta<<<blocks_for(S.n), kBlock, 0, st>>>(S.x64, S.n, lp, sup);
    const int grid = std::min(lp.n_bricks, 8192);
    if (lp.R == 1) k_lat_image<1><<<grid, kBlock, 0, st>>>(lp, (float)sup);
    else if (lp.R == 2) k_lat_image<2><<<grid, kBlock, 0, st>>>(lp, (float)sup);
    else k_lat_image<3><<<grid, kBlock, 0, st>>>(lp, (float)sup);
}

void launch_lattice_scatter(const DeviceState& S, const LatticeParams& lp, const void* in, cudaStream_t st)
{
    k_lat_scatter<<<blocks_for(S.n), kBlock, 0, st>>>(S.n, lp.dense, lp.grid_w, (const float4*)in);
}

void launch_lattice_xpby(const DeviceState& S, const LatticeParams& lp, const void* r, int grid, cudaStream_t st)
{
    k_lat_xpby<<<grid, kBlock, 0, st>>>(S.n, lp.dense, lp.grid_w, S.sc, (const float4*)r, (float4*)S.p);
}

template <int R>
int lattice_blocks(size_t smem)
{
    int m = 1 << 30;
    for (const void* k : {(const void*)k_spmv_lattice<R, false>, (const void*)k_spmv_lattice<R, true>}) {
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        int a = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k, 32 * lat_warps(R), smem);
        m = std::min(m, a);
    }
    return m > 0 ? m : 1;
}

int lattice_spmv_blocks_per_sm(const LatticeParams& lp)
{
    const size_t smem = lattice_smem_bytes(lp);
    return lp.R == 1 ? lattice_blocks<1>(smem) : lp.R == 2 ? lattice_blocks<2>(smem) : lattice_blocks<3>(smem);
}

template <int R>
void launch_lattice_t(bool dot, const StepParams& P, const DeviceState& S, const LatticeParams& lp, void* out,
                      ReduceSlot slot, CgScalars* cg, double* dot_out, int grid, size_t smem, cudaStream_t st)
{
    float4* y = (float4*)out;
    const int threads = 32 * lat_warps(R);
    if (dot) k_spmv_lattice<R, true><<<grid, threads, smem, st>>>(P, S, lp, y, slot, cg, dot_out);
    else k_spmv_lattice<R, false><<<grid, threads, smem, st>>>(P, S, lp, y, slot, nullptr, nullptr);
}

void launch_spmv_lattice(bool dot, const StepParams& P, const DeviceState& S, const LatticeParams& lp, void* out,
                         ReduceSlot slot, CgScalars* cg, double* dot_out, cudaStream_t st)
{
    const size_t smem = lattice_smem_bytes(lp);
    const int grid = std::max(1, std::min(lp.grid, std::max(lp.n_bricks, 1)));
    if (lp.R == 1) launch_lattice_t<1>(dot, P, S, lp, out, slot, cg, dot_out, grid, smem, st);
    else if (lp.R == 2) launch_lattice_t<2>(dot, P, S, lp, out, slot, cg, dot_out, grid, smem, st);
    else launch_lattice_t<3>(dot, P, S, lp, out, slot, cg, dot_out, grid, smem, st);
}

// the direction's grid as a TMA tensor of 4 floats per site, in boxes of a brick's halo
static cudaError_t grid_box(LatticeParams* lp)
{
    using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    const cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q);
    if (e != cudaSuccess) return e;
    if (q != cudaDriverEntryPointSuccess || !fn) return cudaErrorNotSupported;
    const int R = lp->R;
    const cuuint64_t dims[4] = {4, (cuuint64_t)lp->map_dim[0], (cuuint64_t)lp->map_dim[1], (cuuint64_t)lp->map_dim[2]};
    const cuuint64_t strides[3] = {16, 16 * dims[1], 16 * dims[1] * dims[2]};
    const cuuint32_t box[4] = {4, (cuuint32_t)(lat_bx(R) + 2 * R), (cuuint32_t)(kLatBY + 2 * R),
                               (cuuint32_t)(kLatBZ + 2 * R)};
    const cuuint32_t one[4] = {1, 1, 1, 1};
    const CUresult r = ((EncodeFn)fn)(&lp->box_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, lp->grid_w, dims, strides, box, one,
                                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                      CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

void launch_lattice_ell(const DeviceState& S, const LatticeParams& lp, int force, int grid, cudaStream_t st)
{
    k_lat_ell<<<grid, kBlock, 0, st>>>(S, lp, force);
}

void lattice_free(LatticeBuffers* lb)
{
    cudaFree(lb->brick_start);
    cudaFree(lb->brick_corner);
    cudaFree(lb->chunk_start);
    cudaFree(lb->pair_base);
    cudaFree(lb->pair_slot);
    cudaFree(lb->row_pair);
    cudaFree(lb->site);
    cudaFree(lb->offk);
    cudaFree(lb->ell);
    cudaFree(lb->dense);
    cudaFree(lb->grid_w);
    cudaFree(lb->grid_d);
    cudaFree(lb->image);
    cudaFree(lb->sched);
    *lb = LatticeBuffers{};
}

cudaError_t lattice_build(int n, double spacing, dbl4* x64, float4* X32, int* perm, int* row_ptr, int* cnt, int** col,
                          long long total_slots, LatticeParams* lp, LatticeBuffers* lb, int* ok, cudaStream_t st)
{
    *ok = 0;
    // (spacings below 1e-6 would take 2^100 / d0 out of the FP32 range)
    if (n < 1 || !(spacing > 1e-6) || total_slots >= (1LL << 31) - 64) return cudaSuccess;
    // every temporary in one owner, freed on every return path
    struct Tmp {
        int* ext = nullptr;
        int* tab = nullptr;
        unsigned* key = nullptr;
        int* n2o = nullptr;
        int* o2n = nullptr;
        unsigned* len = nullptr;
        void* buf = nullptr;
        int* col_new = nullptr;
        LatticeBuffers lb{};
        ~Tmp()
        {
            cudaFree(ext); cudaFree(tab); cudaFree(key); cudaFree(n2o); cudaFree(o2n); cudaFree(len); cudaFree(buf);
            cudaFree(col_new);
            lattice_free(&lb);
        }
    } t;
    const int G = blocks_for(n);
    LT_TRY(cudaMalloc(&t.lb.site, sizeof(int4) * (size_t)n));
    LT_TRY(cudaMalloc(&t.ext, sizeof(int) * 8));
    LT_TRY(cudaMalloc(&t.tab, sizeof(int) * kLatTab * kLatTab * kLatTab));
    int ext_init[8] = {INT_MAX, INT_MAX, INT_MAX, INT_MIN, INT_MIN, INT_MIN, 0, 0};
    LT_TRY(cudaMemcpyAsync(t.ext, ext_init, sizeof(ext_init), cudaMemcpyHostToDevice, st));
    LT_TRY(cudaMemsetAsync(t.tab, 0, sizeof(int) * kLatTab * kLatTab * kLatTab, st));
    // the lattice anchor: slot 0's position
    dbl4 anchor;
    LT_TRY(cudaMemcpyAsync(&anchor, x64, sizeof(dbl4), cudaMemcpyDeviceToHost, st));
    LT_TRY(cudaStreamSynchronize(st));
    k_lat_sites<<<G, kBlock, 0, st>>>(x64, n, anchor.x, anchor.y, anchor.z, 1.0 / spacing, t.lb.site, t.ext);
    LT_TRY(cudaGetLastError());
    int ext[8];
    LT_TRY(cudaMemcpyAsync(ext, t.ext, sizeof(ext), cudaMemcpyDeviceToHost, st));
    LT_TRY(cudaStreamSynchronize(st));
    if (ext[6]) return cudaSuccess;   // not a lattice fill
    k_lat_offsets<<<G, kBlock, 0, st>>>(n, t.lb.site, row_ptr, cnt, *col, t.tab, t.ext + 7);
    LT_TRY(cudaGetLastError());
    std::vector<int> tab(kLatTab * kLatTab * kLatTab);
    LT_TRY(cudaMemcpyAsync(tab.data(), t.tab, sizeof(int) * tab.size(), cudaMemcpyDeviceToHost, st));
    LT_TRY(cudaMemcpyAsync(ext, t.ext, sizeof(ext), cudaMemcpyDeviceToHost, st));
    LT_TRY(cudaStreamSynchronize(st));
    if (ext[7]) return cudaSuccess;   // a bond longer than the stencil reach
    // the stencil: the bonds' offsets as z columns (dx, dy), a column of reach
    // r covering dz = -r .. r (entries without a bond, the row itself among
    // them, hold 0), columns of the smallest reach first and, of one reach, the
    // farthest from the row's own (the order of their terms' size)
    LatticeParams L{};
    int R = 1, offsets = 0;
    int reach[kLatTab * kLatTab];
    for (int dy = -kLatRmax; dy <= kLatRmax; ++dy)
        for (int dx = -kLatRmax; dx <= kLatRmax; ++dx) {
            int& r = reach[(dy + kLatRmax) * kLatTab + dx + kLatRmax];
            r = -1;
            for (int dz = -kLatRmax; dz <= kLatRmax; ++dz)
                if (tab[((dz + kLatRmax) * kLatTab + (dy + kLatRmax)) * kLatTab + (dx + kLatRmax)]) {
                    r = std::max(r, std::abs(dz));
                    R = std::max(R, std::max(std::abs(dx), std::max(std::abs(dy), std::abs(dz))));
                    ++offsets;
                }
        }
    if (offsets > kLatMaxOffsets) return cudaSuccess;
    // the sites' pitch: the spacing in 21 bits, so that h v_k is exact in FP32 (the
    // deviations take up the difference, 2^-21 of a spacing per site at most)
    int exponent = 0;
    const double mantissa = std::frexp(spacing, &exponent);
    const double pitch = std::ldexp(std::rint(std::ldexp(mantissa, 21)), exponent - 21);
    L.R = R;
    const int BX = lat_bx(R), HX = BX + 2 * R, HY = kLatBY + 2 * R;
    std::vector<int> offk(tab.size(), -1);
    int cols = 0;
    std::vector<std::pair<int, int>> column;
    for (int dy = -kLatRmax; dy <= kLatRmax; ++dy)
        for (int dx = -kLatRmax; dx <= kLatRmax; ++dx)
            if (reach[(dy + kLatRmax) * kLatTab + dx + kLatRmax] >= 0) column.emplace_back(dx, dy);
    std::stable_sort(column.begin(), column.end(), [](const auto& a, const auto& b) {
        return a.first * a.first + a.second * a.second > b.first * b.first + b.second * b.second;
    });
    for (int r = 0; r <= kLatRmax; ++r)
        for (const auto& [dx, dy] : column) {
            if (reach[(dy + kLatRmax) * kLatTab + dx + kLatRmax] != r) continue;
            for (int dz = -r; dz <= r; ++dz)
                offk[((dz + kLatRmax) * kLatTab + (dy + kLatRmax)) * kLatTab + (dx + kLatRmax)] = L.K++;
            L.coff[cols] = dy * HX + dx;
            L.ccx[cols] = (float)(pitch * dx);
            L.ccy[cols] = (float)(pitch * dy);
            ++cols;
            ++L.ncol[r];
        }
    for (int k = 0; k < kLatTab; ++k) L.cz[k] = (float)(pitch * (k - kLatRmax));
    for (int r = 0, k = 0; r <= kLatRmax; ++r)
        for (int left = L.ncol[r]; left > 0; left -= lat_slab_columns(r)) {
            k += (2 * r + 1) * std::min(left, lat_slab_columns(r));
            L.slab_entry[++L.slabs] = k;
        }
    if (L.slabs < 2) return cudaSuccess;   // (bonds along one axis only)
    // site s (from the minimum site) lies at anchor + h (s + min)
    L.h = pitch;
    L.org[0] = anchor.x + pitch * ext[0];
    L.org[1] = anchor.y + pitch * ext[1];
    L.org[2] = anchor.z + pitch * ext[2];
    const long long D[3] = {(long long)ext[3] - ext[0] + 1, (long long)ext[4] - ext[1] + 1,
                            (long long)ext[5] - ext[2] + 1};
    const long long NB[3] = {(D[0] + BX - 1) / BX, (D[1] + kLatBY - 1) / kLatBY, (D[2] + kLatBZ - 1) / kLatBZ};
    const long long M[3] = {NB[0] * BX + 2 * R, NB[1] * kLatBY + 2 * R, NB[2] * kLatBZ + 2 * R};
    const long long map_size = M[0] * M[1] * M[2];
    const long long bricks_total = NB[0] * NB[1] * NB[2];
    // dense grids of modest size: 32 bytes per site (grid_w, grid_d), so 512 per
    // particle at most, where a particle of 80 bonds has some 2,000 elsewhere, and
    // 134 MB for a body of few particles asked for by spmv_path 3
    if (map_size > std::max<long long>(16LL * n, 1LL << 22) || map_size >= (1LL << 31) ||
        bricks_total * BX * kLatBY * kLatBZ >= (1LL << 32))
        return cudaSuccess;
    for (int k = 0; k < 3; ++k) L.map_dim[k] = (int)M[k];
    // brick-major keys, sorted; two particles on one site: not a lattice fill
    LT_TRY(cudaMalloc(&t.key, sizeof(unsigned) * (size_t)n));
    LT_TRY(cudaMalloc(&t.n2o, sizeof(int) * (size_t)n));
    k_lat_keys<<<G, kBlock, 0, st>>>(n, t.lb.site, make_int3(ext[0], ext[1], ext[2]), BX,
                                     make_int3((int)NB[0], (int)NB[1], (int)NB[2]), t.key, t.n2o);
    LT_TRY(cudaGetLastError());
    int key_bits = 0;
    while (key_bits < 32 && (1ULL << key_bits) < (unsigned long long)(bricks_total * BX * kLatBY * kLatBZ)) ++key_bits;
    key_bits = (key_bits + 7) / 8 * 8;
    LT_TRY(sort_pairs_u32(t.key, t.n2o, n, std::max(key_bits, 8), st));
    LT_TRY(cudaMemsetAsync(t.ext + 7, 0, sizeof(int), st));
    k_lat_dups<<<G, kBlock, 0, st>>>(t.key, n, t.ext + 7);
    LT_TRY(cudaMemcpyAsync(ext + 7, t.ext + 7, sizeof(int), cudaMemcpyDeviceToHost, st));
    std::vector<unsigned> keys(n);
    LT_TRY(cudaMemcpyAsync(keys.data(), t.key, sizeof(unsigned) * (size_t)n, cudaMemcpyDeviceToHost, st));
    LT_TRY(cudaStreamSynchronize(st));
    if (ext[7]) return cudaSuccess;
    // bricks, their pairs of z-adjacent rows (rows of a brick come z, then y,
    // then x) and the chunks of 32 pairs: a body so thin along z that most pairs
    // lack a row, or so scattered that most bricks hold a few rows, keeps the
    // gather product
    const unsigned bxy = (unsigned)(BX * kLatBY), bsz = bxy * kLatBZ;
    std::vector<int> bstart, bcorner, chunk_start(1, 0), pair_base, pair_slot, row_pair(n);
    for (int i = 0; i < n;) {
        const unsigned brick = keys[i] / bsz;
        const auto pair_of = [&](unsigned local) { return (int)(local / bxy / kLatRZ * bxy + local % bxy); };
        int e = i;
        unsigned char seen[kLatMaxPairs] = {};
        for (; e < n && keys[e] / bsz == brick; ++e) seen[pair_of(keys[e] % bsz)] = 1;
        int index[kLatMaxPairs];
        for (int t = 0; t < kLatMaxPairs; ++t)
            if (seen[t]) {
                const int xy = t % (int)bxy, z = t / (int)bxy * kLatRZ;
                index[t] = (int)pair_base.size();
                pair_base.push_back(((z + R) * HY + (xy / BX + R)) * HX + (xy % BX + R));
                pair_slot.insert(pair_slot.end(), kLatRZ, -1);
            }
        while (pair_base.size() % 32) {   // spare lanes repeat a pair and write nothing
            pair_base.push_back(pair_base.back());
            pair_slot.insert(pair_slot.end(), kLatRZ, -1);
        }
        for (int k = i; k < e; ++k) {
            const unsigned local = keys[k] % bsz;
            row_pair[(size_t)k] = kLatRZ * index[pair_of(local)] + (int)(local / bxy % kLatRZ);
            pair_slot[(size_t)row_pair[(size_t)k]] = k;
        }
        bstart.push_back(i);
        const long long bxi = brick % NB[0], byi = (brick / NB[0]) % NB[1], bzi = brick / (NB[0] * NB[1]);
        bcorner.push_back((int)(((bzi * kLatBZ) * M[1] + byi * kLatBY) * M[0] + bxi * BX));
        chunk_start.push_back((int)(pair_base.size() / 32));
        i = e;
    }
    L.n_bricks = (int)bstart.size();
    const size_t n_pairs = pair_base.size();
    if (n_pairs * kLatRZ > std::max<size_t>((size_t)n * 5 / 2, 8192) || n_pairs >= (1u << 30)) return cudaSuccess;
    // ---- from here on the particles are renumbered: no more early returns ----
    LT_TRY(cudaMalloc(&t.o2n, sizeof(int) * (size_t)n));
    LT_TRY(cudaMalloc(&t.len, sizeof(unsigned) * ((size_t)n + 1)));
    LT_TRY(cudaMalloc(&t.buf, sizeof(dbl4) * (size_t)n));
    k_lat_inverse<<<G, kBlock, 0, st>>>(t.n2o, t.o2n, n);
    k_lat_gather<dbl4><<<G, kBlock, 0, st>>>(x64, t.n2o, (dbl4*)t.buf, n);
    LT_TRY(cudaMemcpyAsync(x64, t.buf, sizeof(dbl4) * (size_t)n, cudaMemcpyDeviceToDevice, st));
    k_lat_gather<float4><<<G, kBlock, 0, st>>>(X32, t.n2o, (float4*)t.buf, n);
    LT_TRY(cudaMemcpyAsync(X32, t.buf, sizeof(float4) * (size_t)n, cudaMemcpyDeviceToDevice, st));
    k_lat_gather<int4><<<G, kBlock, 0, st>>>(t.lb.site, t.n2o, (int4*)t.buf, n);
    LT_TRY(cudaMemcpyAsync(t.lb.site, t.buf, sizeof(int4) * (size_t)n, cudaMemcpyDeviceToDevice, st));
    k_lat_gather<int><<<G, kBlock, 0, st>>>(perm, t.n2o, (int*)t.buf, n);
    LT_TRY(cudaMemcpyAsync(perm, t.buf, sizeof(int) * (size_t)n, cudaMemcpyDeviceToDevice, st));
    k_lat_gather<int><<<G, kBlock, 0, st>>>(cnt, t.n2o, (int*)t.buf, n);
    LT_TRY(cudaMemcpyAsync(cnt, t.buf, sizeof(int) * (size_t)n, cudaMemcpyDeviceToDevice, st));
    // CSR: rows keep their padded lengths and bond order; columns renamed
    k_lat_lengths<<<G, kBlock, 0, st>>>(row_ptr, t.n2o, t.len, n);
    LT_TRY(scan_exclusive_u32(t.len, t.len, (long long)n + 1, st));
    LT_TRY(cudaMalloc(&t.col_new, sizeof(int) * ((size_t)total_slots + 8)));
    LT_TRY(cudaMemsetAsync(t.col_new, 0, sizeof(int) * ((size_t)total_slots + 8), st));
    k_lat_remap_col<<<G, kBlock, 0, st>>>(row_ptr, *col, t.len, t.n2o, t.o2n, t.col_new, n);
    LT_TRY(cudaMemcpyAsync(row_ptr, t.len, sizeof(int) * ((size_t)n + 1), cudaMemcpyDeviceToDevice, st));
    LT_TRY(cudaGetLastError());
    std::swap(*col, t.col_new);   // the old column array is freed with the temporaries
    LT_TRY(cudaMalloc(&t.lb.brick_start, sizeof(int) * bstart.size()));
    LT_TRY(cudaMalloc(&t.lb.brick_corner, sizeof(int) * bcorner.size()));
    LT_TRY(cudaMalloc(&t.lb.chunk_start, sizeof(int) * chunk_start.size()));
    LT_TRY(cudaMalloc(&t.lb.pair_base, sizeof(int) * n_pairs));
    LT_TRY(cudaMalloc(&t.lb.pair_slot, sizeof(int) * pair_slot.size()));
    LT_TRY(cudaMalloc(&t.lb.row_pair, sizeof(int) * (size_t)n));
    LT_TRY(cudaMalloc(&t.lb.offk, sizeof(int) * offk.size()));
    LT_TRY(cudaMalloc(&t.lb.ell, sizeof(float2) * (size_t)L.K * n_pairs));
    LT_TRY(cudaMemsetAsync(t.lb.ell, 0, sizeof(float2) * (size_t)L.K * n_pairs, st));   // rows that do not exist stay 0
    LT_TRY(cudaMalloc(&t.lb.dense, sizeof(int) * (size_t)n));
    LT_TRY(cudaMalloc(&t.lb.grid_w, sizeof(float4) * (size_t)map_size));
    LT_TRY(cudaMemsetAsync(t.lb.grid_w, 0, sizeof(float4) * (size_t)map_size, st));
    LT_TRY(cudaMalloc(&t.lb.grid_d, sizeof(float4) * (size_t)map_size));
    LT_TRY(cudaMemsetAsync(t.lb.grid_d, 0, sizeof(float4) * (size_t)map_size, st));
    LT_TRY(cudaMalloc(&t.lb.image, (size_t)lat_image_bytes(R) * (size_t)L.n_bricks));
    LT_TRY(cudaMalloc(&t.lb.sched, sizeof(unsigned) * 2));
    LT_TRY(cudaMemsetAsync(t.lb.sched, 0, sizeof(unsigned) * 2, st));
    LT_TRY(cudaMemcpyAsync(t.lb.brick_start, bstart.data(), sizeof(int) * bstart.size(), cudaMemcpyHostToDevice, st));
    LT_TRY(cudaMemcpyAsync(t.lb.brick_corner, bcorner.data(), sizeof(int) * bcorner.size(), cudaMemcpyHostToDevice, st));
    LT_TRY(cudaMemcpyAsync(t.lb.chunk_start, chunk_start.data(), sizeof(int) * chunk_start.size(), cudaMemcpyHostToDevice, st));
    LT_TRY(cudaMemcpyAsync(t.lb.pair_base, pair_base.data(), sizeof(int) * n_pairs, cudaMemcpyHostToDevice, st));
    LT_TRY(cudaMemcpyAsync(t.lb.pair_slot, pair_slot.data(), sizeof(int) * pair_slot.size(), cudaMemcpyHostToDevice, st));
    LT_TRY(cudaMemcpyAsync(t.lb.row_pair, row_pair.data(), sizeof(int) * (size_t)n, cudaMemcpyHostToDevice, st));
    LT_TRY(cudaMemcpyAsync(t.lb.offk, offk.data(), sizeof(int) * offk.size(), cudaMemcpyHostToDevice, st));
    k_lat_dense<<<G, kBlock, 0, st>>>(t.lb.site, n, R, (int)M[0], (int)M[1], t.lb.dense);
    LT_TRY(cudaGetLastError());
    LT_TRY(cudaStreamSynchronize(st));   // the host vectors above are read by the copies
    L.brick_start = t.lb.brick_start;
    L.brick_corner = t.lb.brick_corner;
    L.chunk_start = t.lb.chunk_start;
    L.pair_base = t.lb.pair_base;
    L.pair_slot = t.lb.pair_slot;
    L.row_pair = t.lb.row_pair;
    L.site = t.lb.site;
    L.offk = t.lb.offk;
    L.ell = t.lb.ell;
    L.sched = t.lb.sched;
    L.dense = t.lb.dense;
    L.grid_w = t.lb.grid_w;
    L.grid_d = t.lb.grid_d;
    L.image = t.lb.image;
    LT_TRY(grid_box(&L));
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    L.grid = std::max(1, std::min(L.n_bricks, lattice_spmv_blocks_per_sm(L) * sms));
    L.wait_ns = kWaitLatticeNs;
    *lp = L;
    *lb = t.lb;
    t.lb = LatticeBuffers{};
    *ok = 1;
    return cudaGetLastError();
}

}  // namespace pdgb
