// cg_persist.cu -- the CG iterations of a small body in one cooperative launch.
//
// The solve of the reference (CUSP krylov::cg, driven by
// Simulator::solveLinearSystem, src/core/simulator.cu:735-799) needs two
// grid-wide sums per iteration.  As separate launches (product, solution
// update, direction update) an iteration of a body of a few thousand particles
// costs the launches and the tails of three nearly empty kernels; here every
// block keeps its rows for the whole solve:
//   * x, r, p and A p of the block's own rows stay in shared memory, and so
//     does p of its halo (the distinct neighbours of its rows);
//   * what a bond contributes to the product does not change inside a solve
//     (the positions do not move): where they fit, every bond's geometry (FP64:
//     its Jacobian) and halo index are kept in shared memory;
//   * a grid-wide sum is one exchange of (partial sum, epoch) records, one
//     16-byte store from every block into every block's inbox: a block polls
//     only its own inbox and adds the partials in block order, so the sum and
//     the barrier are the same round trip and no line is polled by two blocks;
//   * the residual r is the only vector that travels: each row publishes (r,
//     epoch) in 16-byte records, which the blocks that have it in their halo
//     poll while <r, r> is being summed, and p = r + beta p of the halo is then
//     formed by every block for itself.
// An iteration takes two exchanges (<p, A p>, <r, r>) and no memory fence.
//
// Memory ordering.  Every value that another block reads is in a record of
// one 16-byte access together with the epoch it belongs to, so a reader never
// needs what was written before or after it.  A record is overwritten only
// after all its readers have it: the next r of a row follows the exchange of
// <p, A p>, whose partials depend on every record read for them, and inbox
// records alternate by epoch parity.  Every wait is bounded (kWaitSolveNs): a
// thread whose wait runs out records the error and its block returns, and so
// does every block that sees the error, in this launch and in later ones.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "batch.h"
#include "step_rows.cuh"

namespace pdgb {

namespace {

constexpr int kPersistThreads = 512;
constexpr int kPersistWarps = kPersistThreads / 32;
constexpr int kPersistMaxGrid = 256;
constexpr int kTileLanes = 4;        // lanes per row where the bonds are read from global memory
constexpr int kTileBlock = 1024;     // threads of a product outside a solve

__device__ __forceinline__ unsigned long long now_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// 16 bytes in one access: a reader sees the value that belongs to the epoch
__device__ __forceinline__ void publish(ulonglong2* slot, unsigned long long value, unsigned long long epoch)
{
    asm volatile("{ .reg .b128 v; mov.b128 v, {%1, %2}; st.relaxed.gpu.global.b128 [%0], v; }"
                 ::"l"(slot), "l"(value), "l"(epoch)
                 : "memory");
}
__device__ __forceinline__ ulonglong2 observe(const ulonglong2* slot)
{
    ulonglong2 v;
    asm volatile("{ .reg .b128 v; ld.relaxed.gpu.global.b128 v, [%2]; mov.b128 {%0, %1}, v; }"
                 : "=l"(v.x), "=l"(v.y)
                 : "l"(slot)
                 : "memory");
    return v;
}

struct PersistArgs {
    StepParams P;
    DeviceState S;
    ulonglong2* rec;            // published r: one record per row (FP64: two)
    ulonglong2* inbox;          // [2][grid][grid]: records by epoch parity, reader, writer
    unsigned long long epoch;   // the last epoch of earlier launches
    int rows;                   // rows per block
    int halo;                   // halo entries of a block at most
    int bonds;                  // bond slots kept in shared memory per block (0: none)
    int max_iters;              // iterations of this launch at most
    int profile;
    int start;                  // form r = p = b - y and its test first (y: A x of the guess)
    int finish;                 // advance the rows when the solve has ended
    unsigned long long wait_ns; // limit of a wait
};

// A block's part in a solve.
struct PersistRun {
    ulonglong2* rec;
    ulonglong2* inbox;
    int rows, halo, bonds, max_iters;
    int block, grid;            // this block among those of the solve
    bool start;
    int* error;                 // set when a wait ran out of time
    unsigned long long wait_ns; // limit of a wait (0: it runs out at once)
};
__device__ __forceinline__ PersistRun persist_run(const PersistArgs& A)
{
    return PersistRun{A.rec, A.inbox, A.rows, A.halo, A.bonds, A.max_iters, (int)blockIdx.x, (int)gridDim.x,
                      A.start != 0, &A.S.sc->wait_error, A.wait_ns};
}

// Bits of the sums within a warp: double-float for FP32 data.
__device__ __forceinline__ unsigned long long pack(DF v)
{
    return ((unsigned long long)__float_as_uint(v.hi) << 32) | __float_as_uint(v.lo);
}
__device__ __forceinline__ unsigned long long pack(double v) { return (unsigned long long)__double_as_longlong(v); }
template <typename T> __device__ __forceinline__ T unpack(unsigned long long v);
template <> __device__ __forceinline__ DF unpack<DF>(unsigned long long v)
{
    return DF{__uint_as_float((unsigned)(v >> 32)), __uint_as_float((unsigned)v)};
}
template <> __device__ __forceinline__ double unpack<double>(unsigned long long v)
{
    return __longlong_as_double((long long)v);
}
__device__ __forceinline__ void add_to(DF& a, DF b) { df_add(a, b); }
__device__ __forceinline__ void add_to(double& a, double b) { a = __dadd_rn(a, b); }
__device__ __forceinline__ DF shfl_xor(DF a, int off)
{
    return DF{__shfl_xor_sync(0xffffffffu, a.hi, off), __shfl_xor_sync(0xffffffffu, a.lo, off)};
}
__device__ __forceinline__ double shfl_xor(double a, int off) { return __shfl_xor_sync(0xffffffffu, a, off); }
// sum over the lanes whose index is a multiple of `step` (a power of two)
template <typename T>
__device__ __forceinline__ void warp_sum(T& v, int step)
{
    for (int off = 16; off >= step; off >>= 1) add_to(v, shfl_xor(v, off));
}

// Beyond the warp, sums of FP32 data are integers times 2^(top - kTopOffset), `top`
// the largest exponent among the terms of a sum: 53 bits of the largest term.
// Double-float holds 48: with it throughout, <r, r> of 2,500 to 30,000 rows was
// 1.2e-15 to 1.9e-15 off the sum of separate launches (FP64 from the warp on), root
// mean square over bodies; with integers it is 0.8e-16 to 2.4e-16 off.  A warp adds
// 32 such terms with 4 reductions (22 cycles for a maximum, 49 for a sum) where
// double-float takes 5 steps of 60, and FP64 5 of 100 and 19 cycles of its pipe for
// every warp; and the warps that poll form the sum once for the block.  With
// double-float an iteration of 512 particles took 7.9 us instead of 7.3, of 16k 10.8
// instead of 10.25, of 100k 23.9 instead of 23.3 (steps included).
constexpr int kTopOffset = 256;
constexpr int kTopSpecial = 511;   // not a finite number
struct WideSum {                   // (hi 2^44 + mid 2^22 + lo) 2^(top - kTopOffset); mid, lo of 22 bits
    int hi, mid, lo, top;
};
__device__ __forceinline__ float power_of_two(int k) { return __int_as_float((k + 127) << 23); }   // -126 .. 127
__device__ __forceinline__ int top_of(DF v)
{
    const int field = (__float_as_int(v.hi) >> 23) & 255;   // hi is a 24-bit integer times 2^(field - 150)
    return field == 255 ? kTopSpecial : max(field, 1) - 179 + kTopOffset;
}
// v 2^-(e) rounded to an integer (53 bits and the sign), e = top_of(v) - kTopOffset
__device__ __forceinline__ long long mantissa_of(DF v)
{
    const int bits = __float_as_int(v.hi), field = (bits >> 23) & 255, e = max(field, 1) - 179, k = -e / 2;
    const long long mant = (bits & 0x7fffff) | (field > 0 ? 0x800000 : 0);
    const int lo = __float2int_rn(v.lo * power_of_two(k) * power_of_two(-e - k));   // (2^28 at most)
    return ((bits < 0 ? -mant : mant) << 29) + lo;
}
// The sum over the warp of m 2^-(down), down >= 0, each term rounded to an integer
// below 2^58; the carries are left in the sums of `mid` and `lo`.
__device__ __forceinline__ WideSum warp_total(long long m, int down, int top)
{
    const int d = min(down, 63);
    m = (m + (long long)((1ull << d) >> 1)) >> d;
    return WideSum{__reduce_add_sync(0xffffffffu, (int)(m >> 44)),
                   (int)__reduce_add_sync(0xffffffffu, (unsigned)(m >> 22) & 0x3fffffu),
                   (int)__reduce_add_sync(0xffffffffu, (unsigned)m & 0x3fffffu), top};
}
__device__ __forceinline__ void carry(WideSum& s)
{
    s.mid += s.lo >> 22;
    s.lo &= 0x3fffff;
    s.hi += s.mid >> 22;
    s.mid &= 0x3fffff;
}
__device__ __forceinline__ DF to_df(const WideSum& s)   // (carried)
{
    if (s.top == kTopSpecial) return DF{__int_as_float(0x7fffffff), 0.f};
    const auto exact = [](int v) { return __int_as_float(0x4B000000 | v) - 8388608.f; };   // 22 bits
    const float x = small_int_to_float(s.hi) * 17592186044416.f, y = exact(s.mid) * 4194304.f;   // 2^44, 2^22
    const float t = __fadd_rn(x, y);
    const float rest = __fadd_rn(__fsub_rn(y, __fsub_rn(t, x)), exact(s.lo));
    const float hi = __fadd_rn(t, rest), lo = __fsub_rn(rest, __fsub_rn(hi, t));
    const int e = s.top - kTopOffset, k = e / 2;
    const float a = power_of_two(k), b = power_of_two(e - k);
    return DF{hi * a * b, lo * a * b};
}
__device__ __forceinline__ double to_double(const WideSum& s)
{
    if (s.top == kTopSpecial) return __longlong_as_double(0x7ff8000000000000ll);
    const double v = __fma_rn((double)(((long long)s.hi << 22) + s.mid), 4194304.0, (double)s.lo);
    return v * __longlong_as_double((long long)(s.top - kTopOffset + 1023) << 52);
}

struct Exchange {
    unsigned long long warp[kPersistWarps];
    unsigned long long from[kPersistMaxGrid];      // FP64: the blocks' sums
    WideSum part[kPersistMaxGrid / 32];            // FP32 data: those of 32 blocks, carried
    int top[kPersistMaxGrid / 32];
    WideSum total;                                 // their sum, and as double-float
    DF sum;
    PersistRun run;
    int error;
};

// Polls a record until `arrived` accepts it; false when the wait ran out of
// time (here or in another thread).
template <typename Ok>
__device__ __forceinline__ bool await(const ulonglong2* rec, int* error, unsigned long long limit, Exchange& e, ulonglong2& r,
                                      Ok arrived)
{
    r = observe(rec);
    if (limit != 0 && arrived(r)) return true;
    unsigned spins = limit != 0 ? 0u : ~0u;
    const unsigned long long t0 = now_ns();
    for (;;) {
        if ((++spins & 255u) == 0) {
            if (limit == 0 || *(volatile int*)error || now_ns() - t0 > limit) {
                *(volatile int*)error = 1;
                e.error = 1;
                return false;
            }
        }
        r = observe(rec);
        if (arrived(r)) return true;
    }
}

// A block's own part goes into every block's inbox, and the part of block
// threadIdx.x comes back (threads beyond the grid: nothing).  The low nine bits of a
// record's second word belong to its value.
__device__ __forceinline__ ulonglong2 round_trip(Exchange& e, const PersistRun& A, unsigned long long epoch,
                                                 unsigned long long value, unsigned nine)
{
    ulonglong2 r = make_ulonglong2(0ull, 0ull);
    const int b = threadIdx.x, grid = A.grid;
    if (b < grid) {
        ulonglong2* box = A.inbox + (size_t)(epoch & 1) * grid * grid;
        publish(box + (size_t)b * grid + A.block, value, (epoch << 9) | nine);
        await(box + (size_t)A.block * grid + b, A.error, A.wait_ns, e, r,
              [epoch](const ulonglong2& x) { return x.y >> 9 == epoch; });
    }
    return r;
}
__device__ __forceinline__ int polling_threads(int grid) { return (grid + 31) / 32 * 32; }   // whole warps
__device__ __forceinline__ void polling_barrier(int threads)
{
    __syncwarp();
    asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}

// The exchange of the warps that poll: from the warps' sums to e.total and e.sum.
// (A call: inlined, it takes registers from the loops around it, 11.6 us at 16k.)
__device__ __noinline__ void exchange_wide(Exchange& e, unsigned long long epoch)
{
    const PersistRun& A = e.run;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, polling = polling_threads(A.grid);
    const DF w = lane < kPersistWarps ? unpack<DF>(e.warp[lane]) : DF{0.f, 0.f};
    const int own = top_of(w), block_top = __reduce_max_sync(0xffffffffu, own);
    const WideSum t = warp_total(mantissa_of(w), block_top - own, block_top);
    const ulonglong2 r = round_trip(
        e, A, epoch, (unsigned long long)(((long long)t.hi << 44) + ((long long)t.mid << 22) + t.lo), (unsigned)block_top);
    const int its = (int)(r.y & 511u), warp_top = __reduce_max_sync(0xffffffffu, its);
    if (lane == 0) e.top[warp] = warp_top;
    polling_barrier(polling);
    int top = e.top[0];
    for (int k = 1; k < polling / 32; ++k) top = max(top, e.top[k]);
    WideSum s = warp_total((long long)r.x, top - its, top);
    carry(s);
    if (lane == 0) e.part[warp] = s;
    polling_barrier(polling);
    if (threadIdx.x == 0) {
        for (int k = 1; k < polling / 32; ++k) {
            const WideSum p = e.part[k];
            s.hi += p.hi;
            s.mid += p.mid;
            s.lo += p.lo;
        }
        carry(s);
        e.total = s;
        e.sum = to_df(s);
    }
}

// The sum over all blocks of v (which only lanes at multiples of `step` hold) in
// `total` (FP32 data: in 48 bits, and e.total in 53); every thread of the block
// calls it and gets the sum.  The warps that do not poll the inbox run help(thread,
// threads) meanwhile.  Returns false when a wait ran out of time.
template <typename Help>
__device__ __forceinline__ bool exchange_sum(Exchange& e, DF v, DF& total, int step, const PersistRun& A,
                                             unsigned long long epoch, Help help)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, polling = polling_threads(A.grid);
    warp_sum(v, step);
    if (lane == 0) e.warp[warp] = pack(v);
    __syncthreads();
    if ((int)threadIdx.x < polling) {
        exchange_wide(e, epoch);
    } else {
        help((int)threadIdx.x - polling, kPersistThreads - polling);
    }
    __syncthreads();
    total = e.sum;
    return e.error == 0;
}
template <typename Help>
__device__ __forceinline__ bool exchange_sum(Exchange& e, double v, double& total, int step, const PersistRun& A,
                                             unsigned long long epoch, Help help)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, polling = polling_threads(A.grid);
    warp_sum(v, step);
    if (lane == 0) e.warp[warp] = pack(v);
    __syncthreads();
    if ((int)threadIdx.x < polling) {
        double t = unpack<double>(e.warp[lane & (kPersistWarps - 1)]);   // both halves of the warp form the same sum
#pragma unroll
        for (int off = kPersistWarps / 2; off > 0; off >>= 1) add_to(t, shfl_xor(t, off));
        const ulonglong2 r = round_trip(e, A, epoch, pack(t), 0u);
        if ((int)threadIdx.x < A.grid) e.from[threadIdx.x] = r.x;
    } else {
        help((int)threadIdx.x - polling, kPersistThreads - polling);
    }
    __syncthreads();
    total = 0.0;
    for (int b = lane; b < A.grid; b += 32) add_to(total, unpack<double>(e.from[b]));
    warp_sum(total, 1);
    return e.error == 0;
}

// The quotient a / b rounded to FP32 (a, b in double-float): the FP32 quotient and
// one correction by its remainder, at a fifth of an FP64 division's latency (573
// cycles).  Of 10^8 pairs, on the CPU, 11 differ from the rounded FP64 quotient, all
// within 0.0002 units of a tie: at most 0.5002 units off where that is 0.5.
// Sums whose FP32 words leave the range of the steps take the FP64 division.
__device__ __forceinline__ float df_quotient(DF a, DF b)
{
    const float fa = fabsf(a.hi), fb = fabsf(b.hi);
    if (!(fa > 1e-25f && fa < 1e25f && fb > 1e-25f && fb < 1e25f)) return (float)(df_to_double(a) / df_to_double(b));
    const float q = __fdiv_rn(a.hi, b.hi);
    const float p = __fmul_rn(q, b.hi);
    const float pe = __fmaf_rn(q, b.hi, -p);
    // a - q b: the leading words cancel exactly
    const float r = __fadd_rn(__fsub_rn(a.hi, p), __fsub_rn(__fsub_rn(a.lo, pe), __fmul_rn(q, b.lo)));
    return __fadd_rn(q, __fdividef(r, b.hi));
}

// One iteration's convergence test (as cg_fin_axpy): ||r|| <= tol, the square
// root only where the squares are too near to tell.
__device__ __forceinline__ bool below_tolerance(double rr, double tol)
{
    const double t2 = tol * tol;
    if (rr > t2 * (1.0 + 1e-12)) return false;
    if (rr < t2 * (1.0 - 1e-12)) return true;
    return sqrt(rr) <= tol;
}

struct __align__(16) BondGeometry {   // one bond of the mixed-precision product, formed once per solve
    float x, y, z;   // x_q - x_p
    float i3;        // 1 / d^3
};
__device__ __forceinline__ BondGeometry bond_geometry(const float4& Xq, const float4& xp, float sup, float inv_d0,
                                                      float& a1)
{
    BondGeometry g;
    float cx, cy, cz;
    supercell_delta(__float_as_int(Xq.w), __float_as_int(xp.w), sup, cx, cy, cz);
    g.x = (Xq.x - xp.x) + cx;
    g.y = (Xq.y - xp.y) + cy;
    g.z = (Xq.z - xp.z) + cz;
    const float inv_d = rsqrtf(fmaf(g.x, g.x, fmaf(g.y, g.y, g.z * g.z)));
    g.i3 = inv_d * inv_d * inv_d;
    a1 = inv_d0 - inv_d;
    return g;
}

// A halo position as 32-bit fixed point, supercell edge = 2^25, wrapping: the
// difference of two positions less than 64 supercells apart is exact, in three
// integer subtractions instead of the decoding of two words of supercell
// coordinates (59 instructions per bond of the tile product, 77 with it).  An FP32
// offset (0 to 1 edge) is finer than 2^-25 below a quarter of the edge, but the
// decoded difference rounds again when the cells' distance is added: over horizons
// of 2 to 3 spacings, edges of 1 to 1.95 horizons and jitters of 0.05 and 0.4, the
// product's error from its geometry is 0.93 to 1.00 of the decoding form's (root
// mean square, against 64 bits, emulated).  Blocks whose rows and halo reach farther
// than kFixedReach supercells from their first row keep the decoding form.
constexpr int kFixedBits = 25;
constexpr int kFixedReach = 31;
__device__ __forceinline__ float4 fixed_position(const float4& X, float per_edge)
{
    const unsigned c = (unsigned)__float_as_int(X.w);
    const auto fix = [per_edge](float off, unsigned cell) {
        return __int_as_float((int)((cell << kFixedBits) + (unsigned)__float2int_rn(off * per_edge)));
    };
    return make_float4(fix(X.x, c & 1023u), fix(X.y, (c >> 10) & 1023u), fix(X.z, (c >> 20) & 1023u), 0.f);
}
// (an offset outside its cell: the body has left the supercells' window)
__device__ __forceinline__ bool farther(const float4& X, int ref, float sup)
{
    const int w = __float_as_int(X.w);
    const bool inside = fabsf(X.x) <= sup && fabsf(X.y) <= sup && fabsf(X.z) <= sup;
    return !inside || abs((w & 1023) - (ref & 1023)) > kFixedReach || abs(((w >> 10) & 1023) - ((ref >> 10) & 1023)) > kFixedReach ||
           abs(((w >> 20) & 1023) - ((ref >> 20) & 1023)) > kFixedReach;
}
// `per_edge` is 2^25 / edge (a power of two): the bond vector is in units of
// 1 / per_edge, and so is i3, which the product takes with it twice.
__device__ __forceinline__ BondGeometry bond_geometry_fixed(const float4& Xq, const float4& xp, float per_edge,
                                                            float inv_d0, float& a1)
{
    BondGeometry g;
    g.x = (float)(__float_as_int(Xq.x) - __float_as_int(xp.x));
    g.y = (float)(__float_as_int(Xq.y) - __float_as_int(xp.y));
    g.z = (float)(__float_as_int(Xq.z) - __float_as_int(xp.z));
    float inv;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(fmaf(g.x, g.x, fmaf(g.y, g.y, g.z * g.z))));
    const float inv_d = inv * per_edge;
    g.i3 = inv * inv * inv_d;
    a1 = inv_d0 - inv_d;
    return g;
}

// Four consecutive bonds' halo indices and 1/d0.
__device__ __forceinline__ void load_bonds(const DeviceState& S, int slot, int (&l)[4], float (&id0)[4])
{
    const ushort4 i = __ldg((const ushort4*)(S.lidx + slot));
    const float4 d = __ldg((const float4*)(S.inv_d0 + slot));
    l[0] = i.x; l[1] = i.y; l[2] = i.z; l[3] = i.w;
    id0[0] = d.x; id0[1] = d.y; id0[2] = d.z; id0[3] = d.w;
}

// The residual of the guess (residual_elem): zero on Dirichlet rows.
template <typename V4>
__device__ __forceinline__ V4 first_residual(const DeviceState& S, int p)
{
    V4 r = make_v4<V4>(0.0, 0.0, 0.0);
    if (is_dirichlet(S.act[p] & kActMask)) return r;
    const V4 b = ((const V4*)S.rhs)[p], y = ((const V4*)S.y)[p];
    r.x = b.x - y.x;
    r.y = b.y - y.y;
    r.z = b.z - y.z;
    return r;
}

template <int N>
using Lanes = std::integral_constant<int, N>;

// Mixed precision, G lanes per row, U bonds in flight per lane.  The halo is
// S.halo of a tile per block, a bond's index into it S.lidx.
// CACHED: the bonds' geometry stays in shared memory; else the halo's
// positions do, and the index and 1/d0 of a bond are read from global memory
// (6 bytes per bond, from L2).  Not cached, the product is bound by the
// shared-memory pipe (7.2 wavefronts per step of 32 bonds and array when bonds
// stood in build order) and by latency (one block per SM).  An iteration at 100k
// particles (76 bonds) takes 25.3 us: 38.2 with scalar loads of the bonds, 31.2
// with four per lane and load and the next four in flight, 30.4 with a round of
// their own for the rows left over, 30.0 with fixed-point positions, 25.3 with
// the order of k_bank_order.  Eight lanes per row: 34.9 against 31.2; 1024
// threads 30.3 (but 24.0 against 21.8 at 50k and 104 bonds); 23.3 with the sums of
// WideSum (steps included).
// `epoch` is the last epoch used in the inbox and the records.  Blocks beyond the
// last row only exchange.  Returns false when a wait ran out of time.
template <bool CACHED, int G, int U>
__device__ __forceinline__ bool persist_solve32(const StepParams& P, const DeviceState& S, const PersistRun& A,
                                                unsigned char* smem, Exchange& ex, unsigned long long& epoch, bool timed)
{
    CgScalars* sc = S.sc;
    // (the scalars change only after every block's last exchange; an error may come
    // from a block of this launch, which the others learn of in their waits)
    if (__syncthreads_or(*(volatile int*)A.error)) return false;
    if (!A.start && ((volatile CgScalars*)sc)->done) return true;
    const int lo = A.block * A.rows;
    const int nr = max(0, min(A.rows, P.n - lo));
    float4* sx = (float4*)smem;
    float4* sr = sx + A.rows;
    float4* sp = sr + A.rows;
    float4* sy = sp + A.rows;
    float4* sw = sy + A.rows;                            // the halo's p
    float4* sh = sw + A.halo;                            // the halo's r
    float4* shx = sh + A.halo;                           // the halo's positions (not CACHED)
    BondGeometry* sg = (BondGeometry*)(CACHED ? shx : shx + A.halo);
    float* sa1 = (float*)(sg + A.bonds);                 // 1/d0 - 1/d
    int* srow = (int*)(sa1 + A.bonds);                   // first slot of the row
    int* scnt = srow + A.rows;                           // live bonds << 8 | activity, -1 for a Dirichlet row
    int* sq = scnt + A.rows;                             // the halo's slots
    uint16_t* sl = (uint16_t*)(sq + A.halo);             // a bond's halo index

    const int lane = threadIdx.x & (G - 1);
    const unsigned gmask = group_mask<G>();
    constexpr int NG = kPersistThreads / G;
    const int slot0 = CACHED && nr > 0 ? S.row_ptr[lo] : 0;
    DotAcc32 first;   // <r, r> of the guess
    for (int t = threadIdx.x; t < nr; t += kPersistThreads) {
        const int p = lo + t;
        sx[t] = ((const float4*)S.sol)[p];
        sr[t] = A.start ? first_residual<float4>(S, p) : ((const float4*)S.r)[p];
        sp[t] = A.start ? sr[t] : ((const float4*)S.p)[p];
        if (A.start) {
            first.fma(sr[t].x, sr[t].x);
            first.fma(sr[t].y, sr[t].y);
            first.fma(sr[t].z, sr[t].z);
        }
        const uint8_t ab = S.act[p];
        scnt[t] = is_dirichlet(ab & kActMask) ? -1 : S.cnt[p] << 8 | ab;
        srow[t] = S.row_ptr[p] - slot0;
    }
    const int h0 = nr > 0 ? S.halo_ptr[A.block] : 0, nh = nr > 0 ? S.halo_ptr[A.block + 1] - h0 : 0;
    for (int h = threadIdx.x; h < nh; h += kPersistThreads) {
        const int q = S.halo[h0 + h];
        sq[h] = q;
        sh[h] = A.start ? first_residual<float4>(S, q) : ((const float4*)S.r)[q];
        sw[h] = A.start ? sh[h] : ((const float4*)S.p)[q];
        if (!CACHED) shx[h] = S.xs4[q];
    }
    if (threadIdx.x == 0) {
        ex.error = 0;
        ex.run = A;
    }
    const float sup = (float)P.sup, per_edge = (float)(1 << kFixedBits) / sup;
    bool fixed = false;
    if (!CACHED) {   // the entries that this thread has staged
        const int ref = nr > 0 ? __float_as_int(S.xs4[lo].w) : 0;
        bool far = false;
        for (int t = threadIdx.x; t < nr; t += kPersistThreads) far |= farther(S.xs4[lo + t], ref, sup);
        for (int h = threadIdx.x; h < nh; h += kPersistThreads) far |= farther(shx[h], ref, sup);
        fixed = !__syncthreads_or(far);
        if (fixed)
            for (int h = threadIdx.x; h < nh; h += kPersistThreads) shx[h] = fixed_position(shx[h], per_edge);
    }
    __syncthreads();
    if (CACHED) {
        for (int i = threadIdx.x / G; i < nr; i += NG) {
            const int cn = scnt[i] < 0 ? 0 : scnt[i] >> 8, base = srow[i];
            const float4 xp = S.xs4[lo + i];
            for (int j = lane; j < cn; j += G) {
                const int l = S.lidx[slot0 + base + j];
                sg[base + j] = bond_geometry(S.xs4[sq[l]], xp, sup, S.inv_d0[slot0 + base + j], sa1[base + j]);
                sl[base + j] = (uint16_t)l;
            }
        }
    }
    const double tol = sc->tol;
    const float tol2_far = (float)(tol * tol * 1.0001);   // a sum of squares above it is above tol^2
    const int max_iter = sc->max_iter;
    const double rz0 = sc->rz;
    DF rz{(float)rz0, (float)(rz0 - (double)(float)rz0)}, pAp{0.f, 0.f};   // for the quotients (48 bits)
    float alpha = 0.f, beta = A.start ? 0.f : (float)sc->beta;
    int iter = sc->iter;
    bool done = false, converged = false;
    if (A.start) {
        if (!exchange_sum(ex, first.v, rz, 1, A, ++epoch, [](int, int) {})) return false;
        converged = below_tolerance(to_double(ex.total), tol);
        done = converged || iter >= max_iter;
    }

    unsigned long long t_mark = 0, ns_spmv = 0, ns_vec = 0;
    for (int it = 0; it < A.max_iters && !done; ++it) {
        if (timed) t_mark = now_ns();
        // ---- p = r + beta p of the halo and the own rows; y = A p
        for (int h = threadIdx.x; h < nh; h += kPersistThreads) {
            const float4 r = sh[h], w = sw[h];
            sw[h] = make_float4(r.x + beta * w.x, r.y + beta * w.y, r.z + beta * w.z, 0.f);
        }
        __syncthreads();
        DotAcc32 acc;
        const auto rows = [&](auto width, auto form, int from, int to) {
            constexpr int R = decltype(width)::value;   // lanes per row
            constexpr bool FIXED = decltype(form)::value;
            const int rl = threadIdx.x & (R - 1);
            const unsigned rmask = group_mask<R>();
            for (int i = from + threadIdx.x / R; i < to; i += kPersistThreads / R) {
                const int cn = scnt[i] >> 8, base = srow[i], p = lo + i;
                int l[U];
                float a1[U];
                // the bond records of one step: index, and 1/d0 - 1/d (CACHED) or
                // 1/d0; U consecutive slots in one load each (not CACHED: rows start
                // 32-byte aligned and hold a multiple of 8 slots)
                const auto load = [&](int j0) {
                    if constexpr (CACHED) {
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            const int j = j0 + u * R;
                            l[u] = 0;
                            a1[u] = 0.f;
                            if (j < cn) {
                                l[u] = sl[base + j];
                                a1[u] = sa1[base + j];
                            }
                        }
                    } else if (j0 < cn) {
                        load_bonds(S, base + j0, l, a1);
                    }
                };
                constexpr int LS = CACHED ? 1 : U, US = CACHED ? R : 1;   // slots between lanes, between a lane's bonds
                load(rl * LS);
                float4 xp = make_float4(0.f, 0.f, 0.f, 0.f);
                if (!CACHED && cn > 0) xp = __ldg(S.xs4 + p);
                if (FIXED) xp = fixed_position(xp, per_edge);
                float4 w = sp[i];
                const float4 r = sr[i];
                w = make_float4(r.x + beta * w.x, r.y + beta * w.y, r.z + beta * w.z, 0.f);
                float ax = 0.f, ay = 0.f, az = 0.f;
                for (int j0 = rl * LS; j0 < cn; j0 += R * U) {
                    int lc[U];
                    float ac[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        lc[u] = l[u];
                        ac[u] = a1[u];
                    }
                    load(j0 + R * U);   // in flight while this step's bonds are added
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int j = j0 + u * US;
                        if (!FIXED && j >= cn) continue;
                        const float4 Wq = sw[lc[u]];
                        BondGeometry g;
                        float a = ac[u];
                        if constexpr (CACHED) g = sg[base + j];
                        else if constexpr (FIXED) g = bond_geometry_fixed(shx[lc[u]], xp, per_edge, ac[u], a);
                        else g = bond_geometry(shx[lc[u]], xp, sup, ac[u], a);
                        // (every slot of a row has a halo index; a w that is not finite there
                        // makes no row wrong that <p, A p> has not made so already)
                        if (FIXED && j >= cn) a = g.i3 = 0.f;
                        const float wx = w.x - Wq.x, wy = w.y - Wq.y, wz = w.z - Wq.z;
                        const float d = fmaf(g.x, wx, fmaf(g.y, wy, g.z * wz)) * g.i3;
                        ax = fmaf(a, wx, fmaf(d, g.x, ax));
                        ay = fmaf(a, wy, fmaf(d, g.y, ay));
                        az = fmaf(a, wz, fmaf(d, g.z, az));
                    }
                }
                if (cn >= 0) spmv_finish_mixed<R, true>(P, S, p, (uint8_t)scnt[i], w, ax, ay, az, rl, rmask, sy - lo, acc);
                else if (rl == 0) sy[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                __syncwarp(rmask);   // every lane has read sp[i]
                if (rl == 0) sp[i] = w;
            }
        };
        // The rows left over from whole rounds of the block's groups take a round of
        // their own with more lanes each.
        const int whole = CACHED ? nr : nr / NG * NG, left = nr - whole;
        const auto all_rows = [&](auto form) {
            rows(Lanes<G>(), form, 0, 2 * left > NG ? nr : whole);
            if (!CACHED && left > 0 && 2 * left <= NG) {
                if (4 * left <= NG) rows(Lanes<4 * kTileLanes>(), form, whole, nr);
                else rows(Lanes<2 * kTileLanes>(), form, whole, nr);
            }
        };
        if constexpr (CACHED) all_rows(std::false_type());
        else if (fixed) all_rows(std::true_type());
        else all_rows(std::false_type());
        if (!exchange_sum(ex, acc.v, pAp, G, A, ++epoch, [](int, int) {})) return false;
        alpha = df_quotient(rz, pAp);
        if (timed) {
            const unsigned long long t = now_ns();
            ns_spmv += t - t_mark;
            t_mark = t;
        }
        // ---- x += alpha p ; r -= alpha A p, by the lanes that formed the rows
        ++epoch;
        const unsigned tag = (unsigned)epoch;
        DotAcc32 rr;
        if (lane == 0) {
            for (int i = threadIdx.x / G; i < nr; i += NG) {
                const float4 pv = sp[i], yv = sy[i];
                float4 xv = sx[i], rv = sr[i];
                xv.x += alpha * pv.x; xv.y += alpha * pv.y; xv.z += alpha * pv.z;
                rv.x -= alpha * yv.x; rv.y -= alpha * yv.y; rv.z -= alpha * yv.z;
                sx[i] = xv;
                sr[i] = rv;
                publish(A.rec + lo + i, pack(DF{rv.y, rv.x}), ((unsigned long long)tag << 32) | __float_as_uint(rv.z));
                rr.fma(rv.x, rv.x);
                rr.fma(rv.y, rv.y);
                rr.fma(rv.z, rv.z);
            }
        }
        const auto gather = [&](int t, int threads) {   // the halo's new r
            for (int h = t; h < nh; h += threads) {
                ulonglong2 v;
                if (!await(A.rec + sq[h], A.error, A.wait_ns, ex, v, [tag](const ulonglong2& x) { return (unsigned)(x.y >> 32) == tag; }))
                    return;
                const DF yx = unpack<DF>(v.x);
                sh[h] = make_float4(yx.lo, yx.hi, __uint_as_float((unsigned)v.y), 0.f);
            }
        };
        DF total;
        if (!exchange_sum(ex, rr.v, total, G, A, epoch, gather)) return false;
        beta = df_quotient(total, rz);
        rz = total;
        ++iter;
        if (!(total.hi > tol2_far)) converged = below_tolerance(to_double(ex.total), tol);
        done = converged || iter >= max_iter;
        if (timed) ns_vec += now_ns() - t_mark;
    }
    for (int t = threadIdx.x; t < nr; t += kPersistThreads) {
        ((float4*)S.sol)[lo + t] = sx[t];
        ((float4*)S.r)[lo + t] = sr[t];
        ((float4*)S.p)[lo + t] = sp[t];
    }
    if (A.block == 0 && threadIdx.x == 0) {
        sc->pAp = df_to_double(pAp);
        sc->rz = to_double(ex.total);
        sc->alpha = alpha;
        sc->beta = beta;
        sc->rnorm = sqrt(sc->rz);
        sc->iter = iter;
        sc->converged = converged;
        sc->done = done;
        sc->ns_spmv = (double)ns_spmv;
        sc->ns_vec = (double)ns_vec;
    }
    return true;
}

template <bool CACHED, int G, int U>
__global__ void __launch_bounds__(kPersistThreads, 1) k_cg_persist32(PersistArgs A)
{
    extern __shared__ __align__(32) unsigned char smem[];
    __shared__ Exchange ex;
    unsigned long long epoch = A.epoch;
    const PersistRun run = persist_run(A);
    if (!persist_solve32<CACHED, G, U>(A.P, A.S, run, smem, ex, epoch, A.profile && blockIdx.x == 0 && threadIdx.x == 0)) return;
    if (A.finish) {
        __syncthreads();   // the block's rows of the solution
        const int lo = blockIdx.x * A.rows, hi = min(A.P.n, lo + A.rows);
        for (int r = lo + (int)threadIdx.x; r < hi; r += kPersistThreads) update_elem<false>(A.P, A.S, r);
    }
}

// One product y = A w outside a solve by the same rows and halos, bonds read as
// the uncached solve reads them, and bound like it.  The gather product, whose
// every bond reads two 16-byte records through L1, takes 35.3 us at 100k
// particles of 76 bonds, this one 26.7.
template <bool DOT>
__global__ void __launch_bounds__(kTileBlock, 1)
    k_tile_product32(StepParams P, DeviceState S, int rows, int halo, const float4* __restrict__ in,
                     float4* __restrict__ out, ReduceSlot slot, CgScalars* cg, double* dot_out)
{
    if (DOT && cg && ((volatile CgScalars*)cg)->done) return;
    constexpr int G = kTileLanes;
    extern __shared__ __align__(32) unsigned char smem[];
    float4* sw = (float4*)smem;
    float4* shx = sw + halo;
    const int lo = blockIdx.x * rows;
    const int nr = min(rows, P.n - lo);
    // a row's own data and its first bonds, in flight while the halo is staged
    // (the block's later rows: while the row before them is finished)
    int rs = 0, cn = -1, l[4];
    float id0[4];
    uint8_t ab = 0;
    float4 w, xp;
    const auto fetch = [&](int i, int end, int lane) {
        if (i >= end) return;
        const int p = lo + i;
        rs = __ldg(S.row_ptr + p);
        cn = S.cnt[p];
        ab = S.act[p];
        w = __ldg(in + p);
        xp = __ldg(S.xs4 + p);
        if (is_dirichlet(ab & kActMask)) cn = -1;
        if (lane * 4 < cn) load_bonds(S, rs + lane * 4, l, id0);
    };
    // (the rows left over from whole rounds: with more lanes each, as in the solve)
    constexpr int NG = kTileBlock / G;
    const int left = nr % NG, whole = 2 * left > NG ? nr : nr - left;
    if (whole > 0) fetch(threadIdx.x / G, whole, threadIdx.x & (G - 1));
    const int h0 = S.halo_ptr[blockIdx.x], nh = S.halo_ptr[blockIdx.x + 1] - h0;
    const float sup = (float)P.sup, per_edge = (float)(1 << kFixedBits) / sup;
    const int ref = nr > 0 ? __float_as_int(__ldg(S.xs4 + lo).w) : 0;
    bool far = false;
    for (int t = threadIdx.x; t < nr; t += kTileBlock) far |= farther(__ldg(S.xs4 + lo + t), ref, sup);
    for (int h = threadIdx.x; h < nh; h += kTileBlock) {
        const int q = __ldg(S.halo + h0 + h);
        const float4 X = __ldg(S.xs4 + q);
        const float4 w = __ldg(in + q);
        sw[h] = w;
        // (the fixed-point form takes 0 times w for a slot without a live bond, so a
        // block that reads a w that is not finite keeps to the other, which skips it)
        far |= farther(X, ref, sup) || !(fabsf(w.x) + fabsf(w.y) + fabsf(w.z) < INFINITY);
        shx[h] = fixed_position(X, per_edge);
    }
    const bool fixed = !__syncthreads_or(far);
    if (!fixed) {
        for (int h = threadIdx.x; h < nh; h += kTileBlock) shx[h] = __ldg(S.xs4 + __ldg(S.halo + h0 + h));
        __syncthreads();
    }
    DotAcc32 acc;
    const auto tile_rows = [&](auto width, auto form, int from, int to) {
        constexpr int R = decltype(width)::value;
        constexpr bool FIXED = decltype(form)::value;
        const int lane = threadIdx.x & (R - 1);
        const unsigned gmask = group_mask<R>();
        if (from > 0 || R != G) fetch(from + threadIdx.x / R, to, lane);
        for (int i = from + threadIdx.x / R; i < to; i += kTileBlock / R) {
            float ax = 0.f, ay = 0.f, az = 0.f;
            const float4 x = FIXED ? fixed_position(xp, per_edge) : xp;
            for (int j0 = lane * 4; j0 < cn; j0 += R * 4) {
                int lc[4];
                float ic[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    lc[u] = l[u];
                    ic[u] = id0[u];
                }
                if (j0 + R * 4 < cn) load_bonds(S, rs + j0 + R * 4, l, id0);   // in flight while this step's bonds are added
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (!FIXED && j0 + u >= cn) continue;
                    const float4 Wq = sw[lc[u]];
                    float a1;
                    BondGeometry g;
                    if constexpr (FIXED) g = bond_geometry_fixed(shx[lc[u]], x, per_edge, ic[u], a1);
                    else g = bond_geometry(shx[lc[u]], x, sup, ic[u], a1);
                    if (FIXED && j0 + u >= cn) a1 = g.i3 = 0.f;
                    const float wx = w.x - Wq.x, wy = w.y - Wq.y, wz = w.z - Wq.z;
                    const float d = fmaf(g.x, wx, fmaf(g.y, wy, g.z * wz)) * g.i3;
                    ax = fmaf(a1, wx, fmaf(d, g.x, ax));
                    ay = fmaf(a1, wy, fmaf(d, g.y, ay));
                    az = fmaf(a1, wz, fmaf(d, g.z, az));
                }
            }
            const int p = lo + i;
            const uint8_t row_ab = ab;
            const float4 row_w = w;
            const bool fixed = cn < 0;
            fetch(i + kTileBlock / R, to, lane);
            if (!fixed) spmv_finish_mixed<R, DOT>(P, S, p, row_ab, row_w, ax, ay, az, lane, gmask, out, acc);
            else if (lane == 0) out[p] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    const auto all_rows = [&](auto form) {
        tile_rows(Lanes<G>(), form, 0, whole);
        if (whole < nr) {
            if (4 * left <= NG) tile_rows(Lanes<4 * G>(), form, whole, nr);
            else tile_rows(Lanes<2 * G>(), form, whole, nr);
        }
    };
    if (fixed) all_rows(std::true_type());
    else all_rows(std::false_type());
    if (DOT)
        block_reduce_finish(acc, slot, [cg, dot_out](double pAp) {
            if (cg) cg_fin_alpha(cg, pAp);
            if (dot_out) *dot_out = pAp;
        });
}

struct __align__(8) Vec3d {
    double x, y, z;
};

// FP64, G lanes per row (at least 4), U bonds in flight per lane.  The product
// is bound by the FP64 pipe (1.7 multiply-adds per cycle and SM measured, 9 per
// bond).
template <bool CACHED, int G, int U>
__global__ void __launch_bounds__(kPersistThreads, 1) k_cg_persist64(PersistArgs A)
{
    CgScalars* sc = A.S.sc;
    if (__syncthreads_or(((volatile CgScalars*)sc)->wait_error) || (!A.start && ((volatile CgScalars*)sc)->done)) return;
    extern __shared__ __align__(32) unsigned char smem[];
    __shared__ Exchange ex;
    const PersistRun run = persist_run(A);
    __shared__ double s_alpha, s_beta, s_rz;
    __shared__ int s_done, s_converged;
    const StepParams& P = A.P;
    const DeviceState& S = A.S;
    const int lo = blockIdx.x * A.rows;
    const int nr = min(A.rows, P.n - lo);
    double2* sJ = (double2*)smem;                        // three per bond: xx yy | zz xy | xz yz
    Vec3d* sx = (Vec3d*)(sJ + 3 * (size_t)A.bonds);
    Vec3d* sr = sx + A.rows;
    Vec3d* sp = sr + A.rows;
    Vec3d* sy = sp + A.rows;
    Vec3d* sw = sy + A.rows;                             // the halo's p
    Vec3d* sh = sw + A.halo;                             // the halo's r
    int* srow = (int*)(sh + A.halo);
    int* scnt = srow + A.rows;
    int* sq = scnt + A.rows;
    uint16_t* sl = (uint16_t*)(sq + A.halo);

    const int lane = threadIdx.x & (G - 1);
    const unsigned gmask = group_mask<G>();
    constexpr int NG = kPersistThreads / G;
    const int slot0 = CACHED ? S.row_ptr[lo] : 0;
    double first = 0.0;   // <r, r> of the guess
    const auto load3 = [](const void* v, int p) {
        const dbl4 a = ((const dbl4*)v)[p];
        return Vec3d{a.x, a.y, a.z};
    };
    for (int t = threadIdx.x; t < nr; t += kPersistThreads) {
        const int p = lo + t;
        sx[t] = load3(S.sol, p);
        if (A.start) {
            const dbl4 r = first_residual<dbl4>(S, p);
            sr[t] = Vec3d{r.x, r.y, r.z};
            sp[t] = sr[t];
            first = fma(r.x, r.x, fma(r.y, r.y, fma(r.z, r.z, first)));
        } else {
            sr[t] = load3(S.r, p);
            sp[t] = load3(S.p, p);
        }
        scnt[t] = is_dirichlet(S.act[p] & kActMask) ? -1 : S.cnt[p];
        srow[t] = S.row_ptr[p] - slot0;
    }
    const int h0 = S.halo_ptr[blockIdx.x], nh = S.halo_ptr[blockIdx.x + 1] - h0;
    for (int h = threadIdx.x; h < nh; h += kPersistThreads) {
        const int q = S.halo[h0 + h];
        sq[h] = q;
        if (A.start) {
            const dbl4 r = first_residual<dbl4>(S, q);
            sh[h] = Vec3d{r.x, r.y, r.z};
            sw[h] = sh[h];
        } else {
            sw[h] = load3(S.p, q);
            sh[h] = load3(S.r, q);
        }
    }
    if (threadIdx.x == 0) {
        ex.error = 0;
        s_rz = sc->rz;
        s_beta = A.start ? 0.0 : sc->beta;
        s_done = 0;
        s_converged = 0;
    }
    __syncthreads();
    if (CACHED) {
        for (int i = threadIdx.x / G; i < nr; i += NG) {
            const int cn = scnt[i], base = srow[i];
            for (int j = lane; j < cn; j += G) {
                const double2* J = (const double2*)(S.jac + 6ll * (slot0 + base + j));
                sJ[3 * (base + j)] = J[0];
                sJ[3 * (base + j) + 1] = J[1];
                sJ[3 * (base + j) + 2] = J[2];
                sl[base + j] = S.lidx[slot0 + base + j];
            }
        }
    }
    const double tol = sc->tol;
    const int max_iter = sc->max_iter;
    int iter = sc->iter;

    unsigned long long epoch = A.epoch;
    if (A.start) {
        __syncthreads();   // (s_rz and s_done before thread 0 sets them again)
        if (!exchange_sum(ex, first, first, 1, run, ++epoch, [](int, int) {})) return;
        if (threadIdx.x == 0) {
            s_rz = first;
            s_converged = below_tolerance(first, tol);
            s_done = s_converged || iter >= max_iter;
        }
        __syncthreads();
    }
    unsigned long long t_mark = 0, ns_spmv = 0, ns_vec = 0;
    const bool timed = A.profile && blockIdx.x == 0 && threadIdx.x == 0;
    double pAp = 0.0;
    const auto next_p = [](const Vec3d& r, const Vec3d& p, double beta) {
        return Vec3d{r.x + beta * p.x, r.y + beta * p.y, r.z + beta * p.z};
    };
    for (int it = 0; it < A.max_iters && !s_done; ++it) {
        if (timed) t_mark = now_ns();
        const double beta = s_beta;
        for (int h = threadIdx.x; h < nh; h += kPersistThreads) sw[h] = next_p(sh[h], sw[h], beta);
        for (int t = threadIdx.x; t < nr; t += kPersistThreads) sp[t] = next_p(sr[t], sp[t], beta);
        __syncthreads();
        double acc = 0.0;
        for (int i = threadIdx.x / G; i < nr; i += NG) {
            const int cn = scnt[i], base = srow[i], p = lo + i;
            double ax = 0, ay = 0, az = 0;
            for (int j0 = lane; j0 < cn; j0 += G * U) {
                int l[U];
                double2 J[U][3];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int j = j0 + u * G;
                    if (j < cn) {
                        l[u] = CACHED ? sl[base + j] : __ldg(S.lidx + base + j);
                        const double2* s = CACHED ? sJ + 3 * (base + j) : (const double2*)(S.jac + 6ll * (base + j));
#pragma unroll
                        for (int k = 0; k < 3; ++k) J[u][k] = CACHED ? s[k] : __ldg(s + k);
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (j0 + u * G >= cn) continue;
                    const Vec3d w = sw[l[u]];
                    const double2 a = J[u][0], b = J[u][1], c = J[u][2];
                    ax = fma(a.x, w.x, fma(b.y, w.y, fma(c.x, w.z, ax)));
                    ay = fma(b.y, w.x, fma(a.y, w.y, fma(c.y, w.z, ay)));
                    az = fma(c.x, w.x, fma(c.y, w.y, fma(b.x, w.z, az)));
                }
            }
            if (cn < 0) {
                if (lane < 3) ((double*)(sy + i))[lane] = 0.0;
                continue;
            }
            const double s = component_sum<G>(ax, ay, az, lane, gmask);
            if (lane < 3) {
                const Vec3d w = sp[i];
                double wk;
                const double y = fp64_row_result(P, S, p, lane, w.x, w.y, w.z, s, wk);
                ((double*)(sy + i))[lane] = y;
                acc = fma(wk, y, acc);
            }
        }
        if (!exchange_sum(ex, acc, pAp, 1, run, ++epoch, [](int, int) {})) return;
        if (threadIdx.x == 0) s_alpha = s_rz / pAp;
        __syncthreads();
        if (timed) {
            const unsigned long long t = now_ns();
            ns_spmv += t - t_mark;
            t_mark = t;
        }
        ++epoch;
        const unsigned tag = (unsigned)epoch;
        const double alpha = s_alpha;
        double rr = 0.0;
        for (int t = threadIdx.x; t < nr; t += kPersistThreads) {
            const Vec3d pv = sp[t], yv = sy[t];
            Vec3d xv = sx[t], rv = sr[t];
            xv.x += alpha * pv.x; xv.y += alpha * pv.y; xv.z += alpha * pv.z;
            rv.x -= alpha * yv.x; rv.y -= alpha * yv.y; rv.z -= alpha * yv.z;
            sx[t] = xv;
            sr[t] = rv;
            // 24 bytes and the tag in two records: (x, y low), (z, y high)
            const unsigned long long y = (unsigned long long)__double_as_longlong(rv.y), hi = (unsigned long long)tag << 32;
            ulonglong2* rec = A.rec + 2 * (size_t)(lo + t);
            publish(rec, pack(rv.x), hi | (y & 0xffffffffull));
            publish(rec + 1, pack(rv.z), hi | (y >> 32));
            rr = fma(rv.x, rv.x, fma(rv.y, rv.y, fma(rv.z, rv.z, rr)));
        }
        const auto gather = [&](int t, int threads) {
            const auto arrived = [tag](const ulonglong2& x) { return (unsigned)(x.y >> 32) == tag; };
            for (int h = t; h < nh; h += threads) {
                const ulonglong2* rec = A.rec + 2 * (size_t)sq[h];
                ulonglong2 a, b;
                if (!await(rec, run.error, run.wait_ns, ex, a, arrived) ||
                    !await(rec + 1, run.error, run.wait_ns, ex, b, arrived))
                    return;
                sh[h] = Vec3d{unpack<double>(a.x), unpack<double>((b.y << 32) | (a.y & 0xffffffffull)), unpack<double>(b.x)};
            }
        };
        if (!exchange_sum(ex, rr, rr, 1, run, epoch, gather)) return;
        ++iter;
        if (threadIdx.x == 0) {
            s_beta = rr / s_rz;
            s_rz = rr;
            s_converged = below_tolerance(rr, tol);
            s_done = s_converged || iter >= max_iter;
        }
        __syncthreads();
        if (timed) ns_vec += now_ns() - t_mark;
    }
    for (int t = threadIdx.x; t < nr; t += kPersistThreads) {
        ((dbl4*)S.sol)[lo + t] = make_dbl4(sx[t].x, sx[t].y, sx[t].z, 0.0);
        ((dbl4*)S.r)[lo + t] = make_dbl4(sr[t].x, sr[t].y, sr[t].z, 0.0);
        ((dbl4*)S.p)[lo + t] = make_dbl4(sp[t].x, sp[t].y, sp[t].z, 0.0);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        sc->pAp = pAp;
        sc->rz = s_rz;
        sc->alpha = s_alpha;
        sc->beta = s_beta;
        sc->rnorm = sqrt(s_rz);
        sc->iter = iter;
        sc->converged = s_converged;
        sc->done = s_done;
        sc->ns_spmv = (double)ns_spmv;
        sc->ns_vec = (double)ns_vec;
    }
    if (A.finish) {
        __syncthreads();   // the block's rows of the solution
        for (int t = threadIdx.x; t < nr; t += kPersistThreads) update_elem<true>(P, S, lo + t);
    }
}

// The solves and updates of a batch's scenes (batch.h) in one cooperative launch.
// The blocks form gangs of A.gang; a gang takes the next scene of the list
// (largest first) when it has finished one, solves it as k_cg_persist32 does, and
// advances its rows.  Scenes meet no barrier of other scenes, and each runs only
// its own iterations.  Every block of a gang takes part in every exchange, so
// the epochs of its inbox go on from scene to scene; which scene comes next is
// a record of its own per turn.  Against phases of all scenes between grid
// barriers (k_batch_cg): 12 steps of 24 bodies of 4k to 24k particles take 81.5 ms
// against 208.5, of 8 of 1k to 4k 10.7 against 65.9.
__global__ void __launch_bounds__(kPersistThreads, 1) k_gang_solve32(GangArgs A)
{
    extern __shared__ __align__(32) unsigned char smem[];
    __shared__ Exchange ex;
    __shared__ int s_turn;
    const int gang = blockIdx.x / A.gang, block = blockIdx.x % A.gang;
    ulonglong2* inbox = A.inbox + (size_t)gang * 2 * A.gang * A.gang;
    ulonglong2* turns = A.turns + (size_t)gang * (A.n_scenes + 1);
    unsigned long long epoch = 0;
    for (int turn = 0; turn <= A.n_scenes; ++turn) {
        if (threadIdx.x == 0) {
            if (block == 0) {
                const int i = atomicAdd(A.next, 1);
                s_turn = i < A.n_scenes ? A.order[i] : A.n_scenes;
                publish(turns + turn, (unsigned long long)s_turn, 1ull);
            } else {
                ulonglong2 r;
                s_turn = await(turns + turn, A.error, A.wait_ns, ex, r, [](const ulonglong2& x) { return x.y == 1ull; })
                             ? (int)r.x
                             : A.n_scenes;
            }
        }
        __syncthreads();
        const int scene = s_turn;
        __syncthreads();
        if (scene >= A.n_scenes) return;
        SceneRun& R = A.run[scene];
        if (!*(volatile int*)&R.solving) continue;
        const SceneDesc& D = A.scenes[scene];
        const GangScene g = A.plan[scene];
        const StepParams P = D.P;
        const DeviceState S = D.S;
        const PersistRun run{A.rec + g.rec, inbox, g.rows, g.halo, g.bonds, 0x7fffffff, block, A.gang, false, A.error, A.wait_ns};
        bool ok;
        if (g.bonds == 0) ok = persist_solve32<false, kTileLanes, 4>(P, S, run, smem, ex, epoch, false);
        else if (g.lanes == 4) ok = persist_solve32<true, 4, 4>(P, S, run, smem, ex, epoch, false);
        else if (g.lanes == 8) ok = persist_solve32<true, 8, 4>(P, S, run, smem, ex, epoch, false);
        else if (g.lanes == 16) ok = persist_solve32<true, 16, 4>(P, S, run, smem, ex, epoch, false);
        else ok = persist_solve32<true, 32, 2>(P, S, run, smem, ex, epoch, false);
        if (!ok) return;
        __syncthreads();   // the block's rows of the solution
        const int lo = block * g.rows, hi = min(P.n, lo + g.rows);
        for (int r = lo + (int)threadIdx.x; r < hi; r += kPersistThreads) update_elem<false>(P, S, r);
        if (block == 0 && threadIdx.x == 0) {
            const volatile CgScalars* sc = S.sc;
            R.last_iters = sc->iter;
            R.total_iters += sc->iter;
            R.last_res = sc->rnorm;
            R.last_tol = sc->tol;
            if (!sc->converged) R.cg_converged = 0;
            R.sim_time += P.h;
        }
    }
}

size_t persist_smem(bool fp64, int rows, int halo, int bonds)
{
    const size_t v = fp64 ? sizeof(Vec3d) : sizeof(float4);
    const size_t bond = (fp64 ? 6 * sizeof(double) : sizeof(BondGeometry) + sizeof(float)) + sizeof(uint16_t);
    return (4 * v + 2 * sizeof(int)) * rows + (v * (fp64 || bonds > 0 ? 2 : 3) + sizeof(int)) * halo + bond * (size_t)bonds;
}

const void* persist_kernel32(const CgPersistPlan& pl)
{
    if (pl.bonds == 0) return (const void*)k_cg_persist32<false, kTileLanes, 4>;
    switch (pl.lanes) {
    case 4: return (const void*)k_cg_persist32<true, 4, 4>;
    case 8: return (const void*)k_cg_persist32<true, 8, 4>;
    case 16: return (const void*)k_cg_persist32<true, 16, 4>;
    default: return (const void*)k_cg_persist32<true, 32, 2>;
    }
}

template <bool CACHED>
const void* persist_kernel64(int lanes)
{
    switch (lanes) {
    case 4: return (const void*)k_cg_persist64<CACHED, 4, 4>;
    case 8: return (const void*)k_cg_persist64<CACHED, 8, 4>;
    case 16: return (const void*)k_cg_persist64<CACHED, 16, 4>;
    default: return (const void*)k_cg_persist64<CACHED, 32, 2>;
    }
}

const void* persist_kernel(bool fp64, const CgPersistPlan& pl)
{
    if (!fp64) return persist_kernel32(pl);
    return pl.bonds > 0 ? persist_kernel64<true>(pl.lanes) : persist_kernel64<false>(pl.lanes);
}

// Dynamic shared memory that a block can have in the solves and in the products by
// tiles.  A kernel's limit is an attribute of the kernel, not of a handle: it is
// always set to this same value, so that no handle, in this thread or another,
// lowers it below what another one launches with (or holds in a captured graph).
int room_less(size_t fixed, int device)
{
    int optin = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    return optin - (int)fixed;
}
int persist_room(int device) { return room_less(sizeof(Exchange) + 1024, device); }
int tile_room(int device) { return room_less(2048, device); }

bool set_tile_room(int device)
{
    for (const void* t : {(const void*)k_tile_product32<true>, (const void*)k_tile_product32<false>})
        if (cudaFuncSetAttribute(t, cudaFuncAttributeMaxDynamicSharedMemorySize, tile_room(device)) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
    return true;
}

}  // namespace

CgPersistPlan cg_persist_rows(bool fp64, int n, int sm_count, int device)
{
    CgPersistPlan pl{};
    int coop = 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device);
    if (!coop || n <= 0 || n > kPersistMaxRows) return pl;
    const int most = std::min(sm_count, kPersistMaxGrid);
    // An exchange costs 1.2 us among 64 blocks and 1.8 among 152, so mixed
    // precision spreads thin only down to 32 rows per block: 4096 particles
    // take 6.0 us per iteration at 32 rows, 6.7 at 27 (152 blocks) and 8.6 at
    // 64; 512 take 5.2 (5.5 at 4 rows).  FP64, bound by its pipe, goes down to
    // 8 rows: 3000 particles take 15.0 us at 20 rows and 17.1 at 32.
    pl.rows = std::max(fp64 ? 8 : 32, (n + most - 1) / most);
    pl.grid = (n + pl.rows - 1) / pl.rows;
    return pl;
}

bool cg_persist_plan(bool fp64, int max_halo, int max_bonds, int device, CgPersistPlan* plan)
{
    CgPersistPlan pl = *plan;
    const int room = persist_room(device);
    pl.halo = max_halo;
    const long long bonds = (long long)pl.rows * ((max_bonds + 7) / 8 * 8);
    pl.bonds = bonds < (1 << 20) && persist_smem(fp64, pl.rows, pl.halo, (int)bonds) <= (size_t)room ? (int)bonds : 0;
    pl.smem = persist_smem(fp64, pl.rows, pl.halo, pl.bonds);
    if (pl.smem > (size_t)room) return false;
    // a cached row is spread over as many lanes as one pass of the block allows
    pl.lanes = 32;
    while (pl.lanes > 4 && kPersistThreads / pl.lanes < pl.rows) pl.lanes /= 2;
    pl.tiled_products = !fp64 && pl.bonds == 0;
    if (pl.tiled_products) pl.lanes = kTileLanes;
    const void* k = persist_kernel(fp64, pl);
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, room) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kPersistThreads, pl.smem);
    if (per_sm < 1) return false;
    if (pl.tiled_products && !set_tile_room(device)) return false;
    *plan = pl;
    return true;
}

bool tile_product_may_fit(int rows, double reach, int device)
{
    const double side = std::cbrt((double)rows) + 2.0 * reach;
    return 2 * sizeof(float4) * side * side * side <= (double)tile_room(device);
}

bool tile_product_plan(int max_halo, int device, CgPersistPlan* plan)
{
    if (2 * sizeof(float4) * (size_t)max_halo > (size_t)tile_room(device) || !set_tile_room(device)) return false;
    plan->halo = max_halo;
    return true;
}

bool cg_persist_may_fit(int rows, double reach, int device)
{
    const double side = std::cbrt((double)rows) + 2.0 * reach;   // a compact block of rows and its halo
    return persist_smem(false, rows, (int)std::min(side * side * side, 1e6), 0) <= (size_t)persist_room(device);
}

cudaError_t gang_solve_prepare(int device)
{
    return cudaFuncSetAttribute((const void*)k_gang_solve32, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                persist_room(device));
}

cudaError_t launch_gang_solve(const GangArgs& A, int gangs, size_t smem, cudaStream_t st)
{
    GangArgs a = A;
    void* args[] = {&a};
    return cudaLaunchCooperativeKernel((const void*)k_gang_solve32, dim3(gangs * A.gang), dim3(kPersistThreads), args, smem, st);
}

cudaError_t launch_tile_product(const StepParams& P, const DeviceState& S, const CgPersistPlan& plan, const void* in,
                                void* out, ReduceSlot slot, CgScalars* cg, double* dot_out, cudaStream_t st)
{
    StepParams p = P;
    DeviceState s = S;
    int rows = plan.rows, halo = plan.halo;
    void* args[] = {&p, &s, &rows, &halo, &in, &out, &slot, &cg, &dot_out};
    const void* k = cg || dot_out ? (const void*)k_tile_product32<true> : (const void*)k_tile_product32<false>;
    return cudaLaunchKernel(k, dim3(plan.grid), dim3(kTileBlock), args, 2 * sizeof(float4) * (size_t)plan.halo, st);
}

cudaError_t launch_cg_persist(bool fp64, const StepParams& P, const DeviceState& S, const CgPersistPlan& plan,
                              ulonglong2* rec, ulonglong2* inbox, unsigned long long epoch, int max_iters, bool profile,
                              bool start, bool finish, unsigned long long wait_ns, cudaStream_t st)
{
    PersistArgs A{P, S, rec, inbox, epoch, plan.rows, plan.halo, plan.bonds, max_iters, profile ? 1 : 0, start ? 1 : 0,
                  finish ? 1 : 0, wait_ns};
    void* args[] = {&A};
    return cudaLaunchCooperativeKernel(persist_kernel(fp64, plan), dim3(plan.grid), dim3(kPersistThreads), args, plan.smem,
                                       st);
}

}  // namespace pdgb
