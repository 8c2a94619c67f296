// h2gpu_ulv.cu -- the ULV solve of an HSS matrix on the device (include/h2gpu.h,
// h2gpu_ulv_*).
//
// The reference solves level by level on the host (H2P_HSS_ULV_Cholesky_solve,
// src/H2Pack_HSS_ULV.c:981-1159; H2P_HSS_ULV_LU_solve, :429-599).  Per node it gathers
// the node's entries of the permuted vector, applies Q^T (or Q), solves with the
// node's triangular factor, updates with the off-diagonal part of the factor and
// scatters back.  Nodes of one level touch disjoint entries, so here each level of a
// sweep is one launch over all its nodes:
//
//   Cholesky, first sweep (levels max .. 0)   b = Q^T b;  b2 = L22 \ b2;  b1 -= L12 b2
//   Cholesky, second sweep (levels 0 .. max)  b2 -= L12^T b1;  b2 = L22^T \ b2;  b = Q b
//   LU, first sweep (levels max .. 0)         b = Q^T b;  b2 = b2(p);  b2 = L0 \ b2 (unit);
//                                             b1 -= DU12 b2
//   LU, second sweep (levels 0 .. max)        b2 -= LD21 b1;  b2 = U0 \ b2;  b = Q b
//
// with b1 / b2 the first Ls / last m - Ls entries and L12, L22, DU12, LD21, L0, U0 the
// blocks of the node's m x m factor.  The root (level 0) has no Q and Ls = 0.
//
// Layout.  Q is kept explicitly (m x m per node, stored as Q^T row-major, i.e. row r
// = column r of Q), formed once from the reflectors at create by k_ulv_form_q, so
// that Q^T b and Q b are plain products instead of a chain of k dependent reflector
// steps; L as H2Pack stores it (m x m row-major).
// FP64 throughout; every sum has a fixed order, so results are deterministic.
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <vector>

#include <cuda_runtime.h>

#include "h2gpu.h"

#define H2G_API extern "C" __attribute__((visibility("default")))

namespace h2gpu {
int set_error(int code, const char* msg);
}

namespace {

constexpr int kUT = 256, kUW = kUT / 32;   // threads and warps of a CTA
constexpr int kB = 64;                     // rows / columns of a unit
constexpr int kDS = kB + 4;                // column stride of a diagonal block in shared memory (apply_diag:
                                           // conflict-free)
constexpr int kMaxNodeRows = 13872;        // larger nodes are refused: the interface's limit (a Q
                                           // product would hold some 19,700 in shared memory)
constexpr unsigned kFull = 0xffffffffu;
constexpr int kPollLimit = 1 << 22;        // polls (a few seconds) before a wait gives up; looked at
                                           // every 2^16 polls
// Largest || |M| |M^-1| || of a diagonal block M that is solved with its inverse E.  One step of
// refinement leaves a residual of about (128 u || |M| |E| ||)^2 of the block's right-hand
// side beside the rounding that substitution has too (u = 2^-53): 2e-18 at this bound.
constexpr double kInverseMax = 1e5;

struct UlvNode {
    long long q_off;     // Q^T (m x m row-major) in the Q arena; -1: no Q
    long long l_off;     // L (m x m row-major) in the L arena
    long long idx_off;   // m indices into the permuted vector, m entries of the tagged vectors
    long long p_off;     // LU: m - I pivots; -1: none
    long long d_off;     // inverses of the diagonal blocks of the triangular factor (64 x 64
                         // row-major each); LU: of L0, then of U0.  Block at d_off + k 64^2 has
                         // its flag at index d_off / 64^2 + k: 1 is solved by substitution
    int m, I, pad0, pad1;
};

// diagonal block at (I + at, I + at) of a node's factor, its inverse at d_off
struct UlvDiagJob {
    long long d_off;
    int node, at, upper, unit;
};

struct UlvQJob {
    long long v_off;     // k reflectors of length m, reflector j at v + j m (1 at j,
                         // zeros above), then tau (k entries)
    long long q_off;
    int m, k, pad0, pad1;
};

enum { CH_UP = 0, CH_DOWN = 1, LU_UP = 2, LU_DOWN = 3 };

// One level of one sweep is a list of units of 64 rows (or columns), each depending on
// units before it in the list only.  CTAs take the units in list order from a counter, so
// a unit that another one waits for is always running or done: no co-residency of the
// whole grid is needed.
//   U_QT    64 rows of Q^T b
//   U_TRI   64 rows of the triangular solve: their product with the solved blocks (the
//           second sweep: and with b1) as those are published, then the diagonal block
//   U_OFF   64 rows of b1 -= L12 b2 (first sweep)
//   U_Q     64 columns of Q^T, i.e. 64 entries of Q b (second sweep)
//   U_PUT   scatter of a node's results, once all of them are published (every unit of
//           the node has read its inputs by then)
enum { U_QT = 0, U_TRI = 1, U_OFF = 2, U_Q = 3, U_PUT = 4 };
struct UlvUnit {
    int node, type, at;   // at: first row / column of the unit
};

// A published entry: value and tag in one 16-byte word, written and read by single
// accesses, so that a reader needs neither a flag nor a fence.  Tag 0: not there yet
// (cleared at the start of every solve).
struct __align__(16) Tagged {
    unsigned long long v, t;
};

__device__ __forceinline__ void tag_put(Tagged* p, double x)
{
    asm volatile("{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], q;\n\t}" ::"l"(p),
                 "l"(__double_as_longlong(x)), "l"(1ull)
                 : "memory");
}
__device__ __forceinline__ Tagged tag_get(const Tagged* p)
{
    Tagged r;
    asm volatile("{\n\t.reg .b128 q;\n\tld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
                 : "=l"(r.v), "=l"(r.t)
                 : "l"(p)
                 : "memory");
    return r;
}
// the value of an entry whose first read gave r; a wait that runs out sets the status word
// and returns zero, and every later wait then gives up soon
__device__ __forceinline__ double tag_wait(const Tagged* p, Tagged r, int* status, int limit)
{
    for (int n = 1; r.t == 0; n++)
    {
        if ((n & 0xffff) == 0 && (n >= limit || *(volatile int*) status != 0))
        {
            *(volatile int*) status = 1;
            return 0.0;
        }
        r = tag_get(p);
    }
    return __longlong_as_double(r.v);
}

// Input vectors of a product: published entries, or plain memory through an index list,
// or shared memory.  issue() starts the read of entry c, wait() gives its value.
struct InTagged {
    const Tagged* x;
    int* status;
    int limit;
    using R = Tagged;
    __device__ R issue(int c) const { return tag_get(x + c); }
    __device__ double wait(int c, R r) const { return tag_wait(x + c, r, status, limit); }
    // entries c0 and c1 (those below n) together: one round trip where both are new
    __device__ void wait2(int c0, int c1, int n, R r0, R r1, double& v0, double& v1) const
    {
        if (c0 >= n) return;
        const bool two = c1 < n;
        for (int k = 1; r0.t == 0 || (two && r1.t == 0); k++)
        {
            if ((k & 0xffff) == 0 && (k >= limit || *(volatile int*) status != 0))
            {
                *(volatile int*) status = 1;
                return;
            }
            r0 = tag_get(x + c0);
            if (two) r1 = tag_get(x + c1);
        }
        v0 = __longlong_as_double(r0.v);
        if (two) v1 = __longlong_as_double(r1.v);
    }
};
struct InIndexed {
    const double* px;
    const int* idx;
    using R = double;
    __device__ R issue(int c) const { return px[idx[c]]; }
    __device__ double wait(int, R r) const { return r; }
    __device__ void wait2(int, int, int, R r0, R r1, double& v0, double& v1) const { v0 = r0; v1 = r1; }
};
struct InShared {
    const double* x;
    using R = double;
    __device__ R issue(int c) const { return x[c]; }
    __device__ double wait(int, R r) const { return r; }
    __device__ void wait2(int, int, int, R r0, R r1, double& v0, double& v1) const { v0 = r0; v1 = r1; }
};

// acc[k] += sum_c A[row][c] x[c] over the 64-column tiles t0, t0 + dt, .. (cnt of them) of nc
// columns, row = 8 warp + k of nr: a lane owns columns c and c + 32 of a tile and eight
// rows, its sums stay in registers over all tiles.  The entries of the next half tile are
// in flight while a half is multiplied, both halves' inputs are awaited together.
template <typename IN>
__device__ __forceinline__ void rows_product(const double* __restrict__ A, int ld, int nr, int nc, int t0, int dt,
                                             int cnt, const IN& in, double (&acc)[8])
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rows = nr - 8 * warp;            // rows of this warp
    if (rows <= 0) return;
    const double* const a = A + (long long) (8 * warp) * ld;
    double u[8], v[8];
    typename IN::R r0{}, r1{};
    auto fetch = [&](int c, double (&b)[8]) {
        if (c < nc)
        {
            const double* p = a + c;
#pragma unroll
            for (int k = 0; k < 8; k++)
            {
                b[k] = __ldg(p);
                if (k + 1 < rows) p += ld;     // past the last row: that row again, its sum unused
            }
        }
    };
    auto start = [&](int c) {
        if (c < nc) r0 = in.issue(c);
        if (c + 32 < nc) r1 = in.issue(c + 32);
    };
    if (cnt > 0)
    {
        start(kB * t0 + lane);
        fetch(kB * t0 + lane, u);
    }
#pragma unroll 1
    for (int i = 0; i < cnt; i++)
    {
        const int c = kB * (t0 + i * dt) + lane;
        fetch(c + 32, v);
        double x0 = 0.0, x1 = 0.0;
        in.wait2(c, c + 32, nc, r0, r1, x0, x1);
        if (i + 1 < cnt) start(c + kB * dt);
        if (c < nc)
#pragma unroll
            for (int k = 0; k < 8; k++) acc[k] = fma(u[k], x0, acc[k]);
        if (i + 1 < cnt) fetch(c + kB * dt, u);
        if (c + 32 < nc)
#pragma unroll
            for (int k = 0; k < 8; k++) acc[k] = fma(v[k], x1, acc[k]);
    }
}

// acc += sum_r A[r][c] x[r] over the 64-row tiles t0, t0 + dt, .. of nr rows, c = lane and
// lane + 32 of nc columns: a warp takes eight rows of a tile (in two halves), its lanes the
// columns
template <typename IN>
__device__ __forceinline__ void cols_product(const double* __restrict__ A, int ld, int nr, int nc, int t0, int dt,
                                             int cnt, const IN& in, double2& acc)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool c0 = lane < nc, c1 = lane + 32 < nc;
    const double* const a = A + (c0 ? lane : 0);
    double2 u[4], v[4];
    typename IN::R q{};
    auto fetch = [&](int r0, double2 (&b)[4]) {
#pragma unroll
        for (int k = 0; k < 4; k++)
        {
            const double* const p = a + (long long) (r0 + k) * ld;
            b[k].x = r0 + k < nr ? __ldg(p) : 0.0;
            b[k].y = r0 + k < nr && c1 ? __ldg(p + 32) : 0.0;
        }
    };
    auto start = [&](int r) {
        if (r < nr) q = in.issue(r);
    };
    auto add = [&](int r0, int j0, double x, const double2 (&b)[4]) {
#pragma unroll
        for (int k = 0; k < 4; k++)
        {
            const double xk = __shfl_sync(kFull, x, j0 + k);
            if (r0 + k < nr)
            {
                acc.x = fma(b[k].x, xk, acc.x);
                acc.y = fma(b[k].y, xk, acc.y);
            }
        }
    };
    if (cnt > 0)
    {
        start(kB * t0 + 8 * warp + (lane & 7));
        fetch(kB * t0 + 8 * warp, u);
    }
#pragma unroll 1
    for (int i = 0; i < cnt; i++)
    {
        const int r0 = kB * (t0 + i * dt) + 8 * warp;
        fetch(r0 + 4, v);
        const double x = r0 + (lane & 7) < nr ? in.wait(r0 + (lane & 7), q) : 0.0;
        if (i + 1 < cnt) start(r0 + kB * dt + (lane & 7));
        add(r0, 0, x, u);
        if (i + 1 < cnt) fetch(r0 + kB * dt, u);
        add(r0 + 4, 4, x, v);
    }
}

// s[row] = the lanes' sums of acc, row = 8 warp + k: a transposed butterfly leaves row k's
// sum with the lanes of bits (16, 8, 4) = k
__device__ __forceinline__ void rows_reduce(double (&acc)[8], double* s)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16, n = 4; n >= 1; o >>= 1, n >>= 1)
    {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (k < n)
            {
                const double send = up ? acc[k] : acc[k + n], keep = up ? acc[k + n] : acc[k];
                acc[k] = keep + __shfl_xor_sync(kFull, send, o);
            }
    }
    acc[0] += __shfl_xor_sync(kFull, acc[0], 2);
    acc[0] += __shfl_xor_sync(kFull, acc[0], 1);
    if ((lane & 3) == 0) s[8 * warp + (lane >> 2)] = acc[0];
}

// sum_j B[i][j] r[j] over the triangle (LOWER: j <= i, else j >= i) of a 64 x 64 block in
// shared memory (element (i, j) at s + j kDS + i) for row i = tid / 4, in every lane of the
// row's four.  Entries outside the triangle are left out rather than multiplied by zero, so
// that an infinite or NaN entry reaches the unknowns that depend on it only.
template <bool LOWER>
__device__ __forceinline__ double apply_diag(const double* s, const double* r)
{
    const int i = threadIdx.x >> 2, q = threadIdx.x & 3;
    double a[2] = {0.0, 0.0};
#pragma unroll
    for (int k = 0; k < 16; k++)
    {
        const int j = q + 4 * k;
        if (LOWER ? j <= i : j >= i) a[k & 1] = fma(s[j * kDS + i], r[j], a[k & 1]);
    }
    a[0] += a[1];
    a[0] += __shfl_xor_sync(kFull, a[0], 1);
    a[0] += __shfl_xor_sync(kFull, a[0], 2);
    return a[0];
}

// x = M^-1 r by substitution, one warp, M as apply_diag has it: lane owns rows lane and lane + 32
template <bool LOWER>
__device__ __forceinline__ void substitute(const double* s, const double* r, double* x)
{
    const int lane = threadIdx.x & 31;
    double r0 = r[lane], r1 = r[lane + 32];
#pragma unroll 1
    for (int t = 0; t < kB; t++)
    {
        const int j = LOWER ? t : kB - 1 - t;
        const double v = __shfl_sync(kFull, j < 32 ? r0 : r1, j & 31) / s[j * kDS + j];
        if (lane == 0) x[j] = v;
        if (LOWER ? lane > j : lane < j) r0 = fma(-s[j * kDS + lane], v, r0);
        if (LOWER ? lane + 32 > j : lane + 32 < j) r1 = fma(-s[j * kDS + lane + 32], v, r1);
    }
}

// The units of one level of one sweep.  What bounds it: the factors are read once a sweep
// (HBM), and the triangular solve of a node is a chain of (m - I) / 64 dependent steps:
// publish a block's 64 entries, read them on another SM through L2, the product with the
// next block's 64 x 64 entries (in registers by then), its reduction, and the diagonal
// block.  A block is solved with its inverse (made at create) and one step of refinement
// against the block itself, three 64 x 64 products, about 0.5 us; substitution by one warp
// (64 dependent shuffle / multiply-add steps) measured 2.15 ms for the solve below, the
// inverse 1.26 ms (3.49e-15 and 3.51e-15 from the 64-bit solve).  That is sound for blocks
// whose inverse is (kInverseMax); the others, which k_ulv_diag flags, are solved by substitution.
// One CTA per node (the earlier form) read the root's 471 MB through one SM.  HSS tree of
// N = 20,000 with 64 leaves, root of 7,700 rows, Cholesky, op 3: 36.8 -> 1.26 ms (2.3 GB of
// factors, 0.36 ms at the copy bandwidth).
template <int MODE>
__global__ void __launch_bounds__(kUT, 2) k_ulv_units(const UlvNode* __restrict__ nodes,
                                                      const UlvUnit* __restrict__ units, int n_units, int* ticket,
                                                      int q_cap, const double* __restrict__ Qt,
                                                      const double* __restrict__ Lf, const double* __restrict__ Dinv,
                                                      const unsigned char* __restrict__ subst,
                                                      const int* __restrict__ idxs, const int* __restrict__ piv,
                                                      double* px, Tagged* W, Tagged* X,
                                                      int* status, int limit)
{
    constexpr bool UP = MODE == CH_UP || MODE == LU_UP;
    extern __shared__ __align__(16) double ulv_sm[];
    double* const sD = ulv_sm;                 // diagonal block, column j at sD + j kDS
    double* const sE = sD + kB * kDS;          // its inverse
    double* const sP = sE + kB * kDS;          // partial sums of the warps (8 x 64)
    double* const sr = sP + kUW * kB;          // right-hand side of the unit
    double* const sx = sr + kB;                // a node's vector (Q products)
    __shared__ int s_unit;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (;;)
    {
        __syncthreads();
        if (tid == 0) s_unit = atomicAdd(ticket, 1);
        __syncthreads();
        const int u = s_unit;
        if (u >= n_units) return;
        const UlvUnit un = units[u];
        const UlvNode N = nodes[un.node];
        const int m = N.m, I = N.I, n2 = m - I, at = un.at;
        const int* const idx = idxs + N.idx_off;
        const double* const L = Lf + N.l_off;
        const double* const T = L + (long long) I * m + I;
        Tagged* const w = W + N.idx_off;
        Tagged* const x = X + N.idx_off;
        const bool hasq = N.q_off >= 0;
        const bool put = hasq || MODE == LU_UP;   // results go through U_PUT
        if (un.type == U_QT)
        {
            for (int i = tid; i < m; i += kUT) sx[i] = px[idx[i]];
            __syncthreads();
            const int nr = min(kB, m - at);
            double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            rows_product(Qt + N.q_off + (long long) at * m, m, nr, m, 0, 1, (m + kB - 1) / kB, InShared{sx}, acc);
            rows_reduce(acc, sr);
            __syncwarp();
            if (lane < 8 && 8 * warp + lane < nr) tag_put(w + at + 8 * warp + lane, sr[8 * warp + lane]);
        }
        else if (un.type == U_TRI)
        {
            const int nr = min(kB, n2 - at);
            const int nt = (n2 + kB - 1) / kB, after = nt - 1 - at / kB;   // blocks; those after this one
            // the diagonal block M (zero outside its triangle, identity past its end) and its
            // inverse, transposed for the second Cholesky sweep
            const long long d_off = N.d_off + (MODE == LU_DOWN ? (long long) ((n2 + kB - 1) / kB) * kB * kB : 0) +
                                    (long long) at * kB;
            const double* const D = Dinv + d_off;
            const bool by_subst = subst[d_off / (kB * kB)] != 0;
#pragma unroll 4
            for (int e = tid; e < kB * kB; e += kUT)
            {
                const int i = e / kB, j = e % kB;      // row, column of the factor block
                double v = 0.0;
                if (MODE == LU_DOWN ? j >= i : j < i || (MODE != LU_UP && j == i))
                    if (i < nr && j < nr) v = __ldg(T + (long long) (at + i) * m + at + j);
                if (i == j && (MODE == LU_UP || i >= nr)) v = 1.0;
                const int k = MODE == CH_DOWN ? i * kDS + j : j * kDS + i;
                sD[k] = v;
                sE[k] = __ldg(D + e);
            }
            double b = 0.0;
            if (tid < nr)
            {
                const int i = at + tid;
                if constexpr (UP)
                {
                    const int k = I + (MODE == LU_UP ? piv[N.p_off + i] : i);
                    b = hasq ? tag_wait(w + k, tag_get(w + k), status, limit) : px[idx[k]];
                } else b = px[idx[I + i]];
            }
            double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            double2 ac = make_double2(0.0, 0.0);
            const InTagged xs{x + I, status, limit};
            if constexpr (UP)
                rows_product(T + (long long) at * m, m, nr, n2, 0, 1, at / kB, xs, acc);
            else if constexpr (MODE == LU_DOWN)
            {
                rows_product(L + (long long) (I + at) * m, m, nr, I, 0, 1, (I + kB - 1) / kB,
                             InIndexed{px, idx}, acc);
                rows_product(T + (long long) at * m, m, nr, n2, nt - 1, -1, after, xs, acc);
            } else {
                cols_product(L + I + at, m, I, nr, 0, 1, (I + kB - 1) / kB, InIndexed{px, idx}, ac);
                cols_product(T + at, m, n2, nr, nt - 1, -1, after, xs, ac);
            }
            if constexpr (MODE == CH_DOWN)
            {
                sP[warp * kB + lane] = ac.x;
                sP[warp * kB + lane + 32] = ac.y;
            } else rows_reduce(acc, sP);
            __syncthreads();
            if (tid < kB)
            {
                double s = sP[tid];
                if constexpr (MODE == CH_DOWN)
                {
#pragma unroll
                    for (int k = 1; k < kUW; k++) s += sP[k * kB + tid];
                }
                sr[tid] = tid < nr ? b - s : 0.0;
            }
            __syncthreads();
            const int i = tid >> 2;
            double y;
            if (by_subst)
            {
                if (warp == 0) substitute<UP>(sD, sr, sP);
                __syncthreads();
                y = sP[i];
            } else {
                // y = M^-1 r, then one step of refinement: y += M^-1 (r - M y)
                y = apply_diag<UP>(sE, sr);
                if ((tid & 3) == 0) sP[i] = y;
                __syncthreads();
                const double d = sr[i] - apply_diag<UP>(sD, sP);
                if ((tid & 3) == 0) sP[kB + i] = d;
                __syncthreads();
                const double c = apply_diag<UP>(sE, sP + kB);
                if (fabs(c) < HUGE_VAL) y += c;     // not for infinite or NaN unknowns
            }
            if ((tid & 3) == 0 && i < nr)
            {
                const int k = I + at + i;
                tag_put(x + k, y);
                if (!put) px[idx[k]] = y;
            }
        }
        else if (un.type == U_OFF)
        {
            const int nr = min(kB, I - at);
            double b = 0.0;
            if (tid < nr) b = hasq ? tag_wait(w + at + tid, tag_get(w + at + tid), status, limit) : px[idx[at + tid]];
            double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            rows_product(L + (long long) at * m + I, m, nr, n2, 0, 1, (n2 + kB - 1) / kB, InTagged{x + I, status, limit}, acc);
            rows_reduce(acc, sP);
            __syncthreads();
            if (tid < nr)
            {
                const double v = b - sP[tid];
                if (put) tag_put(x + at + tid, v);
                else px[idx[at + tid]] = v;
            }
        }
        else if (un.type == U_Q)
        {
            for (int i = tid; i < m; i += kUT) sx[i] = i < I ? px[idx[i]] : tag_wait(x + i, tag_get(x + i), status, limit);
            __syncthreads();
            const int nc = min(kB, m - at);
            double2 ac = make_double2(0.0, 0.0);
            cols_product(Qt + N.q_off + at, m, m, nc, 0, 1, (m + kB - 1) / kB, InShared{sx}, ac);
            sP[warp * kB + lane] = ac.x;
            sP[warp * kB + lane + 32] = ac.y;
            __syncthreads();
            if (tid < nc)
            {
                double s = sP[tid];
#pragma unroll
                for (int k = 1; k < kUW; k++) s += sP[k * kB + tid];
                tag_put(w + at + tid, s);
            }
        }
        else
        {
            // U_PUT: the first sweep's results are in x (b1 and b2), the second's in w
            const Tagged* const r = UP ? x : w;
            for (int i = tid; i < m; i += kUT) tag_wait(r + i, tag_get(r + i), status, limit);
            __syncthreads();
            for (int i = tid; i < m; i += kUT) px[idx[i]] = __longlong_as_double(tag_get(r + i).v);
        }
    }
}

__device__ __forceinline__ double warp_sum(double s)
{
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
    return s;
}

// Q^T of each job: warp w of CTA (x, y) forms column c = 8 x + w of job y's Q, i.e.
// Q e_c = H(0) H(1) .. H(k-1) e_c, into row c of Q^T
__global__ void __launch_bounds__(kUT) k_ulv_form_q(const UlvQJob* __restrict__ jobs, const double* __restrict__ V,
                                                    double* __restrict__ Qt)
{
    const UlvQJob J = jobs[blockIdx.y];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = blockIdx.x * kUW + warp;
    if (c >= J.m) return;
    const int m = J.m;
    double* const x = Qt + J.q_off + (long long) c * m;
    for (int i = lane; i < m; i += 32) x[i] = i == c ? 1.0 : 0.0;
    __syncwarp();
    const double* const v = V + J.v_off;
    const double* const tau = v + (long long) J.k * m;
    for (int j = J.k - 1; j >= 0; j--)
    {
        const double* const vj = v + (long long) j * m;
        double s = 0.0;
        for (int i = j + lane; i < m; i += 32) s += vj[i] * x[i];
        s = warp_sum(s) * tau[j];
        for (int i = j + lane; i < m; i += 32) x[i] -= s * vj[i];
        __syncwarp();
    }
}

// Inverse E of a diagonal block M by substitution, thread c its column c (64 threads), and the
// block's flag: the largest row sum of |M| |E| (for Cholesky also of |M^T| |E^T|, which the
// second sweep solves with) above kInverseMax, or not a number.  A block that ends inside the
// 64 rows is continued with the identity.
__global__ void __launch_bounds__(kB) k_ulv_diag(const UlvDiagJob* __restrict__ jobs, const UlvNode* __restrict__ nodes,
                                                 const double* __restrict__ Lf, double* __restrict__ Dinv,
                                                 unsigned char* __restrict__ subst)
{
    extern __shared__ __align__(16) double ulv_sm[];
    double* const sD = ulv_sm;                  // the block, row i at sD + i kB
    double* const sx = sD + kB * kB;            // the inverse, the same
    const UlvDiagJob J = jobs[blockIdx.x];
    const UlvNode N = nodes[J.node];
    const int nr = min(kB, N.m - N.I - J.at), c = threadIdx.x;
    const double* const T = Lf + N.l_off + (long long) (N.I + J.at) * N.m + N.I + J.at;
    for (int i = 0; i < kB; i++) sD[i * kB + c] = i < nr && c < nr ? T[(long long) i * N.m + c] : (i == c ? 1.0 : 0.0);
    __syncthreads();
    for (int t = 0; t < kB; t++)
    {
        const int i = J.upper ? kB - 1 - t : t;
        double s = i == c ? 1.0 : 0.0;
        if (J.upper)
            for (int j = i + 1; j < kB; j++) s = fma(-sD[i * kB + j], sx[j * kB + c], s);
        else
            for (int j = 0; j < i; j++) s = fma(-sD[i * kB + j], sx[j * kB + c], s);
        sx[i * kB + c] = J.unit ? s : s / sD[i * kB + i];
    }
    for (int i = 0; i < kB; i++) Dinv[J.d_off + i * kB + c] = sx[i * kB + c];
    __shared__ double sum[2][kB];               // row and column sums of |E|
    __syncthreads();
    double er = 0.0, ec = 0.0;
    for (int j = 0; j < kB; j++)
    {
        if (J.upper ? j >= c : j <= c) er += fabs(sx[c * kB + j]);
        if (J.upper ? j <= c : j >= c) ec += fabs(sx[j * kB + c]);
    }
    sum[0][c] = er;
    sum[1][c] = ec;
    __syncthreads();
    const double diag = J.unit ? 1.0 : fabs(sD[c * kB + c]);
    double fr = diag * er, fc = diag * ec;
    for (int j = 0; j < kB; j++)
    {
        if (J.upper ? j > c : j < c) fr = fma(fabs(sD[c * kB + j]), sum[0][j], fr);
        if (J.upper ? j < c : j > c) fc = fma(fabs(sD[j * kB + c]), sum[1][j], fc);
    }
    const bool chol = !J.upper && !J.unit;
    const double f = chol && !(fc <= fr) ? fc : fr;
    const int bad = __syncthreads_or(!(f <= kInverseMax));
    if (c == 0) subst[J.d_off / (kB * kB)] = (unsigned char) (bad != 0);
}

__global__ void k_ulv_gather(int n, const double* __restrict__ src, const int* __restrict__ map,
                             double* __restrict__ dst)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[i] = src[map[i]];
}

// the permuted right-hand side, and the tags and unit counters of the solve cleared
__global__ void k_ulv_start(int n, const double* __restrict__ src, const int* __restrict__ map, double* __restrict__ dst,
                            Tagged* __restrict__ tags, long long n_tags, int* __restrict__ tickets, int n_tickets)
{
    const long long t0 = blockIdx.x * (long long) blockDim.x + threadIdx.x, step = (long long) gridDim.x * blockDim.x;
    for (long long i = t0; i < n; i += step) dst[i] = src[map[i]];
    for (long long i = t0; i < n_tags; i += step) tags[i].t = 0;
    for (long long i = t0; i < n_tickets; i += step) tickets[i] = 0;
}

int smem_bytes(int q_cap) { return (int) sizeof(double) * (2 * kB * kDS + kUW * kB + kB + q_cap); }

}  // namespace

struct h2gpu_ulv {
    int lu = 0, device = 0, n = 0, max_level = 0;
    int q_cap = 0;                       // entries of the longest vector a unit keeps in shared memory
    long long ni = 0;                    // entries of all nodes (one tagged vector)
    cudaStream_t stream = nullptr;
    std::vector<int> beg[2];             // first / second sweep: unit ranges of levels 0 .. max_level
    UlvNode* d_nodes = nullptr;
    UlvUnit* d_units = nullptr;
    Tagged* d_tag = nullptr;             // four tagged vectors: two per sweep
    int* d_ticket = nullptr;             // unit counters, one per level and sweep
    int* h_status = nullptr;             // pinned; set by a wait that ran out
    unsigned char* d_subst = nullptr;    // per diagonal block: solved by substitution
    double *d_Q = nullptr, *d_L = nullptr, *d_D = nullptr, *d_px = nullptr, *d_b = nullptr, *d_x = nullptr;
    int *d_idx = nullptr, *d_p = nullptr, *d_fwd = nullptr, *d_bwd = nullptr;
    size_t bytes = 0;
};

namespace {

int ulv_fail(int code, const char* fmt, ...) __attribute__((format(printf, 2, 3)));
int ulv_fail(int code, const char* fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    return h2gpu::set_error(code, buf);
}

int cuda_status(cudaError_t e, const char* what)
{
    if (e == cudaSuccess) return H2GPU_OK;
    return ulv_fail(e == cudaErrorMemoryAllocation ? H2GPU_ERR_NOMEM : H2GPU_ERR_CUDA, "ULV %s: %s", what,
                    cudaGetErrorString(e));
}

void free_ulv(h2gpu_ulv* u)
{
    for (void* p : {(void*) u->d_nodes, (void*) u->d_units, (void*) u->d_tag, (void*) u->d_ticket, (void*) u->d_subst, (void*) u->d_Q, (void*) u->d_L, (void*) u->d_D, (void*) u->d_px,
                    (void*) u->d_b, (void*) u->d_x, (void*) u->d_idx, (void*) u->d_p, (void*) u->d_fwd,
                    (void*) u->d_bwd})
        if (p) cudaFree(p);
    if (u->h_status) cudaFreeHost(u->h_status);
    if (u->stream) cudaStreamDestroy(u->stream);
    delete u;
}

struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev)
    {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        if (prev != dev) cudaSetDevice(dev);
    }
    ~DeviceGuard()
    {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

// skip, limit: the level's first units left out, and the polls of a wait (h2gpu_ulv_wait_check)
template <int MODE>
cudaError_t launch_level(h2gpu_ulv* u, int l, cudaStream_t st, int skip = 0, int limit = kPollLimit)
{
    constexpr int down = MODE == CH_DOWN || MODE == LU_DOWN;
    const int b = u->beg[down][l] + skip, n = u->beg[down][l + 1] - b;
    if (n <= 0) return cudaSuccess;
    Tagged* const w = u->d_tag + 2 * down * u->ni;
    // two CTAs per SM (the launch bound); fewer when the level has fewer units
    k_ulv_units<MODE><<<std::min(n, 2 * 148), kUT, smem_bytes(u->q_cap), st>>>(
        u->d_nodes, u->d_units + b, n, u->d_ticket + down * (u->max_level + 1) + l, u->q_cap, u->d_Q, u->d_L, u->d_D, u->d_subst,
        u->d_idx, u->d_p, u->d_px, w, w + u->ni, u->h_status, limit);
    return cudaGetLastError();
}

// the status word of waits that ran out: reported once, by the first call that sees it
int check_waits(h2gpu_ulv* u)
{
    if (*(volatile int*) u->h_status == 0) return H2GPU_OK;
    *(volatile int*) u->h_status = 0;
    return ulv_fail(H2GPU_ERR_DEVICE, "ULV solve: a bounded wait between units expired");
}

cudaError_t start_solve(h2gpu_ulv* u, const double* d_b, cudaStream_t st)
{
    const int gs = (int) std::max<long long>(1, std::min<long long>((std::max<long long>(u->n, 4 * u->ni) + 255) / 256, 148 * 8));
    k_ulv_start<<<gs, 256, 0, st>>>(u->n, d_b, u->d_fwd, u->d_px, u->d_tag, 4 * u->ni, u->d_ticket, 2 * (u->max_level + 1));
    return cudaGetLastError();
}

int enqueue_solve(h2gpu_ulv* u, int op, const double* d_b, double* d_x, cudaStream_t st)
{
    const int st0 = check_waits(u);
    if (st0 != H2GPU_OK) return st0;
    const int gb = std::max(1, std::min((u->n + 255) / 256, 4096));
    cudaError_t e = start_solve(u, d_b, st);
    if (op & 1)
        for (int l = u->max_level; l >= 0 && e == cudaSuccess; l--)
            e = u->lu ? launch_level<LU_UP>(u, l, st) : launch_level<CH_UP>(u, l, st);
    if (op & 2)
        for (int l = 0; l <= u->max_level && e == cudaSuccess; l++)
            e = u->lu ? launch_level<LU_DOWN>(u, l, st) : launch_level<CH_DOWN>(u, l, st);
    if (e != cudaSuccess) return cuda_status(e, "solve launch");
    k_ulv_gather<<<gb, 256, 0, st>>>(u->n, u->d_px, u->d_bwd, d_x);
    return cuda_status(cudaGetLastError(), "solve launch");
}

// cudaMemcpy from pageable memory may return once the data is staged, with the transfer itself
// still on its way in the legacy stream, which the object's non-blocking stream does not wait
// for: kernels on that stream read uploads after this only.
cudaError_t uploads_landed() { return cudaStreamSynchronize(cudaStreamLegacy); }

// Units of one level of a sweep, in an order in which every unit depends on earlier ones
// only; the triangular chains of a level's nodes advance side by side.
void level_units(const std::vector<UlvNode>& nodes, const int* list, int cnt, bool up, bool lu, std::vector<UlvUnit>& out)
{
    auto all = [&](int type, auto&& rows, auto&& add) {
        int most = 0;
        for (int j = 0; j < cnt; j++) most = std::max(most, rows(nodes[list[j]]));
        for (int a = 0; a < most; a += kB)
            for (int j = 0; j < cnt; j++)
                if (a < rows(nodes[list[j]])) add(type, list[j], a, rows(nodes[list[j]]));
    };
    auto plain = [&](int type, int node, int a, int) { out.push_back(UlvUnit{node, type, a}); };
    auto q_rows = [](const UlvNode& N) { return N.q_off >= 0 ? N.m : 0; };
    auto tri = [](const UlvNode& N) { return N.m - N.I; };
    if (up)
    {
        all(U_QT, q_rows, plain);
        all(U_TRI, tri, plain);
        all(U_OFF, [](const UlvNode& N) { return N.I; }, plain);
    } else {
        // last block first
        all(U_TRI, tri, [&](int type, int node, int a, int n) { out.push_back(UlvUnit{node, type, (n - 1) / kB * kB - a}); });
        all(U_Q, q_rows, plain);
    }
    for (int j = 0; j < cnt; j++)
        if (nodes[list[j]].m > 0 && (nodes[list[j]].q_off >= 0 || (up && lu))) out.push_back(UlvUnit{list[j], U_PUT, 0});
}

}  // namespace

H2G_API int h2gpu_ulv_create(const h2gpu_ulv_desc* d, h2gpu_ulv** out)
{
    if (!out) return ulv_fail(H2GPU_ERR_INVALID, "out is NULL");
    *out = nullptr;
    if (!d || d->n_node <= 0 || d->max_level < 0 || d->n_leaf_node <= 0 || d->krnl_mat_size <= 0 ||
        !d->level_n_node || !d->level_nodes || !d->fwd_pmt_idx || !d->bwd_pmt_idx || !d->Ls || !d->m ||
        !d->q_ncol || !d->l_ld || !d->idx || !d->Q || !d->L || (d->lu && !d->p))
        return ulv_fail(H2GPU_ERR_INVALID, "malformed ULV descriptor");
    const int n = d->krnl_mat_size;
    for (int i = 0; i < n; i++)
        if (d->fwd_pmt_idx[i] < 0 || d->fwd_pmt_idx[i] >= n || d->bwd_pmt_idx[i] < 0 || d->bwd_pmt_idx[i] >= n)
            return ulv_fail(H2GPU_ERR_INVALID, "permutation entry %d out of range", i);
    // nodes in level order, and their arena offsets
    std::vector<int> list, lvl_off(1, 0), level_of(d->n_node, -1);
    for (int l = 0; l <= d->max_level; l++)
    {
        const int cnt = d->level_n_node[l];
        if (cnt < 0 || cnt > d->n_leaf_node) return ulv_fail(H2GPU_ERR_INVALID, "level %d: %d nodes", l, cnt);
        if (l == 0 && cnt != 1) return ulv_fail(H2GPU_ERR_INVALID, "level 0 must hold the root alone");
        for (int j = 0; j < cnt; j++)
        {
            const int node = d->level_nodes[(size_t) l * d->n_leaf_node + j];
            if (node < 0 || node >= d->n_node || level_of[node] >= 0)
                return ulv_fail(H2GPU_ERR_INVALID, "level %d: bad or repeated node %d", l, node);
            level_of[node] = l;
            list.push_back(node);
        }
        lvl_off.push_back((int) list.size());
    }
    std::vector<UlvNode> nodes(d->n_node);
    std::vector<UlvQJob> jobs;
    std::vector<UlvDiagJob> djobs;
    long long nd = 0;
    long long nq = 0, nl = 0, ni = 0, np = 0, nv = 0;
    int m_cap = 1, q_cap = 1;
    for (int node : list)
    {
        const int m = d->m[node], I = d->Ls[node], k = d->q_ncol[node];
        const bool root = level_of[node] == 0;
        if (m < 0 || I < 0 || I > m) return ulv_fail(H2GPU_ERR_INVALID, "node %d: m %d, Ls %d", node, m, I);
        if (m > 0 && (!d->idx[node] || !d->L[node] || d->l_ld[node] < m))
            return ulv_fail(H2GPU_ERR_INVALID, "node %d: factor or index set missing", node);
        for (int i = 0; i < m; i++)
            if (d->idx[node][i] < 0 || d->idx[node][i] >= n)
                return ulv_fail(H2GPU_ERR_INVALID, "node %d: index %d out of range", node, d->idx[node][i]);
        UlvNode& N = nodes[node];
        N.m = m; N.I = I;
        N.l_off = nl; nl += (long long) m * m;
        N.idx_off = ni; ni += m;
        N.d_off = nd;
        for (int up = 0; up <= (d->lu ? 1 : 0); up++)
            for (int a = 0; a < m - I; a += kB, nd += kB * kB)
                djobs.push_back(UlvDiagJob{nd, node, a, up, d->lu && !up});
        N.q_off = -1;
        N.p_off = -1;
        if (!root && k > 0 && m > 0)
        {
            if (k > m) return ulv_fail(H2GPU_ERR_UNSUPPORTED, "node %d: %d reflectors of length %d", node, k, m);
            if (!d->Q[node]) return ulv_fail(H2GPU_ERR_INVALID, "node %d: Q missing", node);
            N.q_off = nq; nq += (long long) m * m;
            q_cap = std::max(q_cap, m);
            jobs.push_back(UlvQJob{nv, N.q_off, m, k, 0, 0});
            nv += (long long) k * m + k;
        }
        if (d->lu)
        {
            if (m - I > 0 && !d->p[node]) return ulv_fail(H2GPU_ERR_INVALID, "node %d: pivots missing", node);
            for (int j = 0; j < m - I; j++)
                if (d->p[node][j] < 0 || d->p[node][j] >= m - I)
                    return ulv_fail(H2GPU_ERR_INVALID, "node %d: pivot %d out of range", node, d->p[node][j]);
            N.p_off = np; np += m - I;
        }
        m_cap = std::max(m_cap, m);
    }
    for (int i = 0; i < d->n_node; i++)
        if (level_of[i] < 0) { nodes[i] = UlvNode{}; nodes[i].q_off = nodes[i].p_off = -1; }
    if (m_cap > kMaxNodeRows)
        return ulv_fail(H2GPU_ERR_UNSUPPORTED, "a node of %d rows, more than %d", m_cap, kMaxNodeRows);
    int dev = d->device;
    if (dev < 0 && cudaGetDevice(&dev) != cudaSuccess) return ulv_fail(H2GPU_ERR_CUDA, "no CUDA device");
    DeviceGuard guard(dev);
    h2gpu_ulv* u = new h2gpu_ulv;
    u->lu = d->lu ? 1 : 0; u->device = dev; u->n = n; u->max_level = d->max_level; u->ni = ni;
    u->q_cap = q_cap;
    std::vector<UlvUnit> units;
    for (int down = 0; down < 2; down++)
    {
        u->beg[down].push_back((int) units.size());
        for (int l = 0; l <= d->max_level; l++)
        {
            level_units(nodes, list.data() + lvl_off[l], lvl_off[l + 1] - lvl_off[l], !down, u->lu, units);
            u->beg[down].push_back((int) units.size());
        }
    }
    // host staging of the small arrays and of the reflectors (transposed: reflector j
    // contiguous, with its implicit 1 and the zeros above it written out)
    std::vector<int> hidx((size_t) std::max<long long>(ni, 1)), hp((size_t) std::max<long long>(np, 1));
    std::vector<double> hv((size_t) std::max<long long>(nv, 1));
    size_t ji = 0;
    for (int node : list)
    {
        const UlvNode& N = nodes[node];
        if (N.m > 0) memcpy(&hidx[N.idx_off], d->idx[node], sizeof(int) * N.m);
        if (N.p_off >= 0 && N.m - N.I > 0) memcpy(&hp[N.p_off], d->p[node], sizeof(int) * (N.m - N.I));
        if (N.q_off >= 0)
        {
            const UlvQJob& J = jobs[ji++];
            const double* A = d->Q[node];
            const int m = J.m, k = J.k;
            double* v = &hv[J.v_off];
            for (int j = 0; j < k; j++)
                for (int i = 0; i < m; i++)
                    v[(size_t) j * m + i] = i < j ? 0.0 : i == j ? 1.0 : A[(size_t) i * k + j];
            for (int j = 0; j < k; j++) v[(size_t) k * m + j] = A[(size_t) m * k + j];   // tau: the last row
        }
    }
    double* d_v = nullptr;
    UlvQJob* d_jobs = nullptr;
    UlvDiagJob* d_djobs = nullptr;
    int st = H2GPU_OK;
    auto step = [&](cudaError_t e, const char* what) {
        if (st == H2GPU_OK) st = cuda_status(e, what);
        return st == H2GPU_OK;
    };
    auto alloc = [&](void** p, size_t b) {
        if (!step(cudaMalloc(p, std::max<size_t>(b, 16)), "device allocation")) return false;
        u->bytes += std::max<size_t>(b, 16);
        return true;
    };
    if (step(cudaStreamCreateWithFlags(&u->stream, cudaStreamNonBlocking), "stream") &&
        alloc((void**) &u->d_nodes, sizeof(UlvNode) * nodes.size()) &&
        alloc((void**) &u->d_units, sizeof(UlvUnit) * units.size()) &&
        alloc((void**) &u->d_tag, 4 * sizeof(Tagged) * (size_t) ni) &&
        alloc((void**) &u->d_ticket, 2 * sizeof(int) * (size_t) (d->max_level + 1)) &&
        alloc((void**) &u->d_Q, 8 * (size_t) nq) && alloc((void**) &u->d_L, 8 * (size_t) nl) &&
        alloc((void**) &u->d_D, 8 * (size_t) nd) && alloc((void**) &u->d_subst, (size_t) nd / (kB * kB)) &&
        alloc((void**) &u->d_idx, 4 * (size_t) ni) && alloc((void**) &u->d_p, 4 * (size_t) np) &&
        alloc((void**) &u->d_fwd, 4 * (size_t) n) && alloc((void**) &u->d_bwd, 4 * (size_t) n) &&
        alloc((void**) &u->d_px, 8 * (size_t) n) && alloc((void**) &u->d_b, 8 * (size_t) n) &&
        alloc((void**) &u->d_x, 8 * (size_t) n) &&
        step(cudaMemcpy(u->d_nodes, nodes.data(), sizeof(UlvNode) * nodes.size(), cudaMemcpyHostToDevice), "upload") &&
        step(cudaMemcpy(u->d_units, units.data(), sizeof(UlvUnit) * units.size(), cudaMemcpyHostToDevice), "upload") &&
        step(cudaHostAlloc((void**) &u->h_status, sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped), "status word") &&
        step(cudaMemcpy(u->d_idx, hidx.data(), 4 * (size_t) ni, cudaMemcpyHostToDevice), "upload") &&
        step(np ? cudaMemcpy(u->d_p, hp.data(), 4 * (size_t) np, cudaMemcpyHostToDevice) : cudaSuccess, "upload") &&
        step(cudaMemcpy(u->d_fwd, d->fwd_pmt_idx, 4 * (size_t) n, cudaMemcpyHostToDevice), "upload") &&
        step(cudaMemcpy(u->d_bwd, d->bwd_pmt_idx, 4 * (size_t) n, cudaMemcpyHostToDevice), "upload"))
    {
        *u->h_status = 0;
        for (int node : list)
        {
            const UlvNode& N = nodes[node];
            if (N.m == 0) continue;
            if (!step(cudaMemcpy2D(u->d_L + N.l_off, 8 * (size_t) N.m, d->L[node], 8 * (size_t) d->l_ld[node],
                                   8 * (size_t) N.m, (size_t) N.m, cudaMemcpyHostToDevice), "factor upload"))
                break;
        }
    }
    if (st == H2GPU_OK && !djobs.empty() && step(cudaMalloc(&d_djobs, sizeof(UlvDiagJob) * djobs.size()), "diagonal blocks") &&
        step(cudaMemcpy(d_djobs, djobs.data(), sizeof(UlvDiagJob) * djobs.size(), cudaMemcpyHostToDevice), "diagonal blocks") &&
        step(uploads_landed(), "diagonal blocks") &&
        step(cudaFuncSetAttribute(k_ulv_diag, cudaFuncAttributeMaxDynamicSharedMemorySize, 16 * kB * kB), "diagonal blocks"))
    {
        k_ulv_diag<<<(unsigned) djobs.size(), kB, 16 * kB * kB, u->stream>>>(d_djobs, u->d_nodes, u->d_L, u->d_D, u->d_subst);
        step(cudaGetLastError(), "diagonal blocks");
        step(cudaStreamSynchronize(u->stream), "diagonal blocks");
    }
    if (st == H2GPU_OK && !jobs.empty() && step(cudaMalloc(&d_v, 8 * (size_t) nv), "reflector staging") &&
        step(cudaMalloc(&d_jobs, sizeof(UlvQJob) * jobs.size()), "reflector staging") &&
        step(cudaMemcpy(d_v, hv.data(), 8 * (size_t) nv, cudaMemcpyHostToDevice), "reflector upload") &&
        step(cudaMemcpy(d_jobs, jobs.data(), sizeof(UlvQJob) * jobs.size(), cudaMemcpyHostToDevice), "reflector upload") &&
        step(uploads_landed(), "reflector upload"))
    {
        int mq = 1;
        for (const UlvQJob& J : jobs) mq = std::max(mq, J.m);
        for (size_t j0 = 0; j0 < jobs.size() && st == H2GPU_OK; j0 += 65535)
        {
            const unsigned cnt = (unsigned) std::min<size_t>(65535, jobs.size() - j0);
            k_ulv_form_q<<<dim3((unsigned) ((mq + kUW - 1) / kUW), cnt), kUT, 0, u->stream>>>(d_jobs + j0, d_v, u->d_Q);
            step(cudaGetLastError(), "forming Q");
        }
        step(cudaStreamSynchronize(u->stream), "forming Q");
    }
    if (d_v) cudaFree(d_v);
    if (d_jobs) cudaFree(d_jobs);
    if (d_djobs) cudaFree(d_djobs);
    // the first solve may come on any stream (no diagonal block and no reflector: nothing has waited yet)
    step(uploads_landed(), "upload");
    if (st == H2GPU_OK)
    {
        // The limit is a per-function setting of the process: it is set to the device's
        // opt-in maximum, the same value for every object, so that creating a
        // factorization with smaller nodes never lowers it under another's launches.
        int optin = 0;
        if (step(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev), "device query") &&
            smem_bytes(u->q_cap) > (optin -= 128))      // the kernels' static part is within 128 bytes
            st = ulv_fail(H2GPU_ERR_UNSUPPORTED, "a node of %d rows with a Q exceeds one CTA's shared memory", u->q_cap);
        for (auto kern : {k_ulv_units<CH_UP>, k_ulv_units<CH_DOWN>, k_ulv_units<LU_UP>, k_ulv_units<LU_DOWN>})
            if (st == H2GPU_OK)
                step(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, optin),
                     "shared memory of the solve kernels");
    }
    if (st != H2GPU_OK)
    {
        free_ulv(u);
        return st;
    }
    *out = u;
    return H2GPU_OK;
}

H2G_API int h2gpu_ulv_destroy(h2gpu_ulv* u)
{
    if (!u) return H2GPU_OK;
    DeviceGuard guard(u->device);
    cudaStreamSynchronize(u->stream);
    free_ulv(u);
    return H2GPU_OK;
}

H2G_API int h2gpu_ulv_solve_device(h2gpu_ulv* u, int op, const double* d_b, double* d_x, void* stream)
{
    if (!u || !d_b || !d_x) return ulv_fail(H2GPU_ERR_INVALID, "ULV solve: NULL argument");
    if (op < 1 || op > 3) return ulv_fail(H2GPU_ERR_INVALID, "ULV solve: op %d, should be 1, 2 or 3", op);
    DeviceGuard guard(u->device);
    return enqueue_solve(u, op, d_b, d_x, stream ? (cudaStream_t) stream : u->stream);
}

H2G_API int h2gpu_ulv_solve(h2gpu_ulv* u, int op, const double* b, double* x)
{
    if (!u || !b || !x) return ulv_fail(H2GPU_ERR_INVALID, "ULV solve: NULL argument");
    if (op < 1 || op > 3) return ulv_fail(H2GPU_ERR_INVALID, "ULV solve: op %d, should be 1, 2 or 3", op);
    DeviceGuard guard(u->device);
    const size_t nb = 8 * (size_t) u->n;
    int st = cuda_status(cudaMemcpyAsync(u->d_b, b, nb, cudaMemcpyHostToDevice, u->stream), "upload");
    if (st == H2GPU_OK) st = enqueue_solve(u, op, u->d_b, u->d_x, u->stream);
    if (st == H2GPU_OK) st = cuda_status(cudaMemcpyAsync(x, u->d_x, nb, cudaMemcpyDeviceToHost, u->stream), "download");
    const int s2 = cuda_status(cudaStreamSynchronize(u->stream), "solve");
    if (st == H2GPU_OK) st = s2;
    return st != H2GPU_OK ? st : check_waits(u);
}

H2G_API int h2gpu_ulv_wait_check(h2gpu_ulv* u)
{
    if (!u) return ulv_fail(H2GPU_ERR_INVALID, "ULV wait check: NULL argument");
    DeviceGuard guard(u->device);
    const int st0 = check_waits(u);
    if (st0 != H2GPU_OK) return st0;
    cudaError_t e = start_solve(u, u->d_x, u->stream);      // the values do not matter
    for (int l = u->max_level; l >= 0 && e == cudaSuccess; l--)
        if (u->beg[0][l + 1] - u->beg[0][l] > 1)
        {
            e = u->lu ? launch_level<LU_UP>(u, l, u->stream, 1, 1) : launch_level<CH_UP>(u, l, u->stream, 1, 1);
            break;
        }
    const cudaError_t es = cudaStreamSynchronize(u->stream);
    const int st = cuda_status(e != cudaSuccess ? e : es, "wait check");
    return st != H2GPU_OK ? st : check_waits(u);
}

H2G_API size_t h2gpu_ulv_bytes(const h2gpu_ulv* u) { return u ? u->bytes : 0; }
