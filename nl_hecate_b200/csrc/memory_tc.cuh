// Frozen-M0 chunkwise Titans / Delta rule in CHUNK-PARALLEL (matrix) form on the 5th-generation tensor
// cores, head dimension 64.
//
// A problem's tokens are cut into tiles of one chunk, up to 64. Inside a tile the errors come from the
// tile-start state (M0, S0) and everything is linear in it and in them (E: rows e_t). With r_t = 1 - alpha_t
// and, for t >= j,
//     h(j,t)  = prod_{i=j+1..t} eta_i ,  rho(j,t) = prod_{i=j+1..t} r_i
//     Om(t,j) = sum_{i=j..t} h(j,i) rho(i,t)        (weight of -theta_j e_j k_j^T in the state M_t)
//     A_t = prod_{i<=t} r_i,  H_t = prod_{i<=t} eta_i,  B_t = eta_0 Om(t,0)   (weights of M0, S0)
//     W(t,j) = theta_j Om(t,j)
//     E   = K M0^T - V ,  P = Q K^T
//     Y   = diag(A) Q M0^T + diag(B) Q S0^T - (W o P) E
//     M_C = A_L M0 + B_L S0 - E^T diag(W(L-1,:)) K ,       S_C = H_L S0 - E^T diag(theta_j h(j,L-1)) K
// and backward (G_M, G_S: gradients of the tile-end states)
//     F = -[ (W o P)^T dY + diag(W(L-1,:)) K G_M^T + diag(theta h) K G_S^T ] ,  dV = -F ,  R = dY E^T
//     dQ  = diag(A) dY M0 + diag(B) dY S0 - (W o R) K
//     dK  = F M0 - diag(W(L-1,:)) E G_M - diag(theta h) E G_S - (W o R)^T Q
//     G_M' = dY^T diag(A) Q + F^T K + A_L G_M ,            G_S' = dY^T diag(B) Q + B_L G_M + H_L G_S
// The gate gradients contract the states with their adjoints and reduce to two decayed scans down
// the columns of X = R o P, plus two columns for M0 and S0. Only W's recurrences over tokens are
// sequential, and they are 64 scalar steps.
// Same semantics as the per-token statement core/kernels/titans_chunkwise_{forward,backward}.cu.
//
// Precision. Operands are fp32 and stay so: each is stored as THREE bf16 planes x = hi + mid + lo,
// which hold all 24 bits of the significand, and a product is the six plane products
// hi.hi, hi.mid, mid.hi, mid.mid, hi.lo, lo.hi accumulated in fp32 in TMEM, the small ones first (the
// dropped ones are below 2^-24 of the product). Scans and gate tables are fp32 FMA. Against float64, 16
// problems x 333 tokens, chunk 64: y 1.25e-7, dK 2.0e-7, dV 1.8e-7, d_eta 2.0e-7 (fp32 FMA contractions, which
// these replace: 1.6e-7, 3.1e-7, 2.1e-7, 2.4e-7). All 24 bits are there while the low plane is a normal bf16: an
// operand below 2^-110 keeps fewer. One that rounds above the largest bf16 (3.39e38), and an infinity, become NaN.
// Values that are not finite reach the tokens that the per-token statement lets them reach and no others
// (NonFinite below). The exact rule has the same form with a triangular solve per
// tile, but there it replaces per-token kernels at 1.0e-7 and came to 2.1e-7: it stays with those.
//
// What bounds it. One CTA (256 threads) walks one problem, so a launch is bound by the chain of a
// tile's stages: tensor products (55 cycles per 128x64x16 plane product, 64 per 128x128x16, the A operand is
// read from shared memory for each; the 312 of a Titans backward tile take 17.6k of its 47k cycles), loads
// and the conversion of every intermediate into planes with two warps per scheduler. The stage times are the
// same with 4 problems as with 128, so neither memory nor the other SMs bound them. Forward and backward,
// 128 problems x 2048 tokens, chunk 64: 1802 us with fp32 FMA contractions in shared memory, 1172 us so (Delta,
// 24 x 1000, chunk 48: 903 -> 633).
//
// Shared-memory matrices: element (row, col) of an R-row plane at (col/8)*(R*16) + row*16 + (col%8)*2,
// the canonical no-swizzle core-matrix layout with the 8-column chunk outermost. The same bytes serve
// as K-major operand (rows = M/N index) and as MN-major operand (rows = contraction index), so no
// transposed copy of anything exists. Every MMA has M = 128; where a product has 64 rows the other
// 64 lanes compute garbage from whatever follows in shared memory and are never read.
#pragma once

#include "nlh_common.cuh"
#include "tc_common.cuh"

namespace nlh {
namespace mtc {

using namespace nlh::tc;

constexpr int D = 64, DD = D * D;
constexpr int TMAX = 64;          // tokens per tile
constexpr int NT = 256;
constexpr int LDX = 68;           // leading dimension of the fp32 staging buffers
constexpr int LDS = 67;           // leading dimension of the scan buffers (64 columns + M0 + S0)
constexpr unsigned TCOLS = 512;
constexpr int MIN_TILE = 16;      // shorter tiles run the per-token register kernels

__device__ int g_mtc_timeout = 0;

// ── fp32 <-> three bf16 planes ──
__device__ __forceinline__ unsigned pack2(float a, float b)
{
    const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const unsigned*>(&t);
}
__device__ __forceinline__ float lo_f(unsigned p) { return __uint_as_float(p << 16); }
__device__ __forceinline__ float hi_f(unsigned p) { return __uint_as_float(p & 0xffff0000u); }
// 8 consecutive columns (chunk cc) of one row
__device__ __forceinline__ void store8(unsigned char* t, int R, int plane, int row, int cc, const float* v)
{
    unsigned h[4], m[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float x = v[2 * i], y = v[2 * i + 1];
        h[i] = pack2(x, y);
        const float x1 = x - lo_f(h[i]), y1 = y - hi_f(h[i]);
        m[i] = pack2(x1, y1);
        l[i] = pack2(x1 - lo_f(m[i]), y1 - hi_f(m[i]));
    }
    unsigned char* p = t + cc * (R * 16) + row * 16;
    *reinterpret_cast<uint4*>(p) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4*>(p + plane) = make_uint4(m[0], m[1], m[2], m[3]);
    *reinterpret_cast<uint4*>(p + 2 * plane) = make_uint4(l[0], l[1], l[2], l[3]);
}
__device__ __forceinline__ void load8(float* v, const unsigned char* t, int R, int plane, int row, int cc)
{
    const unsigned char* p = t + cc * (R * 16) + row * 16;
    const uint4 h = *reinterpret_cast<const uint4*>(p);
    const uint4 m = *reinterpret_cast<const uint4*>(p + plane);
    const uint4 l = *reinterpret_cast<const uint4*>(p + 2 * plane);
    const unsigned hh[4] = {h.x, h.y, h.z, h.w}, mm[4] = {m.x, m.y, m.z, m.w}, ll[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        v[2 * i] = (lo_f(ll[i]) + lo_f(mm[i])) + lo_f(hh[i]);
        v[2 * i + 1] = (hi_f(ll[i]) + hi_f(mm[i])) + hi_f(hh[i]);
    }
}
// 32 columns starting at chunk cc0
__device__ __forceinline__ void store32(unsigned char* t, int R, int plane, int row, int cc0, const float (&v)[32])
{
#pragma unroll
    for (int c = 0; c < 4; c++) store8(t, R, plane, row, cc0 + c, v + 8 * c);
}

// ── tensor product of split operands, issued by one thread ──
// D[128, N] (+)= A B with contraction length 16 * KSTEPS. a_mn / b_mn: the operand's rows are the
// contraction index (MN-major), otherwise its rows are the M / N index (K-major).
template <bool AMN, bool BMN, int KSTEPS = 4>
__device__ __forceinline__ void mma6(unsigned d, unsigned a, int a_plane, int a_R, unsigned b, int b_plane, int b_R,
                                     int N)
{
    const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((AMN ? 1u : 0u) << 15) | ((BMN ? 1u : 0u) << 16) |
                           ((unsigned)(N >> 3) << 17) | (8u << 24);
    const uint64_t ab = AMN ? make_desc(0, 128, a_R * 16) : make_desc(0, a_R * 16, 128);
    const uint64_t bb = BMN ? make_desc(0, 128, b_R * 16) : make_desc(0, b_R * 16, 128);
    const unsigned as = AMN ? 256 : a_R * 32, bs = BMN ? 256 : b_R * 32;    // bytes per 16 contraction steps
    unsigned acc = 0;
#pragma unroll 1
    for (int p = 0; p < 6; p++) {
        // plane pairs (2,0) (0,2) (1,1) (1,0) (0,1) (0,0)
        const unsigned pa = p == 0 ? 2u : (p == 2 || p == 3) ? 1u : 0u;
        const unsigned pb = p == 1 ? 2u : (p == 2 || p == 4) ? 1u : 0u;
        const unsigned a0 = a + pa * a_plane, b0 = b + pb * b_plane;
#pragma unroll 4
        for (int k = 0; k < KSTEPS; k++) {
            mma_bf16(d, ab + ((a0 + k * as) >> 4), bb + ((b0 + k * bs) >> 4), idesc, acc);
            acc = 1;
        }
    }
}

// ── gates of a tile ──
struct Tables {
    float4 gt[TMAX];            // r_t, eta_t, theta_t of the tile's tokens (padding: 1, 0, 0)
    float wM[TMAX], wS[TMAX];   // W(L-1,j), theta_j h(j,L-1)
    float tot[8];               // A_L, B_L, H_L
    float2 ab[TMAX];            // A_t, B_t
    float z[4][2 * TMAX];       // backward: row dots of the two column halves (zM, zS, gm, gs)
    float part[2][2 * TMAX];
    float red[8][4];
    unsigned long long bar[4];
    unsigned tmem;
};

// W of the tile as a table [TMAX][LDX], row t: W(t, j), of no meaning above the diagonal; tb.ab[t] = A_t, B_t;
// tb.wS[j] = theta_j h(j, L-1); tb.tot = A_L, B_L, H_L; tb.wM = W(L-1, .). One thread per column j, the
// recurrence runs over t: h' = eta_t h, Om' = r_t Om + h'. With one row per thread (63 unrolled steps in
// every warp) this stage took the MMA-issuing warp, which the others wait for, 4.6k cycles a tile; 2.8k so.
template <bool HAS_S>
__device__ __forceinline__ void decay_table(Tables& tb, float* Wt, int tid, int L)
{
    if (tid >= 0 && tid < TMAX) {
        const int j = tid;
        const float th = tb.gt[j].z;
        float om = 0.f, h = 0.f;
#pragma unroll 8
        for (int t = 0; t < TMAX; t++) {
            const float4 g = tb.gt[t];
            h = t == j ? 1.f : g.y * h;
            om = t == j ? 1.f : fmaf(g.x, om, h);      // starts here, whatever the gates before j hold
            Wt[t * LDX + j] = th * om;
            if (t == L - 1) { tb.wM[j] = t >= j ? th * om : 0.f; if (HAS_S) tb.wS[j] = t >= j ? th * h : 0.f; }
        }
    } else if (tid == TMAX) {
        float aa = 1.f, h = 1.f, om = 0.f;
#pragma unroll 8
        for (int t = 0; t < TMAX; t++) {
            const float4 g = tb.gt[t];
            aa *= g.x; h *= g.y; om = t == 0 ? h : fmaf(g.x, om, h);
            tb.ab[t] = make_float2(aa, HAS_S ? om : 0.f);
            if (t == L - 1) { tb.tot[0] = aa; tb.tot[1] = HAS_S ? om : 0.f; tb.tot[2] = h; }
        }
    }
}
// Row u of the table for this thread's 32 columns (half hf), and A_u, B_u; u = -1: no token before
__device__ __forceinline__ void decay_row(const Tables& tb, const float* Wt, int u, int hf, float (&w)[32], float& au, float& bu)
{
    if (u < 0) {
#pragma unroll
        for (int i = 0; i < 32; i++) w[i] = 0.f;
        au = 1.f; bu = 0.f;
        return;
    }
    const float* row = Wt + u * LDX + hf * 32;
    const float2 ab = tb.ab[u];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const float4 x = *reinterpret_cast<const float4*>(row + 4 * i);
        w[4 * i] = x.x; w[4 * i + 1] = x.y; w[4 * i + 2] = x.z; w[4 * i + 3] = x.w;
    }
    au = ab.x; bu = ab.y;
}

__device__ __forceinline__ void ld32(float (&v)[32], const float* __restrict__ p, bool ok)
{
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const float4 x = ok ? *reinterpret_cast<const float4*>(p + 4 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
    }
}
__device__ __forceinline__ void st32(float* p, const float (&v)[32])
{
#pragma unroll
    for (int i = 0; i < 8; i++)
        *reinterpret_cast<float4*>(p + 4 * i) = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
}
// Global memory is read and written in units of 8 rows x 32 columns per warp (a lane: 8 columns of one
// row): 8 lines of 128 bytes per instruction, where one row per lane touches 32. Unit i of a warp:
// rows 32 i + 8 (warp / 2) .. + 7, columns 32 (warp % 2) .. + 31; 64 rows are units 0 and 1.
struct Unit {
    int row0, cc;              // row of unit 0; 8-column chunk
    __device__ __forceinline__ Unit(int warp, int lane) : row0((warp >> 1) * 8 + (lane & 7)), cc((warp & 1) * 4 + (lane >> 3)) {}
    __device__ __forceinline__ int row(int i) const { return row0 + 32 * i; }
};
__device__ __forceinline__ void ld8(float* v, const float* __restrict__ p)
{
    const float4 x = *reinterpret_cast<const float4*>(p), y = *reinterpret_cast<const float4*>(p + 4);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
}
// rows past the tile's L tokens: row 0 is read and dropped, so that every load is in flight at once
__device__ __forceinline__ void ld8_row(float* v, const float* __restrict__ tile, int r, int L)
{
    ld8(v, tile + (r < L ? r : 0) * D);
}
__device__ __forceinline__ void zero_past(float* v, int r, int L)
{
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = r < L ? v[j] : 0.f;
}
__device__ __forceinline__ void st8(float* p, const float* v)
{
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
// 8 columns of one row of a staged matrix to global memory
__device__ __forceinline__ void copy8(float* g, const float* s)
{
    const float4 x = *reinterpret_cast<const float4*>(s), y = *reinterpret_cast<const float4*>(s + 4);
    *reinterpret_cast<float4*>(g) = x; *reinterpret_cast<float4*>(g + 4) = y;
}
// asks for `bytes` (a multiple of 16) of global memory to be brought into L2
__device__ __forceinline__ void l2_prefetch(const float* p, unsigned bytes)
{
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(p), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tload(float (&v)[32], unsigned taddr)
{
    unsigned r[32];
    tmem_ld_32x32b_x32(r, taddr);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

// Bounded wait on one of the CTA's barriers; each barrier is waited on once per commit.
struct Waiter {
    unsigned bar0, phases;
    bool dead;
    __device__ __forceinline__ void operator()(int i)
    {
        if (!dead) dead = !mbar_wait(bar0 + 8 * i, (phases >> i) & 1u, WAIT_LIMIT);
        phases ^= 1u << i;
        fence_after_sync();
    }
};
// ── values that are not finite ──
// W is zero above the diagonal, but 0 x NaN in a 64-token product would carry a token's NaN or infinity to
// the tokens on the wrong side of it. Elementwise products with W select; a product over tokens whose
// other operand holds such a value is formed again over the tokens that belong to it, in fp32 FMA.
struct NonFinite {
    float z = 0.f;
    __device__ __forceinline__ void add(const float (&v)[8])
    {
#pragma unroll
        for (int j = 0; j < 8; j++) z = fmaf(v[j], 0.f, z);
    }
    __device__ __forceinline__ bool any() const { return !(z == 0.f); }
};
__device__ __forceinline__ float plane_element(const unsigned char* t, int R, int plane, int row, int col)
{
    const unsigned char* p = t + (col >> 3) * (R * 16) + row * 16 + (col & 7) * 2;
    auto f = [](const unsigned char* q) { return __uint_as_float((unsigned)*reinterpret_cast<const unsigned short*>(q) << 16); };
    return (f(p + 2 * plane) + f(p + plane)) + f(p);
}
// s = sum over tokens j0 <= j < j1 of a(j) times 32 columns of token j; b(v, j, c): 8 columns from chunk c of 4
template <class A, class B>
__device__ __forceinline__ void sum_tokens(float (&s)[32], int j0, int j1, A a, B b)
{
#pragma unroll
    for (int i = 0; i < 32; i++) s[i] = 0.f;
#pragma unroll 1
    for (int j = j0; j < j1; j++) {
        const float w = a(j);
#pragma unroll
        for (int c = 0; c < 4; c++) {
            float v[8];
            b(v, j, c);
#pragma unroll
            for (int i = 0; i < 8; i++) s[8 * c + i] = fmaf(w, v[i], s[8 * c + i]);
        }
    }
}

// all generic-proxy writes to shared memory and TMEM reads so far are ordered before the MMAs that one
// thread issues after it
__device__ __forceinline__ void publish()
{
    fence_async_proxy();
    fence_before_sync();
    __syncthreads();
}
// the same, and whether any thread found something
__device__ __forceinline__ bool publish_or(bool found)
{
    fence_async_proxy();
    fence_before_sync();
    return __syncthreads_or(found) != 0;
}

// ───────────────────────────────── forward ─────────────────────────────────
constexpr int F_KQ = 0, F_MS = 49152, F_WP = 98304, F_E = 122880, F_EW = 147456, F_X = 196608;
constexpr int F_TAB = F_X + TMAX * LDX * 4;
constexpr int FWD_SMEM = F_TAB + (int)sizeof(Tables);

// T tokens per tile = per frozen chunk.
// States are stored at every tile start and after the last token.
template <int RULE>
__global__ void __launch_bounds__(NT, 1) tile_fwd_kernel(FwdArgs a, int T)
{
    constexpr bool HAS_S = (RULE == RULE_TITANS);
    extern __shared__ __align__(1024) unsigned char sm[];
    Tables& tb = *reinterpret_cast<Tables*>(sm + F_TAB);
    float* Xb = reinterpret_cast<float*>(sm + F_X);      // right-hand side, then E, fp32
    float* Wt = reinterpret_cast<float*>(sm + F_E);      // table of W until the errors take its place
    const int tid = threadIdx.x, warp = uniform_warp();
    const int R = (warp & 3) * 32 + (tid & 31), hf = warp >> 2;     // TMEM lane, column half
    const int dt = tid - 160;                                       // columns of the decay table: warps 5 to 7
    const int tr = R & 63;                                          // token (or state row) of this thread
    const bool krow = R < 64;                                       // K / M rows, else Q / S rows
    const int b = blockIdx.x;
    const Unit un(warp, tid & 31);
    const size_t su = (size_t)b * a.in_stride_tok * D + un.cc * 8;
    const float* alg = a.alpha + (size_t)b * a.in_stride_tok;
    const float* thg = a.theta + (size_t)b * a.in_stride_tok;
    const float* etg = HAS_S ? a.eta + (size_t)b * a.in_stride_tok : nullptr;
    float* yg = a.y + (size_t)b * a.seq_len * D + un.cc * 8;
    const size_t sgo = (size_t)b * a.out_stride + un.cc * 8;
    float* Sb = reinterpret_cast<float*>(sm + F_EW);     // tile-end states on their way out, fp32
    float* Yb = reinterpret_cast<float*>(sm + F_E);      // outputs on their way out, fp32
    const int ntile = (a.seq_len + T - 1) / T;

    if (tid == 0) { mbar_init(smem_u32(&tb.bar[0]), 1); mbar_init(smem_u32(&tb.bar[1]), 1); mbar_init(smem_u32(&tb.bar[2]), 1); }
    if (warp == 0) tmem_alloc_cols(reinterpret_cast<unsigned char*>(&tb.tmem), TCOLS);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const unsigned tm = tb.tmem;
    const unsigned trow = tm + ((unsigned)((warp & 3) * 32) << 16) + hf * 32;
    Waiter wait{smem_u32(&tb.bar[0]), 0u, false};
    const unsigned kq = smem_u32(sm + F_KQ), ms = smem_u32(sm + F_MS), wp = smem_u32(sm + F_WP), ep = smem_u32(sm + F_E),
                   ew = smem_u32(sm + F_EW);

    float st[32];                     // fp32 row of M (krow) or S
    if (HAS_S || krow) {
        ld32(st, (krow ? a.m_init : a.s_init) + (size_t)b * a.init_stride + tr * D + hf * 32, true);
        store32(sm + F_MS, 128, 16384, R, hf * 4, st);
        st32((krow ? a.m_out : a.s_out) + (size_t)b * a.out_stride + tr * D + hf * 32, st);
    }
    float x[4][8], v[2][8], gal = 0.f, gth = 0.f, get = 0.f;
    auto fetch = [&](int c) {         // this thread's units (K 0, 1, Q 2, 3, V) and gates of tile c
        const int t0 = c * T, L = min(T, a.seq_len - t0);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = un.row(i & 1);
            ld8_row(x[i], (i < 2 ? a.k : a.q) + su + (size_t)t0 * D, r, L);
            if (i < 2) ld8_row(v[i], a.v + su + (size_t)t0 * D, r, L);
        }
        if (tid < TMAX) {
            gal = (tid < L) ? alg[t0 + tid] : 0.f;
            gth = (tid < L) ? thg[t0 + tid] : 0.f;
            get = (HAS_S && tid < L) ? etg[t0 + tid] : 0.f;
        }
    };
    if (ntile > 0) fetch(0);

    for (int c = 0; c < ntile; c++) {
        const int t0 = c * T, L = min(T, a.seq_len - t0);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            zero_past(x[i], un.row(i & 1), L);
            if (i < 2) zero_past(v[i], un.row(i), L);
            store8(sm + F_KQ, 128, 16384, un.row(i), un.cc, x[i]);
            if (i < 2) st8(Xb + un.row(i) * LDX + un.cc * 8, v[i]);
        }
        if (tid < TMAX) tb.gt[tid] = make_float4(1.0f - gal, get, gth, 0.f);
        publish();
        if (warp == 0 && elect_one()) {
            fence_after_sync();
            mma6<false, false>(tm, kq, 16384, 128, ms, 16384, 128, HAS_S ? 128 : 64);     // K,Q x M0,S0
            mma6<false, false>(tm + 128, kq, 16384, 128, kq, 16384, 128, 64);             // K,Q x K
            mma_commit(smem_u32(&tb.bar[0]));
        }
        float w[32], au, bu;
        const int u = krow ? -1 : tr;
        decay_table<HAS_S>(tb, Wt, dt, L);
        __syncthreads();
        decay_row(tb, Wt, u, hf, w, au, bu);
        wait(0);
        float acc[32], p[32];
        tload(acc, trow);
#pragma unroll
        for (int i = 0; i < 32; i++) acc[i] *= au;
        if (HAS_S && !krow) {
            tload(p, trow + 64);
#pragma unroll
            for (int i = 0; i < 32; i++) acc[i] = fmaf(bu, p[i], acc[i]);
        }
        tload(p, trow + 128);
        if (krow) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float4 v4 = *reinterpret_cast<const float4*>(Xb + tr * LDX + hf * 32 + 4 * i);
                acc[4 * i] -= v4.x; acc[4 * i + 1] -= v4.y; acc[4 * i + 2] -= v4.z; acc[4 * i + 3] -= v4.w;
            }
            st32(Xb + tr * LDX + hf * 32, acc);
        } else {
#pragma unroll
            for (int i = 0; i < 32; i++) p[i] = hf * 32 + i <= tr ? p[i] * -w[i] : 0.f;
            store32(sm + F_WP, 64, 8192, tr, hf * 4, p);
        }
        if (c + 1 < ntile) fetch(c + 1);         // lands under the products
        __syncthreads();
        // E and its tile-end weighted copies as planes
        NonFinite nf;
#pragma unroll 1
        for (int i = 0; i < 2; i++) {
            const int row = un.row(i);
            const float wm = tb.wM[row], wsv = HAS_S ? tb.wS[row] : 0.f;
            float e[8], s[8];
            ld8(e, Xb + row * LDX + un.cc * 8);
            nf.add(e);
            store8(sm + F_E, 64, 8192, row, un.cc, e);
#pragma unroll
            for (int j = 0; j < 8; j++) s[j] = e[j] * wm;
            store8(sm + F_EW, 64, 16384, row, un.cc, s);
            if (HAS_S) {
#pragma unroll
                for (int j = 0; j < 8; j++) s[j] = e[j] * wsv;
                store8(sm + F_EW, 64, 16384, row, 8 + un.cc, s);
            }
        }
        const bool again = publish_or(nf.any());
        if (warp == 0 && elect_one()) {
            fence_after_sync();
            mma6<true, true>(tm + 256, ew, 16384, 64, kq, 16384, 128, 64);              // [Ew Es]^T K
            mma_commit(smem_u32(&tb.bar[1]));
            mma6<false, true>(tm + 192, wp - 1024, 8192, 64, ep, 8192, 64, 64);         // rows 64..127: -(W o P) E
            mma_commit(smem_u32(&tb.bar[2]));
        }
        // tile-end states while the outputs' product runs (the partner row is read before anyone
        // overwrites the planes)
        const float At = tb.tot[0], Bt = tb.tot[1], Ht = tb.tot[2];
#pragma unroll
        for (int i = 0; i < 32; i++) st[i] *= krow ? At : Ht;
        if (HAS_S && krow) {
#pragma unroll
            for (int c8 = 0; c8 < 4; c8++) {
                float s[8];
                load8(s, sm + F_MS, 128, 16384, 64 + tr, hf * 4 + c8);
#pragma unroll
                for (int i = 0; i < 8; i++) st[8 * c8 + i] = fmaf(Bt, s[i], st[8 * c8 + i]);
            }
        }
        wait(1);
        tload(p, trow + 256);
        __syncthreads();
        if (HAS_S || krow) {
#pragma unroll
            for (int i = 0; i < 32; i++) st[i] -= p[i];
            store32(sm + F_MS, 128, 16384, R, hf * 4, st);
            st32(Sb + R * LDX + hf * 32, st);          // the weighted errors have been consumed
        }
        wait(2);
        tload(p, trow + 192);
        if (!krow) {
            if (again)
                sum_tokens(p, 0, tr + 1, [&](int j) { return plane_element(sm + F_WP, 64, 8192, tr, j); },
                           [&](float (&v8)[8], int j, int c8) { ld8(v8, Xb + j * LDX + hf * 32 + c8 * 8); });
#pragma unroll
            for (int i = 0; i < 32; i++) p[i] += acc[i];
            st32(Yb + tr * LDX + hf * 32, p);          // and so have the errors
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int r = un.row(i);
            copy8(a.m_out + sgo + (size_t)(c + 1) * DD + r * D, Sb + r * LDX + un.cc * 8);
            if (HAS_S) copy8(a.s_out + sgo + (size_t)(c + 1) * DD + r * D, Sb + (64 + r) * LDX + un.cc * 8);
            if (r < L) copy8(yg + (size_t)(t0 + r) * D, Yb + r * LDX + un.cc * 8);
        }
    }
    if (wait.dead && (tid & 31) == 0) atomicExch(&g_mtc_timeout, 1);
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_free_cols(tm, TCOLS);
}

// ───────────────────────────────── backward ────────────────────────────────
constexpr int B_KQ = 0, B_YF = 49152, B_WZ = 98304, B_X = 147456, B_E = 196608;
constexpr int B_TAB = B_E + 24576;
constexpr int BWD_SMEM = B_TAB + (int)sizeof(Tables);

// Chunk-boundary states are DD floats apart.
template <int RULE>
__global__ void __launch_bounds__(NT, 1) tile_bwd_kernel(BwdArgs a, int T)
{
    constexpr bool HAS_S = (RULE == RULE_TITANS);
    extern __shared__ __align__(1024) unsigned char sm[];
    Tables& tb = *reinterpret_cast<Tables*>(sm + B_TAB);
    float* Xb = reinterpret_cast<float*>(sm + B_WZ);                  // right-hand sides, fp32
    float* Ob = Xb + 2 * TMAX * LDX;                                  // dK and dQ on their way out, fp32
    float* Sd = reinterpret_cast<float*>(sm + B_X);                   // scan buffers X -> Xd, and Xs
    float* Ss = reinterpret_cast<float*>(sm + B_X + 17408);
    float* Gx = reinterpret_cast<float*>(sm + B_E);                   // G_M rows for the S rows
    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    const int R = (warp & 3) * 32 + lane, hf = warp >> 2;
    const int dt = tid - 160;          // columns of the decay table: warps 5 to 7
    const int tr = R & 63;
    const bool krow = R < 64;
    const int b = blockIdx.x;
    const Unit un(warp, lane);
    const size_t so = (size_t)b * a.seq_len * D, go = (size_t)b * a.seq_len;
    const size_t su = so + un.cc * 8;
    const float* mtraj = a.m_traj + (size_t)b * a.traj_stride;
    const float* straj = HAS_S ? a.s_traj + (size_t)b * a.traj_stride : nullptr;
    const int n = a.t_end - a.t_start;
    const int ntile = (n + T - 1) / T;

    if (tid == 0) { mbar_init(smem_u32(&tb.bar[0]), 1); mbar_init(smem_u32(&tb.bar[1]), 1); }
    if (warp == 0) tmem_alloc_cols(reinterpret_cast<unsigned char*>(&tb.tmem), TCOLS);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const unsigned tm = tb.tmem;
    const unsigned trow = tm + ((unsigned)((warp & 3) * 32) << 16) + hf * 32;
    Waiter wait{smem_u32(&tb.bar[0]), 0u, false};
    const unsigned kq = smem_u32(sm + B_KQ), yf = smem_u32(sm + B_YF), wz = smem_u32(sm + B_WZ), xx = smem_u32(sm + B_X),
                   ep = smem_u32(sm + B_E);
    unsigned char* const kqp = sm + B_KQ;
    unsigned char* const yfp = sm + B_YF;
    unsigned char* const xxp = sm + B_X;

    float g[32];                       // row of G_M (krow) or G_S, columns of this half
    {
        const float* seed = krow ? a.d_m_seed : a.d_s_seed;
        ld32(g, seed + (size_t)b * DD + tr * D + hf * 32, (HAS_S || krow) && seed != nullptr);
    }

    float gal = 0.f, gth = 0.f, get = 0.f;             // gates of the tile to come, one token per thread
    auto fetch_gates = [&](int c) {
        const int t0 = a.t_start + c * T, L = min(T, n - c * T);
        const bool in = tid < L;
        gal = in ? a.alpha[go + t0 + tid] : 0.f;
        gth = in ? a.theta[go + t0 + tid] : 0.f;
        get = (in && HAS_S) ? a.eta[go + t0 + tid] : 0.f;
    };
    if (tid < TMAX) fetch_gates(ntile - 1);

    for (int c = ntile - 1; c >= 0; c--) {
        const int t0 = a.t_start + c * T, L = min(T, n - c * T);
        auto state_unit = [&](float (&x3)[8], int i) {   // unit i of M0 (0, 1) or S0 (2, 3)
            const float* mp = mtraj + (size_t)c * DD;
            const int r = un.row(i & 1), ofs = r * D + un.cc * 8;
            if (i < 2) ld8(x3, mp + ofs);
            else if (HAS_S) ld8(x3, straj + (size_t)c * DD + ofs);
            else {
#pragma unroll
                for (int j = 0; j < 8; j++) x3[j] = 0.f;
            }
        };
        // ── stage 1: operands; K K^T | Q K^T and K,Q x M0,S0 ──
        // The four units of each matrix go round one loop with the next unit's loads in flight (as fast as
        // straight-line code with all 24 loads at once, 8k cycles a tile, and a third of its size).
        NonFinite nf;                                // in K, Q, dY
        {
            float x[8], y[8], x3[8];
            auto get = [&](int i) {                  // K, V, M0 rows, then Q, dY, S0 rows
                const int r = un.row(i & 1);
                ld8_row(x, (i < 2 ? a.k : a.q) + su + (size_t)t0 * D, r, L);
                ld8_row(y, (i < 2 ? a.v : a.d_y) + su + (size_t)t0 * D, r, L);
                state_unit(x3, i);
            };
            get(0);
#pragma unroll 1
            for (int i = 0; i < 4; i++) {
                float xc[8], yc[8], x3c[8];
                const int r = un.row(i);
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const bool in = un.row(i & 1) < L;
                    xc[j] = in ? x[j] : 0.f; yc[j] = in ? y[j] : 0.f; x3c[j] = x3[j];
                }
                if (i < 3) get(i + 1);
                nf.add(xc);
                if (i >= 2) nf.add(yc);
                store8(kqp, 128, 16384, r, un.cc, xc);
                store8(xxp, 128, 16384, r, un.cc, x3c);
                if (i < 2) st8(Xb + r * LDX + un.cc * 8, yc);
                else store8(yfp, 128, 16384, r, un.cc, yc);
            }
        }
        if (tid < TMAX) {
            tb.gt[tid] = make_float4(1.0f - gal, get, gth, 0.f);
            if (c > 0) fetch_gates(c - 1);
        }
        const bool again = publish_or(nf.any());
        if (warp == 0 && elect_one()) {
            fence_after_sync();
            mma6<false, false>(tm, kq, 16384, 128, kq, 16384, 128, 64);
            mma6<false, false>(tm + 64, kq, 16384, 128, xx, 16384, 128, HAS_S ? 128 : 64);
            mma_commit(smem_u32(&tb.bar[0]));
        }
        if (c > 0 && tid < 4) {                       // the next tile's streams, while this one is worked on
            const float* nx = (tid == 0 ? a.k : tid == 1 ? a.q : tid == 2 ? a.v : a.d_y) + so + (size_t)(t0 - T) * D;
            l2_prefetch(nx, (unsigned)T * D * 4);
        } else if (c > 0 && tid < 6) {
            if (tid == 4) l2_prefetch(mtraj + (size_t)(c - 1) * DD, DD * 4);
            else if (HAS_S) l2_prefetch(straj + (size_t)(c - 1) * DD, DD * 4);
        }
        float w[32], p[32], au, bu;
        const int u = krow ? -1 : tr;
        float dots[2] = {0.f, 0.f};                   // <M0, G_M> or <S0, G_S>; <S0, G_M>
#pragma unroll
        for (int c8 = 0; c8 < 4; c8++) {
            float m[8];
            if (HAS_S || krow) {
                load8(m, xxp, 128, 16384, R, hf * 4 + c8);
#pragma unroll
                for (int i = 0; i < 8; i++) dots[0] = fmaf(g[8 * c8 + i], m[i], dots[0]);
            }
            if (HAS_S && krow) {
                load8(m, xxp, 128, 16384, 64 + tr, hf * 4 + c8);
#pragma unroll
                for (int i = 0; i < 8; i++) dots[1] = fmaf(g[8 * c8 + i], m[i], dots[1]);
            }
        }
        decay_table<HAS_S>(tb, Gx, dt, L);            // the errors' planes are free until stage 2
        dots[0] = warp_sum(dots[0]); dots[1] = warp_sum(dots[1]);
        if (lane == 0) { tb.red[warp][0] = dots[0]; tb.red[warp][1] = dots[1]; }
        __syncthreads();
        decay_row(tb, Gx, u, hf, w, au, bu);
        wait(0);
        tload(p, trow);                               // k_t . k_j or q_t . k_j
        {
            float acc[32];
            tload(acc, trow + 64);
            if (krow) {
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float4 v4 = *reinterpret_cast<const float4*>(Xb + tr * LDX + hf * 32 + 4 * i);
                    acc[4 * i] -= v4.x; acc[4 * i + 1] -= v4.y; acc[4 * i + 2] -= v4.z; acc[4 * i + 3] -= v4.w;
                }
                st32(Xb + tr * LDX + hf * 32, acc);
            } else {
                float zm = 0.f, zs = 0.f, y[32];
#pragma unroll
                for (int c8 = 0; c8 < 4; c8++) load8(y + 8 * c8, yfp, 128, 16384, R, hf * 4 + c8);
#pragma unroll
                for (int i = 0; i < 32; i++) zm = fmaf(y[i], acc[i], zm);
                if (HAS_S) {
                    tload(acc, trow + 128);
#pragma unroll
                    for (int i = 0; i < 32; i++) zs = fmaf(y[i], acc[i], zs);
                }
                tb.z[0][hf * 64 + tr] = zm; tb.z[1][hf * 64 + tr] = zs;
            }
        }
        __syncthreads();
        // ── stage 2: E planes, W o P, G planes; right-hand side of F, E x G ──
#pragma unroll 1
        for (int i = 0; i < 2; i++) {
            float e[8];
            ld8(e, Xb + un.row(i) * LDX + un.cc * 8);
            store8(sm + B_E, 64, 8192, un.row(i), un.cc, e);
        }
        if (!krow) {
            float wpv[32];
#pragma unroll
            for (int i = 0; i < 32; i++) wpv[i] = hf * 32 + i <= tr ? w[i] * p[i] : 0.f;
            store32(sm + B_WZ + 24576, 64, 8192, tr, hf * 4, wpv);
        }
        store32(xxp, 128, 16384, R, hf * 4, g);
        publish();
        if (warp == 0 && elect_one()) {
            fence_after_sync();
            mma6<false, false>(tm, kq, 16384, 128, xx, 16384, 128, HAS_S ? 128 : 64);              // K G^T
            mma6<true, true>(tm + 128, wz + 24576, 8192, 64, yf + 1024, 16384, 128, 64);           // (W o P)^T dY
            mma_commit(smem_u32(&tb.bar[0]));
            mma6<false, true>(tm + 192, ep, 8192, 64, xx, 16384, 128, 64);                         // E G_M
            if (HAS_S) mma6<false, true>(tm + 256, ep, 8192, 64, xx + 1024, 16384, 128, 64);       // E G_S
            mma_commit(smem_u32(&tb.bar[1]));
        }
        wait(0);
        float dx[32];                                  // gradient of this thread's K or Q row
        if (krow) {
            const float wm = tb.wM[tr], wsv = HAS_S ? tb.wS[tr] : 0.f;
            float s[32];
            tload(dx, trow);
            tload(s, trow + 128);
            if (again)
                sum_tokens(s, tr, L, [&](int t) { return plane_element(sm + B_WZ + 24576, 64, 8192, t, tr); },
                           [&](float (&v8)[8], int t, int c8) { load8(v8, yfp, 128, 16384, 64 + t, hf * 4 + c8); });
#pragma unroll
            for (int i = 0; i < 32; i++) dx[i] = -fmaf(wm, dx[i], s[i]);
            if (HAS_S) {
                tload(s, trow + 64);
#pragma unroll
                for (int i = 0; i < 32; i++) dx[i] = fmaf(-wsv, s[i], dx[i]);
            }
            st32(Xb + tr * LDX + hf * 32, dx);
        }
        __syncthreads();
        wait(1);
        if (krow) {
            const float wm = tb.wM[tr], wsv = HAS_S ? tb.wS[tr] : 0.f;
            float gm = 0.f, gs = 0.f, s[32], s2[32];
            tload(s, trow + 192);
            if (HAS_S) tload(s2, trow + 256);
#pragma unroll
            for (int c8 = 0; c8 < 4; c8++) {
                float kk[8];
                load8(kk, kqp, 128, 16384, R, hf * 4 + c8);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    gm = fmaf(kk[i], s[8 * c8 + i], gm);
                    if (HAS_S) gs = fmaf(kk[i], s2[8 * c8 + i], gs);
                }
            }
#pragma unroll
            for (int i = 0; i < 32; i++) {
                dx[i] = -wm * s[i];
                if (HAS_S) dx[i] = fmaf(-wsv, s2[i], dx[i]);
            }
            tb.z[2][hf * 64 + tr] = gm; tb.z[3][hf * 64 + tr] = gs;
        }
        // ── stage 3: F planes, dV, M0/S0 planes again; N | R, F and dY x M0,S0 ──
#pragma unroll 1
        for (int i = 0; i < 2; i++) {
            const int r = un.row(i);
            float e[8];
            ld8(e, Xb + r * LDX + un.cc * 8);
            store8(yfp, 128, 16384, r, un.cc, e);
            if (r < L) {
#pragma unroll
                for (int j = 0; j < 8; j++) e[j] = -e[j];
                st8(a.d_v + su + (size_t)(t0 + r) * D, e);
            }
        }
        {
            float x3[8];
            state_unit(x3, 0);
#pragma unroll 1
            for (int i = 0; i < 4; i++) {
                float x3c[8];
#pragma unroll
                for (int j = 0; j < 8; j++) x3c[j] = x3[j];
                if (i < 3) state_unit(x3, i + 1);
                store8(xxp, 128, 16384, un.row(i), un.cc, x3c);
            }
        }
        publish();
        if (warp == 0 && elect_one()) {
            fence_after_sync();
            mma6<false, false>(tm, yf, 16384, 128, ep, 8192, 64, 64);                       // F,dY x E
            mma_commit(smem_u32(&tb.bar[0]));
            mma6<false, true>(tm + 64, yf, 16384, 128, xx, 16384, 128, 64);                 // F,dY x M0
            if (HAS_S) mma6<false, true>(tm + 128, yf, 16384, 128, xx + 1024, 16384, 128, 64);   // F,dY x S0
            mma_commit(smem_u32(&tb.bar[1]));
        }
        wait(0);
        {
            float s[32];
            tload(s, trow);                            // N row (krow) or R row
#pragma unroll
            for (int i = 0; i < 32; i++) { p[i] *= s[i]; s[i] = hf * 32 + i <= tr ? s[i] * -w[i] : 0.f; }
            if (!krow) store32(sm + B_WZ, 128, 16384, R, hf * 4, s);
            wait(1);
            if (!krow) {
                // every read of the state planes by the tensor cores is over: the scan buffers take their place
#pragma unroll
                for (int i = 0; i < 32; i++) Sd[tr * LDS + hf * 32 + i] = p[i];
                if (hf == 0) Sd[tr * LDS + 64] = tb.z[0][tr] + tb.z[0][64 + tr];
                else Sd[tr * LDS + 65] = tb.z[1][tr] + tb.z[1][64 + tr];
            }
            float s2[32];
            tload(s, trow + 64);
            if (krow) {
#pragma unroll
                for (int i = 0; i < 32; i++) dx[i] += s[i];
            } else {
                if (HAS_S) tload(s2, trow + 128);
#pragma unroll
                for (int i = 0; i < 32; i++) dx[i] = HAS_S ? fmaf(bu, s2[i], au * s[i]) : au * s[i];
            }
        }
        publish();
        // ── stage 4: -(W o R) K and -(W o R)^T Q; gate scans under them ──
        if (warp == 4 && elect_one()) {                // warps 0 to 2 have the scans to do
            fence_after_sync();
            mma6<false, true>(tm + 192, wz, 16384, 128, kq, 16384, 128, 64);        // rows 64..127: -(W o R) K
            mma6<true, true>(tm + 256, wz + 1024, 16384, 128, kq + 1024, 16384, 128, 64);  // -(W o R)^T Q
            mma_commit(smem_u32(&tb.bar[0]));
        }
        if (tid < 66) {                                // decayed scans, one column per thread
            const int j = tid;
            float sM, sS;
            if (j < 64) { sM = tb.z[2][j] + tb.z[2][64 + j]; sS = tb.z[3][j] + tb.z[3][64 + j]; }
            else {
                sM = 0.f; sS = 0.f;
#pragma unroll
                for (int wq = 0; wq < 8; wq++) {
                    const bool kw = (wq & 3) < 2;
                    if (j == 64 && kw) sM += tb.red[wq][0];
                    if (j == 65 && kw) sM += tb.red[wq][1];
                    if (j == 65 && !kw) sS += tb.red[wq][0];
                }
            }
            float xd = sM, xs = sS, gr = 1.f, ge = 1.f;      // r and eta of the row above
#pragma unroll 1
            for (int s0 = 48; s0 >= 0; s0 -= 16) {
                if (s0 >= L) continue;
                float xv[16];
#pragma unroll
                for (int i = 0; i < 16; i++) xv[i] = Sd[(s0 + i) * LDS + j];
#pragma unroll
                for (int i = 15; i >= 0; i--) {
                    const float4 gn = tb.gt[s0 + i];
                    const bool in = s0 + i < L;            // rows past the tile are written but never read
                    xd = in ? fmaf(gr, xd, xv[i]) : xd;
                    xs = in ? fmaf(ge, xs, xd) : xs;
                    gr = in ? gn.x : 1.f; ge = in ? gn.y : 1.f;
                    xv[i] = xd;
                    Ss[(s0 + i) * LDS + j] = xs;
                }
#pragma unroll
                for (int i = 0; i < 16; i++) Sd[(s0 + i) * LDS + j] = xv[i];
            }
            if (j < L) a.d_theta[go + t0 + j] = -Ss[j * LDS + j];
        }
        __syncthreads();
        float s1 = 0.f, s2 = 0.f, hend = 1.f;
        if (!krow) {
            // row t + 1 of the decayed scans against row t of W and of theta_j h(j,t)
            const float* xd = Sd + (tr + 1) * LDS + hf * 32;
            const float* xs = Ss + (tr + 1) * LDS + hf * 32;
            if (tr + 1 < L) {
#pragma unroll
                for (int i = 0; i < 32; i++) s1 = hf * 32 + i <= tr ? fmaf(w[i], xd[i], s1) : s1;
                if (HAS_S) {
                    float hh = 1.f;
                    const int jh = hf * 32;
                    float4 gn = tb.gt[hf == 0 ? 32 : 63];          // gates of column j + 1
                    if (hf == 0) {
#pragma unroll 8
                        for (int j = 62; j >= 32; j--) { const float et = tb.gt[j + 1].y; hh = (j < tr) ? hh * et : hh; }
                    }
#pragma unroll 8
                    for (int j = 31; j >= 0; j--) {
                        const float4 gj = tb.gt[jh + j];
                        hh = (jh + j < tr) ? hh * gn.y : hh;
                        s2 = (jh + j <= tr) ? fmaf(gj.z * hh, xs[j], s2) : s2;
                        gn = gj;
                    }
                    hend = hh * tb.gt[0].y;
                }
            }
            tb.part[0][hf * 64 + tr] = s1; tb.part[1][hf * 64 + tr] = s2;
        }
        // G_M rows for the S rows of the carry
        if (krow && HAS_S) st32(Gx + tr * LDX + hf * 32, g);
        __syncthreads();
        if (!krow && hf == 0 && tr + 1 < L) {
            const int t = tr + 1;
            a.d_alpha[go + t0 + t] = -(fmaf(au, Sd[t * LDS + 64], bu * Sd[t * LDS + 65]) - (tb.part[0][tr] + tb.part[0][64 + tr]));
            if (HAS_S) a.d_eta[go + t0 + t] = hend * Ss[t * LDS + 65] - (tb.part[1][tr] + tb.part[1][64 + tr]);
        }
        if (tid == 0) {
            a.d_alpha[go + t0] = -Sd[64];
            if (HAS_S) a.d_eta[go + t0] = Ss[65];
        }
        wait(0);
        {
            float s[32];
            tload(s, trow + (krow ? 256 : 192));
            if (again)                                 // dK: tokens from this one on; dQ: tokens up to this one
                sum_tokens(s, krow ? tr : 0, krow ? L : tr + 1,
                           [&](int j) { return plane_element(sm + B_WZ, 128, 16384, 64 + (krow ? j : tr), krow ? tr : j); },
                           [&](float (&v8)[8], int j, int c8) { load8(v8, kqp, 128, 16384, (krow ? 64 : 0) + j, hf * 4 + c8); });
#pragma unroll
            for (int i = 0; i < 32; i++) dx[i] += s[i];
        }
        __syncthreads();                               // the scan buffers have been read
        // ── stage 5: carry. [diag(a) F ; diag(A) dY | diag(b) F ; diag(B) dY]^T [K ; Q] ──
#pragma unroll 1
        for (int c8 = 0; c8 < 4; c8++) {
            float f[8], s[8];
            load8(f, yfp, 128, 16384, R, hf * 4 + c8);
#pragma unroll
            for (int i = 0; i < 8; i++) s[i] = f[i] * au;
            store8(sm + B_WZ, 128, 32768, R, hf * 4 + c8, s);
            if (HAS_S) {
#pragma unroll
                for (int i = 0; i < 8; i++) s[i] = krow ? 0.f : f[i] * bu;
                store8(sm + B_WZ, 128, 32768, R, 8 + hf * 4 + c8, s);
            }
        }
        publish();
        if (warp == 0 && elect_one()) {
            fence_after_sync();
            mma6<true, true, 8>(tm + 320, wz, 32768, 128, kq, 16384, 128, 64);
            mma_commit(smem_u32(&tb.bar[0]));
        }
        const float At = tb.tot[0], Bt = tb.tot[1], Ht = tb.tot[2];
        if (krow) {
#pragma unroll
            for (int i = 0; i < 32; i++) g[i] *= At;
        } else if (HAS_S) {
            const float* gr = Gx + tr * LDX + hf * 32;
#pragma unroll
            for (int i = 0; i < 32; i++) g[i] = fmaf(Bt, gr[i], Ht * g[i]);
        }
        wait(0);
        {
            float s[32];
            tload(s, trow + 320);
            if (again && HAS_S) {
                if (!krow)                             // without the K rows, whose weights for G_S are zero
                    sum_tokens(s, 0, L, [&](int t) { return plane_element(sm + B_WZ, 128, 32768, 64 + t, 64 + tr); },
                               [&](float (&v8)[8], int t, int c8) { load8(v8, kqp, 128, 16384, 64 + t, hf * 4 + c8); });
                __syncthreads();                       // the staged rows below go over those weights
            }
            if (HAS_S || krow) {
#pragma unroll
                for (int i = 0; i < 32; i++) g[i] += s[i];
            }
        }
        st32(Ob + R * LDX + hf * 32, dx);
        fence_before_sync();
        __syncthreads();
#pragma unroll 1
        for (int i = 0; i < 4; i++) {
            const int r = un.row(i & 1);
            if (r < L) copy8((i < 2 ? a.d_k : a.d_q) + su + (size_t)(t0 + r) * D, Ob + un.row(i) * LDX + un.cc * 8);
        }
        __syncthreads();                               // the next tile's planes go over the staged rows
    }

    if ((HAS_S || krow) && a.d_m_out != nullptr) {
        float* o = (krow ? a.d_m_out : a.d_s_out) + tr * D + hf * 32;
        if (a.atomic_out) {
#pragma unroll
            for (int i = 0; i < 32; i++) atomicAdd(o + i, g[i]);
        } else st32(o + (size_t)b * DD, g);
    }
    if (wait.dead && lane == 0) atomicExch(&g_mtc_timeout, 1);
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_free_cols(tm, TCOLS);
}

}  // namespace mtc
}  // namespace nlh
