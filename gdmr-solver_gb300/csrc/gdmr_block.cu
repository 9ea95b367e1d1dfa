// Blocked Krylov steps of the complex64 refined cycles.
//
// The Krylov loop (arnoldiDMR, gDMR.cu:2069-2328) reads the whole own basis V twice a step: once for
// the coefficients V^H w, once for w - V c.  For a batch with resident bases of a few gigabytes
// those two passes were two thirds of a restart cycle, at 0.9-1.06 of the copy peak: nothing to
// gain per pass, only by making fewer passes.  Here BK_S = 3 steps share them.  From the last basis vector v_j
//   y_1 = s (I - W W^H)(A - t) v_j,   y_{b+1} = s (I - W W^H)(A - t) y_b
// are formed first (operator and shared deflation vectors only), then one pass over V gives
// C = V^H Y and G = Y^H Y, and a second writes the three new vectors (Y - V C) R^-1 with
// R^H R = G - C^H C (Cholesky).  The Hessenberg columns follow from the recurrence
//   A y_b = W a_{b+1} / s + (y_{b+1} / s + t y_b)   with   y_b = V C_b + V_new R_b
// in FP64.  The space is the classical loop's; t (the mean of the Hessenberg's Krylov diagonal, the
// centre of the spectrum the basis sees) and s (one over the last subdiagonal) keep Y well conditioned:
// on the Helmholtz operators the smallest squared pivot is 0.05 of its column's squared norm.
// In complex64 on a 24^3 Helmholtz operator, m = 48, k = 24: largest
// departure of [W V] from orthonormality 4e-4 (3.6e-3 step by step) and of A V = [W V] H from
// equality 8e-7 of ||H|| (4.6e-6 step by step), the same number of cycles.  Four steps a block have pivots of
// 0.013 and an orthogonality of 1.4e-2, so three it is.
//
// Measured (whole solves to 1e-10, the same cycle counts): 96^3, 64 systems, m = 48, k = 24: 1850 to
// 1250 ms; 64^3, 16 systems: 663 to 515 ms; one system at 128^3, m = 60, k = 20: 655 to 612 ms.
//
// A block whose pivot falls below BK_ILL of its column (an exhausted or badly scaled Krylov space) sets
// SysState::ill: the caller drops the cycle's correction of that system and runs step by step while the system
// is in flight.  (s-step bases: Chronopoulos and Gear 1989; Hoemmen 2010.)
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "gdmr_kernels.cuh"

namespace gdmr {

namespace {

constexpr int NTB = 256, NWB = NTB / 32;
constexpr int BK_S = KRYLOV_BLOCK;
constexpr int BK_C = 2 * BK_S;          // real components a basis vector contributes to the projection
constexpr int BK_QMAX = 164;            // own basis vectors plus the block's (basisDim <= 160)
constexpr double BK_ILL = 1e-4;         // smallest squared pivot over squared column norm
static_assert(BK_S == 3, "the reduction below is laid out for blocks of three");

template <int VEC> struct Pk {
    float2 v[VEC];
};
template <int VEC> __device__ __forceinline__ Pk<VEC> ld(const float2 *p, long i0, int n) {
    Pk<VEC> r;
    if constexpr (VEC == 2) {
        float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i0 < n) f = *reinterpret_cast<const float4 *>(p + i0);   // n even: both elements or neither
        r.v[0] = make_float2(f.x, f.y);
        r.v[1] = make_float2(f.z, f.w);
    } else {
        r.v[0] = i0 < n ? p[i0] : make_float2(0.f, 0.f);
    }
    return r;
}
template <int VEC> __device__ __forceinline__ void st(float2 *p, long i0, int n, const Pk<VEC> &r) {
    if (i0 >= n) return;
    if constexpr (VEC == 2)
        *reinterpret_cast<float4 *>(p + i0) = make_float4(r.v[0].x, r.v[0].y, r.v[1].x, r.v[1].y);
    else
        p[i0] = r.v[0];
}
__device__ __forceinline__ void dotacc(float2 &acc, float2 a, float2 b) {   // acc += conj(a) b
    acc.x = fmaf(a.x, b.x, acc.x);
    acc.x = fmaf(a.y, b.y, acc.x);
    acc.y = fmaf(a.x, b.y, acc.y);
    acc.y = fmaf(-a.y, b.x, acc.y);
}
__device__ __forceinline__ void mulacc(float2 &acc, float2 a, float2 b) {   // acc += a b
    acc.x = fmaf(a.x, b.x, acc.x);
    acc.x = fmaf(-a.y, b.y, acc.x);
    acc.y = fmaf(a.x, b.y, acc.y);
    acc.y = fmaf(a.y, b.x, acc.y);
}
__device__ __forceinline__ void mulsub(float2 &acc, float2 a, float2 b) {   // acc -= a b
    acc.x = fmaf(-a.x, b.x, acc.x);
    acc.x = fmaf(a.y, b.y, acc.x);
    acc.y = fmaf(-a.x, b.y, acc.y);
    acc.y = fmaf(-a.y, b.x, acc.y);
}

// Warp sums of the 12 components v[6 u + 2 b + (re | im)] of two basis vectors u against three
// block vectors b, as a reduce-scatter butterfly: 13 shuffles instead of 60.  On return lane l
// with an even l holds the sum of component 6 [l & 16] + 3 [l & 8] + 2 [l & 4] + [l & 2] (not the
// lanes with both l & 4 and l & 2 set: they hold padding).
__device__ __forceinline__ float scatter12(float (&v)[12], int lane) {
    float a[6], b[3], c[2];
    {
        const bool hi = lane & 16;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const float keep = hi ? v[6 + i] : v[i], send = hi ? v[i] : v[6 + i];
            a[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
        }
    }
    {
        const bool hi = lane & 8;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const float keep = hi ? a[3 + i] : a[i], send = hi ? a[i] : a[3 + i];
            b[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
        }
    }
    {
        const bool hi = lane & 4;
        const float k0 = hi ? b[2] : b[0], k1 = hi ? 0.f : b[1], s0 = hi ? b[0] : b[2], s1 = hi ? b[1] : 0.f;
        c[0] = k0 + __shfl_xor_sync(0xffffffffu, s0, 4);
        c[1] = k1 + __shfl_xor_sync(0xffffffffu, s1, 4);
    }
    {
        const bool hi = lane & 2;
        const float keep = hi ? c[1] : c[0], send = hi ? c[0] : c[1];
        c[0] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
    }
    return c[0] + __shfl_xor_sync(0xffffffffu, c[0], 1);
}

// part[slot][G][6 i + 2 b + (re | im)]: <v_i, y_b> for the nv basis vectors, then <y_a, y_b>; y_b is
// basis slot nv + b.  HBM-bound: a CTA keeps the block's elements of a chunk in registers and streams
// the basis past them two vectors at a time: 96^3, 64 systems, nv = 13: 1083 us with the finish, 6.69 TB/s of its
// bytes (1185 us with four elements a thread).  FP32 sums over 256 elements a warp, then double-float.
template <int EPT, int VEC>
__global__ void __launch_bounds__(NTB, 2)
    k_block_proj(int n, int nv, const float2 *__restrict__ V0, size_t strideV, const int *__restrict__ act,
                 const SysState *__restrict__ state, double *__restrict__ part, int nch) {
    constexpr int NP = EPT / VEC;
    extern __shared__ dfr bp_ws[];                      // [warp][6 (nv + 3)]
    const int slot = blockIdx.x, s = act[slot], G = gridDim.y;
    if (state[s].broken) return;
    const float2 *V = V0 + (size_t)s * strideV;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, ncomp = BK_C * (nv + BK_S);
    dfr *ws = bp_ws + (size_t)warp * ncomp;
    for (int c = lane; c < ncomp; c += 32) ws[c] = dfr(0.f, 0.f);
    __syncwarp();
    // the component this lane ends up with (see scatter12)
    const int low = ((lane & 4) ? 2 : 0) + ((lane & 2) ? 1 : 0);
    const int u_of = (lane & 16) ? 1 : 0, c_of = ((lane & 8) ? 3 : 0) + low;
    const bool holds = !(lane & 1) && low < 3;
    for (int ch = blockIdx.y; ch < nch; ch += G) {
        const long c0 = (long)ch * NTB * EPT + (long)tid * VEC;
        Pk<VEC> y[BK_S][NP];
#pragma unroll
        for (int b = 0; b < BK_S; ++b)
#pragma unroll
            for (int e = 0; e < NP; ++e) y[b][e] = ld<VEC>(V + (size_t)(nv + b) * n, c0 + (long)e * NTB * VEC, n);
        auto pair = [&](const Pk<VEC>(&p)[NP], const Pk<VEC>(&q)[NP], int i0, bool two) {
            float2 a[2][BK_S];
#pragma unroll
            for (int b = 0; b < BK_S; ++b) {
                a[0][b] = a[1][b] = make_float2(0.f, 0.f);
#pragma unroll
                for (int e = 0; e < NP; ++e)
#pragma unroll
                    for (int j = 0; j < VEC; ++j) {
                        dotacc(a[0][b], p[e].v[j], y[b][e].v[j]);
                        dotacc(a[1][b], q[e].v[j], y[b][e].v[j]);
                    }
            }
            float v[12];
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int b = 0; b < BK_S; ++b) {
                    v[6 * u + 2 * b] = a[u][b].x;
                    v[6 * u + 2 * b + 1] = a[u][b].y;
                }
            const float sum = scatter12(v, lane);
            if (holds && (u_of == 0 || two)) {
                dfr &w = ws[BK_C * (i0 + u_of) + c_of];
                w = w + dfr(sum, 0.f);
            }
        };
        for (int i0 = 0; i0 < nv; i0 += 2) {
            Pk<VEC> p[NP], q[NP];
            const float2 *vp = V + (size_t)i0 * n, *vq = V + (size_t)(i0 + 1) * n;   // slot nv at most: y_1
#pragma unroll
            for (int e = 0; e < NP; ++e) {
                p[e] = ld<VEC>(vp, c0 + (long)e * NTB * VEC, n);
                q[e] = ld<VEC>(vq, c0 + (long)e * NTB * VEC, n);
            }
            pair(p, q, i0, i0 + 1 < nv);
        }
        pair(y[0], y[1], nv, true);
        pair(y[2], y[2], nv + 2, false);
    }
    __syncthreads();
    double *pp = part + (size_t)slot * ncomp * G;
    for (int c = tid; c < ncomp; c += NTB) {
        dfr t(0.f, 0.f);
#pragma unroll
        for (int w = 0; w < NWB; ++w) t = t + bp_ws[(size_t)w * ncomp + c];
        *reinterpret_cast<dfr *>(pp + (size_t)blockIdx.y * ncomp + c) = t;
    }
}

// v_new_b = sum_a y_a T_ab - sum_i v_i D_ib in place of y_b (basis slots nv .. nv + 2).  HBM-bound:
// reads nv + 3 vectors, writes three.  96^3, 64 systems, nv = 13: 1220 us, 7.06 TB/s of its bytes (1258 us with two
// vectors in flight; four elements a thread instead of eight: 1225-1390).  A zero T_bb (a system that broke down earlier) stores zeros.
template <int EPT, int VEC>
__global__ void __launch_bounds__(NTB, 2)
    k_block_update(int n, int nv, float2 *__restrict__ V0, size_t strideV, const int *__restrict__ act,
                   const float2 *__restrict__ dco, size_t dstride) {
    constexpr int NP = EPT / VEC, PU = 4;
    __shared__ float2 ds[BK_S * BK_QMAX], ts[BK_S * BK_S];
    const int slot = blockIdx.x, s = act[slot], tid = threadIdx.x;
    float2 *V = V0 + (size_t)s * strideV;
    const float2 *d = dco + (size_t)slot * dstride;
    if (tid < BK_S * BK_S) ts[tid] = d[tid];
    for (int i = tid; i < BK_S * nv; i += NTB) ds[i] = d[BK_S * BK_S + i];
    __syncthreads();
    const long c0 = (long)blockIdx.y * NTB * EPT + (long)tid * VEC;
    Pk<VEC> a[BK_S][NP];
#pragma unroll
    for (int b = 0; b < BK_S; ++b)
#pragma unroll
        for (int e = 0; e < NP; ++e) a[b][e] = ld<VEC>(V + (size_t)(nv + b) * n, c0 + (long)e * NTB * VEC, n);
    // T is upper triangular: the last vector first, each then free to be overwritten
#pragma unroll
    for (int b = BK_S - 1; b >= 0; --b)
#pragma unroll
        for (int e = 0; e < NP; ++e)
#pragma unroll
            for (int j = 0; j < VEC; ++j) {
                float2 r = make_float2(0.f, 0.f);
#pragma unroll
                for (int q = 0; q <= b; ++q) mulacc(r, ts[q * BK_S + b], a[q][e].v[j]);
                a[b][e].v[j] = r;
            }
    for (int i0 = 0; i0 < nv; i0 += PU) {
        Pk<VEC> p[PU][NP];
#pragma unroll
        for (int u = 0; u < PU; ++u) {
            const float2 *vp = V + (size_t)min(i0 + u, nv - 1) * n;
#pragma unroll
            for (int e = 0; e < NP; ++e) p[u][e] = ld<VEC>(vp, c0 + (long)e * NTB * VEC, n);
        }
#pragma unroll
        for (int u = 0; u < PU; ++u) {
            if (i0 + u < nv) {
#pragma unroll
                for (int b = 0; b < BK_S; ++b) {
                    const float2 c = ds[BK_S * (i0 + u) + b];
#pragma unroll
                    for (int e = 0; e < NP; ++e)
#pragma unroll
                        for (int j = 0; j < VEC; ++j) mulsub(a[b][e].v[j], c, p[u][e].v[j]);
                }
            }
        }
    }
#pragma unroll
    for (int b = 0; b < BK_S; ++b) {
        const bool zero = ts[b * BK_S + b].x == 0.f;
#pragma unroll
        for (int e = 0; e < NP; ++e) {
            if (zero)
#pragma unroll
                for (int j = 0; j < VEC; ++j) a[b][e].v[j] = make_float2(0.f, 0.f);
            st<VEC>(V + (size_t)(nv + b) * n, c0 + (long)e * NTB * VEC, n, a[b][e]);
        }
    }
}

__device__ __forceinline__ double2 zfma(double2 a, double2 b, double2 c) {
    return make_double2(::fma(a.x, b.x, ::fma(-a.y, b.y, c.x)), ::fma(a.x, b.y, ::fma(a.y, b.x, c.y)));
}
__device__ __forceinline__ double wsum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One CTA a system: the block's coefficients from the partial sums, the Cholesky factor, the
// update's coefficients (dco: T then D) and the block's Hessenberg columns.  Latency-bound.
template <int NTF>
__global__ void __launch_bounds__(NTF) k_block_finish(int nv, int kk, int m, int G, const double *__restrict__ part,
                                                      const int *__restrict__ act, SysState *state,
                                                      double2 *__restrict__ H0, size_t strideH,
                                                      const double2 *__restrict__ a0, const double2 *__restrict__ a1,
                                                      const double2 *__restrict__ a2, size_t strideC, double tol,
                                                      float2 *__restrict__ dco, size_t dstride) {
    const int slot = blockIdx.x, s = act[slot], tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, ld = m + 1;
    SysState &stt = state[s];
    float2 *d = dco + (size_t)slot * dstride;
    double2 *H = H0 + (size_t)s * strideH;
    __shared__ double2 q[BK_S + 1][BK_QMAX + BK_S];   // q[b + 1]: y_{b+1} in the basis; q[0]: v_j
    __shared__ double2 gs[BK_S][BK_S], ss[BK_S][BK_S], tt[BK_S][BK_S];
    __shared__ double2 hc[BK_S][2 * BK_QMAX];         // the block's columns (kk + nv + 3 rows)
    __shared__ int s_ok;
    const int ncomp = BK_C * (nv + BK_S), nown = nv + BK_S;
    if (stt.broken) {
        if (tid < BK_S * BK_S) d[tid] = make_float2(0.f, 0.f);
        for (int i = tid; i < BK_S * nv; i += NTF) d[BK_S * BK_S + i] = make_float2(0.f, 0.f);
        return;
    }
    // the CTAs' sums: a thread a component (coalesced across components), the CTAs split over as many
    // thread groups as fit, four loads in flight, then the groups in order.  (A warp a component, a
    // butterfly each, was most of 38 us a block for 16 systems at 64^3.)
    const double *pp = part + (size_t)slot * ncomp * G;
    __shared__ dfr gsum[NTF];
    const int per = ncomp < NTF ? ncomp : NTF, groups = NTF / per, grp = tid / per;
    for (int c0 = 0; c0 < ncomp; c0 += per) {
        const int c = c0 + tid % per;
        dfr t(0.f, 0.f);
        if (grp < groups && c < ncomp)
            for (int g = grp; g < G; g += 4 * groups) {
                float2 f[4];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    f[u] = g + u * groups < G
                               ? __ldcg(reinterpret_cast<const float2 *>(pp + (size_t)(g + u * groups) * ncomp + c))
                               : make_float2(0.f, 0.f);
#pragma unroll
                for (int u = 0; u < 4; ++u) t = t + dfr(f[u].x, f[u].y);
            }
        gsum[tid] = t;
        __syncthreads();
        if (grp == 0 && c < ncomp) {
            for (int h = 1; h < groups; ++h) t = t + gsum[h * per + tid];
            const int i = c / BK_C, b = (c % BK_C) >> 1;
            double2 &z = i < nv ? q[b + 1][i] : gs[i - nv][b];
            if (c & 1) z.y = (double)t;
            else z.x = (double)t;
        }
        __syncthreads();
    }
    for (int i = tid; i < nown; i += NTF) q[0][i] = make_double2(i == nv - 1 ? 1.0 : 0.0, 0.0);
    __syncthreads();
    // G - C^H C, upper triangle, one warp an entry
    if (warp < 6) {
        const int b = warp < 1 ? 0 : warp < 3 ? 1 : 2, a = warp - (b * (b + 1)) / 2;
        double2 z = make_double2(0.0, 0.0);
        for (int i = lane; i < nv; i += 32) {
            const double2 u = q[a + 1][i], v = q[b + 1][i];
            z.x += u.x * v.x + u.y * v.y;
            z.y += u.x * v.y - u.y * v.x;
        }
        z.x = wsum(z.x);
        z.y = wsum(z.y);
        if (lane == 0) ss[a][b] = make_double2(gs[a][b].x - z.x, gs[a][b].y - z.y);
    }
    __syncthreads();
    const double sig = (double)stt.bs_sigma, isig = 1.0 / sig;
    const double2 th = make_double2((double)stt.bs_tr, (double)stt.bs_ti);
    if (tid == 0) {
        bool ok = true;
        double ri[BK_S];
        double2 r[BK_S][BK_S];
#pragma unroll
        for (int b = 0; b < BK_S; ++b) {
            for (int a = 0; a < b; ++a) {
                double2 z = ss[a][b];
                for (int l = 0; l < a; ++l)   // conj(r_la) r_lb
                    z = make_double2(z.x - (r[l][a].x * r[l][b].x + r[l][a].y * r[l][b].y),
                                     z.y - (r[l][a].x * r[l][b].y - r[l][a].y * r[l][b].x));
                r[a][b] = make_double2(z.x * ri[a], z.y * ri[a]);
            }
            double piv = ss[b][b].x;
            for (int l = 0; l < b; ++l) piv -= r[l][b].x * r[l][b].x + r[l][b].y * r[l][b].y;
            // also false for NaN and for an infinite column norm
            if (!(piv > BK_ILL * gs[b][b].x) || !(gs[b][b].x < 1e30)) ok = false;
            ri[b] = ok ? rsqrt(piv) : 1.0;
            r[b][b] = make_double2(ok ? piv * ri[b] : 1.0, 0.0);
            // the subdiagonal of the column this vector completes, in the operator's units
            const double beta = r[b][b].x * isig * (b == 0 ? 1.0 : ri[b - 1]);
            if (!(beta >= tol) || !(beta < 1e300)) ok = false;
        }
        // T = R^-1, upper triangular
#pragma unroll
        for (int b = 0; b < BK_S; ++b) {
            tt[b][b] = make_double2(ri[b], 0.0);
            for (int a = b - 1; a >= 0; --a) {
                double2 z = make_double2(0.0, 0.0);
                for (int l = a + 1; l <= b; ++l) z = zfma(r[a][l], tt[l][b], z);
                tt[a][b] = make_double2(-z.x * ri[a], -z.y * ri[a]);
            }
            for (int a = b + 1; a < BK_S; ++a) tt[a][b] = make_double2(0.0, 0.0);
        }
        for (int b = 0; b < BK_S; ++b)
            for (int a = 0; a < BK_S; ++a) q[b + 1][nv + a] = a <= b ? r[a][b] : make_double2(0.0, 0.0);
        if (!ok) {
            stt.ill = 1;
            stt.broken = nv;
        }
        s_ok = ok ? 1 : 0;
    }
    __syncthreads();
    if (!s_ok) {
        if (tid < BK_S * BK_S) d[tid] = make_float2(0.f, 0.f);
        for (int i = tid; i < BK_S * nv; i += NTF) d[BK_S * BK_S + i] = make_float2(0.f, 0.f);
        return;
    }
    if (tid < BK_S * BK_S) {
        const double2 t = tt[tid / BK_S][tid % BK_S];
        d[tid] = make_float2((float)t.x, (float)t.y);
    }
    for (int e = tid; e < BK_S * nv; e += NTF) {   // D = C T
        const int i = e / BK_S, b = e % BK_S;
        double2 z = make_double2(0.0, 0.0);
        for (int a = 0; a <= b; ++a) z = zfma(q[a + 1][i], tt[a][b], z);
        d[BK_S * BK_S + e] = make_float2((float)z.x, (float)z.y);
    }
    // the columns nv - 1 + b of A V = [W V] H: four lanes a row, row = tid / 4, tid / 4 + NTF / 4, ...
    const int part4 = tid & 3;
    for (int b = 0; b < BK_S; ++b) {
        const int col = nv - 1 + b;                       // own column; rows kk + 0 .. col + 1
        const double2 *ab = (b == 0 ? a0 : b == 1 ? a1 : a2) + (size_t)s * strideC;
        const double ir = tt[b > 0 ? b - 1 : 0][b > 0 ? b - 1 : 0].x;   // 1 / R_bb of q[b] (b > 0)
        for (int r0 = tid >> 2; r0 < ((kk + col + 2 + NTF / 4 - 1) & ~(NTF / 4 - 1)); r0 += NTF / 4) {   // warp-uniform
            double2 z = make_double2(0.0, 0.0);
            const int own = r0 - kk;
            if (b > 0 && r0 < kk + col + 2)
                for (int i = max(0, own - 1) + part4; i < col; i += 4) {
                    const double2 h = i >= nv - 1 ? hc[i - (nv - 1)][r0] : H[(size_t)(kk + i) * ld + r0];
                    const double2 c = q[b][i];
                    z = zfma(make_double2(-c.x, -c.y), h, z);
                }
            z.x += __shfl_xor_sync(0xffffffffu, z.x, 1);
            z.y += __shfl_xor_sync(0xffffffffu, z.y, 1);
            z.x += __shfl_xor_sync(0xffffffffu, z.x, 2);
            z.y += __shfl_xor_sync(0xffffffffu, z.y, 2);
            if (part4 == 0 && r0 < kk + col + 2) {
                if (own < 0) {
                    z.x = ::fma(ab[r0].x, isig, z.x);
                    z.y = ::fma(ab[r0].y, isig, z.y);
                } else {
                    const double2 y1 = q[b + 1][own];
                    z.x = ::fma(y1.x, isig, z.x);
                    z.y = ::fma(y1.y, isig, z.y);
                    z = zfma(th, q[b][own], z);
                }
                if (b > 0) z = make_double2(z.x * ir, z.y * ir);
                hc[b][r0] = z;
                H[(size_t)(kk + col) * ld + r0] = z;
            }
        }
        for (int r0 = kk + col + 2 + tid; r0 < kk + nown + 1; r0 += NTF) hc[b][r0] = make_double2(0.0, 0.0);
        __syncthreads();
    }
    if (tid == 0) {
        double2 sum = make_double2(stt.bs_sumr, stt.bs_sumi);
        for (int b = 0; b < BK_S; ++b) {
            const double2 h = hc[b][kk + nv - 1 + b];
            sum = make_double2(sum.x + h.x, sum.y + h.y);
        }
        stt.bs_sumr = sum.x;
        stt.bs_sumi = sum.y;
        const double inv = 1.0 / (double)(nv - 1 + BK_S);
        stt.bs_tr = (float)(sum.x * inv);
        stt.bs_ti = (float)(sum.y * inv);
        stt.bs_sigma = (float)(1.0 / hc[BK_S - 1][kk + nv + BK_S - 1].x);
    }
}

// Shift and scale of the first block from the `cols` Hessenberg columns of the steps before it.
__global__ void k_block_init(int cols, int kk, int m, const int *__restrict__ act, int nsys, SysState *state,
                             const double2 *__restrict__ H0, size_t strideH) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nsys; i += gridDim.x * blockDim.x) {
        SysState &st = state[act[i]];
        if (st.broken) continue;
        const double2 *H = H0 + (size_t)act[i] * strideH;
        double2 sum = make_double2(0.0, 0.0);
        for (int c = 0; c < cols; ++c) {
            const double2 h = H[(size_t)(kk + c) * (m + 1) + kk + c];
            sum = make_double2(sum.x + h.x, sum.y + h.y);
        }
        const double2 b = H[(size_t)(kk + cols - 1) * (m + 1) + kk + cols];
        const double beta = sqrt(b.x * b.x + b.y * b.y);
        st.bs_sumr = sum.x;
        st.bs_sumi = sum.y;
        st.bs_tr = (float)(sum.x / cols);
        st.bs_ti = (float)(sum.y / cols);
        st.bs_sigma = (float)(1.0 / beta);
        if (!(beta > 1e-30 && beta < 1e30)) {
            st.ill = 1;
            st.broken = cols;
        }
    }
}

// Elements a thread: the largest whose chunks still give every SM a CTA of the launch.
constexpr int EPT_BIG = 8, EPT_SMALL = 2;
int block_ept(int n, int nsys, int sms) {
    return (long)nsys * ((n + NTB * EPT_BIG - 1) / (NTB * EPT_BIG)) >= sms ? EPT_BIG : EPT_SMALL;
}

}  // namespace

size_t krylov_block_scratch(int m, int nsys) {   // doubles at the scratch's end: T and D of every system
    return (size_t)nsys * (BK_S * BK_S + BK_S * (m + 1));
}

bool krylov_block_fits(int m, int n, int nsys, size_t capacity) {
    // the projection's partials for the finest grid, then the coefficients
    const int sms = device_sm_count(), ept = block_ept(n, nsys, sms);
    const size_t nch = ((size_t)n + NTB * ept - 1) / (NTB * ept);
    return nch <= 65535 && (size_t)nsys * BK_C * (m + 1 + BK_S) * nch + krylov_block_scratch(m, nsys) <= capacity;
}

void launch_block_init(int cols, int kk, int m, const int *act, int nsys, SysState *state, const double2 *H,
                       size_t strideH, cudaStream_t st) {
    ProfScope p(KC_OTHER, 0.0, st, 1);
    k_block_init<<<(nsys + 63) / 64, 64, 0, st>>>(cols, kk, m, act, nsys, state, H, strideH);
}

void launch_block_step(int n, int nv, int kk, int m, float2 *V, size_t strideV, const int *act, int nsys,
                       SysState *state, double2 *H, size_t strideH, const double2 *const (&a)[KRYLOV_BLOCK],
                       size_t strideC, double tol, double *scratch, size_t capacity, cudaStream_t st) {
    const int sms = device_sm_count(), ept = block_ept(n, nsys, sms);
    const int nch = (n + NTB * ept - 1) / (NTB * ept);
    const bool v2 = n % 2 == 0 && strideV % 2 == 0 && (reinterpret_cast<uintptr_t>(V) & 15) == 0;
    // about eight CTAs an SM over the launch, two a system and SM at most: a CTA's chunks share one set of
    // partial sums, and one CTA adds a system's (one system at 128^3, nv = 21: 150 us with 1024 sets; 64 systems
    // at 96^3 1335 us with half as many, 1083 as is)
    const int G = (int)std::min<long>(nch, std::min<long>(2 * sms, ((long)sms * 8 + nsys - 1) / nsys));
    const size_t smem = sizeof(dfr) * NWB * BK_C * (size_t)(nv + BK_S);
    float2 *dco = reinterpret_cast<float2 *>(scratch + capacity - krylov_block_scratch(m, nsys));
    const size_t dstride = BK_S * BK_S + (size_t)BK_S * (m + 1);
    {
        ProfScope p(KC_MDOT, sizeof(float2) * (double)n * nsys * (nv + BK_S), st, 2);
        auto go = [&](auto kernel) {
            block_allow_smem((const void *)kernel, smem);
            kernel<<<dim3(nsys, G), NTB, smem, st>>>(n, nv, V, strideV, act, state, scratch, nch);
        };
        if (ept == EPT_BIG) v2 ? go(k_block_proj<EPT_BIG, 2>) : go(k_block_proj<EPT_BIG, 1>);
        else v2 ? go(k_block_proj<EPT_SMALL, 2>) : go(k_block_proj<EPT_SMALL, 1>);
        // more threads only where there are many sets to add (12 systems, 49 sets: 57 us with the projection at 512
        // threads, 61 at 1024)
        auto fin = [&](auto kernel, int threads) {
            kernel<<<nsys, threads, 0, st>>>(nv, kk, m, G, scratch, act, state, H, strideH, a[0], a[1], a[2], strideC,
                                             tol, dco, dstride);
        };
        if (G > 128) fin(k_block_finish<1024>, 1024);
        else fin(k_block_finish<512>, 512);
    }
    ProfScope p(KC_UPDATE, sizeof(float2) * (double)n * nsys * (nv + 2 * BK_S), st, 1);
    const dim3 grid(nsys, nch);
    if (ept == EPT_BIG) {
        if (v2) k_block_update<EPT_BIG, 2><<<grid, NTB, 0, st>>>(n, nv, V, strideV, act, dco, dstride);
        else k_block_update<EPT_BIG, 1><<<grid, NTB, 0, st>>>(n, nv, V, strideV, act, dco, dstride);
    } else {
        if (v2) k_block_update<EPT_SMALL, 2><<<grid, NTB, 0, st>>>(n, nv, V, strideV, act, dco, dstride);
        else k_block_update<EPT_SMALL, 1><<<grid, NTB, 0, st>>>(n, nv, V, strideV, act, dco, dstride);
    }
}

}  // namespace gdmr
