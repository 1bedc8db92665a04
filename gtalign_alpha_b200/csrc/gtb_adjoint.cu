// gtb_adjoint.cu -- TM-score adjoint for fixed alignments and projected-
// gradient polishing of superpositions on SO(3) x R^3.
//
// For a pair with aligned residues (q_i, r_i), transform (R, t) and d0:
//   e_i = R q_i + t - r_i,  u_i = d0^2 + |e_i|^2,  TM = sum_i d0^2 / u_i
//   dTM/de_i = -2 d0^2 e_i / u_i^2
//   dTM/dt      = sum_i dTM/de_i
//   dTM/domega  = sum_i (R q_i) x dTM/de_i     (R <- exp([omega]x) R)
//   dTM/dq_i    = R^T dTM/de_i
// One warp per pair; lanes stride over residues; FP32 arithmetic with
// per-lane compensated sums and a fixed butterfly reduction.
#include <cuda_runtime.h>
#include <cstdio>
#include "gtb200.h"
#include "gtb_device.cuh"
#include "gtb_kernels.cuh"

namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

struct Kahan {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float x) {
        float y = x - c;
        float t = s + y;
        c = (t - s) - y;
        s = t;
    }
    // c holds the rounding excess of the last additions: the compensated
    // total is s - c
    __device__ __forceinline__ float value() const { return s - c; }
};

// 1 / u within an ulp, without the branches of the IEEE division: the
// approximate reciprocal and one Newton step (0 for u = inf and for u above 2^126,
// where the score term is below 10^-34; NaN stays).  Errors against 64 bits
// before and after: scores and gradients 4.9e-7 and 4.5e-7, polishing 2.4e-6.
__device__ __forceinline__ float recip(float u) {
    float b, y;
    asm("min.NaN.f32 %0, %1, 0f7F7FFFFF;" : "=f"(b) : "f"(u));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
    return __fmaf_rn(y, __fmaf_rn(-b, y, 1.f), y);
}

// TM-score and gradient for one pair; omega about the origin
__device__ void tm_grad(const float* q, const float* r, int n, const float* T, float d0,
                        float* gq, float& tm, float* g6) {
    int lane = threadIdx.x & 31;
    float d02 = d0 * d0;
    Kahan s, gw[3], gt[3];
#pragma unroll 2
    for (int i = lane; i < n; i += 32) {
        float qx = q[3 * i], qy = q[3 * i + 1], qz = q[3 * i + 2];
        float px = fmaf(T[0], qx, fmaf(T[1], qy, T[2] * qz));
        float py = fmaf(T[3], qx, fmaf(T[4], qy, T[5] * qz));
        float pz = fmaf(T[6], qx, fmaf(T[7], qy, T[8] * qz));
        float ex = px + T[9] - r[3 * i], ey = py + T[10] - r[3 * i + 1], ez = pz + T[11] - r[3 * i + 2];
        float iu = recip(fmaf(ex, ex, fmaf(ey, ey, fmaf(ez, ez, d02))));
        s.add(d02 * iu);
        float k = -2.f * d02 * iu * iu;
        float gx = k * ex, gy = k * ey, gz = k * ez;
        gt[0].add(gx); gt[1].add(gy); gt[2].add(gz);
        gw[0].add(fmaf(py, gz, -(pz * gy)));
        gw[1].add(fmaf(pz, gx, -(px * gz)));
        gw[2].add(fmaf(px, gy, -(py * gx)));
        if (gq) {
            gq[3 * i] = fmaf(T[0], gx, fmaf(T[3], gy, T[6] * gz));
            gq[3 * i + 1] = fmaf(T[1], gx, fmaf(T[4], gy, T[7] * gz));
            gq[3 * i + 2] = fmaf(T[2], gx, fmaf(T[5], gy, T[8] * gz));
        }
    }
    tm = warp_sum(s.value());
    for (int k = 0; k < 3; k++) {
        g6[k] = warp_sum(gw[k].value());
        g6[3 + k] = warp_sum(gt[k].value());
    }
}

__global__ void k_tm_adjoint(int npairs, const long long* off, const int* n, const float* qxyz,
                             const float* rxyz, const float* tfm, const float* d0, float* tm,
                             float* grad, float* gq) {
    int p = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (p >= npairs) return;
    int lane = threadIdx.x & 31;
    long long o = off[p];
    float T[12];
    for (int f = 0; f < 12; f++) T[f] = tfm[p * 12 + f];
    float t, g6[6];
    tm_grad(qxyz + 3 * o, rxyz + 3 * o, n[p], T, d0[p], gq ? gq + 3 * o : nullptr, t, g6);
    if (lane == 0) {
        if (tm) tm[p] = t;
        if (grad) for (int k = 0; k < 6; k++) grad[p * 6 + k] = g6[k];
    }
}

// The backward pass of the scores (adjoint.TMScore), a warp per pair: with the
// forward pass's gq (dTM/dq) and g (dTM/domega, dTM/dt) and the incoming
// gradient gout, grad_q = gout gq and grad_tfm = gout (dTM/dR, dTM/dt) with
// dTM/dR = sum (dTM/de) q^T = R sum gq q^T.  One read of q and gq and one write
// of grad_q: bound by HBM.  (Gathers, a scatter and atomic additions by torch
// operations took 1.6 ms for 20,000 pairs of 60 to 600 residues.)
__global__ void k_tm_backward(int npairs, const long long* off, const int* n, const float* qxyz,
                              const float* gq, const float* tfm, const float* grad,
                              const float* gout, float* grad_q, float* grad_tfm) {
    int p = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (p >= npairs) return;
    const int lane = threadIdx.x & 31, m = n[p];
    const long long o = 3 * off[p];
    const float go = gout[p];
    Kahan s[9];
#pragma unroll 2
    for (int i = lane; i < m; i += 32) {
        float g[3], x[3];
        for (int k = 0; k < 3; k++) { g[k] = gq[o + 3 * i + k]; x[k] = qxyz[o + 3 * i + k]; }
        for (int k = 0; k < 3; k++) grad_q[o + 3 * i + k] = g[k] * go;
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++) s[3 * a + b].add(g[a] * x[b]);
    }
    float v[9];
    for (int k = 0; k < 9; k++) v[k] = warp_sum(s[k].value());
    if (lane < 12) {
        float x;
        if (lane < 9) {
            const int a = lane / 3, b = lane % 3;
            const float* R = tfm + p * 12LL + 3 * a;
            const float v0 = b == 0 ? v[0] : b == 1 ? v[1] : v[2];
            const float v1 = b == 0 ? v[3] : b == 1 ? v[4] : v[5];
            const float v2 = b == 0 ? v[6] : b == 1 ? v[7] : v[8];
            x = fmaf(R[0], v0, fmaf(R[1], v1, R[2] * v2));
        } else {
            x = grad[p * 6LL + 3 + (lane - 9)];
        }
        grad_tfm[p * 12LL + lane] = x * go;
    }
}

template <int S>
__device__ float tm_only(const float* q, const float* r, int n, const float* T, float d0) {
    int lane = threadIdx.x & 31;
    float d02 = d0 * d0;
    Kahan s;
    for (int i = lane; i < n; i += 32) {
        float qx = q[S * i], qy = q[S * i + 1], qz = q[S * i + 2];
        float ex = fmaf(T[0], qx, fmaf(T[1], qy, fmaf(T[2], qz, T[9]))) - r[S * i];
        float ey = fmaf(T[3], qx, fmaf(T[4], qy, fmaf(T[5], qz, T[10]))) - r[S * i + 1];
        float ez = fmaf(T[6], qx, fmaf(T[7], qy, fmaf(T[8], qz, T[11]))) - r[S * i + 2];
        s.add(d02 * recip(fmaf(ex, ex, fmaf(ey, ey, fmaf(ez, ez, d02)))));
    }
    return warp_sum(s.value());
}

// gradient and the curvature scales of a step in one sweep: g6 as tm_grad's
// about the point cen, h_t = sum 2 d0^2/u^2, h_w = sum 2 d0^2 |a|^2/u^2
template <int S>
__device__ __forceinline__ void grad_curv(const float* q, const float* r, int n, const float* T,
                                          float d0, const float* cen, float* g6, float& ht, float& hw) {
    int lane = threadIdx.x & 31;
    float d02 = d0 * d0;
    Kahan gw[3], gt[3];
    float a1 = 0.f, a2 = 0.f;
    for (int i = lane; i < n; i += 32) {
        float qx = q[S * i], qy = q[S * i + 1], qz = q[S * i + 2];
        float px = fmaf(T[0], qx, fmaf(T[1], qy, fmaf(T[2], qz, T[9])));
        float py = fmaf(T[3], qx, fmaf(T[4], qy, fmaf(T[5], qz, T[10])));
        float pz = fmaf(T[6], qx, fmaf(T[7], qy, fmaf(T[8], qz, T[11])));
        float ex = px - r[S * i], ey = py - r[S * i + 1], ez = pz - r[S * i + 2];
        float iu = recip(fmaf(ex, ex, fmaf(ey, ey, fmaf(ez, ez, d02))));
        float w = 2.f * d02 * iu * iu;
        float gx = -w * ex, gy = -w * ey, gz = -w * ez;
        gt[0].add(gx); gt[1].add(gy); gt[2].add(gz);
        float ax = px - cen[0], ay = py - cen[1], az = pz - cen[2];
        gw[0].add(fmaf(ay, gz, -(az * gy)));
        gw[1].add(fmaf(az, gx, -(ax * gz)));
        gw[2].add(fmaf(ax, gy, -(ay * gx)));
        a1 += w;
        a2 = fmaf(w, fmaf(ax, ax, fmaf(ay, ay, az * az)), a2);
    }
    for (int k = 0; k < 3; k++) {
        g6[k] = warp_sum(gw[k].value());
        g6[3 + k] = warp_sum(gt[k].value());
    }
    ht = warp_sum(a1);
    hw = warp_sum(a2);
}

// apply x -> exp([w]x)(x - c) + c + dt to the transform (Rodrigues, FP64)
__device__ void apply_step(const float* T, const float* w, const float* dt, const float* c,
                           float* Tn) {
    const double x = (double)w[0] * w[0] + (double)w[1] * w[1] + (double)w[2] * w[2];
    double K[9] = {0, -w[2], w[1], w[2], 0, -w[0], -w[1], w[0], 0};
    double A, Bc;                     // sin(th)/th and (1 - cos(th))/th^2, x = th^2
    if (x <= 0.25) {
        // their Taylor series: the first term left out is below 2^-60
        A = 1.0; Bc = 0.5;
        double ta = 1.0, tb = 0.5;
#pragma unroll
        for (int k = 1; k <= 8; k++) {
            ta *= x * (-1.0 / (2 * k * (2 * k + 1)));
            tb *= x * (-1.0 / ((2 * k + 1) * (2 * k + 2)));
            A += ta;
            Bc += tb;
        }
    } else {
        const double th = sqrt(x);
        A = sin(th) / th;
        Bc = (1.0 - cos(th)) / x;
    }
    double K2[9];
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) {
            double s = 0;
            for (int k = 0; k < 3; k++) s += K[3 * i + k] * K[3 * k + j];
            K2[3 * i + j] = s;
        }
    double E[9];
    for (int k = 0; k < 9; k++) E[k] = ((k % 4) == 0 ? 1.0 : 0.0) + A * K[k] + Bc * K2[k];
    double Rn[9];
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) {
            double s = 0;
            for (int k = 0; k < 3; k++) s += E[3 * i + k] * (double)T[3 * k + j];
            Rn[3 * i + j] = s;
        }
    for (int i = 0; i < 3; i++) {
        double s = 0;
        for (int k = 0; k < 3; k++) s += E[3 * i + k] * ((double)T[9 + k] - c[k]);
        Tn[9 + i] = (float)(s + c[i] + dt[i]);
    }
    for (int k = 0; k < 9; k++) Tn[k] = (float)Rn[k];
}

// Projected-gradient ascent of TM (d0) over (R, t) for one pair, from T;
// a step is kept only if it raises the score.  Returns the final score.
template <int S>
__device__ float polish_pair(const float* q, const float* r, int m, float d0, float* T, int steps,
                             float* before) {
    float Tn[12];
    float cur = tm_only<S>(q, r, m, T, d0);
    if (before) *before = cur;
    int lane = threadIdx.x & 31;
    // the query's centroid, which each step's transform carries along
    float cq[3] = {0.f, 0.f, 0.f};
    if (steps > 0 && m > 0) {
        for (int i = lane; i < m; i += 32)
            for (int k = 0; k < 3; k++) cq[k] += q[S * i + k];
        for (int k = 0; k < 3; k++) cq[k] = warp_sum(cq[k]) / m;
    }
    for (int it = 0; it < steps && m > 0; it++) {
        float c[3], g6[6], ht, hw;
        for (int k = 0; k < 3; k++)
            c[k] = fmaf(T[3 * k], cq[0], fmaf(T[3 * k + 1], cq[1], fmaf(T[3 * k + 2], cq[2], T[9 + k])));
        grad_curv<S>(q, r, m, T, d0, c, g6, ht, hw);
        if (!(ht > 0.f) || !(hw > 0.f)) break;
        float w[3] = {g6[0] / hw, g6[1] / hw, g6[2] / hw};
        float dt[3] = {g6[3] / ht, g6[4] / ht, g6[5] / ht};
        bool acc = false;
        for (int bt = 0; bt < 10 && !acc; bt++) {
            apply_step(T, w, dt, c, Tn);
            float nv = tm_only<S>(q, r, m, Tn, d0);
            if (nv > cur) {
                acc = true;
                cur = nv;
                for (int f = 0; f < 12; f++) T[f] = Tn[f];
            } else {
                for (int k = 0; k < 3; k++) { w[k] *= 0.5f; dt[k] *= 0.5f; }
            }
        }
        if (!acc) break;
    }
    return cur;
}

__global__ void k_polish(int npairs, const long long* off, const int* n, const float* qxyz,
                         const float* rxyz, float* tfm, const float* d0v, int steps,
                         float* tmb, float* tma) {
    int p = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (p >= npairs) return;
    int lane = threadIdx.x & 31;
    long long o = off[p];
    float T[12], before;
    for (int f = 0; f < 12; f++) T[f] = tfm[p * 12 + f];
    float cur = polish_pair<3>(qxyz + 3 * o, rxyz + 3 * o, n[p], d0v[p], T, steps, &before);
    if (lane == 0) {
        for (int f = 0; f < 12; f++) tfm[p * 12 + f] = T[f];
        if (tmb) tmb[p] = before;
        if (tma) tma[p] = cur;
    }
}

// Polishing inside the search, after the production scores: each pair's
// final transform is polished against TM with the search's d0 (that of the
// shorter structure) over its final alignment (the aligned coordinates the
// traceback stored, 6 floats per aligned pair); when a step was kept, the
// FP32 TM-scores by both lengths are recomputed for the new transform (the
// FP64 recomputation and error record follow in the final kernel).
__global__ void k_polish_final(gtb::Blk B, gtb::Bat T, int steps) {
    int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (i >= T.np) return;
    int lane = threadIdx.x & 31;
    if (T.flags[i] & gtb::CONV_LOWTMSC) return;
    int m = T.naln[i];
    if (m < 3) return;
    int qi = (int)((T.p0 + i) / B.nr), ri = (int)((T.p0 + i) % B.nr);
    int lq = B.qlen[qi], lr = B.rlen[ri];
    int ml = lq < lr ? lq : lr;
    const float* q = T.alc + 6 * T.off_aln[i];
    const float* r = q + 3;
    float Tm[12], before;
    for (int f = 0; f < 12; f++) Tm[f] = T.tfm_gr[i * 12 + f];
    float cur = polish_pair<6>(q, r, m, B.t_d0fin[ml], Tm, steps, &before);
    if (!(cur > before)) return;
    float tq = tm_only<6>(q, r, m, Tm, B.t_d0fin[lq]);
    float tr = tm_only<6>(q, r, m, Tm, B.t_d0fin[lr]);
    if (lane == 0) {
        for (int f = 0; f < 12; f++) T.tfm_gr[i * 12 + f] = Tm[f];
        T.out[i * 16 + 9] = tq / (float)lq;
        T.out[i * 16 + 10] = tr / (float)lr;
    }
}

}  // namespace

namespace gtb {
void launch_polish_final(const Blk& B, const Bat& T, int steps, cudaStream_t st) {
    if (steps <= 0 || T.np <= 0) return;
    k_polish_final<<<(T.np + 3) / 4, 128, 0, st>>>(B, T, steps);
    if (T.launches) (*T.launches)++;
}
}  // namespace gtb

struct gtb_handle;
extern "C" gtb_status gtb_tm_adjoint(gtb_handle* h, int npairs, const long long* off, const int* n,
                                     const float* qxyz, const float* rxyz, const float* tfm,
                                     const float* d0, float* tm, float* grad, float* gq, void* stream) {
    (void)h;
    if (npairs < 0 || !off || !n || !qxyz || !rxyz || !tfm || !d0) return GTB_ERR_ARG;
    if (npairs == 0) return GTB_OK;
    int blocks = (npairs + 3) / 4;
    k_tm_adjoint<<<blocks, 128, 0, (cudaStream_t)stream>>>(npairs, off, n, qxyz, rxyz, tfm, d0, tm, grad, gq);
    return cudaGetLastError() == cudaSuccess ? GTB_OK : GTB_ERR_CUDA;
}

extern "C" gtb_status gtb_polish(gtb_handle* h, int npairs, const long long* off, const int* n,
                                 const float* qxyz, const float* rxyz, float* tfm, const float* d0,
                                 int steps, float* tm_before, float* tm_after, void* stream) {
    (void)h;
    if (npairs < 0 || !off || !n || !qxyz || !rxyz || !tfm || !d0 || steps < 0) return GTB_ERR_ARG;
    if (npairs == 0) return GTB_OK;
    int blocks = (npairs + 3) / 4;
    k_polish<<<blocks, 128, 0, (cudaStream_t)stream>>>(npairs, off, n, qxyz, rxyz, tfm, d0, steps,
                                                       tm_before, tm_after);
    return cudaGetLastError() == cudaSuccess ? GTB_OK : GTB_ERR_CUDA;
}

extern "C" gtb_status gtb_tm_backward(gtb_handle* h, int npairs, const long long* off, const int* n,
                                      const float* qxyz, const float* gq, const float* tfm,
                                      const float* grad, const float* gout, float* grad_q,
                                      float* grad_tfm, void* stream) {
    (void)h;
    if (npairs < 0 || !off || !n || !qxyz || !gq || !tfm || !grad || !gout || !grad_q || !grad_tfm)
        return GTB_ERR_ARG;
    if (npairs == 0) return GTB_OK;
    k_tm_backward<<<(npairs + 3) / 4, 128, 0, (cudaStream_t)stream>>>(npairs, off, n, qxyz, gq, tfm, grad,
                                                                      gout, grad_q, grad_tfm);
    return cudaGetLastError() == cudaSuccess ? GTB_OK : GTB_ERR_CUDA;
}
