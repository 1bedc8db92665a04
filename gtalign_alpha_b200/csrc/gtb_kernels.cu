// gtb_kernels.cu -- sm_100a kernels of the per-pair superposition search.
//
// Work decomposition (one launch covers every pair of a batch):
//  * seed (stage 1, fragment search): one CTA per pair (a long pair's
//    offsets are split over several CTAs, 512 each), one thread per diagonal
//    offset; each thread runs the whole covariance -> rotation -> score ->
//    threshold loop of its offset sequentially and keeps its best; the CTA
//    reduces (max score, lowest offset index), across CTAs through a packed
//    64-bit atomic maximum.
//  * refinement (every fragment-based superposition refinement): pairs taken
//    from a work list sorted by position count.  Where few pairs take part
//    (after the --pre-score filter, small batches) and for pairs of 512+
//    positions, a warp makes each pass of a variant and a cluster of CTAs
//    takes a pair (k_refine_coop); the shorter pairs of a large batch's first
//    launches take 16 lanes each, a variant per lane from the pair's pool
//    (k_refine), and pairs of 1,536+ positions many warps.  The winner is the
//    larger score, then the lower variant index.  The distance-threshold
//    covariance pass of iteration k+1 is fused into the scoring pass of
//    iteration k.
//  * DP: pairs from a work list (largest matrices first), one warp per pair;
//    the warp sweeps strips of 32*R rows along anti-diagonals (R rows per
//    lane, register-blocked), left/up/diagonal values move between lanes by
//    shuffles, each lane packs the 2-bit directions of its cells into
//    traceback words.  A long pair's strips run as a wavefront over several
//    single-warp CTAs (cooperative launch, bounded waits on progress counters).
//  * traceback, alignment rows, final scores: a warp per pair.
// All floating-point reductions are sequential per thread in forward position
// order (blocks of BLK positions, Neumaier-compensated), so results do not
// depend on the launch geometry.
#include <algorithm>
#include <type_traits>
#include <cooperative_groups.h>
#include "gtb200.h"
#include "gtb_device.cuh"
#include "gtb_kernels.cuh"
#include "gtb_gonnet.h"

namespace gtb {
namespace cg = cooperative_groups;

// Residue exchange scores of the --add-search-by-ss DP (log2 Gonnet ratios
// over the letters A..Z, built on the host by gtb_gonnet_scores); a global
// array read through L1: the lanes of a warp look up different residues.
__device__ float g_gonnet[GTB_GONNET_NA * GTB_GONNET_NA];
constexpr float DPSS_C = -1048576.0f;     // offset of a diagonally reached cell
constexpr float DPSS_CMP = -524288.0f;    // stored values below this carry it

__device__ __forceinline__ float gonnet(unsigned char a, unsigned char b) {
    return ('A' <= a && a <= 'Z' && 'A' <= b && b <= 'Z')
               ? __ldg(g_gonnet + (a - 'A') * GTB_GONNET_NA + (b - 'A')) : 0.f;
}


#define GTB_LAUNCHED(T) do { if ((T).launches) (*(T).launches)++; } while (0)

void KTimer::begin(int f, cudaStream_t st) {
    if (used + 2 > ev.size()) {
        for (int k = 0; k < 64; k++) {
            cudaEvent_t e;
            if (cudaEventCreate(&e) != cudaSuccess) return;
            ev.push_back(e);
        }
    }
    if (fam.size() < ev.size() / 2) fam.resize(ev.size() / 2);
    fam[used / 2] = f;
    cudaEventRecord(ev[used], st);
}

void KTimer::end(cudaStream_t st) {
    if (used + 2 > ev.size()) return;       // begin could not create events
    cudaEventRecord(ev[used + 1], st);
    used += 2;
}

cudaError_t KTimer::collect(float* ms) {
    cudaError_t e = cudaSuccess;
    for (size_t k = 0; k + 1 < used; k += 2) {
        float t = 0.f;
        cudaError_t r = cudaEventElapsedTime(&t, ev[k], ev[k + 1]);
        if (r == cudaSuccess) ms[fam[k / 2]] += t;
        else if (e == cudaSuccess) e = r;
    }
    used = 0;
    return e;
}

KTimer::~KTimer() {
    for (cudaEvent_t e : ev) cudaEventDestroy(e);
}

// algorithmic work counters (Bat::work): one atomic per caller, spread over
// WORK_SLOTS addresses by CTA
__device__ __forceinline__ void work_add(const Bat& T, int kind, unsigned long long v) {
    if (T.work && v)
        atomicAdd(T.work + kind * WORK_SLOTS + (blockIdx.x & (WORK_SLOTS - 1)), v);
}

// the transform a DP of pair i uses (DpTfm)
__device__ __forceinline__ const float* dp_tfm(const Bat& T, int i, int tfmsrc) {
    if (tfmsrc == DP_TFM_GRAND) return T.tfm_gr + i * 12;
    if (tfmsrc == DP_TFM_ALT) return T.f3alt + ((long long)i * T.f3br + T.alt_rci) * 12;
    if (tfmsrc == DP_TFM_2ND) return T.tfm_2nd + i * 12;
    return T.tfm_ib + i * 12;
}
// the detailed search's branch T.alt_rci of pair i is empty
__device__ __forceinline__ bool alt_empty(const Bat& T, int i) {
    return T.f3ok && T.alt_rci >= 0 && !T.f3ok[(long long)i * T.f3br + T.alt_rci];
}

__device__ __forceinline__ int pair_qi(const Blk& B, const Bat& T, int i) {
    return (int)((T.p0 + i) / B.nr);
}
__device__ __forceinline__ int pair_ri(const Blk& B, const Bat& T, int i) {
    return (int)((T.p0 + i) % B.nr);
}

// ---------------------------------------------------------------------------
// secondary structure: MpSecStr.cpp:26-118 / MpSecStr.h:218-249
__device__ __forceinline__ float ss_dst(const float* x, const float* y, const float* z, int i, int j) {
    float dx = __fsub_rn(x[i], x[j]), dy = __fsub_rn(y[i], y[j]), dz = __fsub_rn(z[i], z[j]);
    float a = __fmul_rn(dx, dx), b = __fmul_rn(dy, dy), c = __fmul_rn(dz, dz);
    return __fsqrt_rn(__fadd_rn(__fadd_rn(a, b), c));
}

__global__ void k_secstr(char* ss, const float* X, const float* Y, const float* Z,
                         const int* len, const int* off, const int* mol, int nstr) {
    int si = blockIdx.x;
    if (si >= nstr) return;
    int L = len[si];
    const float* x = X + off[si];
    const float* y = Y + off[si];
    const float* z = Z + off[si];
    char* s = ss + off[si];
    int prot = mol ? (mol[si] == 0) : 1;
    for (int p = threadIdx.x; p < L; p += blockDim.x) {
        char c = ' ';
        if (prot && p >= 2 && p + 2 < L) {
            float d13 = ss_dst(x, y, z, p - 2, p);
            float d14 = ss_dst(x, y, z, p - 2, p + 1);
            float d15 = ss_dst(x, y, z, p - 2, p + 2);
            float d24 = ss_dst(x, y, z, p - 1, p + 1);
            float d25 = ss_dst(x, y, z, p - 1, p + 2);
            float d35 = ss_dst(x, y, z, p, p + 2);
            float e = 2.1f;
            if (fabsf(d15 - 6.37f) < e && fabsf(d14 - 5.18f) < e && fabsf(d25 - 5.18f) < e &&
                fabsf(d13 - 5.45f) < e && fabsf(d24 - 5.45f) < e && fabsf(d35 - 5.45f) < e)
                c = 'h';
            else {
                e = 1.42f;
                if (fabsf(d15 - 13.0f) < e && fabsf(d14 - 10.4f) < e && fabsf(d25 - 10.4f) < e &&
                    fabsf(d13 - 6.1f) < e && fabsf(d24 - 6.1f) < e && fabsf(d35 - 6.1f) < e)
                    c = 'e';
                else if (d15 < 8.0f)
                    c = 't';
            }
        }
        s[p] = c;
    }
}

void launch_secstr(char* ss, const float* x, const float* y, const float* z,
                   const int* len, const int* off, const int* mol, int nstr,
                   cudaStream_t st, long long* launches) {
    if (nstr <= 0) return;
    k_secstr<<<nstr, 128, 0, st>>>(ss, x, y, z, len, off, mol, nstr);
    if (launches) (*launches)++;
}

// ---------------------------------------------------------------------------
// A structure's residues as (x, y, z, 0), and its mark: some coordinate is not
// ordinary (not a number, or above 10^9, from where on squared distances could
// leave the range that the DP's fast form takes).  The marks have an array of
// their own: the residue ranges of two structures may overlap, and then share
// the copies.
__global__ void k_pack4s(float4* out, unsigned char* mark, const float* x, const float* y,
                         const float* z, const int* off, const int* len, const int* coff, int n) {
    int si = blockIdx.x;
    if (si >= n) return;
    int o = off[si], L = len[si], c = coff[si];
    bool odd = false;
    for (int p = threadIdx.x; p < L; p += blockDim.x) {
        const float4 v = make_float4(x[o + p], y[o + p], z[o + p], 0.f);
        odd = odd || !(fabsf(v.x) <= 1.e9f && fabsf(v.y) <= 1.e9f && fabsf(v.z) <= 1.e9f);
        out[c + p] = v;
    }
    odd = __syncthreads_or(odd);
    if (threadIdx.x == 0) mark[si] = odd ? 1 : 0;
}

__device__ __forceinline__ bool coords_ordinary(const Blk& B, int qi, int ri) {
    return (__ldg(B.qodd + qi) | __ldg(B.rodd + ri)) == 0;
}

void launch_pack4_structs(float4* out, unsigned char* mark, const float* x, const float* y,
                          const float* z, const int* off, const int* len, const int* coff, int n,
                          cudaStream_t st) {
    if (n <= 0) return;
    k_pack4s<<<n, 128, 0, st>>>(out, mark, x, y, z, off, len, coff, n);
}

// ---------------------------------------------------------------------------
// pair initialisation: MpStage1.cpp:28-167
// the clustering run's prefilter of a pair (CheckMaxCoverage)
__device__ __forceinline__ bool cls_pass(const Blk& B, int qi, int ri) {
    const float lq = (float)B.qlen[qi], lr = (float)B.rlen[ri];
    return B.rtype[ri] < B.clsqend && __fmul_rn(fmaxf(lq, lr), B.clscov) <= fminf(lq, lr);
}

// a thread per node; the residue index is relative to the structure, its SS
// byte at the structure's offset + residue
__global__ void k_pack_nodes(float4* nd, int2* nc, const float* x, const float* y, const float* z,
                             const int* l, const int* r, const int* o, const int* off,
                             const int* len, const char* ss, int nstr) {
    const int s = blockIdx.y;
    if (s >= nstr) return;
    const int L = len[s], a = off[s];
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < L; k += gridDim.x * blockDim.x) {
        const int p = a + k, org = o[p];
        const unsigned w = (unsigned)org | ((unsigned)(unsigned char)ss[a + org] << 16);
        nd[p] = make_float4(x[p], y[p], z[p], __uint_as_float(w));
        nc[p] = make_int2(l[p], r[p]);
    }
}

void launch_pack_nodes(float4* nd, int2* nc, const float* x, const float* y, const float* z,
                       const int* l, const int* r, const int* o, const int* off, const int* len,
                       const char* ss, long long n, int nstr, cudaStream_t st) {
    (void)n;
    for (int s0 = 0; s0 < nstr; s0 += 65535) {
        const int ns = nstr - s0 < 65535 ? nstr - s0 : 65535;
        k_pack_nodes<<<dim3(4, ns), 128, 0, st>>>(nd, nc, x, y, z, l, r, o, off + s0, len + s0, ss, ns);
    }
}

__global__ void k_init(Blk B, Bat T) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= T.np) return;
    int qi = pair_qi(B, T, i), ri = pair_ri(B, T, i);
    // with the --pre-similarity screen or in a clustering run every pair starts
    // filtered, with no molecule-type check (custage1.cu:74-82); a clustering
    // run releases the pairs of its triangle whose lengths can reach the
    // coverage (CheckMaxCoverage, coverage.cu:28-52), and k_presim then
    // releases, of the rest, the ones that pass its screen
    if (B.cls) T.flags[i] = cls_pass(B, qi, ri) ? 0 : CONV_LOWTMSC;
    else T.flags[i] = (B.presim > 0.f || B.qmol[qi] != B.rmol[ri]) ? CONV_LOWTMSC : 0;
    T.grand[i] = 0.f; T.best[i] = 0.f; T.best0[i] = 0.f; T.rmsd32[i] = -1.f;
    T.seedq[i] = 0; T.seedr[i] = 0; T.naln[i] = 0;
    T.sfndx[i] = T.sfpos[i] = T.sfndx_cur[i] = T.sfpos_cur[i] = 0;
#pragma unroll
    for (int f = 0; f < 12; f++) {
        float v = (f == 0 || f == 4 || f == 8) ? 1.f : 0.f;
        T.tfm_ib[i * 12 + f] = v;
        T.tfm_gr[i * 12 + f] = v;
    }
#pragma unroll
    for (int f = 0; f < 16; f++) T.out[i * 16 + f] = (f == 8) ? 9999.9f : 0.f;
#pragma unroll
    for (int f = 0; f < 4; f++) T.err[i * 4 + f] = 0.f;
}

void launch_init(const Blk& B, const Bat& T, cudaStream_t st) {
    k_init<<<(T.np + 127) / 128, 128, 0, st>>>(B, T);
    GTB_LAUNCHED(T);
}

// --pre-similarity (MpStage1.cpp:175-248, PMBatchStrData.inl:37-95; the
// reference's GPU form similarity.cu): a pair passes when some diagonal,
// every 2nd one at least PRESIM_EDGE residues from either end, has an
// ungapped run whose Gonnet scores sum to the threshold or more.  Diagonals
// are numbered over the block's longest query and reference: diagonal di
// starts at query position 2*di or, past the query's last admissible start,
// at reference position ((2*di - (lq - 20)) rounded down to even) + 2.  A
// warp per pair, its lanes on 32 diagonals at a time, each summing its run
// in position order (prefix sum minus the smallest prefix so far).
__global__ void __launch_bounds__(128) k_presim(Blk B, Bat T) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (i >= T.np) return;                        // the same for the whole warp
    int qi = pair_qi(B, T, i), ri = pair_ri(B, T, i);
    if (B.cls && cls_pass(B, qi, ri)) return;     // released already (similarity.cu:60-65)
    const int ql = B.qlen[qi], rl = B.rlen[ri];
    const unsigned char* qa = B.qa + B.qoff[qi];
    const unsigned char* ra = B.ra + B.roff[ri];
    const int ndiag = (B.qmax + B.rmax - 2 * PRESIM_EDGE) >> 1;
    bool pass = false;
    for (int d0 = 0; d0 < ndiag; d0 += 32) {
        const int di = d0 + lane;
        if (di < ndiag && !pass) {
            int qp = di * 2, rp = 0;
            if (ql - PRESIM_EDGE <= qp) { rp = ((qp - (ql - PRESIM_EDGE)) & ~1) + 2; qp = 0; }
            if (!(ql - PRESIM_EDGE <= qp || rl - PRESIM_EDGE <= rp)) {
                const int n1 = ql - qp < rl ? ql - qp : rl, n2 = rl - rp < ql ? rl - rp : ql;
                const int n = n1 < n2 ? n1 : n2;
                float s = 0.f, mn = 0.f, best = 0.f;
                for (int k = 0; k < n; k++) {
                    s = __fadd_rn(s, gonnet(qa[qp + k], ra[rp + k]));
                    mn = s < mn ? s : mn;
                    const float loc = __fsub_rn(s, mn);
                    best = loc > best ? loc : best;
                }
                pass = B.presim <= best;
            }
        }
        if (__any_sync(FULL, pass)) {
            if (lane == 0) T.flags[i] = 0;
            return;
        }
    }
}

void launch_presim(const Blk& B, const Bat& T, cudaStream_t st) {
    k_presim<<<(T.np + 3) / 4, 128, 0, st>>>(B, T);
    GTB_LAUNCHED(T);
}

// ---------------------------------------------------------------------------
// position spaces: a gapless diagonal from (q0, r0), or DP-aligned pairs
// stored in traceback (reverse) order.
// (The aligned space is read from the coordinates the traceback stored
// with each aligned pair, 6 floats per pair in traceback order.)
struct PairGeom {
    const float4 *q4, *r4;  // the pair's structures, (x, y, z, 0) per residue
    const float2* alc;      // aligned coordinates, reverse order; null: diagonal
    int q0, r0, n;
    __device__ __forceinline__ void at(int k, float& a, float& b, float& c,
                                       float& d, float& e, float& f) const {
        if (alc) {
            const float2* p = alc + 3 * (n - 1 - k);
            float2 u = __ldg(p), v = __ldg(p + 1), w = __ldg(p + 2);
            a = u.x; b = u.y; c = v.x; d = v.y; e = w.x; f = w.y;
        } else {
            float4 u = __ldg(q4 + q0 + k), v = __ldg(r4 + r0 + k);
            a = u.x; b = u.y; c = u.z; d = v.x; e = v.y; f = v.z;
        }
    }
    // bring line `ln` (0..7) of the positions [k, k+32) into L1 ahead of use
    __device__ __forceinline__ void prefetch(int k, int ln) const {
        const char* p;
        if (alc) {
            int hi = n - 1 - k;                       // positions run backwards in memory
            if (hi < 0) return;
            int lo = hi - 31 < 0 ? 0 : hi - 31;
            const char* base = (const char*)(alc + 3 * lo);
            const char* end = (const char*)(alc + 3 * (hi + 1));
            p = base + 128 * ln;
            if (p >= end) return;
        } else {
            if (k >= n) return;
            int k1 = k + 32 < n ? k + 32 : n;         // stay inside the pair's residues
            const char* base = ln < 4 ? (const char*)(q4 + q0 + k) : (const char*)(r4 + r0 + k);
            const char* end = ln < 4 ? (const char*)(q4 + q0 + k1) : (const char*)(r4 + r0 + k1);
            p = base + 128 * (ln & 3);
            if (p >= end) return;
        }
        asm volatile("prefetch.global.L1 [%0];" :: "l"(p));
    }
};

// Every pass below walks its range in blocks of BLK positions (folded into
// the compensated totals after each block); the block boundaries count from
// the start of the range, as in the oracle.
__device__ void cov_range(const PairGeom& G, int k0, int k1, float* v) {
    CovAcc a;
    a.init();
    for (int b0 = k0; b0 < k1; b0 += BLK) {
        int b1 = b0 + BLK < k1 ? b0 + BLK : k1;
#pragma unroll 4
        for (int k = b0; k < b1; k++) {
            float qx, qy, qz, rx, ry, rz;
            G.at(k, qx, qy, qz, rx, ry, rz);
            a.add(qx, qy, qz, rx, ry, rz);
        }
        a.fold();
    }
    a.final(v);
}

__device__ void cov_ext(const PairGeom& G, const float* tfm, float thr, float* v) {
    CovAcc a;
    a.init();
    for (int b0 = 0; b0 < G.n; b0 += BLK) {
        int b1 = b0 + BLK < G.n ? b0 + BLK : G.n;
#pragma unroll 4
        for (int k = b0; k < b1; k++) {
            float qx, qy, qz, rx, ry, rz;
            G.at(k, qx, qy, qz, rx, ry, rz);
            float d = dist2_tf(tfm, qx, qy, qz, rx, ry, rz);
            if (d <= thr) a.add(qx, qy, qz, rx, ry, rz);
        }
        a.fold();
    }
    a.final(v);
}

// three smallest distances; m3mode 0 none, 1 distinct values, 2 multiset
__device__ __forceinline__ void track3(int m3mode, float d, float& m1, float& m2, float& m3) {
    if (m3mode == 2) {
        if (d < m1) { m3 = m2; m2 = m1; m1 = d; }
        else if (d < m2) { m3 = m2; m2 = d; }
        else if (d < m3) m3 = d;
    } else if (m3mode == 1) {
        if (d < m1) { m3 = m2; m2 = m1; m1 = d; }
        else if (d > m1 && d < m2) { m3 = m2; m2 = d; }
        else if (d > m2 && d < m3) m3 = d;
    }
}

// score pass under tfm (chk: only distances within d82 count)
__device__ float score_pass(const PairGeom& G, const float* tfm, float d02, int chk, float d82,
                            int m3mode, float& m3out) {
    float ss = 0.f, sc = 0.f, sb = 0.f;
    float m1 = LARGEDST, m2 = LARGEDST, m3 = LARGEDST;
    for (int b0 = 0; b0 < G.n; b0 += BLK) {
        int b1 = b0 + BLK < G.n ? b0 + BLK : G.n;
#pragma unroll 4
        for (int k = b0; k < b1; k++) {
            float qx, qy, qz, rx, ry, rz;
            G.at(k, qx, qy, qz, rx, ry, rz);
            float d = dist2_tf(tfm, qx, qy, qz, rx, ry, rz);
            if (!chk || d <= d82) sb = __fadd_rn(sb, tmterm(d02, d));
            track3(m3mode, d, m1, m2, m3);
        }
        nfold(ss, sc, sb);
    }
    nfold(ss, sc, sb);
    m3out = m3;
    return __fadd_rn(ss, sc);
}

// every one of the 16 sums changed by less than RM_CONVEPS relative (b strided)
__device__ __forceinline__ int converged16(const float* a, const float* b, int bstr) {
    int cnt = 0;
#pragma unroll
    for (int f = 0; f < 16; f++) {
        float x = a[f], y = b[f * bstr];
        float m = fabsf(x) < fabsf(y) ? fabsf(x) : fabsf(y);
        if (fabsf(__fsub_rn(x, y)) < __fmul_rn(m, RM_CONVEPS)) cnt++;
    }
    return cnt >= 16;
}

// ---------------------------------------------------------------------------
// stage 1 seed: MpStage1.cpp:289-440

// The seed's fused pass: score (no d8 check), the three smallest distinct
// distances, the covariance of d <= thr, and the SEED_K smallest distances
// with their positions (ascending; ties keep the earlier position first).
// When the next threshold turns out to be above thr, the positions within
// it are usually these few (three in almost every case), and their
// covariance is rebuilt from the list instead of another pass.
constexpr int SEED_K = 6;

__device__ float seed_score_ext(const PairGeom& G, const float* tfm, float d02, float thr,
                                float* v, float& m3out, float* kd, int* kk) {
    float ss = 0.f, sc = 0.f, sb = 0.f;
    float m1 = LARGEDST, m2 = LARGEDST, m3 = LARGEDST;
#pragma unroll
    for (int j = 0; j < SEED_K; j++) { kd[j] = LARGEDST; kk[j] = 0; }
    CovAcc a;
    a.init();
    for (int b0 = 0; b0 < G.n; b0 += BLK) {
        int b1 = b0 + BLK < G.n ? b0 + BLK : G.n;
#pragma unroll 2
        for (int k = b0; k < b1; k++) {
            float qx, qy, qz, rx, ry, rz;
            G.at(k, qx, qy, qz, rx, ry, rz);
            float d = dist2_tf(tfm, qx, qy, qz, rx, ry, rz);
            sb = __fadd_rn(sb, tmterm(d02, d));
            {   // three smallest distinct distances, branch-free
                bool c1 = d < m1, c2 = d > m1 && d < m2, c3 = d > m2 && d < m3;
                m3 = (c1 || c2) ? m2 : (c3 ? d : m3);
                m2 = c1 ? m1 : (c2 ? d : m2);
                m1 = c1 ? d : m1;
            }
            if (d < kd[SEED_K - 1]) {
                // insert (d, k) keeping kd ascending
                float cd = d;
                int ck = k;
#pragma unroll
                for (int j = 0; j < SEED_K; j++) {
                    bool sw = cd < kd[j];
                    float td = kd[j];
                    int tk = kk[j];
                    kd[j] = sw ? cd : td; kk[j] = sw ? ck : tk;
                    cd = sw ? td : cd; ck = sw ? tk : ck;
                }
            }
            if (d <= thr) a.add(qx, qy, qz, rx, ry, rz);
        }
        nfold(ss, sc, sb);
        a.fold();
    }
    nfold(ss, sc, sb);
    a.final(v);
    m3out = m3;
    return __fadd_rn(ss, sc);
}

// covariance of the listed positions with kd <= thr, in position order
// with the block folds of a full pass (folding an empty block changes
// nothing); valid when every position with d <= thr is listed.
__device__ void seed_cov_list(const PairGeom& G, const float* kd, const int* kk, float thr,
                              float* v) {
    int sel[SEED_K], m = 0;
#pragma unroll
    for (int j = 0; j < SEED_K; j++)
        if (kd[j] <= thr) sel[m++] = kk[j];
    for (int x = 1; x < m; x++) {            // position order
        int y = sel[x], z = x - 1;
        while (z >= 0 && sel[z] > y) { sel[z + 1] = sel[z]; z--; }
        sel[z + 1] = y;
    }
    CovAcc a;
    a.init();
    int blk = -1;
    for (int x = 0; x < m; x++) {
        int k = sel[x];
        if (blk >= 0 && k / BLK != blk) a.fold();
        blk = k / BLK;
        float qx, qy, qz, rx, ry, rz;
        G.at(k, qx, qy, qz, rx, ry, rz);
        a.add(qx, qy, qz, rx, ry, rz);
    }
    a.final(v);
}

// vis: position visits of the passes made (the algorithmic work count)
__device__ float findfrag_variant(const PairGeom& G, float d02, float d0s, int swap,
                                  unsigned long long& vis) {
    float v[16], tfm[12], m3, best = 0.f;
    float d02s0 = __fmul_rn(d0s, d0s);
    cov_range(G, 0, G.n, v);
    vis += G.n;
    for (int it = 0; it < 3; it++) {
        solve_sums(v, swap, tfm);
        vis += G.n;
        if (it == 2) {
            float sc = score_pass(G, tfm, d02, 0, 0.f, 0, m3);
            if (best < sc) best = sc;
            break;
        }
        float d02s = __fadd_rn(d02s0, (it == 1 ? 1.0f : 0.0f));
        // the next threshold is d02s unless the third-smallest distance is
        // above it: accumulate for d02s while scoring, redo in the rare case
        float kd[SEED_K];
        int kk[SEED_K];
        float sc = seed_score_ext(G, tfm, d02, d02s, v, m3, kd, kk);
        if (best < sc) best = sc;
        float dst32;
        if (LARGEDST_CMP < m3 || m3 < d02s || G.n <= 3) dst32 = d02s;
        else dst32 = __fadd_rn(d02s, __fmul_rn(ceilf(__fmul_rn(__fsub_rn(m3, d02s), 2.0f)), 0.5f));
        if (dst32 != d02s) {
            if (dst32 < kd[SEED_K - 1]) seed_cov_list(G, kd, kk, dst32, v);
            else { cov_ext(G, tfm, dst32, v); vis += G.n; }
        }
        if (v[15] < 1.0f) break;
        if ((int)v[15] == G.n) break;
    }
    return best;
}

// The same for ordinary coordinates (coords_ordinary), without branches in the
// sweeps.  findfrag_variant's fused pass kept the six smallest distances with
// their positions and added to the covariance as it went: with 32 offsets a
// warp, some lane took nearly every branch (about 60 issued instructions a
// visit).  Here a pass scores and keeps the three smallest distances by five
// minima and maxima; the threshold then known, a second sweep marks the
// positions within it in a 32-bit mask per block and only the marked ones are
// added.  What bounds it: issue, and the L1 reads of 32 offsets' residues.
struct SeedCov {                       // covariance sums, CovAcc's order of operations
    float s[15], c[15], b[15];
    int n;
    __device__ __forceinline__ void init() {
#pragma unroll
        for (int f = 0; f < 15; f++) { s[f] = 0.f; c[f] = 0.f; b[f] = 0.f; }
        n = 0;
    }
    __device__ __forceinline__ void add(const float4& u, const float4& v) {
        b[0] = __fmaf_rn(u.x, v.x, b[0]); b[1] = __fmaf_rn(u.x, v.y, b[1]); b[2] = __fmaf_rn(u.x, v.z, b[2]);
        b[3] = __fmaf_rn(u.y, v.x, b[3]); b[4] = __fmaf_rn(u.y, v.y, b[4]); b[5] = __fmaf_rn(u.y, v.z, b[5]);
        b[6] = __fmaf_rn(u.z, v.x, b[6]); b[7] = __fmaf_rn(u.z, v.y, b[7]); b[8] = __fmaf_rn(u.z, v.z, b[8]);
        b[9] = __fadd_rn(b[9], u.x); b[10] = __fadd_rn(b[10], u.y); b[11] = __fadd_rn(b[11], u.z);
        b[12] = __fadd_rn(b[12], v.x); b[13] = __fadd_rn(b[13], v.y); b[14] = __fadd_rn(b[14], v.z);
    }
    __device__ __forceinline__ void fold() {
#pragma unroll
        for (int f = 0; f < 15; f++) { tfold(s[f], c[f], b[f]); b[f] = 0.f; }
    }
    __device__ __forceinline__ void final(float* v) const {
#pragma unroll
        for (int f = 0; f < 15; f++) v[f] = __fadd_rn(s[f], c[f]);
        v[15] = (float)n;
    }
};

__device__ __forceinline__ float seed_d2(const float* tfm, const float4& u, const float4& v) {
    return dist2_tf(tfm, u.x, u.y, u.z, v.x, v.y, v.z);
}

// score under tfm and, M3, the three smallest distances (a multiset)
template <bool M3>
__device__ __forceinline__ float seed_score(const float4* q, const float4* r, int n, const float* tfm,
                                            float d02, float& m1, float& m2, float& m3) {
    float ss = 0.f, sc = 0.f;
    m1 = m2 = m3 = LARGEDST;
    auto visit = [&](int k, float& sb) {
        const float d = seed_d2(tfm, __ldg(q + k), __ldg(r + k));
        sb = __fadd_rn(sb, div_ord(d02, __fadd_rn(d02, d)));
        if (M3) {
            const float a = fmaxf(m1, d);
            m1 = fminf(m1, d);
            m3 = fminf(m3, fmaxf(m2, a));
            m2 = fminf(m2, a);
        }
    };
    int b0 = 0;
    for (; b0 + BLK <= n; b0 += BLK) {
        float sb = 0.f;
#pragma unroll 8
        for (int k = 0; k < BLK; k++) visit(b0 + k, sb);
        tfold(ss, sc, sb);
    }
    float sb = 0.f;
#pragma unroll 2
    for (int k = b0; k < n; k++) visit(k, sb);
    tfold(ss, sc, sb);
    return __fadd_rn(ss, sc);
}

// covariance of the positions with d <= thr
__device__ __forceinline__ void seed_cov(const float4* q, const float4* r, int n, const float* tfm,
                                         float thr, float* v) {
    SeedCov A;
    A.init();
    for (int b0 = 0; b0 < n; b0 += BLK) {
        unsigned mask = 0u;
        if (b0 + BLK <= n) {
#pragma unroll 1
            for (int k = 0; k < BLK; k += 8) {
                unsigned m8 = 0u;
#pragma unroll
                for (int e = 0; e < 8; e++)
                    if (seed_d2(tfm, __ldg(q + b0 + k + e), __ldg(r + b0 + k + e)) <= thr) m8 |= 1u << e;
                mask |= m8 << k;
            }
        } else {
#pragma unroll 2
            for (int k = b0; k < n; k++)
                if (seed_d2(tfm, __ldg(q + k), __ldg(r + k)) <= thr) mask |= 1u << (k - b0);
        }
        if (mask) {
            A.n += __popc(mask);
            do {
                const int k = b0 + __ffs(mask) - 1;
                mask &= mask - 1;
                A.add(__ldg(q + k), __ldg(r + k));
            } while (mask);
            A.fold();
        }
    }
    A.final(v);
}

// the third smallest distinct distance (ties among the smallest: rare)
__device__ __noinline__ float seed_third_distinct(const float4* q, const float4* r, int n, const float* tfm) {
    float m1 = LARGEDST, m2 = LARGEDST, m3 = LARGEDST;
    for (int k = 0; k < n; k++) track3(1, seed_d2(tfm, __ldg(q + k), __ldg(r + k)), m1, m2, m3);
    return m3;
}

// vis counts what findfrag_variant's fused passes visit (the covariance sweep is
// the same visit's second half)
__device__ __forceinline__ float findfrag_variant_fast(const float4* q, const float4* r, int n, float d02,
                                                       float d0s, int swap, unsigned long long& vis) {
    float v[16], tfm[12], best = 0.f;
    const float d02s0 = __fmul_rn(d0s, d0s);
    {
        SeedCov A;
        A.init();
        for (int b0 = 0; b0 < n; b0 += BLK) {
            const int b1 = b0 + BLK < n ? b0 + BLK : n;
#pragma unroll 4
            for (int k = b0; k < b1; k++) A.add(__ldg(q + k), __ldg(r + k));
            A.fold();
        }
        A.n = n;
        A.final(v);
    }
    vis += n;
#pragma unroll 1
    for (int it = 0; it < 3; it++) {
        solve_sums(v, swap, tfm);
        float m1, m2, m3;
        vis += n;
        if (it == 2) {
            const float sc = seed_score<false>(q, r, n, tfm, d02, m1, m2, m3);
            if (best < sc) best = sc;
            break;
        }
        const float d02s = __fadd_rn(d02s0, (it == 1 ? 1.0f : 0.0f));
        const float sc = seed_score<true>(q, r, n, tfm, d02, m1, m2, m3);
        if (best < sc) best = sc;
        if ((m1 == m2 || m2 == m3) && m1 < LARGEDST) m3 = seed_third_distinct(q, r, n, tfm);
        float dst32;
        if (LARGEDST_CMP < m3 || m3 < d02s || n <= 3) dst32 = d02s;
        else dst32 = __fadd_rn(d02s, __fmul_rn(ceilf(__fmul_rn(__fsub_rn(m3, d02s), 2.0f)), 0.5f));
        seed_cov(q, r, n, tfm, dst32, v);
        if (v[15] < 1.0f) break;
        if ((int)v[15] == n) break;
    }
    return best;
}

__global__ void __launch_bounds__(128) k_findfrag(Blk B, Bat T) {
    const int item = blockIdx.x;
    int i = item, c = 0, nch = 1;
    if (T.ff_pair) {
        if (item >= T.nff) return;
        i = T.ff_pair[item];
        c = T.ff_chunk[item];
        nch = T.ff_nch[i];
    }
    if (i >= T.np) return;
    int flags = T.flags[i];
    if (flags & CONV_LOWTMSC) return;
    int qi = pair_qi(B, T, i), ri = pair_ri(B, T, i);
    int lq = B.qlen[qi], lr = B.rlen[ri];
    const int step = B.stepinit;
    int n1, silo, sihi, prv;
    seed_range(lq, lr, B.qmax, B.qmin, B.rmax, B.rmin, step, n1, silo, sihi, prv);
    const int ml = lq < lr ? lq : lr;
    // this CTA's share of the offsets
    int s0 = silo, s1 = sihi;
    if (nch > 1) {
        const int chunk = T.ff_span > 0 ? T.ff_span : FF_CHUNK;
        s0 = silo + c * chunk;
        s1 = s0 + chunk - 1 < sihi ? s0 + chunk - 1 : sihi;
    }
    float d0 = B.t_d0[ml];
    float d02 = __fmul_rn(d0, d0);
    float d0s = d0s_of(d0);
    int swap = B.symmetric && (lq < lr);
    PairGeom G;
    G.q4 = B.q4 + B.q4off[qi]; G.r4 = B.r4 + B.r4off[ri];
    G.alc = nullptr;
    const bool fast = coords_ordinary(B, qi, ri);
    float lbest = 0.f;
    int lsi = 0x7fffffff;
    unsigned long long vis = 0;
    // offsets handed out one at a time (a thread's offsets still come in
    // increasing order, so its strict-improvement rule keeps the lowest index)
    __shared__ int s_next;
    if (threadIdx.x == 0) s_next = s0 + (int)blockDim.x;
    __syncthreads();
    for (int si = s0 + (int)threadIdx.x; si <= s1; si = atomicAdd(&s_next, 1)) {
        int ab = n1 + si * step;
        int qpos = ab > 0 ? ab : 0;
        int rpos = -ab > 0 ? -ab : 0;
        if (lq <= qpos || lr <= rpos) continue;
        if (lq - qpos < prv || lr - rpos < prv) continue;
        G.q0 = qpos; G.r0 = rpos;
        G.n = (lq - qpos) < (lr - rpos) ? (lq - qpos) : (lr - rpos);
        const float b = fast ? findfrag_variant_fast(G.q4 + qpos, G.r4 + rpos, G.n, d02, d0s, swap, vis)
                             : findfrag_variant(G, d02, d0s, swap, vis);
        if (b > 0.f && lbest < b) { lbest = b; lsi = si; }
    }
    __shared__ float sb[128];
    __shared__ int ssi[128];
    __shared__ unsigned long long s_vis;
    if (threadIdx.x == 0) s_vis = 0;
    sb[threadIdx.x] = lbest;
    ssi[threadIdx.x] = lsi;
    __syncthreads();
    if (T.work) atomicAdd(&s_vis, vis);
    for (int s = blockDim.x >> 1; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) {
            float o = sb[threadIdx.x + s];
            int os = ssi[threadIdx.x + s];
            if (o > sb[threadIdx.x] || (o == sb[threadIdx.x] && os < ssi[threadIdx.x])) {
                sb[threadIdx.x] = o;
                ssi[threadIdx.x] = os;
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        work_add(T, WK_SEED, s_vis);
        float b = sb[0];
        if (nch > 1) {
            // larger score, then lower offset index, over the pair's CTAs
            if (b > 0.f) {
                unsigned long long key = ((unsigned long long)__float_as_uint(b) << 32) |
                                         (unsigned long long)(0xffffffffu - (unsigned)ssi[0]);
                atomicMax(T.ff_key + i, key);
            }
            return;
        }
        T.best[i] = b;
        if (b > 0.f) {
            int ab = n1 + ssi[0] * step;
            T.seedq[i] = ab > 0 ? ab : 0;
            T.seedr[i] = -ab > 0 ? -ab : 0;
        } else {
            T.seedq[i] = 0;
            T.seedr[i] = 0;
        }
    }
}

// seeds of the pairs split over several CTAs
__global__ void k_findfrag_fin(Blk B, Bat T) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= T.np || T.ff_nch[i] <= 1) return;
    if (T.flags[i] & CONV_LOWTMSC) return;
    unsigned long long key = T.ff_key[i];
    float b = __uint_as_float((unsigned)(key >> 32));
    T.best[i] = b;
    if (b > 0.f) {
        int qi = pair_qi(B, T, i), ri = pair_ri(B, T, i);
        int n1, silo, sihi, prv;
        seed_range(B.qlen[qi], B.rlen[ri], B.qmax, B.qmin, B.rmax, B.rmin, B.stepinit, n1, silo,
                   sihi, prv);
        int si = (int)(0xffffffffu - (unsigned)(key & 0xffffffffu));
        int ab = n1 + si * B.stepinit;
        T.seedq[i] = ab > 0 ? ab : 0;
        T.seedr[i] = -ab > 0 ? -ab : 0;
    } else {
        T.seedq[i] = 0;
        T.seedr[i] = 0;
    }
}

void launch_findfrag(const Blk& B, const Bat& T, cudaStream_t st) {
    KtScope kts(T, KF_SEED, st);
    if (T.ff_pair) {
        cudaMemsetAsync(T.ff_key, 0, (size_t)T.np * sizeof(unsigned long long), st);
        k_findfrag<<<T.nff, 128, 0, st>>>(B, T);
        k_findfrag_fin<<<(T.np + 255) / 256, 256, 0, st>>>(B, T);
        if (T.launches) (*T.launches) += 2;
        return;
    }
    k_findfrag<<<T.np, 128, 0, st>>>(B, T);
    GTB_LAUNCHED(T);
}

// ---------------------------------------------------------------------------
// Refinement work list.  Before each refinement launch the pairs that take
// part (mode's convergence flags clear, a non-empty position space) are
// listed in decreasing order of their position count (buckets of 16), so
// that the pairs sharing a warp have passes of about the same length and
// finished pairs cost nothing.  Pairs left out get the mode's outputs for
// "no variant scored" here.
constexpr int RL_SHIFT = 4;
// up to here one CTA builds a list (4 pairs a thread): one pair 4.9 -> 4.2 ms,
// 1 x 1,000 at the fastest preset 7.5 -> 7.2
constexpr int LIST_SMALL = 4096;
constexpr int RL_NB = 65536 >> RL_SHIFT;   // buckets; rhist[RL_NB] = list length

// position count of pair i in mode `mode`, or -1 when the pair is skipped
__device__ __forceinline__ int refine_span(const Blk& B, const Bat& T, int mode, int i) {
    int flags = T.flags[i];
    if (mode == RM_DP ? flags != 0 : (flags & CONV_LOWTMSC) != 0) return -1;
    if (mode != RM_INIT) return T.naln[i];
    int qi = pair_qi(B, T, i), ri = pair_ri(B, T, i);
    int lq = B.qlen[qi], lr = B.rlen[ri];
    int sq = T.seedq[i], sr = T.seedr[i];
    if (lq <= sq || lr <= sr) return 0;
    return (lq - sq) < (lr - sr) ? (lq - sq) : (lr - sr);
}

// pair i's bucket, or -1: left out (with its outputs for "no variant scored"
// here), or put on the long pairs' list
__device__ __forceinline__ int rlist_bucket(const Blk& B, const Bat& T, int i, int mode) {
    int n = refine_span(B, T, mode, i);
    if (n >= T.rl_min && T.rl_long) {          // many warps for this pair
        int slot = atomicAdd(T.rl_count, 1);
        if (slot < T.rl_nlmax) { T.rl_long[slot] = i; return -1; }
    }
    if (n > 0) return RL_NB - 1 - (n >> RL_SHIFT);
    // no variant: MpStage1.cpp:700-716 with nothing scored
    bool skipped = n < 0;
    if (mode == RM_INIT || mode == RM_DP || (!skipped && (mode == RM_FIN1 || mode == RM_FIN2)))
        T.best[i] = 0.f;
    if (!skipped && mode == RM_FIN1) { T.sfndx[i] = T.sfndx_cur[i]; T.sfpos[i] = T.sfpos_cur[i]; }
    return -1;
}

__global__ void k_rlist_count(Blk B, Bat T, int mode) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= T.np) return;
    int b = rlist_bucket(B, T, i, mode);
    if (b >= 0) atomicAdd(&T.rhist[b], 1);
}

// exclusive scan of the bucket counts (one CTA of 1024 threads)
__global__ void __launch_bounds__(1024) k_rlist_scan(Bat T) {
    __shared__ int part[1024];
    constexpr int PER = RL_NB / 1024;
    int t = threadIdx.x, loc[PER], s = 0;
#pragma unroll
    for (int j = 0; j < PER; j++) { loc[j] = T.rhist[t * PER + j]; s += loc[j]; }
    part[t] = s;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        int v = t >= o ? part[t - o] : 0;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    int run = part[t] - s;
#pragma unroll
    for (int j = 0; j < PER; j++) { T.rhist[t * PER + j] = run; run += loc[j]; }
    if (t == 1023) T.rhist[RL_NB] = part[1023];
}

// skipmode & DL_KEEPALN: the pairs left out keep their aligned pairs (before a
// constrained traceback); else they have none
constexpr int DL_KEEPALN = 2;
// DP work list: the pairs a DP launch works on (flags clear, not on the
// wavefront path), largest matrices first; kept in the same buffers as the
// refinement list (a DP launch is over before the next list is built).
__device__ __forceinline__ int dlist_bucket(const Blk& B, const Bat& T, int i, int skipmode) {
    int skipmask = (skipmode & 1) == 0 ? (CONV_LOWTMSC | CONV_SCOREDP) : CONV_LOWTMSC;
    if (T.flags[i] & skipmask) return -1;
    if (T.dw_mark && T.dw_mark[i]) return -1;
    if (alt_empty(T, i)) return -1;
    int qi = pair_qi(B, T, i), ri = pair_ri(B, T, i);
    long long cells = (long long)B.qlen[qi] * B.rlen[ri];
    long long b = cells >> 8;
    return RL_NB - 1 - (int)(b < RL_NB - 1 ? b : RL_NB - 1);
}

__global__ void k_dlist_count(Blk B, Bat T, int skipmode) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= T.np) return;
    int b = dlist_bucket(B, T, i, skipmode);
    if (b >= 0) atomicAdd(&T.rhist[b], 1);
    else if (!(skipmode & DL_KEEPALN)) T.naln[i] = 0;
}

__global__ void k_dlist_fill(Blk B, Bat T, int skipmode) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= T.np) return;
    int b = dlist_bucket(B, T, i, skipmode);
    if (b >= 0) T.rlist[atomicAdd(&T.rhist[b], 1)] = i;
}

// pair list without any flag of skipmask (every size, wavefront pairs too)
__device__ __forceinline__ int plist_bucket(const Blk& B, const Bat& T, int i, int skipmask) {
    if (T.flags[i] & skipmask) return -1;
    int qi = pair_qi(B, T, i), ri = pair_ri(B, T, i);
    long long b = ((long long)B.qlen[qi] * B.rlen[ri]) >> 8;
    return RL_NB - 1 - (int)(b < RL_NB - 1 ? b : RL_NB - 1);
}
__global__ void k_plist_count(Blk B, Bat T, int skipmask) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= T.np) return;
    int b = plist_bucket(B, T, i, skipmask);
    if (b >= 0) atomicAdd(&T.rhist[b], 1);
}
__global__ void k_plist_fill(Blk B, Bat T, int skipmask) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= T.np) return;
    int b = plist_bucket(B, T, i, skipmask);
    if (b >= 0) T.rlist[atomicAdd(&T.rhist[b], 1)] = i;
}

__global__ void k_rlist_fill(Blk B, Bat T, int mode) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= T.np) return;
    int n = refine_span(B, T, mode, i);
    if (n >= T.rl_min && T.rl_long) return;      // listed by k_rlist_count
    if (n > 0) T.rlist[atomicAdd(&T.rhist[RL_NB - 1 - (n >> RL_SHIFT)], 1)] = i;
}

// The work list of a batch of at most LIST_SMALL pairs by one CTA, buckets in
// shared memory, in place of a memset and three launches (KIND: LK_*; arg: the
// refinement mode, the DP's skip mode or the flag mask).
enum ListKind { LK_REFINE = 0, LK_DP = 1, LK_PAIRS = 2 };
template <int KIND>
__global__ void __launch_bounds__(1024) k_list_small(Blk B, Bat T, int arg) {
    __shared__ int hist[RL_NB], part[1024];
    constexpr int PER = RL_NB / 1024, IPT = LIST_SMALL / 1024;
    const int t = threadIdx.x;
#pragma unroll
    for (int j = 0; j < PER; j++) hist[t * PER + j] = 0;
    if (KIND == LK_REFINE && T.rl_long) {
        if (t == 0) *T.rl_count = 0;
        for (int k = t; k < T.rl_nlmax; k += 1024) T.rl_next[k] = 0;
    }
    __syncthreads();
    int b[IPT];
#pragma unroll
    for (int j = 0; j < IPT; j++) {
        const int i = t + 1024 * j;
        b[j] = -1;
        if (i < T.np) {
            b[j] = KIND == LK_REFINE ? rlist_bucket(B, T, i, arg)
                 : KIND == LK_DP ? dlist_bucket(B, T, i, arg) : plist_bucket(B, T, i, arg);
            if (b[j] >= 0) atomicAdd(&hist[b[j]], 1);
            else if (KIND == LK_DP && !(arg & DL_KEEPALN)) T.naln[i] = 0;
        }
    }
    __syncthreads();
    int loc[PER], s = 0;
#pragma unroll
    for (int j = 0; j < PER; j++) { loc[j] = hist[t * PER + j]; s += loc[j]; }
    part[t] = s;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const int v = t >= o ? part[t - o] : 0;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    int run = part[t] - s;
#pragma unroll
    for (int j = 0; j < PER; j++) { hist[t * PER + j] = run; run += loc[j]; }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < IPT; j++)
        if (b[j] >= 0) T.rlist[atomicAdd(&hist[b[j]], 1)] = t + 1024 * j;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < PER; j++) T.rhist[t * PER + j] = hist[t * PER + j];
    if (t == 0) T.rhist[RL_NB] = part[1023];
    if (t < RL_NHIST - RL_NB - 1) T.rhist[RL_NB + 1 + t] = 0;
}

// Variant list of one pair, enumerated compactly (admissible variants only).
// VK_STAGE (6 fragment lengths x step 40): variant si = fct*6 + ndx is
// admissible when frag_length(n, ndx) >= 1 and 40*fct + fraglen < n + 40
// (MpStage1.cpp:635-641).  VK_P2ONE (phase 2, one length: the phase-1
// winner's, 0 promoted to 1): si in [0, nf), pos = pos1 - nf/2 + si, with
// 0 <= pos and pos + fraglen <= n (MpStageFin.cpp:380-396).  VK_P2ALL (phase
// 2, every length: --refinement 2 in production, 3 in both final phases):
// si = fct*6 + ndx, pos = pos1 - nf/2 + fct, the same bounds
// (covariance_production_dp_refn_complete.cu:381-530,
// covariance_fin_dp_refn_complete.cu:464-630).  VK_LOG (one round of the
// log search, covariance_production_dp_refn_complete.cu:836-880): lengths
// 1..5 at pos = pos1 + step, si = ndx, admissible when 0 <= pos and
// pos + fraglen < n + max(step, 0); a fragment reaching past the end is
// shifted back to end at n.
enum VariantKind { VK_STAGE = 0, VK_P2ONE = 1, VK_P2ALL = 2, VK_LOG = 3 };

// the variants of a refinement launch
__device__ __forceinline__ int refine_variants(int mode, const Blk& B) {
    return mode == RM_PLOG ? VK_LOG
         : mode == RM_FIN2 ? (B.refinement == GTB_REFINEMENT_FULLA ? VK_P2ALL : VK_P2ONE)
         : mode == RM_PROD2 ? (B.refinement >= GTB_REFINEMENT_FULL ? VK_P2ALL : VK_P2ONE)
         : VK_STAGE;
}

struct VariantList {
    int total;
    int cnt[FRAG_NSUB], fl[FRAG_NSUB], lo[FRAG_NSUB];
    int base;                 // phase 2: position of si (or fct) = base + si; log: the round's position
};

// the step of log-search round r: +32, -32, +16, -16, ..., +1, -1
__device__ __forceinline__ int plog_step(int r) {
    int st = 32 >> (r >> 1);
    return (r & 1) ? -st : st;
}

__device__ __forceinline__ void variants_init(VariantList& V, int vk, int n, int maxalnmax,
                                              int sfndx0, int sfpos0, int round) {
    V.total = 0;
    V.base = 0;
#pragma unroll
    for (int d = 0; d < FRAG_NSUB; d++) { V.cnt[d] = 0; V.fl[d] = 0; V.lo[d] = 0; }
    if (n <= 0) return;
    if (vk == VK_STAGE) {
        int NF = (int)ceilf((float)(maxalnmax + FRAG_STEP - MINFRAGLEN) / FRAG_STEP);
#pragma unroll
        for (int d = 0; d < FRAG_NSUB; d++) {
            int fl = frag_length(n, d);
            int c = 0;
            if (fl >= 1) {
                c = (n + FRAG_STEP - fl + FRAG_STEP - 1) / FRAG_STEP;
                if (c > NF) c = NF;
                if (c < 0) c = 0;
            }
            V.fl[d] = fl;
            V.cnt[d] = c;
            V.total += c;
        }
        return;
    }
    if (vk == VK_LOG) {
        int step = plog_step(round);
        int pos = sfpos0 + step;
        int ext = step > 0 ? step : 0;
        V.base = pos;
#pragma unroll
        for (int d = 1; d < FRAG_NSUB; d++) {
            int fl = frag_length(n, d);
            int c = (fl >= 1 && pos >= 0 && pos + fl < n + ext) ? 1 : 0;
            V.fl[d] = fl;
            V.cnt[d] = c;
            V.total += c;
        }
        return;
    }
    int nf = 2 * maxalnmax < FIN_MAXNPOS ? 2 * maxalnmax : FIN_MAXNPOS;
    V.base = sfpos0 - (nf >> 1);                // pos = base + fct
    const int lo = -V.base > 0 ? -V.base : 0;   // pos >= 0
#pragma unroll
    for (int d = 0; d < FRAG_NSUB; d++) {
        bool use = vk == VK_P2ALL || d == (sfndx0 == 0 ? 1 : sfndx0);
        int fl = use ? frag_length(n, d) : 0;
        int c = 0;
        if (fl >= 1) {
            int hi = n - fl - V.base;           // pos + fl <= n
            if (hi > nf - 1) hi = nf - 1;
            c = hi >= lo ? hi - lo + 1 : 0;
        }
        V.fl[d] = fl;
        V.lo[d] = lo;
        V.cnt[d] = c;
        V.total += c;
    }
}

// k-th admissible variant (0 <= k < total) -> (si, length index, position,
// length, first position of the refined fragment); variants are grouped by
// length index, so ties are broken by si, not by k
__device__ __forceinline__ void variants_get(const VariantList& V, int vk, int n, int k,
                                             int& si, int& ndx, int& pos, int& fl, int& kf) {
    // the group is selected inside the unrolled loop (no run-time array index)
    int d = 0, c = V.cnt[0], fcl = V.fl[0], lol = V.lo[0];
#pragma unroll
    for (int e = 1; e < FRAG_NSUB; e++) {
        if (k >= c) { k -= c; d = e; c = V.cnt[e]; fcl = V.fl[e]; lol = V.lo[e]; }
    }
    ndx = d;
    fl = fcl;
    if (vk == VK_STAGE) {
        si = k * FRAG_NSUB + d;
        pos = k * FRAG_STEP;
    } else if (vk == VK_LOG) {
        si = d;
        pos = V.base;
    } else {
        int fct = lol + k;
        si = vk == VK_P2ALL ? fct * FRAG_NSUB + d : fct;
        pos = V.base + fct;
    }
    int delta = pos + fl - n;
    kf = pos - (delta > 0 ? delta : 0);
}

// ---------------------------------------------------------------------------
// Refinement.  RF_LPP lanes share one pair and take the pair's admissible
// variants from a pool in list order; a lane whose variant is done takes
// the next one, so the lanes stay busy while variants last.  All lanes
// advance together one pass at a time (a pass = one sweep of the pair's
// positions); what a lane does in a pass depends on where its variant is
// in the refinement loop of MpStage1.cpp:640-700 (and its copies in
// RefineFragDPKernel and MpStageFin.cpp):
enum PassKind {
    PK_IDLE = 0,    // no variant left for this lane
    PK_FRAG = 1,    // covariance of the fragment [k0, k1)
    PK_SCORE = 2,   // score under tfm, fused with the covariance of d <= thr
    PK_EXT = 3,     // covariance of d <= thr only (iteration 1's threshold
                    // when it differs from the one fused into iteration 0)
    PK_GSCORE = 4,  // score of the variant's best transform with another d0
};

// One pass of one lane.  Blocks of BLK positions are the absolute blocks
// of the position space for every kind, so lanes fold together.
// M3 / FR / SC: whether any lane of the warp tracks the three smallest
// distances, covers a fragment, or scores in this pass; the code for what
// no lane does is left out.
template <bool M3, bool FR, bool SC>
__device__ __forceinline__ float lane_pass_t(const PairGeom& G, int kind, int k0, int k1,
                                             const float* tfm, float d02, int chk, float d82,
                                             float thr, int m3on, float* v, float& m3out, int pl) {
    float ss = 0.f, sc = 0.f, sb = 0.f;
    float m1 = LARGEDST, m2 = LARGEDST, m3 = LARGEDST;
    const bool frag = FR && kind == PK_FRAG;
    const bool scr = SC && (kind == PK_SCORE || kind == PK_GSCORE);
    const bool cov = kind == PK_SCORE || kind == PK_EXT;
    const int n = kind == PK_IDLE ? 0 : (frag ? k1 : G.n);
    CovAcc a;
    a.init();
    for (int b0 = frag ? (k0 & ~(BLK - 1)) : 0; b0 < n; b0 += BLK) {
        int b1 = b0 + BLK < n ? b0 + BLK : n;
        if (pl < 8) G.prefetch(b0 + BLK, pl);    // the next block, one line per lane
#pragma unroll 2
        for (int k = b0; k < b1; k++) {
            float qx, qy, qz, rx, ry, rz;
            G.at(k, qx, qy, qz, rx, ry, rz);
            float d = dist2_tf(tfm, qx, qy, qz, rx, ry, rz);
            // branch-free: adding +0 and zero coordinates leaves the sums unchanged
            if (SC) {
                float tm = tmterm(d02, d);
                sb = __fadd_rn(sb, (scr && (!chk || d <= d82)) ? tm : 0.f);
            }
            if (M3) {
                bool c1 = m3on && d < m1, c2 = m3on && d < m2, c3 = m3on && d < m3;
                m3 = c2 ? m2 : (c3 ? d : m3);
                m2 = c1 ? m1 : (c2 ? d : m2);
                m1 = c1 ? d : m1;
            }
            bool inc = FR ? (frag ? (k0 <= k) : (cov && d <= thr)) : (cov && d <= thr);
            a.add(inc ? qx : 0.f, inc ? qy : 0.f, inc ? qz : 0.f,
                  inc ? rx : 0.f, inc ? ry : 0.f, inc ? rz : 0.f);
            a.n += inc ? 0 : -1;
        }
        nfold(ss, sc, sb);
        a.fold();
    }
    nfold(ss, sc, sb);
    a.final(v);
    m3out = m3;
    return __fadd_rn(ss, sc);
}

__device__ __forceinline__ float lane_pass(const PairGeom& G, int kind, int k0, int k1,
                                           const float* tfm, float d02, int chk, float d82,
                                           float thr, int m3on, float* v, float& m3out, int pl) {
    const unsigned FULL = 0xffffffffu;
    const bool sc = __any_sync(FULL, kind == PK_SCORE || kind == PK_GSCORE);
    const bool m3 = __any_sync(FULL, kind == PK_SCORE && m3on);
    const bool fr = __any_sync(FULL, kind == PK_FRAG);
    if (m3)
        return fr ? lane_pass_t<true, true, true>(G, kind, k0, k1, tfm, d02, chk, d82, thr, m3on, v, m3out, pl)
                  : lane_pass_t<true, false, true>(G, kind, k0, k1, tfm, d02, chk, d82, thr, m3on, v, m3out, pl);
    if (sc)
        return fr ? lane_pass_t<false, true, true>(G, kind, k0, k1, tfm, d02, chk, d82, thr, m3on, v, m3out, pl)
                  : lane_pass_t<false, false, true>(G, kind, k0, k1, tfm, d02, chk, d82, thr, m3on, v, m3out, pl);
    return fr ? lane_pass_t<false, true, false>(G, kind, k0, k1, tfm, d02, chk, d82, thr, m3on, v, m3out, pl)
              : lane_pass_t<false, false, false>(G, kind, k0, k1, tfm, d02, chk, d82, thr, m3on, v, m3out, pl);
}

// The pair's result of a refinement launch (MpStage1.cpp:700-716 and the
// final/production copies): winner score, transform and fragment, or the
// "nothing scored" outputs.  tb: the winner's transform, stride tstr.
template <int MODE>
__device__ __forceinline__ void refine_commit(const Blk& B, const Bat& T, int i, int lq, int lr,
                                              bool havewin, float wb, float lgbest, int wndx,
                                              int wpos, const float* tb, int tstr) {
    if (MODE == RM_PROD1 || MODE == RM_PROD2 || MODE == RM_PLOG) {
        if (!havewin) return;
        float grand = T.grand[i];
        bool write = (MODE == RM_PROD1) || (grand < wb);
        if (write) {
            T.grand[i] = wb;
            float bs = wb, gb = lgbest;
            if ((float)lr < (float)lq) { float t = bs; bs = gb; gb = t; }
            T.out[i * 16 + 9] = __fdiv_rn(bs, (float)lq);
            T.out[i * 16 + 10] = __fdiv_rn(gb, (float)lr);
            T.out[i * 16 + 11] = B.t_d0fin[lq];
            T.out[i * 16 + 12] = B.t_d0fin[lr];
#pragma unroll
            for (int f = 0; f < 12; f++) T.tfm_gr[i * 12 + f] = tb[f * tstr];
            if (MODE == RM_PROD1) { T.sfndx[i] = wndx; T.sfpos[i] = wpos; }
            if (MODE == RM_PLOG) T.sfpos[i] = wpos;   // the search moves to the round's position
        }
        return;
    }
    T.best[i] = havewin ? wb : 0.f;
    if (havewin) {
#pragma unroll
        for (int f = 0; f < 12; f++) T.tfm_ib[i * 12 + f] = tb[f * tstr];
        if (T.grand[i] < wb) {
            T.grand[i] = wb;
#pragma unroll
            for (int f = 0; f < 12; f++) T.tfm_gr[i * 12 + f] = tb[f * tstr];
        }
    }
    if (MODE == RM_FIN1) {
        // the winner's fragment, or the previous one when no variant scored
        int nd = havewin ? wndx : T.sfndx_cur[i];
        int np_ = havewin ? wpos : T.sfpos_cur[i];
        T.sfndx_cur[i] = nd; T.sfpos_cur[i] = np_;
        T.sfndx[i] = nd; T.sfpos[i] = np_;
    }
}

// RF_LPP lanes per pair: 16 (two pairs per warp), or a warp (long pairs).
// Warps per CTA: 4 (1 and 2, with an SM refilling a finished warp's slot at
// once, measured the same on the benchmark step: the concurrent sub-batch
// streams fill those slots already).
constexpr int RF_WARPS_SHORT = 4;
constexpr int RF_WARPS_LONG = RLW_CTA_WARPS;

// LONG: the pairs with at least RL_LONG positions, RLW_CTAS CTAs each; every
// warp of them takes the pair's variants from one counter in global memory
// and leaves its best variant as a candidate; k_refine_long_fin picks the
// pair's winner among them.
// One slot of a refinement launch: a short pair (slot of the length-sorted
// list) or, LONG, warp `wlong` of the warps working on long pair `slot`.
template <int MODE, int RF_LPP, bool LONG>
__device__ __forceinline__ void refine_slot(const Blk& B, const Bat& T, int slot, int wlong, int slot_end = 0) {
    constexpr int RF_WARPS = LONG ? RF_WARPS_LONG : RF_WARPS_SHORT;
    __shared__ float s_last[16 * RF_WARPS * 32];   // previous iteration's sums
    __shared__ float s_tb[12 * RF_WARPS * 32];     // best transform of the current variant
    __shared__ float s_tbest[12 * RF_WARPS * 32];  // best transform over the lane's variants
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int sub = lane / RF_LPP;
    const unsigned smask = RF_LPP == 32 ? 0xffffffffu : ((1u << (RF_LPP & 31)) - 1u) << (sub * RF_LPP);
    const bool valid = LONG ? slot < *T.rl_count : slot < slot_end;
    if (__ballot_sync(FULL, valid) == 0) return;
    const int i = valid ? (LONG ? T.rl_long[slot] : T.rlist[slot]) : 0;
    const int str = RF_WARPS * 32;
    float* last = s_last + threadIdx.x;
    float* tbs = s_tb + threadIdx.x;
    float* tbest = s_tbest + threadIdx.x;
    int qi = pair_qi(B, T, i), ri = pair_ri(B, T, i);
    int lq = B.qlen[qi], lr = B.rlen[ri];
    int ml = lq < lr ? lq : lr;
    int swap = B.symmetric && (lq < lr);
    PairGeom G;
    G.q4 = B.q4 + B.q4off[qi]; G.r4 = B.r4 + B.r4off[ri];
    if (MODE == RM_INIT) {
        int sq = T.seedq[i], sr = T.seedr[i];
        G.alc = nullptr;
        G.q0 = sq; G.r0 = sr;
        if (lq <= sq || lr <= sr) G.n = 0;
        else G.n = (lq - sq) < (lr - sr) ? (lq - sq) : (lr - sr);
    } else {
        G.alc = (const float2*)(T.alc + 6 * T.off_aln[i]);
        G.q0 = G.r0 = 0;
        G.n = T.naln[i];
    }
    if (!valid) G.n = 0;
    const int n = G.n;
    const bool prod = (MODE == RM_PROD1 || MODE == RM_PROD2 || MODE == RM_PLOG);
    const bool phase2 = (MODE == RM_FIN2 || MODE == RM_PROD2 || MODE == RM_PLOG);
    const int vk = refine_variants(MODE, B);
    const float d0 = prod ? B.t_d0fin[ml] : B.t_d0[ml];
    const float d02 = __fmul_rn(d0, d0);
    const float d82 = B.t_d82[ml];
    const int chk = prod ? 0 : 1;
    // the log search carries the best score so far (phase 1's to begin with)
    // into every variant; the other modes start each variant afresh
    const float best_init = (MODE == RM_INIT || MODE == RM_DP) ? 0.f
                          : MODE == RM_PLOG ? T.grand[i] : -1.f;
    const int maxalnmax = B.qmax < B.rmax ? B.qmax : B.rmax;
    const float d0s = d0s_of(d0);
    const float d0sm = __fsub_rn(d0s, 1.0f);
    const float d02s = __fmul_rn(d0sm, d0sm);       // iteration 1's usual threshold
    const float d0sp = __fadd_rn(d0s, 1.0f);
    const float thr2 = __fmul_rn(d0sp, d0sp);       // threshold of iterations >= 2
    const bool gscore = prod && lq != lr;           // also scored by the longer length
    float g02 = 0.f;
    if (gscore) { float g0 = B.t_d0fin[lq > lr ? lq : lr]; g02 = __fmul_rn(g0, g0); }
    VariantList V;
    variants_init(V, vk, n, maxalnmax, phase2 ? T.sfndx[i] : 0, phase2 ? T.sfpos[i] : 0, T.plog_round);
    if (MODE == RM_PROD1 && (lane % RF_LPP) == 0 && V.total > 0 && wlong == 0) {
        // RMSD over the whole alignment (variant 0: fragment [0, n)) from
        // compensated FP32 sums, MpStageFin.cpp production phase 1
        int s0, nd0, ps0, fl0, kf0;
        variants_get(V, vk, n, 0, s0, nd0, ps0, fl0, kf0);
        CovAcc a;
        a.init();
        float sq[6], cq[6], bq[6];
#pragma unroll
        for (int f = 0; f < 6; f++) { sq[f] = 0.f; cq[f] = 0.f; bq[f] = 0.f; }
        int blk = 0;
        for (int kk = kf0; kk < kf0 + fl0; kk++) {
            float qx, qy, qz, rx, ry, rz;
            G.at(kk, qx, qy, qz, rx, ry, rz);
            a.add(qx, qy, qz, rx, ry, rz);
            bq[0] = __fmaf_rn(qx, qx, bq[0]); bq[1] = __fmaf_rn(qy, qy, bq[1]); bq[2] = __fmaf_rn(qz, qz, bq[2]);
            bq[3] = __fmaf_rn(rx, rx, bq[3]); bq[4] = __fmaf_rn(ry, ry, bq[4]); bq[5] = __fmaf_rn(rz, rz, bq[5]);
            if (++blk == BLK) {
                a.fold();
#pragma unroll
                for (int f = 0; f < 6; f++) nfold(sq[f], cq[f], bq[f]);
                blk = 0;
            }
        }
        float vv[16];
        a.final(vv);
        double dv[21];
#pragma unroll
        for (int f = 0; f < 15; f++) dv[f] = (double)vv[f];
#pragma unroll
        for (int f = 0; f < 6; f++) { nfold(sq[f], cq[f], bq[f]); dv[15 + f] = (double)__fadd_rn(sq[f], cq[f]); }
        T.rmsd32[i] = (float)rmsd_from_sums(dv, (double)fl0);
    }
    float lbest = 0.f, lgbest = 0.f;              // this lane's best variant so far
    int lsi = 0x7fffffff, lndx = 0, lpos = 0;
    int kind = PK_IDLE, si = 0, vndx = 0, vpos = 0, k0 = 0, k1 = 0, cit = 0, m3mode = 0, pchk = chk;
    float best = 0.f, thr = 0.f, pd02 = d02;
    float tfm[12];
#pragma unroll
    for (int f = 0; f < 12; f++) tfm[f] = 0.f;
    bool need = true;
    int nextk = 0;                                // the pair's next variant to hand out
    unsigned long long vis = 0;                   // position visits of this lane's passes
    for (;;) {
        const unsigned nm = __ballot_sync(FULL, need) & smask;
        if (nm) {
            if (LONG) {                           // the pair's counter, shared by its warps
                int base = 0;
                if (lane == 0) base = atomicAdd(T.rl_next + slot, __popc(nm));
                nextk = __shfl_sync(FULL, base, 0);
            }
            int kv = nextk + __popc(nm & ((1u << lane) - 1u));
            nextk += __popc(nm);
            if (need) {
                need = false;
                kind = PK_IDLE;
                if (kv < V.total) {
                    int fl, kf;
                    variants_get(V, vk, n, kv, si, vndx, vpos, fl, kf);
                    if (MODE == RM_DP && T.vskip && si < 32 * F3_NSEC &&
                        ((T.vskip[(long long)i * F3_NSEC + (si >> 5)] >> (si & 31)) & 1u)) {
                        need = true;       // a variant the detailed search's slots rule out
                    } else {
                        kind = PK_FRAG; k0 = kf; k1 = kf + fl;
                        best = best_init; cit = 0;
                    }
                }
            }
        }
        if (__ballot_sync(FULL, kind != PK_IDLE) == 0) {
            // lanes that passed over a skipped variant take the next one
            if (MODE == RM_DP && T.vskip && __any_sync(FULL, need && nextk < V.total)) continue;
            break;
        }
        float v[16], m3;
        const float sc = lane_pass(G, kind, k0, k1, tfm, pd02, pchk, d82, thr, m3mode, v, m3, lane % RF_LPP);
        vis += kind == PK_IDLE ? 0u : (kind == PK_FRAG ? (unsigned)(k1 - k0) : (unsigned)n);
        bool havev = false, done = false;
        if (kind == PK_FRAG) {
            if (v[15] < 1.0f) done = true;
            else {
#pragma unroll
                for (int f = 0; f < 16; f++) last[f * str] = v[f];
                solve_sums(v, swap, tfm);
                kind = PK_SCORE; thr = d02s; m3mode = 2; cit = 0; pd02 = d02; pchk = chk;
            }
        } else if (kind == PK_SCORE) {
            if (best < sc) {
                best = sc;
#pragma unroll
                for (int f = 0; f < 12; f++) tbs[f * str] = tfm[f];
            }
            havev = true;
            if (cit == 0) {
                // iteration 1's threshold from iteration 0's three smallest distances
                float dst32;
                if (LARGEDST_CMP < m3 || m3 < d02s || n <= 3) dst32 = d02s;
                else {
                    float t = __fadd_rn(d0sm, __fmul_rn(ceilf(__fmul_rn(__fsub_rn(__fsqrt_rn(m3), d0sm), 2.0f)), 0.5f));
                    dst32 = __fmul_rn(t, t);
                }
                if (dst32 != d02s) { kind = PK_EXT; thr = dst32; m3mode = 0; havev = false; }
            }
            cit++;
        } else if (kind == PK_EXT) {
            havev = true;
        } else if (kind == PK_GSCORE) {
            done = true;
        }
        if (havev) {
            if (cit >= NMAXCONVIT + 2 || converged16(v, last, str) || v[15] < 1.0f) done = true;
            else {
#pragma unroll
                for (int f = 0; f < 16; f++) last[f * str] = v[f];
                solve_sums(v, swap, tfm);
                kind = PK_SCORE; thr = thr2; m3mode = 0;
            }
        }
        if (done) {
            if (kind != PK_GSCORE && gscore && best >= 0.f && (MODE != RM_PLOG || best > best_init)) {
                // one more pass: the variant's best transform scored with the
                // d0 of the longer structure
#pragma unroll
                for (int f = 0; f < 12; f++) tfm[f] = tbs[f * str];
                kind = PK_GSCORE; pd02 = g02; pchk = 0; m3mode = 0;
            } else {
                const float gbest = kind == PK_GSCORE ? sc : best;
                if (best > 0.f && (lbest < best || (lbest == best && si < lsi))) {
                    lbest = best; lgbest = gbest; lsi = si; lndx = vndx; lpos = vpos;
#pragma unroll
                    for (int f = 0; f < 12; f++) tbest[f * str] = tbs[f * str];
                }
                need = true;
                kind = PK_IDLE;
            }
        }
    }
    if (T.work) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) vis += __shfl_xor_sync(FULL, vis, o);
        if (lane == 0) work_add(T, WK_REFINE, vis);
    }
    // arg-max over the pair's lanes: larger score, then lower variant index
    float wb = lbest;
    int wsi = lsi;
#pragma unroll
    for (int o = RF_LPP / 2; o > 0; o >>= 1) {
        float ob = __shfl_xor_sync(FULL, wb, o);
        int os = __shfl_xor_sync(FULL, wsi, o);
        if (ob > wb || (ob == wb && os < wsi)) { wb = ob; wsi = os; }
    }
    const bool havewin = wb > 0.f;
    const unsigned wmask = __ballot_sync(FULL, havewin && lsi == wsi) & smask;
    const int wl = wmask ? __ffs(wmask) - 1 : sub * RF_LPP;
    const int wndx = __shfl_sync(FULL, lndx, wl);
    const int wpos = __shfl_sync(FULL, lpos, wl);
    if (!valid) return;
    if (LONG) {
        if (lane == wl) {
            float* c = T.rl_cand + ((long long)slot * (T.rlw_ctas * RF_WARPS_LONG) + wlong) * RLW_CAND;
            c[0] = havewin ? wb : 0.f;
            c[1] = __int_as_float(wsi);
            c[2] = lgbest;
            c[3] = __int_as_float(wndx);
            c[4] = __int_as_float(wpos);
#pragma unroll
            for (int f = 0; f < 12; f++) c[5 + f] = tbest[f * str];
        }
        return;
    }
    if (lane == wl)
        refine_commit<MODE>(B, T, i, lq, lr, havewin, wb, lgbest, wndx, wpos, tbest, str);
}

// Pairs with lo <= n < hi of the work list (lo, hi multiples of 16, hi 0: no
// upper bound): their range of list slots.
__device__ __forceinline__ void rlist_range(const Bat& T, int lo, int hi, int& first, int& last) {
    first = hi > 0 ? T.rhist[RL_NB - 1 - (hi >> RL_SHIFT)] : 0;
    last = T.rhist[RL_NB - 1 - (lo >> RL_SHIFT)];
}

// LONG: T.rlw_ctas CTAs per long pair; the grid (a multiple of that) walks
// the long pairs listed for this launch.
// Otherwise: the pairs of the work list with lo <= n < hi positions.
template <int MODE, int RF_LPP, bool LONG>
__global__ void __launch_bounds__((LONG ? RF_WARPS_LONG : RF_WARPS_SHORT) * 32) k_refine(Blk B, Bat T, int lo, int hi) {
    if (LONG) {
        const int c = T.rlw_ctas;
        const int wl = (int)(blockIdx.x % c) * RF_WARPS_LONG + (threadIdx.x >> 5);
        const int nlong = *T.rl_count;
        for (int slot = (int)(blockIdx.x / c); slot < nlong; slot += (int)(gridDim.x / c))
            refine_slot<MODE, RF_LPP, LONG>(B, T, slot, wl);
    } else {
        constexpr int RF_PPW = 32 / RF_LPP;        // pairs per warp
        int first, last;
        rlist_range(T, lo, hi, first, last);
        const int slot = first + blockIdx.x * (RF_PPW * RF_WARPS_SHORT) + (threadIdx.x >> 5) * RF_PPW +
                         (int)(threadIdx.x & 31) / RF_LPP;
        refine_slot<MODE, RF_LPP, LONG>(B, T, slot, 0, last);
    }
}

// the winner of each long pair among its warps' candidates
template <int MODE>
__global__ void k_refine_long_fin(Blk B, Bat T) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int slot = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (slot >= *T.rl_count) return;
    const int i = T.rl_long[slot];
    const float* c0 = T.rl_cand + (long long)slot * (T.rlw_ctas * RF_WARPS_LONG) * RLW_CAND;
    float wb = 0.f;
    int wsi = 0x7fffffff, wk = -1;
    const int nw = T.rlw_ctas * RF_WARPS_LONG;      // the warps that left candidates
    for (int k = lane; k < nw; k += 32) {
        float b = c0[k * RLW_CAND];
        int si = __float_as_int(c0[k * RLW_CAND + 1]);
        if (b > 0.f && (wb < b || (wb == b && si < wsi))) { wb = b; wsi = si; wk = k; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        float ob = __shfl_xor_sync(FULL, wb, o);
        int os = __shfl_xor_sync(FULL, wsi, o);
        int ok = __shfl_xor_sync(FULL, wk, o);
        if (ob > wb || (ob == wb && os < wsi)) { wb = ob; wsi = os; wk = ok; }
    }
    if (lane != 0) return;
    int qi = pair_qi(B, T, i), ri = pair_ri(B, T, i);
    const bool havewin = wb > 0.f;
    const float* c = c0 + (havewin ? wk : 0) * RLW_CAND;
    refine_commit<MODE>(B, T, i, B.qlen[qi], B.rlen[ri], havewin, wb, c[2], __float_as_int(c[3]),
                        __float_as_int(c[4]), c + 5, 1);
}

// ---------------------------------------------------------------------------
// Refinement with a warp to a pass.  A lane that sweeps a whole pass by itself
// (refine_slot) makes n dependent position visits, so a launch lasts as long
// as its slowest variant's: ~150 us for one pair of 150 positions, 16 ms where
// pairs of 400 to 1,500 positions share 16 lanes.  Here the 32 lanes of a warp
// take the 32 positions of a block: distances, scores and inclusion masks of
// a block at once (no order matters there), the masked coordinates and score
// terms go to shared memory, and then 16 lanes a block sum its 16 fields, a
// field each, in position order; the block sums are folded in block order by
// the field's lane.  Every sum is the sequence of operations of one lane's
// sweep (a masked position adds a zero), so results are the same bits.
//
// The rotation solve is FP64 and takes as long as several such passes, so a
// warp holds up to CM_MAX variants, lane m the state of variant m: it runs
// their passes one after another and then all their solves at once.
//
// A cluster of CTAs takes a pair (the grid's clusters walk the pairs of the
// launch's length class, longest first); the CTAs copy the pair's coordinates
// to shared memory once, draw variants from a counter each, and the CTAs'
// winners meet in the first one's shared memory.  What bounds it: the latency
// of the pass -> solve chain (about 800 + 2,800 cycles at 150 positions).
// Refinement launches of a call, before -> after: one pair of 150 residues
// 3.5 -> 1.0 ms, 16 x 500 29 -> 16 ms, all against all of 400 structures
// 114 -> 78 ms, 2 x 20,000 115 -> 62 ms (three streams).  Four CTAs a SM (128
// registers) against three: 2 x 8,000 41.8 -> 36.9 ms, 1 x 1,000 4.0 -> 3.5.
constexpr int CM_WARPS = 4;
constexpr int CM_MAX = 8;                    // variants a warp holds at most
constexpr int CM_CMAX = 8;                   // CTAs per cluster at most
constexpr int CM_CHUNK = 4;                  // blocks of positions per step of a pass
constexpr int CM_BST = 36;                   // floats between a block's components (16-byte rows, no bank conflicts)
constexpr int CM_BLKW = 8 * CM_BST;          // floats per block: q xyz, r xyz, score term, ones
constexpr int CM_ROW = 20;                   // floats of a variant's pass parameters
struct CoopWarp {                            // one warp's shared memory
    float buf[CM_CHUNK * CM_BLKW];
    float row[CM_MAX * CM_ROW];              // transform and parameters of each variant's pass
    float tot[CM_MAX * CM_ROW];              // its 15 sums, score, count, third-smallest distance
    float last[16 * CM_MAX], tb[12 * CM_MAX], tbest[12 * CM_MAX];   // as refine_slot's, a column per lane
};
struct alignas(16) CoopSmem {
    CoopWarp w[CM_WARPS];
    float win[CM_CMAX * 32];                 // the CTAs' winners (first CTA)
    float cand[CM_WARPS * 32];               // the warps' winners
    int next, slot;
};
inline size_t coop_smem_bytes(int nmax) {
    return sizeof(CoopSmem) + (size_t)((nmax + BLK - 1) / BLK * BLK) * (sizeof(float4) + sizeof(float2));
}

__device__ __forceinline__ void keep3(float d, float& m1, float& m2, float& m3) {
    const bool c1 = d < m1, c2 = d < m2, c3 = d < m3;
    m3 = c2 ? m2 : (c3 ? d : m3);
    m2 = c1 ? m1 : (c2 ? d : m2);
    m1 = c1 ? d : m1;
}

// One pass of variant m (its parameters in w.row) by the whole warp; its
// sums, score, count and third-smallest distance to w.tot.
__device__ __forceinline__ void coop_pass(CoopWarp& w, int m, int n, const float4* cA,
                                          const float2* cB, int lane) {
    const unsigned FULL = 0xffffffffu;
    const float* row = w.row + m * CM_ROW;
    float tfm[12];
#pragma unroll
    for (int f = 0; f < 12; f++) tfm[f] = row[f];
    const int kind = __float_as_int(row[12]), k0 = __float_as_int(row[13]), k1 = __float_as_int(row[14]);
    const float thr = row[15], d02 = row[16], d82 = row[17];
    const int flg = __float_as_int(row[18]);          // 1: only distances within d82 score, 2: smallest distances
    const bool frag = kind == PK_FRAG;
    const bool scr = kind == PK_SCORE || kind == PK_GSCORE;
    const bool cov = kind == PK_SCORE || kind == PK_EXT;
    const bool chk = flg & 1, trk = flg & 2;
    const int lim = frag ? k1 : n;
    const int nblk = (lim + BLK - 1) / BLK;
    // this lane's sum: field lane & 15 of block 2k + lane / 16
    const int f = lane & 15;
    const int ax = f < 9 ? f / 3 : (f < 12 ? f - 9 : (f < 15 ? f - 9 : 6));
    const int ay = f < 9 ? 3 + f % 3 : 7;
    const float* X = w.buf + (lane >> 4) * CM_BLKW + ax * CM_BST;
    const float* Y = w.buf + (lane >> 4) * CM_BLKW + ay * CM_BST;
    float s = 0.f, c = 0.f;
    float m1 = LARGEDST, m2 = LARGEDST, m3 = LARGEDST;
    int cnt = 0;
    for (int cb = frag ? k0 / BLK : 0; cb < nblk; cb += CM_CHUNK) {
#pragma unroll
        for (int e = 0; e < CM_CHUNK; e++) {
            const int p = (cb + e) * BLK + lane;
            const bool in = p < lim;
            float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
            float2 v = make_float2(0.f, 0.f);
            if (in) { u = cA[p]; v = cB[p]; }
            bool inc = in && k0 <= p;
            float tm = 0.f;
            if (!frag) {
                const float d = dist2_tf(tfm, u.x, u.y, u.z, u.w, v.x, v.y);
                inc = in && cov && d <= thr;
                const float x = tmterm(d02, d);
                tm = in && scr && (!chk || d <= d82) ? x : 0.f;
                if (trk && in) keep3(d, m1, m2, m3);
            }
            float* o = w.buf + e * CM_BLKW + lane;
            o[0] = inc ? u.x : 0.f;          o[CM_BST] = inc ? u.y : 0.f;
            o[2 * CM_BST] = inc ? u.z : 0.f; o[3 * CM_BST] = inc ? u.w : 0.f;
            o[4 * CM_BST] = inc ? v.x : 0.f; o[5 * CM_BST] = inc ? v.y : 0.f;
            o[6 * CM_BST] = tm;
            cnt += __popc(__ballot_sync(FULL, inc));
        }
        __syncwarp();
        float b[CM_CHUNK / 2];
#pragma unroll
        for (int e = 0; e < CM_CHUNK / 2; e++) b[e] = 0.f;
#pragma unroll
        for (int p = 0; p < BLK; p += 4)
#pragma unroll
            for (int e = 0; e < CM_CHUNK / 2; e++) {
                const float4 x = *(const float4*)(X + 2 * e * CM_BLKW + p), y = *(const float4*)(Y + 2 * e * CM_BLKW + p);
                b[e] = __fmaf_rn(x.x, y.x, b[e]); b[e] = __fmaf_rn(x.y, y.y, b[e]);
                b[e] = __fmaf_rn(x.z, y.z, b[e]); b[e] = __fmaf_rn(x.w, y.w, b[e]);
            }
        __syncwarp();
        // folding the zeros of a block past the end changes nothing
#pragma unroll
        for (int e = 0; e < CM_CHUNK / 2; e++) {
            const float odd = __shfl_down_sync(FULL, b[e], 16);
            tfold(s, c, b[e]);
            tfold(s, c, odd);
        }
    }
    float* tot = w.tot + m * CM_ROW;
    if (lane < 16) tot[lane] = __fadd_rn(s, c);
    if (trk) {
        // the three smallest of the pass: the lanes' three smallest merged
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float x1 = __shfl_xor_sync(FULL, m1, o), x2 = __shfl_xor_sync(FULL, m2, o),
                        x3 = __shfl_xor_sync(FULL, m3, o);
            keep3(x1, m1, m2, m3); keep3(x2, m1, m2, m3); keep3(x3, m1, m2, m3);
        }
    }
    if (lane == 0) { tot[16] = (float)cnt; tot[17] = m3; }
}

// The whole alignment's FP32 RMSD (production phase 1, MpStageFin.cpp): the
// 15 covariance sums, then the 6 sums of squares, by a warp; at(p, q): position
// p's six coordinates; buf: a block's components, the eighth all ones.
template <class At>
__device__ __forceinline__ float rmsd_warp(float* buf, int n, At at, int lane) {
    double dv[21];
    for (int part = 0; part < 2; part++) {
        float s = 0.f, c = 0.f;
        const int f = lane & 15;
        const int ax = part ? (f < 6 ? f : 6) : (f < 9 ? f / 3 : (f < 15 ? f - 9 : 6));
        const int ay = part ? ax : (f < 9 ? 3 + f % 3 : 7);
        for (int b0 = 0; b0 * BLK < n; b0++) {
            const int p = b0 * BLK + lane;
            float q[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (p < n) at(p, q);
#pragma unroll
            for (int k = 0; k < 6; k++) buf[k * CM_BST + lane] = q[k];
            buf[6 * CM_BST + lane] = 0.f;
            __syncwarp();
            float b = 0.f;
#pragma unroll 8
            for (int k = 0; k < BLK; k++) b = __fmaf_rn(buf[ax * CM_BST + k], buf[ay * CM_BST + k], b);
            __syncwarp();
            tfold(s, c, b);
        }
        const float t = __fadd_rn(s, c);
        if (part == 0) {
#pragma unroll
            for (int k = 0; k < 15; k++) dv[k] = (double)__shfl_sync(0xffffffffu, t, k);
        } else {
#pragma unroll
            for (int k = 0; k < 6; k++) dv[15 + k] = (double)__shfl_sync(0xffffffffu, t, k);
        }
    }
    return (float)rmsd_from_sums(dv, (double)n);
}

template <int MODE>
__global__ void __launch_bounds__(CM_WARPS * 32, 4) k_refine_coop(Blk B, Bat T, int lo, int hi, int cls) {
    extern __shared__ __align__(16) unsigned char cm_smem[];
    CoopSmem& S = *(CoopSmem*)cm_smem;
    float4* cA = (float4*)(cm_smem + sizeof(CoopSmem));
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    cg::cluster_group cl = cg::this_cluster();
    const int C = (int)cl.num_blocks(), crank = (int)cl.block_rank();
    CoopWarp& w = S.w[warp];
    int first, last;
    rlist_range(T, lo, hi, first, last);
    for (int e = 0; e < CM_CHUNK; e++) w.buf[e * CM_BLKW + 7 * CM_BST + lane] = 1.f;
    // the first pair by position, the next ones as clusters come free
    int* ctr = T.rhist + RL_NB + 1 + cls;
    const int ncl = (int)gridDim.x / C;
    // every CTA of the cluster has started before its shared memory is written
    // from another one (S.win); the later pairs have the barriers at a pair's end
    if (C > 1) cl.sync();
    for (int slot = first + (int)blockIdx.x / C; slot < last;) {
        const int i = T.rlist[slot];
        const int qi = pair_qi(B, T, i), ri = pair_ri(B, T, i);
        const int lq = B.qlen[qi], lr = B.rlen[ri];
        const int ml = lq < lr ? lq : lr;
        const int swap = B.symmetric && (lq < lr);
        const float4* q4 = B.q4 + B.q4off[qi];
        const float4* r4 = B.r4 + B.r4off[ri];
        int n, sq = 0, sr = 0;
        if (MODE == RM_INIT) {
            sq = T.seedq[i]; sr = T.seedr[i];
            n = (lq - sq) < (lr - sr) ? (lq - sq) : (lr - sr);
        } else {
            n = T.naln[i];
        }
        float2* cB = (float2*)(cA + (n + BLK - 1) / BLK * BLK);
        if (MODE == RM_INIT) {
            for (int p = threadIdx.x; p < n; p += blockDim.x) {
                const float4 u = __ldg(q4 + sq + p), v = __ldg(r4 + sr + p);
                cA[p] = make_float4(u.x, u.y, u.z, v.x);
                cB[p] = make_float2(v.y, v.z);
            }
        } else {
            const unsigned* aln = T.aln + T.off_aln[i];
            for (int p = threadIdx.x; p < n; p += blockDim.x) {
                const unsigned wv = aln[n - 1 - p];           // the traceback's order is backwards
                const float4 u = __ldg(q4 + (wv >> 16)), v = __ldg(r4 + (wv & 0xffffu));
                cA[p] = make_float4(u.x, u.y, u.z, v.x);
                cB[p] = make_float2(v.y, v.z);
            }
        }
        if (threadIdx.x == 0) S.next = 0;
        __syncthreads();
        float* lastv = w.last + lane;
        float* tbs = w.tb + lane;
        float* tbest = w.tbest + lane;
        const bool prod = (MODE == RM_PROD1 || MODE == RM_PROD2 || MODE == RM_PLOG);
        const bool phase2 = (MODE == RM_FIN2 || MODE == RM_PROD2 || MODE == RM_PLOG);
        const int vk = refine_variants(MODE, B);
        const float d0 = prod ? B.t_d0fin[ml] : B.t_d0[ml];
        const float d02 = __fmul_rn(d0, d0);
        const float d82 = B.t_d82[ml];
        const int chk = prod ? 0 : 1;
        const float best_init = (MODE == RM_INIT || MODE == RM_DP) ? 0.f
                              : MODE == RM_PLOG ? T.grand[i] : -1.f;
        const int maxalnmax = B.qmax < B.rmax ? B.qmax : B.rmax;
        const float d0s = d0s_of(d0);
        const float d0sm = __fsub_rn(d0s, 1.0f);
        const float d02s = __fmul_rn(d0sm, d0sm);             // iteration 1's usual threshold
        const float d0sp = __fadd_rn(d0s, 1.0f);
        const float thr2 = __fmul_rn(d0sp, d0sp);             // threshold of iterations >= 2
        const bool gscore = prod && lq != lr;                 // also scored by the longer length
        float g02 = 0.f;
        if (gscore) { const float g0 = B.t_d0fin[lq > lr ? lq : lr]; g02 = __fmul_rn(g0, g0); }
        VariantList V;
        variants_init(V, vk, n, maxalnmax, phase2 ? T.sfndx[i] : 0, phase2 ? T.sfpos[i] : 0, T.plog_round);
        if (MODE == RM_PROD1 && warp == CM_WARPS - 1 && crank == 0 && V.total > 0) {
            const float r = rmsd_warp(w.buf, n, [&](int p, float* q) {
                const float4 u = cA[p];
                const float2 v = cB[p];
                q[0] = u.x; q[1] = u.y; q[2] = u.z; q[3] = u.w; q[4] = v.x; q[5] = v.y;
            }, lane);
            if (lane == 0) T.rmsd32[i] = r;
        }
        // variants a warp holds: an even share of the pair's
        int M = (V.total + CM_WARPS * C - 1) / (CM_WARPS * C);
        M = M < 1 ? 1 : (M < CM_MAX ? M : CM_MAX);
        float lbest = 0.f, lgbest = 0.f;                      // this lane's best variant so far
        int lsi = 0x7fffffff, lndx = 0, lpos = 0;
        int kind = PK_IDLE, si = 0, vndx = 0, vpos = 0, k0 = 0, k1 = 0, cit = 0, m3on = 0, pchk = chk;
        float best = 0.f, thr = 0.f, pd02 = d02;
        bool need = lane < M;
        unsigned long long vis = 0;
        for (;;) {
            const unsigned nm = __ballot_sync(FULL, need);
            if (nm) {
                int base = 0;
                if (lane == 0) base = atomicAdd(&S.next, __popc(nm));
                base = __shfl_sync(FULL, base, 0);
                if (need) {
                    need = false;
                    kind = PK_IDLE;
                    const int kv = (base + __popc(nm & ((1u << lane) - 1u))) * C + crank;
                    if (kv < V.total) {
                        int fl, kf;
                        variants_get(V, vk, n, kv, si, vndx, vpos, fl, kf);
                        if (MODE == RM_DP && T.vskip && si < 32 * F3_NSEC &&
                            ((T.vskip[(long long)i * F3_NSEC + (si >> 5)] >> (si & 31)) & 1u)) {
                            need = true;       // a variant the detailed search's slots rule out
                        } else {
                            kind = PK_FRAG; k0 = kf; k1 = kf + fl;
                            best = best_init; cit = 0;
                        }
                    }
                }
            }
            const unsigned act = __ballot_sync(FULL, kind != PK_IDLE);
            if (act == 0) {
                if (__any_sync(FULL, need)) continue;         // variants passed over
                break;
            }
            // a pass of every variant, one after another
            if (kind != PK_IDLE) {
                float* row = w.row + lane * CM_ROW;
                row[12] = __int_as_float(kind);
                row[13] = __int_as_float(kind == PK_FRAG ? k0 : 0);
                row[14] = __int_as_float(k1);
                row[15] = thr; row[16] = pd02; row[17] = d82;
                row[18] = __int_as_float((pchk ? 1 : 0) | (kind == PK_SCORE && m3on ? 2 : 0));
            }
            __syncwarp();
            for (unsigned a = act; a; a &= a - 1) coop_pass(w, __ffs(a) - 1, n, cA, cB, lane);
            __syncwarp();
            vis += kind == PK_IDLE ? 0u : (kind == PK_FRAG ? (unsigned)(k1 - k0) : (unsigned)n);
            // the variants' next steps, a lane each
            if (kind != PK_IDLE) {
                const float* tot = w.tot + lane * CM_ROW;
                float* row = w.row + lane * CM_ROW;
                float v[16];
#pragma unroll
                for (int f = 0; f < 15; f++) v[f] = tot[f];
                v[15] = tot[16];
                const float sc = tot[15], m3 = tot[17];
                bool havev = false, done = false, solve = false;
                if (kind == PK_FRAG) {
                    if (v[15] < 1.0f) done = true;
                    else solve = true;
                } else if (kind == PK_SCORE) {
                    if (best < sc) {
                        best = sc;
#pragma unroll
                        for (int f = 0; f < 12; f++) tbs[f * CM_MAX] = row[f];
                    }
                    havev = true;
                    if (cit == 0) {
                        // iteration 1's threshold from iteration 0's three smallest distances
                        float dst32;
                        if (LARGEDST_CMP < m3 || m3 < d02s || n <= 3) dst32 = d02s;
                        else {
                            const float t = __fadd_rn(d0sm, __fmul_rn(ceilf(__fmul_rn(__fsub_rn(__fsqrt_rn(m3), d0sm), 2.0f)), 0.5f));
                            dst32 = __fmul_rn(t, t);
                        }
                        if (dst32 != d02s) { kind = PK_EXT; thr = dst32; m3on = 0; havev = false; }
                    }
                    cit++;
                } else if (kind == PK_EXT) {
                    havev = true;
                } else if (kind == PK_GSCORE) {
                    done = true;
                }
                if (havev) {
                    if (cit >= NMAXCONVIT + 2 || converged16(v, lastv, CM_MAX) || v[15] < 1.0f) done = true;
                    else solve = true;
                }
                if (solve) {
#pragma unroll
                    for (int f = 0; f < 16; f++) lastv[f * CM_MAX] = v[f];
                    float t2[12];
                    solve_sums(v, swap, t2);
#pragma unroll
                    for (int f = 0; f < 12; f++) row[f] = t2[f];
                    if (kind == PK_FRAG) { thr = d02s; m3on = 1; cit = 0; pd02 = d02; pchk = chk; }
                    else { thr = thr2; m3on = 0; }
                    kind = PK_SCORE;
                }
                if (done) {
                    if (kind != PK_GSCORE && gscore && best >= 0.f && (MODE != RM_PLOG || best > best_init)) {
                        // one more pass: the variant's best transform scored with the
                        // d0 of the longer structure
#pragma unroll
                        for (int f = 0; f < 12; f++) row[f] = tbs[f * CM_MAX];
                        kind = PK_GSCORE; pd02 = g02; pchk = 0; m3on = 0;
                    } else {
                        const float gbest = kind == PK_GSCORE ? sc : best;
                        if (best > 0.f && (lbest < best || (lbest == best && si < lsi))) {
                            lbest = best; lgbest = gbest; lsi = si; lndx = vndx; lpos = vpos;
#pragma unroll
                            for (int f = 0; f < 12; f++) tbest[f * CM_MAX] = tbs[f * CM_MAX];
                        }
                        need = true;
                        kind = PK_IDLE;
                    }
                }
            }
        }
        if (T.work) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) vis += __shfl_xor_sync(FULL, vis, o);
            if (lane == 0) work_add(T, WK_REFINE, vis);
        }
        // the warp's winner, then the CTA's: larger score, then lower variant index
        float wb = lbest;
        int wsi = lsi, wl = lane;
#pragma unroll
        for (int o = CM_MAX / 2; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(FULL, wb, o);
            const int os = __shfl_xor_sync(FULL, wsi, o), ol = __shfl_xor_sync(FULL, wl, o);
            if (ob > wb || (ob == wb && os < wsi)) { wb = ob; wsi = os; wl = ol; }
        }
        wl = __shfl_sync(FULL, wl, 0);
        if (lane == wl) {
            float* x = S.cand + warp * 32;
            x[0] = lbest;
            x[1] = __int_as_float(lsi);
            x[2] = lgbest;
            x[3] = __int_as_float(lndx);
            x[4] = __int_as_float(lpos);
#pragma unroll
            for (int f = 0; f < 12; f++) x[5 + f] = tbest[f * CM_MAX];
        }
        __syncthreads();
        if (warp == 0) {
            int k = 0;
#pragma unroll
            for (int j = 1; j < CM_WARPS; j++) {
                const float ob = S.cand[j * 32], cb = S.cand[k * 32];
                if (ob > cb || (ob == cb && __float_as_int(S.cand[j * 32 + 1]) < __float_as_int(S.cand[k * 32 + 1]))) k = j;
            }
            const float* x = S.cand + k * 32;
            if (C > 1) {
                // to the first CTA
                float* dst = cl.map_shared_rank(S.win, 0) + crank * 32;
                if (lane < 17) dst[lane] = x[lane];
            } else if (lane == 0) {
                refine_commit<MODE>(B, T, i, lq, lr, x[0] > 0.f, x[0], x[2], __float_as_int(x[3]),
                                    __float_as_int(x[4]), x + 5, 1);
            }
        }
        if (C > 1) {
            cl.sync();
            if (crank == 0 && threadIdx.x == 0) {
                int k = 0;
                for (int j = 1; j < C; j++) {
                    const float ob = S.win[j * 32], cb = S.win[k * 32];
                    if (ob > cb || (ob == cb && __float_as_int(S.win[j * 32 + 1]) < __float_as_int(S.win[k * 32 + 1]))) k = j;
                }
                const float* x = S.win + k * 32;
                refine_commit<MODE>(B, T, i, lq, lr, x[0] > 0.f, x[0], x[2], __float_as_int(x[3]),
                                    __float_as_int(x[4]), x + 5, 1);
            }
        }
        if (crank == 0 && threadIdx.x == 0) S.slot = first + ncl + atomicAdd(ctr, 1);
        // the next pair is known; this one's shared data is done with
        if (C > 1) cl.sync();
        else __syncthreads();
        slot = *cl.map_shared_rank(&S.slot, 0);
    }
    if (C > 1) cl.sync();              // the first CTA's shared memory is read until here
}

// ---------------------------------------------------------------------------
// Long pairs, few of them: a CTA to a pass.  The variants of a pair of 5,000
// positions (750) are drawn one at a time by the CTAs of the launch; a pass
// gives each warp every CL_WARPS-th group of CM_CHUNK blocks, as coop_pass sums
// them, the block sums meet in shared memory and 16 lanes fold them in block
// order.  Every thread holds the variant's state.  (A warp to a variant, a block
// per lane, took 28,000 cycles a pass at 5,000 positions; refinement of one such
// pair 47.0 -> 14.6 ms.)
constexpr int CL_WARPS = 4;
constexpr int CL_SEG = 256;                  // blocks between two folds
struct LongSmem {
    float buf[CL_WARPS][CM_CHUNK * CM_BLKW];
    float sums[CL_SEG * 16];                 // block sums of a segment
    float tot[16];
    float m3[CL_WARPS][3];
    int cnt[CL_WARPS];
    float tb[12], tbest[12];
    int kv;
};

// one pass: the sums, the score, the count and the third-smallest distance, on
// every thread (v[0..14], v[15] count; returns the score)
__device__ float long_pass(LongSmem& S, const PairGeom& G, int kind, int k0, int k1, const float* tfm,
                           float d02, int chk, float d82, float thr, int trk, float* v, float& m3out) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const bool frag = kind == PK_FRAG;
    const bool scr = kind == PK_SCORE || kind == PK_GSCORE;
    const bool cov = kind == PK_SCORE || kind == PK_EXT;
    const int lim = frag ? k1 : G.n;
    const int nblk = (lim + BLK - 1) / BLK;
    const int f = lane & 15;
    const int ax = f < 9 ? f / 3 : (f < 12 ? f - 9 : (f < 15 ? f - 9 : 6));
    const int ay = f < 9 ? 3 + f % 3 : 7;
    float* buf = S.buf[wp];
    const float* X = buf + (lane >> 4) * CM_BLKW + ax * CM_BST;
    const float* Y = buf + (lane >> 4) * CM_BLKW + ay * CM_BST;
    float s = 0.f, c = 0.f;
    float m1 = LARGEDST, m2 = LARGEDST, m3 = LARGEDST;
    int cnt = 0;
    for (int sb = frag ? k0 / BLK : 0; sb < nblk; sb += CL_SEG) {
        const int se = sb + CL_SEG < nblk ? sb + CL_SEG : nblk;
        __syncthreads();                     // the last segment's sums are folded
        for (int cb = sb + wp * CM_CHUNK; cb < se; cb += CL_WARPS * CM_CHUNK) {
            float q[CM_CHUNK][6];
#pragma unroll
            for (int e = 0; e < CM_CHUNK; e++) {
                const int p = (cb + e) * BLK + lane;
#pragma unroll
                for (int k = 0; k < 6; k++) q[e][k] = 0.f;
                if (p < lim) G.at(p, q[e][0], q[e][1], q[e][2], q[e][3], q[e][4], q[e][5]);
            }
#pragma unroll
            for (int e = 0; e < CM_CHUNK; e++) {
                const int p = (cb + e) * BLK + lane;
                const bool in = p < lim;
                bool inc = in && k0 <= p;
                float tm = 0.f;
                if (!frag) {
                    const float d = dist2_tf(tfm, q[e][0], q[e][1], q[e][2], q[e][3], q[e][4], q[e][5]);
                    inc = in && cov && d <= thr;
                    const float x = tmterm(d02, d);
                    tm = in && scr && (!chk || d <= d82) ? x : 0.f;
                    if (trk && in) keep3(d, m1, m2, m3);
                }
                float* o = buf + e * CM_BLKW + lane;
#pragma unroll
                for (int k = 0; k < 6; k++) o[k * CM_BST] = inc ? q[e][k] : 0.f;
                o[6 * CM_BST] = tm;
                cnt += __popc(__ballot_sync(FULL, inc));
            }
            __syncwarp();
            float b[CM_CHUNK / 2];
#pragma unroll
            for (int e = 0; e < CM_CHUNK / 2; e++) b[e] = 0.f;
#pragma unroll
            for (int p = 0; p < BLK; p += 4)
#pragma unroll
                for (int e = 0; e < CM_CHUNK / 2; e++) {
                    const float4 x = *(const float4*)(X + 2 * e * CM_BLKW + p), y = *(const float4*)(Y + 2 * e * CM_BLKW + p);
                    b[e] = __fmaf_rn(x.x, y.x, b[e]); b[e] = __fmaf_rn(x.y, y.y, b[e]);
                    b[e] = __fmaf_rn(x.z, y.z, b[e]); b[e] = __fmaf_rn(x.w, y.w, b[e]);
                }
            __syncwarp();
#pragma unroll
            for (int e = 0; e < CM_CHUNK / 2; e++) {
                const int blk = cb + 2 * e + (lane >> 4);
                if (blk < se) S.sums[(blk - sb) * 16 + f] = b[e];
            }
        }
        __syncthreads();
        if (threadIdx.x < 16)
            for (int k = 0; k < se - sb; k++) tfold(s, c, S.sums[k * 16 + threadIdx.x]);
    }
    if (threadIdx.x < 16) S.tot[threadIdx.x] = __fadd_rn(s, c);
    if (trk) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float x1 = __shfl_xor_sync(FULL, m1, o), x2 = __shfl_xor_sync(FULL, m2, o),
                        x3 = __shfl_xor_sync(FULL, m3, o);
            keep3(x1, m1, m2, m3); keep3(x2, m1, m2, m3); keep3(x3, m1, m2, m3);
        }
        if (lane == 0) { S.m3[wp][0] = m1; S.m3[wp][1] = m2; S.m3[wp][2] = m3; }
    }
    if (lane == 0) S.cnt[wp] = cnt;
    __syncthreads();
    m1 = m2 = m3 = LARGEDST;
    cnt = 0;
#pragma unroll
    for (int k = 0; k < CL_WARPS; k++) {
        cnt += S.cnt[k];
        if (trk) { keep3(S.m3[k][0], m1, m2, m3); keep3(S.m3[k][1], m1, m2, m3); keep3(S.m3[k][2], m1, m2, m3); }
    }
    m3out = m3;
#pragma unroll
    for (int k = 0; k < 15; k++) v[k] = S.tot[k];
    v[15] = (float)cnt;
    const float sc = S.tot[15];
    __syncthreads();                         // tot, cnt and m3 are read
    return sc;
}

// The whole alignment's FP32 RMSD (production phase 1): warp 0 from the pair's
// positions.
__device__ float long_rmsd(LongSmem& S, const PairGeom& G) {
    float r = 0.f;
    if (threadIdx.x < 32)
        r = rmsd_warp(S.buf[0], G.n, [&](int p, float* q) { G.at(p, q[0], q[1], q[2], q[3], q[4], q[5]); },
                      (int)threadIdx.x);
    return r;
}

// The CTAs of a long pair (4 * T.rlw_ctas, a candidate each) draw its variants
// from a counter; k_refine_long_fin picks the winner among the candidates.
template <int MODE>
__global__ void __launch_bounds__(CL_WARPS * 32, 4) k_refine_long(Blk B, Bat T) {
    extern __shared__ __align__(16) unsigned char cl_smem[];
    LongSmem& S = *(LongSmem*)cl_smem;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int nc = T.rlw_ctas * RF_WARPS_LONG, nlong = *T.rl_count;
    for (int e = 0; e < CM_CHUNK; e++) S.buf[wp][e * CM_BLKW + 7 * CM_BST + lane] = 1.f;
    for (int slot = (int)blockIdx.x / nc; slot < nlong; slot += (int)gridDim.x / nc) {
        const int cand = (int)blockIdx.x % nc;
        const int i = T.rl_long[slot];
        const int qi = pair_qi(B, T, i), ri = pair_ri(B, T, i);
        const int lq = B.qlen[qi], lr = B.rlen[ri];
        const int ml = lq < lr ? lq : lr;
        const int swap = B.symmetric && (lq < lr);
        PairGeom G;
        G.q4 = B.q4 + B.q4off[qi]; G.r4 = B.r4 + B.r4off[ri];
        G.alc = nullptr;
        G.q0 = G.r0 = 0;
        if (MODE == RM_INIT) {
            G.q0 = T.seedq[i]; G.r0 = T.seedr[i];
            G.n = (lq - G.q0) < (lr - G.r0) ? (lq - G.q0) : (lr - G.r0);
        } else {
            G.alc = (const float2*)(T.alc + 6 * T.off_aln[i]);
            G.n = T.naln[i];
        }
        const int n = G.n;
        const bool prod = (MODE == RM_PROD1 || MODE == RM_PROD2 || MODE == RM_PLOG);
        const bool phase2 = (MODE == RM_FIN2 || MODE == RM_PROD2 || MODE == RM_PLOG);
        const int vk = refine_variants(MODE, B);
        const float d0 = prod ? B.t_d0fin[ml] : B.t_d0[ml];
        const float d02 = __fmul_rn(d0, d0);
        const float d82 = B.t_d82[ml];
        const int chk = prod ? 0 : 1;
        const float best_init = (MODE == RM_INIT || MODE == RM_DP) ? 0.f
                              : MODE == RM_PLOG ? T.grand[i] : -1.f;
        const int maxalnmax = B.qmax < B.rmax ? B.qmax : B.rmax;
        const float d0s = d0s_of(d0);
        const float d0sm = __fsub_rn(d0s, 1.0f);
        const float d02s = __fmul_rn(d0sm, d0sm);             // iteration 1's usual threshold
        const float d0sp = __fadd_rn(d0s, 1.0f);
        const float thr2 = __fmul_rn(d0sp, d0sp);             // threshold of iterations >= 2
        const bool gscore = prod && lq != lr;                 // also scored by the longer length
        float g02 = 0.f;
        if (gscore) { const float g0 = B.t_d0fin[lq > lr ? lq : lr]; g02 = __fmul_rn(g0, g0); }
        VariantList V;
        variants_init(V, vk, n, maxalnmax, phase2 ? T.sfndx[i] : 0, phase2 ? T.sfpos[i] : 0, T.plog_round);
        if (MODE == RM_PROD1 && cand == 0 && V.total > 0) {
            const float r = long_rmsd(S, G);
            if (threadIdx.x == 0) T.rmsd32[i] = r;
        }
        float lbest = 0.f, lgbest = 0.f;                      // this CTA's best variant so far
        int lsi = 0x7fffffff, lndx = 0, lpos = 0;
        unsigned long long vis = 0;
        for (;;) {
            __syncthreads();
            if (threadIdx.x == 0) S.kv = atomicAdd(T.rl_next + slot, 1);
            __syncthreads();
            const int kv = S.kv;
            if (kv >= V.total) break;
            int si, vndx, vpos, fl, kf;
            variants_get(V, vk, n, kv, si, vndx, vpos, fl, kf);
            if (MODE == RM_DP && T.vskip && si < 32 * F3_NSEC &&
                ((T.vskip[(long long)i * F3_NSEC + (si >> 5)] >> (si & 31)) & 1u))
                continue;                      // a variant the detailed search's slots rule out
            float v[16], last[16], tfm[12], m3, best = best_init, thr = d02s;
            long_pass(S, G, PK_FRAG, kf, kf + fl, nullptr, d02, chk, d82, thr, 0, v, m3);
            vis += (unsigned)fl;
            if (v[15] < 1.0f) continue;
            bool more = true, ext = false;
            for (int cit = 0; more;) {
                if (!ext) {
#pragma unroll
                    for (int f = 0; f < 16; f++) last[f] = v[f];
                    solve_sums(v, swap, tfm);
                    const float sc = long_pass(S, G, PK_SCORE, 0, 0, tfm, d02, chk, d82, thr, cit == 0, v, m3);
                    vis += (unsigned)n;
                    if (best < sc) {
                        best = sc;
                        if (threadIdx.x == 0) {
#pragma unroll
                            for (int f = 0; f < 12; f++) S.tb[f] = tfm[f];
                        }
                    }
                    if (cit++ == 0) {
                        // iteration 1's threshold from iteration 0's three smallest distances
                        float dst32;
                        if (LARGEDST_CMP < m3 || m3 < d02s || n <= 3) dst32 = d02s;
                        else {
                            const float t = __fadd_rn(d0sm, __fmul_rn(ceilf(__fmul_rn(__fsub_rn(__fsqrt_rn(m3), d0sm), 2.0f)), 0.5f));
                            dst32 = __fmul_rn(t, t);
                        }
                        if (dst32 != d02s) { ext = true; thr = dst32; continue; }
                    }
                } else {
                    long_pass(S, G, PK_EXT, 0, 0, tfm, d02, chk, d82, thr, 0, v, m3);
                    vis += (unsigned)n;
                    ext = false;
                }
                more = !(cit >= NMAXCONVIT + 2 || converged16(v, last, 1) || v[15] < 1.0f);
                thr = thr2;
            }
            float gbest = best;
            __syncthreads();                                  // tb
            if (gscore && best >= 0.f && (MODE != RM_PLOG || best > best_init)) {
                // one more pass: the variant's best transform scored with the
                // d0 of the longer structure
#pragma unroll
                for (int f = 0; f < 12; f++) tfm[f] = S.tb[f];
                gbest = long_pass(S, G, PK_GSCORE, 0, 0, tfm, g02, 0, d82, thr, 0, v, m3);
                vis += (unsigned)n;
            }
            if (best > 0.f && (lbest < best || (lbest == best && si < lsi))) {
                lbest = best; lgbest = gbest; lsi = si; lndx = vndx; lpos = vpos;
                if (threadIdx.x < 12) S.tbest[threadIdx.x] = S.tb[threadIdx.x];
            }
        }
        if (threadIdx.x == 0) {
            work_add(T, WK_REFINE, vis);
            float* c = T.rl_cand + ((long long)slot * nc + cand) * RLW_CAND;
            c[0] = lbest;
            c[1] = __int_as_float(lsi);
            c[2] = lgbest;
            c[3] = __int_as_float(lndx);
            c[4] = __int_as_float(lpos);
#pragma unroll
            for (int f = 0; f < 12; f++) c[5 + f] = S.tbest[f];
        }
    }
}

// npair: pairs the launch may have at most (a lane form's grid)
template <int LPP, bool LONG>
static void launch_refine_k(int mode, const Blk& B, const Bat& T, cudaStream_t st, int npair = 0,
                            int lo = 0, int hi = 0) {
    constexpr int W = LONG ? RF_WARPS_LONG : RF_WARPS_SHORT;
    // long pairs: at most RLW_GRID CTAs, T.rlw_ctas per pair at a time
    const int nslot = LONG ? std::max(1, std::min(T.rl_nlmax, RLW_GRID / T.rlw_ctas)) : 0;
    const int ng = LONG ? nslot * T.rlw_ctas
                        : (npair + (32 / LPP) * W - 1) / ((32 / LPP) * W);
    const int nt = W * 32;
    switch (mode) {
        case RM_INIT:  k_refine<RM_INIT, LPP, LONG><<<ng, nt, 0, st>>>(B, T, lo, hi); break;
        case RM_DP:    k_refine<RM_DP, LPP, LONG><<<ng, nt, 0, st>>>(B, T, lo, hi); break;
        case RM_FIN1:  k_refine<RM_FIN1, LPP, LONG><<<ng, nt, 0, st>>>(B, T, lo, hi); break;
        case RM_FIN2:  k_refine<RM_FIN2, LPP, LONG><<<ng, nt, 0, st>>>(B, T, lo, hi); break;
        case RM_PROD1: k_refine<RM_PROD1, LPP, LONG><<<ng, nt, 0, st>>>(B, T, lo, hi); break;
        case RM_PROD2: k_refine<RM_PROD2, LPP, LONG><<<ng, nt, 0, st>>>(B, T, lo, hi); break;
        case RM_PLOG:  k_refine<RM_PLOG, LPP, LONG><<<ng, nt, 0, st>>>(B, T, lo, hi); break;
    }
}

// A warp to a pass: the listed pairs with lo <= n < hi (at most npair of
// them), a cluster of C CTAs a pair.
static void launch_refine_coop(int mode, const Blk& B, const Bat& T, cudaStream_t st, int npair,
                               int lo, int hi, int C, int cls) {
    const int nmax = std::min(hi - 1, std::min(B.qmax, B.rmax));
    if (npair <= 0 || nmax < lo) return;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(std::min(npair, RC_GRID / C) * C);
    cfg.blockDim = dim3(CM_WARPS * 32);
    cfg.dynamicSmemBytes = coop_smem_bytes(nmax);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = C > 1 ? 1 : 0;
    cudaError_t e = cudaErrorInvalidValue;
    switch (mode) {
        case RM_INIT:  e = cudaLaunchKernelEx(&cfg, k_refine_coop<RM_INIT>, B, T, lo, hi, cls); break;
        case RM_DP:    e = cudaLaunchKernelEx(&cfg, k_refine_coop<RM_DP>, B, T, lo, hi, cls); break;
        case RM_FIN1:  e = cudaLaunchKernelEx(&cfg, k_refine_coop<RM_FIN1>, B, T, lo, hi, cls); break;
        case RM_FIN2:  e = cudaLaunchKernelEx(&cfg, k_refine_coop<RM_FIN2>, B, T, lo, hi, cls); break;
        case RM_PROD1: e = cudaLaunchKernelEx(&cfg, k_refine_coop<RM_PROD1>, B, T, lo, hi, cls); break;
        case RM_PROD2: e = cudaLaunchKernelEx(&cfg, k_refine_coop<RM_PROD2>, B, T, lo, hi, cls); break;
        case RM_PLOG:  e = cudaLaunchKernelEx(&cfg, k_refine_coop<RM_PLOG>, B, T, lo, hi, cls); break;
    }
    if (e != cudaSuccess && T.lerr && *T.lerr == cudaSuccess) *T.lerr = e;
    GTB_LAUNCHED(T);
}

// The refinement kernels re-read each pair's positions on every pass: ask
// for the smallest shared-memory carve-out that holds as many CTAs as their
// registers allow (static arrays + the 1 kB each CTA reserves), leaving the
// rest of the SM's 256 kB to L1.
template <int LPP, bool LONG>
static void carve_refine() {
    constexpr int W = LONG ? RF_WARPS_LONG : RF_WARPS_SHORT;
    const void* ks[7] = {(const void*)k_refine<RM_INIT, LPP, LONG>, (const void*)k_refine<RM_DP, LPP, LONG>,
                         (const void*)k_refine<RM_FIN1, LPP, LONG>, (const void*)k_refine<RM_FIN2, LPP, LONG>,
                         (const void*)k_refine<RM_PROD1, LPP, LONG>, (const void*)k_refine<RM_PROD2, LPP, LONG>,
                         (const void*)k_refine<RM_PLOG, LPP, LONG>};
    int dev = 0, smem_sm = 0, regs_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev);
    for (const void* k : ks) {
        cudaFuncAttributes fa{};
        int carve = 27;
        if (cudaFuncGetAttributes(&fa, k) == cudaSuccess && smem_sm > 0 && fa.numRegs > 0) {
            const int warp_regs = (fa.numRegs * 32 + 255) / 256 * 256;   // per-warp allocation unit
            int ctas = regs_sm / (warp_regs * W);
            if (ctas > 32) ctas = 32;
            const long long need = (long long)ctas * ((long long)fa.sharedSizeBytes + 1024);
            carve = (int)((need * 100 + smem_sm - 1) / smem_sm);
            if (carve < 1) carve = 1;
            if (carve > 100) carve = 100;
        }
        cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, carve);
    }
}

void configure_kernels() {
    carve_refine<16, false>();
    carve_refine<32, true>();
    const void* kc[7] = {(const void*)k_refine_coop<RM_INIT>, (const void*)k_refine_coop<RM_DP>,
                         (const void*)k_refine_coop<RM_FIN1>, (const void*)k_refine_coop<RM_FIN2>,
                         (const void*)k_refine_coop<RM_PROD1>, (const void*)k_refine_coop<RM_PROD2>,
                         (const void*)k_refine_coop<RM_PLOG>};
    for (const void* k : kc)
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)coop_smem_bytes(RL_LONG - 1));
    float gs[GTB_GONNET_NA * GTB_GONNET_NA];
    gtb_gonnet_scores(gs);
    cudaMemcpyToSymbol(g_gonnet, gs, sizeof(gs));
}

static void launch_refine_long(int mode, const Blk& B, const Bat& T, cudaStream_t st) {
    const int ng = T.rl_nlmax * T.rlw_ctas * RF_WARPS_LONG, nt = CL_WARPS * 32;
    const size_t sm = sizeof(LongSmem);
    switch (mode) {
        case RM_INIT:  k_refine_long<RM_INIT><<<ng, nt, sm, st>>>(B, T); break;
        case RM_DP:    k_refine_long<RM_DP><<<ng, nt, sm, st>>>(B, T); break;
        case RM_FIN1:  k_refine_long<RM_FIN1><<<ng, nt, sm, st>>>(B, T); break;
        case RM_FIN2:  k_refine_long<RM_FIN2><<<ng, nt, sm, st>>>(B, T); break;
        case RM_PROD1: k_refine_long<RM_PROD1><<<ng, nt, sm, st>>>(B, T); break;
        case RM_PROD2: k_refine_long<RM_PROD2><<<ng, nt, sm, st>>>(B, T); break;
        case RM_PLOG:  k_refine_long<RM_PLOG><<<ng, nt, sm, st>>>(B, T); break;
    }
}

static void launch_refine_long_fin(int mode, const Blk& B, const Bat& T, cudaStream_t st) {
    const int ng = (T.rl_nlmax + 3) / 4;
    switch (mode) {
        case RM_INIT:  k_refine_long_fin<RM_INIT><<<ng, 128, 0, st>>>(B, T); break;
        case RM_DP:    k_refine_long_fin<RM_DP><<<ng, 128, 0, st>>>(B, T); break;
        case RM_FIN1:  k_refine_long_fin<RM_FIN1><<<ng, 128, 0, st>>>(B, T); break;
        case RM_FIN2:  k_refine_long_fin<RM_FIN2><<<ng, 128, 0, st>>>(B, T); break;
        case RM_PROD1: k_refine_long_fin<RM_PROD1><<<ng, 128, 0, st>>>(B, T); break;
        case RM_PROD2: k_refine_long_fin<RM_PROD2><<<ng, 128, 0, st>>>(B, T); break;
        case RM_PLOG:  k_refine_long_fin<RM_PLOG><<<ng, 128, 0, st>>>(B, T); break;
    }
}

void launch_refine(int mode, const Blk& B, const Bat& T0, cudaStream_t st, bool few) {
    Bat T = T0;
    T.rl_min = RL_LONG;
    T.rlw_ctas = T0.rlw_ctas > 0 && T0.rlw_ctas <= RLW_CTAS_MAX ? T0.rlw_ctas : RLW_CTAS;
    if (T.np <= LIST_SMALL) {
        k_list_small<LK_REFINE><<<1, 1024, 0, st>>>(B, T, mode);
        GTB_LAUNCHED(T);
    } else {
        cudaMemsetAsync(T.rhist, 0, RL_NHIST * sizeof(int), st);
        if (T.rl_long) {
            cudaMemsetAsync(T.rl_count, 0, sizeof(int), st);
            cudaMemsetAsync(T.rl_next, 0, (size_t)T.rl_nlmax * sizeof(int), st);
        }
        const int nb = (T.np + 255) / 256;
        k_rlist_count<<<nb, 256, 0, st>>>(B, T, mode);
        k_rlist_scan<<<1, 1024, 0, st>>>(T);
        k_rlist_fill<<<nb, 256, 0, st>>>(B, T, mode);
        if (T.launches) (*T.launches) += 3;
    }
    // The longer pairs' launches on the second stream, beside the shorter
    // ones' (all read the lists built above; they write disjoint pairs)
    const bool fork = T.st2 && (T.rl_long || T.nml[2] > 0);
    cudaStream_t sl = fork ? T.st2 : st;
    KtScope kts(T, KF_REFINE, st);   // on st, after the join: both streams' time
    if (fork) {
        cudaEventRecord(T.evfork, st);
        cudaStreamWaitEvent(T.st2, T.evfork, 0);
    }
    if (T.rl_long) {
        if (T.rl_nlmax <= RLW_CTA_MAX) {
            // a CTA to a pass, up to RLW_CTA_GRID CTAs in all; they leave a
            // candidate each, in the room of 4 CTAs' warps
            Bat TL = T;
            TL.rlw_ctas = std::max(4, std::min(T.rlw_ctas, RLW_CTA_GRID / 4 / T.rl_nlmax));
            launch_refine_long(mode, B, TL, sl);
            launch_refine_long_fin(mode, B, TL, sl);
        } else {
            launch_refine_k<32, true>(mode, B, T, sl);
            launch_refine_long_fin(mode, B, T, sl);
        }
        if (T.launches) (*T.launches) += 2;
    } else if (T.nml[3] > 0) {
        launch_refine_k<16, false>(mode, B, T, sl, T.nml[3], RL_LONG, 0);
        GTB_LAUNCHED(T);
    }
    const bool coop = few || T.np <= RC_SMALL;
    launch_refine_coop(mode, B, T, sl, T.nml[2], RC_N2, RL_LONG, 8, 2);
    if (coop) {
        const int c = T.np <= RC_NP8 ? 8 : T.np <= RC_NP4 ? 4 : T.np <= RC_NP2 ? 2 : 1;
        launch_refine_coop(mode, B, T, st, T.nml[1], RC_N1, RC_N2, c < 4 ? 4 : c, 1);
        launch_refine_coop(mode, B, T, st, T.np, 0, RC_N1, c, 0);
    } else {
        launch_refine_k<16, false>(mode, B, T, st, T.np, 0, RC_N2);
        GTB_LAUNCHED(T);
    }
    if (fork) {
        cudaEventRecord(T.evjoin, T.st2);
        cudaStreamWaitEvent(st, T.evjoin, 0);
    }
}

// ---------------------------------------------------------------------------
// DP: MpDPHub.cpp:72-346 and 686-940.  One warp per pair.  Lane l holds the
// R query rows 32*R*s + R*l + r of strip s and, at step t of the strip,
// computes column j = t - l of those rows (one anti-diagonal of the strip
// per step).  The value above a lane's first row comes from lane l-1 (its
// last row, previous step) or, for lane 0, from the previous strip's last
// row kept in `row`.  Stored values are negated when the cell was reached
// diagonally (the reference's state encoding, MpDPHub.cpp:246-262).  Steps
// run in groups of 16/R, one traceback word per lane and group.
// WAVE: the strips of one pair are shared by several CTAs (strip s by CTA
// s mod s_step); a strip waits, with a bounded spin, until the previous one
// has published the steps whose last-row values it is about to read
// (`prog`: steps done per strip), and publishes its own progress every 32
// steps.  Returns false when a wait gave up (error flag set).
// SC, the cell score: DP_SC_TFM (TM-score term under t), DP_SC_TFMSS (plus 0.5
// for equal secondary structure), DP_SC_SSRR (the --add-search-by-ss DP,
// dpssw_btck.cu:280-330: 1 for equal secondary structure + 0.2 x the Gonnet
// score of the residues, no transform; a cell reached diagonally stores its
// value + DPSS_C, a reader takes the offset off again, the gap cost is paid
// once when leaving such a cell; the border reads as a diagonal cell of 0).
// SCOREONLY: no traceback words; the last cell's value goes to *fin.
// This form takes any coordinates and the --add-search-by-ss score; the others
// run dp_pair_fast.
template <int R, bool gap0, int SC, bool WAVE, bool SCOREONLY = false>
__device__ __forceinline__ bool dp_pair(const float* t, float d02, float gcost, int lq, int lr,
                                        const float* qx, const float* qy, const float* qz,
                                        const float4* r4, const char* qs, const char* rs,
                                        const unsigned char* qa, const unsigned char* ra,
                                        float* row, unsigned* bt, int lane, int s_first = 0,
                                        int s_step = 1, volatile int* prog = nullptr,
                                        volatile int* err = nullptr,
                                        long long spin = DP_WAVE_SPIN_DEFAULT, float* fin = nullptr,
                                        bool cta_wave = false) {
    // cta_wave: the strips' warps share one CTA, so the row values and the
    // progress counters need ordering at CTA scope only
    constexpr bool usess = SC == DP_SC_TFMSS, ssrr = SC == DP_SC_SSRR;
    constexpr float BND = ssrr ? DPSS_C : 0.f;   // the matrix border
    constexpr int ROWS = 32 * R, SPW = 16 / R;
    const unsigned FULL = 0xffffffffu;
    const int W = lr + 31;
    const int ngrp = (W + SPW - 1) / SPW;
    const int nstrips = (lq + ROWS - 1) / ROWS;
    for (int s = s_first; s < nstrips; s += s_step) {
        float tx[R], ty[R], tz[R], h[R];
        char qss[R];
        unsigned char qaa[R];
        int nv = 0;  // valid rows of this lane (a prefix of its R rows)
#pragma unroll
        for (int r = 0; r < R; r++) {
            int irow = s * ROWS + lane * R + r;
            tx[r] = ty[r] = tz[r] = 0.f;
            qss[r] = 0;
            qaa[r] = 0;
            h[r] = BND;
            if (irow < lq) {
                if (!ssrr) xform(t, __ldg(qx + irow), __ldg(qy + irow), __ldg(qz + irow), tx[r], ty[r], tz[r]);
                if (usess || ssrr) qss[r] = qs[irow];
                if (ssrr) qaa[r] = qa[irow];
                nv = r + 1;
            }
        }
        float uplast = BND, rb = BND;
        unsigned* bts = SCOREONLY ? nullptr : bt + (long long)s * ngrp * 32 + lane;
        const bool full = (s + 1) * ROWS <= lq;    // every lane has R rows
        const int lastr = (lq - 1) - s * ROWS - lane * R;   // the last row among this lane's (if 0..R-1)
        __syncwarp();
        for (int g = 0; g < ngrp; g++) {
            unsigned acc = 0u;
            if (WAVE && s > 0 && ((g * SPW) & 31) == 0) {
                // row[tt .. tt+31] of strip s-1: written up to its step tt+62
                const int need = g * SPW + 64 < ngrp * SPW ? g * SPW + 64 : ngrp * SPW;
                if (lane == 0) {
                    long long it = 0;
                    while (prog[s - 1] < need) {
                        if (*err || ++it > spin) { *err = 1; break; }
                        __nanosleep(64);
                    }
                }
                __syncwarp();
                if (cta_wave) __threadfence_block();
                else __threadfence();
                if (*err) return false;
            }
            if ((g * SPW & 31) == 0) {            // the previous strip's last row, 32 columns
                int jj = g * SPW + lane;
                if (WAVE) rb = (s > 0 && jj < lr) ? __ldcg(row + jj) : BND;
                else rb = (s > 0 && jj < lr) ? row[jj] : BND;
            }
            // SPW steps; CHK: some lane may be outside the matrix or have
            // fewer than R rows (strip ramps, the last strip)
            auto steps = [&](auto chk) {
                constexpr bool CHK = decltype(chk)::value;
#pragma unroll
                for (int u = 0; u < SPW; u++) {
                    const int tt = g * SPW + u;   // steps past W find j >= lr on every lane
                    const int j = tt - lane;
                    float upv = __shfl_up_sync(FULL, h[R - 1], 1);
                    float up0 = __shfl_sync(FULL, rb, tt & 31);
                    if (lane == 0) upv = (!CHK || j < lr) ? up0 : BND;
                    if (!CHK || (j >= 0 && j < lr && nv > 0)) {
                        float4 c4 = ssrr ? make_float4(0.f, 0.f, 0.f, 0.f) : __ldg(r4 + j);
                        char css = (usess || ssrr) ? rs[j] : 0;
                        unsigned char cra = ssrr ? ra[j] : 0;
                        float up = upv, dg = uplast;
#pragma unroll
                        for (int r = 0; r < R; r++) {
                            if (ssrr && (!CHK || r < nv)) {
                                float v = __fmaf_rn(gonnet(qaa[r], cra), 0.2f, (float)(qss[r] == css));
                                v = __fadd_rn(v, dg < DPSS_CMP ? __fsub_rn(dg, DPSS_C) : dg);
                                int bk = BTW_DIAG;
                                float l = h[r];
                                if (l < DPSS_CMP) l = __fsub_rn(__fadd_rn(gcost, l), DPSS_C);
                                if (v < l) { v = l; bk = BTW_LEFT; }
                                float uu = up;
                                if (uu < DPSS_CMP) uu = __fsub_rn(__fadd_rn(gcost, uu), DPSS_C);
                                if (v < uu) { v = uu; bk = BTW_UP; }
                                float w = bk == BTW_DIAG ? __fadd_rn(v, DPSS_C) : v;
                                dg = h[r];
                                up = w;
                                h[r] = w;
                                acc |= (unsigned)bk << (2 * R * u + 2 * r);
                            } else if (!ssrr && (!CHK || r < nv)) {
                                float v = tmterm(d02, dist2(tx[r], ty[r], tz[r], c4.x, c4.y, c4.z));
                                if (usess) v = __fadd_rn(v, __fmul_rn((float)(qss[r] == css), 0.5f));
                                v = __fadd_rn(v, gap0 ? dg : fabsf(dg));
                                int bk = BTW_DIAG;
                                float l = h[r];
                                if (!gap0 && l < 0.f) l = __fsub_rn(gcost, l);
                                if (v < l) { v = l; bk = BTW_LEFT; }
                                float uu = up;
                                if (!gap0 && uu < 0.f) uu = __fsub_rn(gcost, uu);
                                if (v < uu) { v = uu; bk = BTW_UP; }
                                float w = (gap0 || bk != BTW_DIAG) ? v : -v;
                                dg = h[r];   // (row r, j-1): the next row's diagonal
                                up = w;      // (row r, j):   the next row's up
                                h[r] = w;
                                if (SCOREONLY) { if (r == lastr && j == lr - 1) *fin = w; }
                                else acc |= (unsigned)bk << (2 * R * u + 2 * r);
                            }
                        }
                        if (lane == 31 && (!CHK || nv == R)) row[j] = h[R - 1];
                    }
                    uplast = upv;
                }
            };
            if (full && g * SPW >= 31 && (g + 1) * SPW <= lr) steps(std::false_type{});
            else steps(std::true_type{});
            if (!SCOREONLY) bts[g * 32] = acc;
            // the next strip reads its row values 32 steps at a time, so the
            // count is published at every 32nd step (and the last): one fence
            // per 32 steps instead of per group
            if (WAVE && lane == 31 && ((((g + 1) * SPW) & 31) == 0 || g == ngrp - 1)) {
                if (cta_wave) __threadfence_block();   // the row values before the count
                else __threadfence();
                prog[s] = (g + 1) * SPW;
            }
        }
        __syncwarp();
    }
    return true;
}

// The DP of a pair whose coordinates are ordinary (coords_ordinary), cell
// scores DP_SC_TFM and DP_SC_TFMSS: the values and directions of dp_pair.
// A lone warp of dp_pair took ~600 cycles a step (R cells a lane): each cell's
// score was computed inside the chain of cell values.  Here the score terms
// of a group of steps (16 cells a lane) come first, two steps to a packed
// FP32 operation, and the chain that is left is a shuffle and, per row, one
// maximum (and, with a gap cost, the choice of what a neighbour sees).
//  * The reference's coordinates go through a ring of 64 columns in shared
//    memory, kept twice, the second time shifted by one, so that every lane
//    reads the pairs of columns (j, j+1) of its steps as 8 aligned bytes.
//  * Rows past the query's end and columns past the reference's are computed
//    and never read; before the first column the terms are -inf (stored negated), which leaves
//    the zeros of the border in place.
//  * With a gap cost a cell keeps its value and what its right and lower
//    neighbours see: the value + gap cost if it was reached diagonally.  In the
//    row buffer a diagonally reached value is negative, as in dp_pair.
// What bounds it: a lone pair, the chain; a full GPU, issue.
constexpr int DPR_W = 64;                    // columns of a warp's ring
struct DpRing { float c[2][3][DPR_W]; };

template <int R, bool gap0, int SC, bool WAVE, bool SCOREONLY>
__device__ __forceinline__ bool dp_pair_fast(const float* t, float d02, float gcost, int lq, int lr,
                                             const float4* q4, const float4* r4, const char* qs,
                                             const char* rs, float* row, unsigned* bt, DpRing& ring,
                                             int lane, int s_first = 0, int s_step = 1,
                                             volatile int* prog = nullptr,
                                             volatile int* err = nullptr,
                                             long long spin = DP_WAVE_SPIN_DEFAULT,
                                             float* fin = nullptr, bool cta_wave = false) {
    constexpr bool usess = SC == DP_SC_TFMSS;
    constexpr int ROWS = 32 * R, SPW = 16 / R;
    const unsigned FULL = 0xffffffffu;
    const float INF = __int_as_float(0x7f800000);
    const int ngrp = (lr + 31 + SPW - 1) / SPW;
    const int nstrips = (lq + ROWS - 1) / ROWS;
    const f32x2 D02 = pack2(d02, d02), ONE = pack2(1.f, 1.f);
    const float* cx = ring.c[lane & 1][0];
    const int codd = (lane & 1) - lane;      // a lane's column pairs in its copy: t + codd, even
    for (int s = s_first; s < nstrips; s += s_step) {
        f32x2 nx[R], ny[R], nz[R];
        float h[R], e[R];                    // (row, j-1): value; what a neighbour sees (gap cost)
        char qss[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int irow = s * ROWS + lane * R + r;
            float x = 0.f, y = 0.f, z = 0.f;
            qss[r] = 0;
            h[r] = e[r] = 0.f;
            if (irow < lq) {
                const float4 q = __ldg(q4 + irow);
                xform(t, q.x, q.y, q.z, x, y, z);
                if (usess) qss[r] = qs[irow];
            }
            nx[r] = pack2(-x, -x); ny[r] = pack2(-y, -y); nz[r] = pack2(-z, -z);
        }
        float hup = 0.f;                     // (first row - 1, j-1)
        float rb = 0.f;
        float4 cn = lane < lr ? __ldg(r4 + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
        unsigned* bts = SCOREONLY ? nullptr : bt + (long long)s * ngrp * 32 + lane;
        const int lastr = (lq - 1) - s * ROWS - lane * R;   // the last row among this lane's (if 0..R-1)
        __syncwarp();
        for (int g = 0; g < ngrp; g++) {
            const int t0 = g * SPW;
            if ((t0 & 31) == 0) {
                if (WAVE && s > 0) {
                    // row[t0 .. t0+31] of strip s-1: written up to its step t0+62
                    const int need = t0 + 64 < ngrp * SPW ? t0 + 64 : ngrp * SPW;
                    int ok = 1;
                    if (lane == 0) {
                        long long it = 0;
                        while (prog[s - 1] < need) {
                            if (*err || ++it > spin) { *err = 1; ok = 0; break; }
                            __nanosleep(32);
                        }
                    }
                    if (!__shfl_sync(FULL, ok, 0)) return false;
                    // lane 0's look at the counter before every lane's reads of
                    // the row (a shuffle alone orders no memory)
                    __syncwarp();
                    if (cta_wave) __threadfence_block();
                    else __threadfence();
                }
                const int jj = t0 + lane;
                if (s > 0) rb = jj < lr ? (WAVE ? __ldcg(row + jj) : row[jj]) : 0.f;
                // these 32 columns into the ring, the next 32 on their way
                __syncwarp();                // the columns in their place are read
                const int a = jj & (DPR_W - 1), b = (jj + 1) & (DPR_W - 1);
                ring.c[0][0][a] = cn.x; ring.c[0][1][a] = cn.y; ring.c[0][2][a] = cn.z;
                ring.c[1][0][b] = cn.x; ring.c[1][1][b] = cn.y; ring.c[1][2][b] = cn.z;
                __syncwarp();
                if (jj + 32 < lr) cn = __ldg(r4 + jj + 32);
            }
            float nt[SPW][R];                // the negated score terms
#pragma unroll
            for (int u = 0; u < SPW; u += 2) {
                const int o = (t0 + u + codd) & (DPR_W - 1);
                const float2 x2 = *(const float2*)(cx + o), y2 = *(const float2*)(cx + DPR_W + o),
                             z2 = *(const float2*)(cx + 2 * DPR_W + o);
                const f32x2 X = pack2(x2.x, x2.y), Y = pack2(y2.x, y2.y), Z = pack2(z2.x, z2.y);
                char c0 = 0, c1 = 0;
                if (usess) {
                    const int j = t0 + u - lane;
                    c0 = j >= 0 && j < lr ? rs[j] : 0;
                    c1 = j + 1 >= 0 && j + 1 < lr ? rs[j + 1] : 0;
                }
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const f32x2 dx = add2(X, nx[r]), dy = add2(Y, ny[r]), dz = add2(Z, nz[r]);
                    const f32x2 b = add2(D02, fma2(dx, dx, fma2(dy, dy, mul2(dz, dz))));
                    unpack2(div2_neg(D02, b, ONE), nt[u][r], nt[u + 1][r]);
                    if (usess) {
                        nt[u][r] = __fsub_rn(nt[u][r], qss[r] == c0 ? 0.5f : 0.f);
                        nt[u + 1][r] = __fsub_rn(nt[u + 1][r], qss[r] == c1 ? 0.5f : 0.f);
                    }
                }
            }
            if (t0 < 31) {
#pragma unroll
                for (int u = 0; u < SPW; u++)
                    if (t0 + u < lane) {
#pragma unroll
                        for (int r = 0; r < R; r++) nt[u][r] = INF;
                    }
            }
            unsigned acc = 0u;
#pragma unroll
            for (int u = 0; u < SPW; u++) {
                const int tt = t0 + u;
                const float r0 = __shfl_sync(FULL, rb, tt & 31);
                float hu = __shfl_up_sync(FULL, h[R - 1], 1), eu = 0.f;
                if (gap0) {
                    if (lane == 0) hu = r0;
                } else {
                    eu = __shfl_up_sync(FULL, e[R - 1], 1);
                    if (lane == 0) { hu = fabsf(r0); eu = r0 < 0.f ? __fsub_rn(gcost, r0) : r0; }
                }
                float dg = hup;
                hup = hu;
                float up = gap0 ? hu : eu;
                bool diag = false;           // the last row's cell was reached diagonally
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const float v = __fsub_rn(dg, nt[u][r]);
                    const float l = gap0 ? h[r] : e[r];
                    const bool p1 = v < l;                        // left rather than diagonal
                    const float m = fmaxf(v, l);
                    const bool p2 = m < up;                       // up rather than either
                    const float w = fmaxf(m, up);
                    if (!SCOREONLY) {
                        if (p1) acc |= 1u << (2 * R * u + 2 * r);
                        if (p2) acc |= 2u << (2 * R * u + 2 * r);
                    }
                    dg = h[r];
                    h[r] = w;
                    if (gap0) up = w;
                    else {
                        diag = !(p1 || p2);
                        e[r] = diag ? __fadd_rn(gcost, w) : w;
                        up = e[r];
                    }
                    if (SCOREONLY && t0 + SPW >= lr && r == lastr && tt - lane == lr - 1) *fin = w;
                }
                if (lane == 31 && tt >= 31 && tt - 31 < lr) row[tt - 31] = diag ? -h[R - 1] : h[R - 1];
            }
            if (!SCOREONLY) bts[g * 32] = acc;
            // the count is published at every 32nd step, when the next strip
            // may read 32 more columns, and at the end
            if (WAVE && lane == 31 && (((t0 + SPW) & 31) == 0 || g == ngrp - 1)) {
                if (cta_wave) __threadfence_block();       // the row values before the count
                else __threadfence();
                prog[s] = t0 + SPW;
            }
        }
        __syncwarp();
    }
    return true;
}

// traceback: MpDPHub.cpp:1515-1660 (plain) and 1699-1905 (constrained)
//
// A warp per pair.  The walk is one chain of dependent steps, the same on every
// lane; a thread per pair paid a load from L2 for most of them (580 cycles a
// step: 0.73 ms for a pair of 1,200 residues).  The warp that ran the pair's DP
// (the first of its CTA's) makes the walk right after it, beside other pairs' DPs.
// The 32 words of a (strip,
// step group), one 128-byte line, come in for BT_WIN groups at a time into
// shared memory while the ones the path is likely to enter next (the groups below,
// or the previous strip's where a diagonal path enters it) are on their way to
// registers.  32 aligned pairs at a time are written out, a pair per lane.
constexpr int BT_WIN = 16;        // groups of a window
constexpr int BT_WARPS = 4;
template <int R>
__device__ __forceinline__ int btck_walk(const unsigned* bt, int lq, int lr, const float4* q4,
                                         const float4* r4, bool constrained, const float* t,
                                         float d82, unsigned* aln, float* alc, unsigned* win,
                                         int lane) {
    const unsigned FULL = 0xffffffffu;
    constexpr int ROWS = 32 * R, SPW = 16 / R;
    const long long sw = bt_strip_words(lr, R);
    const int ngrp = (int)(sw / 32);
    int y = lq - 1, x = lr - 1, n = 0, pend = 0;
    unsigned mine = 0;                        // this lane's aligned pair among the last 32
    auto flush = [&](int cnt) {
        bool keep = lane < cnt;
        if (constrained && keep) {
            const float4 cq = __ldg(q4 + (mine >> 16)), cr = __ldg(r4 + (mine & 0xffffu));
            keep = dist2_tf(t, cq.x, cq.y, cq.z, cr.x, cr.y, cr.z) <= d82;
        }
        const unsigned m = __ballot_sync(FULL, keep);
        if (keep) aln[n + __popc(m & ((1u << lane) - 1u))] = mine;
        n += __popc(m);
    };
    // the words of BT_WIN groups, loaded into registers while the walk is in the
    // window before: strip ps, groups pg, pg - 1, ...
    unsigned pw[BT_WIN];
    int ps = -1, pg = 0;
    auto load = [&](int s, int g) {
        const unsigned* line = bt + s * sw + lane;
        ps = s; pg = g;
#pragma unroll
        for (int k = 0; k < BT_WIN; k++) pw[k] = g - k >= 0 ? line[(g - k) * 32] : 0u;
    };
    int cs = -1, wlo = 0;                     // the window's strip and lowest group
    while ((x | y) >= 0) {
        const int s = y / ROWS, l = y % ROWS / R, tt = x + l, g = tt / SPW;
        if (s != cs || g < wlo) {
            if (ps != s || g > pg || g <= pg - BT_WIN / 2) load(s, g);
            cs = s;
            wlo = pg - BT_WIN + 1 > 0 ? pg - BT_WIN + 1 : 0;
            __syncwarp();
#pragma unroll
            for (int k = 0; k < BT_WIN; k++) win[((pg - k) & (BT_WIN - 1)) * 32 + lane] = pw[k];
            __syncwarp();
            // what comes next if the path goes on diagonally: the groups below, or
            // the previous strip's from where the path leaves this one
            const int left = y % ROWS + 1;
            if (left * (R + 1) / R < (g - wlo) * SPW) {
                const int xn = x - left;
                if (s > 0 && xn >= 0) load(s - 1, (xn + 31) / SPW + 1 < ngrp ? (xn + 31) / SPW + 1 : ngrp - 1);
            } else if (wlo > 0) {
                load(s, wlo - 1);
            }
        }
        // the path through one word (R rows x SPW steps): bits 0-4 of pos are the
        // cell's place in the word, row and step above them with a guard bit
        // each that turns when they fall below 0; the column's sign is looked at
        // too (a word can hold steps before the first column)
        const unsigned w = win[(g & (BT_WIN - 1)) * 32 + l];
        const int rr = y % R, uu = tt % SPW;
        unsigned pos = (unsigned)(2 * R * uu + 2 * rr) | (unsigned)rr << 8 | (unsigned)uu << 16;
        do {
            const unsigned b = (w >> (pos & 31)) & 3u;
            const unsigned yx = ((unsigned)y << 16) | (unsigned)x;
            if (b == BTW_DIAG && lane == pend) mine = yx;
            pend += b == BTW_DIAG;
            y -= b != BTW_LEFT;
            x -= b < BTW_UP;
            // diagonal (0), left (1), up (2 or 3): down a row, back a step
            pos -= b >= BTW_UP ? 2u + (1u << 8)
                               : (b == BTW_LEFT ? 2u * R + (1u << 16) : 2u * R + 2u + (1u << 8) + (1u << 16));
        } while (!(pos & 0x80008000u) && x >= 0);
        if (pend > 32 - R) { flush(pend); pend = 0; }     // a word adds at most R
    }
    if (pend > 0) flush(pend);
    // the aligned residues' coordinates, for the passes that read them in a row
    __syncwarp();
#pragma unroll 4
    for (int k = lane; k < n; k += 32) {
        const unsigned m = aln[k];
        const float4 cq = __ldg(q4 + (m >> 16)), cr = __ldg(r4 + (m & 0xffffu));
        float2* c2 = (float2*)(alc + 6 * (long long)k);
        c2[0] = make_float2(cq.x, cq.y); c2[1] = make_float2(cq.z, cr.x); c2[2] = make_float2(cr.y, cr.z);
    }
    return n;
}

// the traceback of pair i by a warp: its aligned pairs and their number
__device__ __forceinline__ void btck_pair(const Blk& B, const Bat& T, int i, int flags, int lq, int lr,
                                          const float4* q4, const float4* r4, int constrained,
                                          unsigned* win, int lane) {
    if (!constrained && (flags & CONV_SCOREDP)) {
        if (lane == 0) T.naln[i] = 0;
        return;
    }
    const unsigned* bt = T.bt + T.off_bt[i];
    unsigned* aln = T.aln + T.off_aln[i];
    float* alc = T.alc + 6 * T.off_aln[i];
    const float d82 = B.t_d82[lq < lr ? lq : lr];
    float t[12];
#pragma unroll
    for (int f = 0; f < 12; f++) t[f] = constrained ? T.tfm_gr[i * 12 + f] : 0.f;
    const int n = dp_r(lq) == 4
        ? btck_walk<4>(bt, lq, lr, q4, r4, constrained != 0, t, d82, aln, alc, win, lane)
        : btck_walk<2>(bt, lq, lr, q4, r4, constrained != 0, t, d82, aln, alc, win, lane);
    if (lane == 0) T.naln[i] = n;
}

// The DP work list (k_dlist_*, largest matrices first): its first dp_kc
// pairs take a CTA each, whose 4 warps run the pair's strips as a wavefront
// (strip s on warp s mod 4, each strip waiting with a bounded spin until the
// previous one has published the row values it reads, the counters in
// shared memory); the other pairs take a warp each.
template <int GAP0, int SC>
__global__ void __launch_bounds__(128) k_dp(Blk B, Bat T, int tfmsrc, float gcost, int dpscan,
                                            int constrained) {
    __shared__ int s_prog[DP_CTA_MAXSTRIPS];
    __shared__ DpRing s_ring[4];
    __shared__ unsigned s_win[4][BT_WIN * 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int len = T.rhist[RL_NB];
    const int dkc = T.dw_err ? T.dp_kc : 0;
    const int kc = dkc < len ? dkc : len;
    const bool cta = (int)blockIdx.x < kc;
    const int slot = cta ? (int)blockIdx.x : kc + ((int)blockIdx.x - kc) * (blockDim.x >> 5) + w;
    if (slot >= len) return;                       // never for a CTA of the first kind
    const int i = T.rlist[slot];
    int qi = pair_qi(B, T, i), ri = pair_ri(B, T, i);
    int lq = B.qlen[qi], lr = B.rlen[ri];
    int ml = lq < lr ? lq : lr;
    const float* tsrc = dp_tfm(T, i, tfmsrc);
    float t[12];
#pragma unroll
    for (int f = 0; f < 12; f++) t[f] = tsrc[f];
    float d0 = B.t_d0[ml];
    float d02;
    if (dpscan) { float a = __fadd_rn(d0, 1.5f); d02 = __fmul_rn(a, a); }
    else d02 = __fmul_rn(d0, d0);
    const float* qx = B.qx + B.qoff[qi];
    const float* qy = B.qy + B.qoff[qi];
    const float* qz = B.qz + B.qoff[qi];
    const float4* q4 = B.q4 + B.q4off[qi];
    const float4* r4 = B.r4 + B.r4off[ri];
    const bool fast = SC != DP_SC_SSRR && coords_ordinary(B, qi, ri);
    const char* qs = B.qs + B.qoff[qi];
    const char* rs = B.rs + B.roff[ri];
    float* row = T.row + T.off_row[i];
    unsigned* bt = T.bt + T.off_bt[i];
    const unsigned char* qa = B.qa + B.qoff[qi];
    const unsigned char* ra = B.ra + B.roff[ri];
    if (cta) {
        if (lane == 0 && w == 0) work_add(T, WK_DPCELL, (unsigned long long)lq * (unsigned long long)lr);
        if (dp_strips(lq) > 1) {
            for (int k = threadIdx.x; k < DP_CTA_MAXSTRIPS; k += blockDim.x) s_prog[k] = 0;
            __syncthreads();
            if (fast) {
                if (dp_r(lq) == 4)
                    dp_pair_fast<4, GAP0 != 0, SC, true, false>(t, d02, gcost, lq, lr, q4, r4, qs, rs, row, bt,
                                                                s_ring[w], lane, w, blockDim.x >> 5, s_prog,
                                                                T.dw_err, T.dw_spin, nullptr, true);
                else
                    dp_pair_fast<2, GAP0 != 0, SC, true, false>(t, d02, gcost, lq, lr, q4, r4, qs, rs, row, bt,
                                                                s_ring[w], lane, w, blockDim.x >> 5, s_prog,
                                                                T.dw_err, T.dw_spin, nullptr, true);
            } else if (dp_r(lq) == 4)
                dp_pair<4, GAP0 != 0, SC, true>(t, d02, gcost, lq, lr, qx, qy, qz, r4, qs, rs, qa, ra, row,
                                                bt, lane, w, blockDim.x >> 5, s_prog, T.dw_err, T.dw_spin,
                                                nullptr, true);
            else
                dp_pair<2, GAP0 != 0, SC, true>(t, d02, gcost, lq, lr, qx, qy, qz, r4, qs, rs, qa, ra, row,
                                                bt, lane, w, blockDim.x >> 5, s_prog, T.dw_err, T.dw_spin,
                                                nullptr, true);
            __syncthreads();                       // every strip's words
            if (w == 0) btck_pair(B, T, i, T.flags[i], lq, lr, q4, r4, constrained, s_win[w], lane);
            return;
        }
        if (w != 0) return;                        // one strip: one warp
    } else if (lane == 0) {
        work_add(T, WK_DPCELL, (unsigned long long)lq * (unsigned long long)lr);
    }
    if (fast) {
        if (dp_r(lq) == 4)
            dp_pair_fast<4, GAP0 != 0, SC, false, false>(t, d02, gcost, lq, lr, q4, r4, qs, rs, row, bt,
                                                         s_ring[w], lane);
        else
            dp_pair_fast<2, GAP0 != 0, SC, false, false>(t, d02, gcost, lq, lr, q4, r4, qs, rs, row, bt,
                                                         s_ring[w], lane);
    } else if (dp_r(lq) == 4)
        dp_pair<4, GAP0 != 0, SC, false>(t, d02, gcost, lq, lr, qx, qy, qz, r4, qs, rs, qa, ra, row, bt, lane);
    else
        dp_pair<2, GAP0 != 0, SC, false>(t, d02, gcost, lq, lr, qx, qy, qz, r4, qs, rs, qa, ra, row, bt, lane);
    __syncwarp();
    btck_pair(B, T, i, T.flags[i], lq, lr, q4, r4, constrained, s_win[w], lane);
}

// One warp per CTA; the CTAs of a long pair take its strips round robin.
// Launched cooperatively so that all CTAs are resident together.
template <int GAP0, int SC>
__global__ void __launch_bounds__(32) k_dp_wave(Blk B, Bat T, int tfmsrc, float gcost, int dpscan,
                                                int skipmode) {
    __shared__ DpRing s_ring;
    const int lane = threadIdx.x & 31;
    const int item = blockIdx.x;
    if (item >= T.ndw) return;
    const int slot = T.dw_item[item], c = T.dw_item[T.ndw + item];
    const int i = T.dw_pair[slot], G = T.dw_G[slot];
    int flags = T.flags[i];
    int skipmask = skipmode == 0 ? (CONV_LOWTMSC | CONV_SCOREDP) : CONV_LOWTMSC;
    if (flags & skipmask) return;                  // the same for every CTA of the pair
    if (alt_empty(T, i)) return;
    int qi = pair_qi(B, T, i), ri = pair_ri(B, T, i);
    int lq = B.qlen[qi], lr = B.rlen[ri];
    int ml = lq < lr ? lq : lr;
    const float* tsrc = dp_tfm(T, i, tfmsrc);
    float t[12];
#pragma unroll
    for (int f = 0; f < 12; f++) t[f] = tsrc[f];
    float d0 = B.t_d0[ml];
    float d02;
    if (dpscan) { float a = __fadd_rn(d0, 1.5f); d02 = __fmul_rn(a, a); }
    else d02 = __fmul_rn(d0, d0);
    const float* qx = B.qx + B.qoff[qi];
    const float* qy = B.qy + B.qoff[qi];
    const float* qz = B.qz + B.qoff[qi];
    const float4* q4 = B.q4 + B.q4off[qi];
    const float4* r4 = B.r4 + B.r4off[ri];
    const bool fast = SC != DP_SC_SSRR && coords_ordinary(B, qi, ri);
    const char* qs = B.qs + B.qoff[qi];
    const char* rs = B.rs + B.roff[ri];
    float* row = T.row + T.off_row[i];
    unsigned* bt = T.bt + T.off_bt[i];
    volatile int* prog = T.dw_prog + T.dw_soff[slot];
    const unsigned char* qa = B.qa + B.qoff[qi];
    const unsigned char* ra = B.ra + B.roff[ri];
    if (lane == 0 && c == 0) work_add(T, WK_DPCELL, (unsigned long long)lq * (unsigned long long)lr);
    if (fast) {
        if (dp_r(lq) == 4)
            dp_pair_fast<4, GAP0 != 0, SC, true, false>(t, d02, gcost, lq, lr, q4, r4, qs, rs, row, bt, s_ring,
                                                        lane, c, G, prog, T.dw_err, T.dw_spin);
        else
            dp_pair_fast<2, GAP0 != 0, SC, true, false>(t, d02, gcost, lq, lr, q4, r4, qs, rs, row, bt, s_ring,
                                                        lane, c, G, prog, T.dw_err, T.dw_spin);
        return;
    }
    if (dp_r(lq) == 4)
        dp_pair<4, GAP0 != 0, SC, true>(t, d02, gcost, lq, lr, qx, qy, qz, r4, qs, rs, qa, ra, row,
                                        bt, lane, c, G, prog, T.dw_err, T.dw_spin);
    else
        dp_pair<2, GAP0 != 0, SC, true>(t, d02, gcost, lq, lr, qx, qy, qz, r4, qs, rs, qa, ra, row,
                                        bt, lane, c, G, prog, T.dw_err, T.dw_spin);
}

int dp_wave_capacity() {
    int dev = 0, nsm = 0, m = 1 << 30, nb = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const void* ks[5] = {(const void*)k_dp_wave<1, DP_SC_TFM>, (const void*)k_dp_wave<0, DP_SC_TFM>,
                         (const void*)k_dp_wave<0, DP_SC_TFMSS>, (const void*)k_dp_wave<1, DP_SC_TFMSS>,
                         (const void*)k_dp_wave<0, DP_SC_SSRR>};
    for (const void* k : ks) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, 32, 0) != cudaSuccess) return 0;
        m = nb < m ? nb : m;
    }
    return m * nsm;
}

template <int GAP0, int SC>
static void launch_dp_wave(const Blk& B, const Bat& T, int tfmsrc, float gcost, int dpscan,
                           int skipmode, cudaStream_t st) {
    Blk b = B;
    Bat t = T;
    void* args[] = {&b, &t, &tfmsrc, &gcost, &dpscan, &skipmode};
    cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_dp_wave<GAP0, SC>, dim3(T.ndw),
                                                dim3(32), args, 0, st);
    if (e != cudaSuccess && T.lerr && *T.lerr == cudaSuccess) *T.lerr = e;
}

// the pairs whose DP ran on several CTAs (dw_mark); the others' walks are in k_dp
__global__ void __launch_bounds__(BT_WARPS * 32) k_btck(Blk B, Bat T, int constrained) {
    __shared__ unsigned s_win[BT_WARPS][BT_WIN * 32];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int i = blockIdx.x * BT_WARPS + wp;
    if (i >= T.np || !T.dw_mark[i]) return;
    const int flags = T.flags[i];
    if (constrained) {
        if (flags & CONV_LOWTMSC) return;
    } else if ((flags & CONV_LOWTMSC) || alt_empty(T, i)) {
        if (lane == 0) T.naln[i] = 0;
        return;
    }
    const int qi = pair_qi(B, T, i), ri = pair_ri(B, T, i);
    btck_pair(B, T, i, flags, B.qlen[qi], B.rlen[ri], B.q4 + B.q4off[qi], B.r4 + B.r4off[ri], constrained,
              s_win[wp], lane);
}

void launch_dp(const Blk& B, const Bat& T, int tfmsrc, int gap0, float gcost, int usess,
               int dpscan, int skipmode, int constrained, cudaStream_t st) {
    const int lmode = skipmode | (constrained ? DL_KEEPALN : 0);
    if (T.np <= LIST_SMALL) {
        k_list_small<LK_DP><<<1, 1024, 0, st>>>(B, T, lmode);
        GTB_LAUNCHED(T);
    } else {
        cudaMemsetAsync(T.rhist, 0, RL_NHIST * sizeof(int), st);
        const int nb = (T.np + 255) / 256;
        k_dlist_count<<<nb, 256, 0, st>>>(B, T, lmode);
        k_rlist_scan<<<1, 1024, 0, st>>>(T);
        k_dlist_fill<<<nb, 256, 0, st>>>(B, T, lmode);
        if (T.launches) (*T.launches) += 3;
    }
    KtScope kts(T, KF_DP, st);
    if (T.ndw > 0) {
        cudaMemsetAsync(T.dw_prog, 0, (size_t)T.dw_nprog * sizeof(int), st);
        if (usess == DP_SC_SSRR) launch_dp_wave<0, DP_SC_SSRR>(B, T, tfmsrc, gcost, dpscan, skipmode, st);
        else if (gap0 && !usess) launch_dp_wave<1, DP_SC_TFM>(B, T, tfmsrc, gcost, dpscan, skipmode, st);
        else if (!gap0 && !usess) launch_dp_wave<0, DP_SC_TFM>(B, T, tfmsrc, gcost, dpscan, skipmode, st);
        else if (!gap0 && usess) launch_dp_wave<0, DP_SC_TFMSS>(B, T, tfmsrc, gcost, dpscan, skipmode, st);
        else launch_dp_wave<1, DP_SC_TFMSS>(B, T, tfmsrc, gcost, dpscan, skipmode, st);
        GTB_LAUNCHED(T);
    }
    // dp_kc CTAs for the largest listed pairs, then a warp per pair
    const int nb = (T.dw_err ? T.dp_kc : 0) + (T.np + 3) / 4;
    if (usess == DP_SC_SSRR) k_dp<0, DP_SC_SSRR><<<nb, 128, 0, st>>>(B, T, tfmsrc, gcost, dpscan, constrained);
    else if (gap0 && !usess) k_dp<1, DP_SC_TFM><<<nb, 128, 0, st>>>(B, T, tfmsrc, gcost, dpscan, constrained);
    else if (!gap0 && !usess) k_dp<0, DP_SC_TFM><<<nb, 128, 0, st>>>(B, T, tfmsrc, gcost, dpscan, constrained);
    else if (!gap0 && usess) k_dp<0, DP_SC_TFMSS><<<nb, 128, 0, st>>>(B, T, tfmsrc, gcost, dpscan, constrained);
    else k_dp<1, DP_SC_TFMSS><<<nb, 128, 0, st>>>(B, T, tfmsrc, gcost, dpscan, constrained);
    GTB_LAUNCHED(T);
    if (T.ndw > 0) {
        k_btck<<<(T.np + BT_WARPS - 1) / BT_WARPS, BT_WARPS * 32, 0, st>>>(B, T, constrained);
        GTB_LAUNCHED(T);
    }
}

void launch_pair_list(const Blk& B, const Bat& T, int skipmask, cudaStream_t st) {
    if (T.np <= LIST_SMALL) {
        k_list_small<LK_PAIRS><<<1, 1024, 0, st>>>(B, T, skipmask);
        GTB_LAUNCHED(T);
        return;
    }
    cudaMemsetAsync(T.rhist, 0, RL_NHIST * sizeof(int), st);
    const int nb = (T.np + 255) / 256;
    k_plist_count<<<nb, 256, 0, st>>>(B, T, skipmask);
    k_rlist_scan<<<1, 1024, 0, st>>>(T);
    k_plist_fill<<<nb, 256, 0, st>>>(B, T, skipmask);
    if (T.launches) (*T.launches) += 3;
}

// Detailed search: the DP scores of a pair's fragment slots
// (ExecDPScore128xKernel, MpDPHub.cpp:389-645): for every slot with a
// positive score, the last cell of the gap-0 DP under the slot's transform
// (search d0), no traceback; 0 for the others.  A warp per (listed pair,
// slot) item, the items walked by a grid of resident warps in list order
// (largest pairs first); each slot's DP keeps its strip row in the pair's
// detailed-search region (the local score matrix is no longer read).
__global__ void __launch_bounds__(128) k_f3_dpscore(Blk B, Bat T) {
    __shared__ DpRing s_ring[4];
    const int lane = threadIdx.x & 31;
    DpRing& ring = s_ring[threadIdx.x >> 5];
    const int nsl = B.f3nsec * F3_NTOP;          // slots per pair
    const long long nitems = (long long)T.rhist[RL_NB] * nsl;
    const long long wstride = (long long)gridDim.x * (blockDim.x >> 5);
    for (long long it = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); it < nitems;
         it += wstride) {
        const int i = T.rlist[it / nsl];
        const int k = (int)(it % nsl);
        const float* sl = T.f3slot + ((long long)i * nsl + k) * 13;
        float* fin = T.f3dps + (long long)i * nsl + k;
        if (!(0.f < sl[0])) {
            if (lane == 0) *fin = 0.f;
            continue;
        }
        int qi = pair_qi(B, T, i), ri = pair_ri(B, T, i);
        int lq = B.qlen[qi], lr = B.rlen[ri];
        int ml = lq < lr ? lq : lr;
        const float d0 = B.t_d0[ml];
        const float d02 = __fmul_rn(d0, d0);
        const float* qx = B.qx + B.qoff[qi];
        const float* qy = B.qy + B.qoff[qi];
        const float* qz = B.qz + B.qoff[qi];
        const float4* q4 = B.q4 + B.q4off[qi];
        const float4* r4 = B.r4 + B.r4off[ri];
        float* row = (float*)(T.lsm + T.off_lsm[i]) + (long long)k * lr;
        float t[12];
#pragma unroll
        for (int f = 0; f < 12; f++) t[f] = sl[1 + f];
        if (lane == 0) work_add(T, WK_F3CELL, (unsigned long long)lq * (unsigned long long)lr);
        if (coords_ordinary(B, qi, ri)) {
            if (dp_r(lq) == 4)
                dp_pair_fast<4, true, DP_SC_TFM, false, true>(t, d02, 0.f, lq, lr, q4, r4, nullptr, nullptr, row,
                                                              nullptr, ring, lane, 0, 1, nullptr, nullptr,
                                                              DP_WAVE_SPIN_DEFAULT, fin);
            else
                dp_pair_fast<2, true, DP_SC_TFM, false, true>(t, d02, 0.f, lq, lr, q4, r4, nullptr, nullptr, row,
                                                              nullptr, ring, lane, 0, 1, nullptr, nullptr,
                                                              DP_WAVE_SPIN_DEFAULT, fin);
        } else if (dp_r(lq) == 4)
            dp_pair<4, true, DP_SC_TFM, false, true>(t, d02, 0.f, lq, lr, qx, qy, qz, r4, nullptr,
                                                     nullptr, nullptr, nullptr, row, nullptr, lane,
                                                     0, 1, nullptr, nullptr, DP_WAVE_SPIN_DEFAULT, fin);
        else
            dp_pair<2, true, DP_SC_TFM, false, true>(t, d02, 0.f, lq, lr, qx, qy, qz, r4, nullptr,
                                                     nullptr, nullptr, nullptr, row, nullptr, lane,
                                                     0, 1, nullptr, nullptr, DP_WAVE_SPIN_DEFAULT, fin);
        __syncwarp();
    }
}

void launch_f3_dpscore(const Blk& B, const Bat& T, cudaStream_t st) {
    // enough warps to fill the GPU (the kernel walks its items)
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const long long need = ((long long)T.np * B.f3nsec * F3_NTOP + 3) / 4;
    const int ng = (int)std::min<long long>(need, (long long)nsm * 8);
    k_f3_dpscore<<<ng > 0 ? ng : 1, 128, 0, st>>>(B, T);
    GTB_LAUNCHED(T);
}

// ---------------------------------------------------------------------------
// ---------------------------------------------------------------------------
// per-iteration bookkeeping of DPRefine: MpStage1.cpp:495-513 and
// CheckScoreConvergence / SaveLastScore0 / SetLowScoreConvergenceFlag
__global__ void k_post(Blk B, Bat T, int dpi, int maxit, int prescreen, float prescore) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= T.np) return;
    int flags = T.flags[i];
    float best = T.best[i];
    if (0 < dpi && !(flags & (CONV_SCOREDP | CONV_LOWTMSC)) &&
        fabsf(__fsub_rn(best, T.best0[i])) < SCORE_CONVEPS)
        flags |= CONV_SCOREDP;
    if (dpi + 1 < maxit && !(flags & (CONV_SCOREDP | CONV_LOWTMSC)))
        T.best0[i] = best;
    if (prescreen && maxit <= dpi + 1 && 0.0f < prescore) {
        int qi = pair_qi(B, T, i), ri = pair_ri(B, T, i);
        int lq = B.qlen[qi], lr = B.rlen[ri];
        int ml = lq < lr ? lq : lr;
        if (T.grand[i] < __fmul_rn(prescore, (float)ml)) flags |= CONV_LOWTMSC;
    }
    if (dpi == maxit - 1) flags &= ~CONV_SCOREDP;
    T.flags[i] = flags;
}

void launch_post(const Blk& B, const Bat& T, int dpi, int maxit, int prescreen, float prescore,
                 cudaStream_t st) {
    k_post<<<(T.np + 255) / 256, 256, 0, st>>>(B, T, dpi, maxit, prescreen, prescore);
    GTB_LAUNCHED(T);
}

__global__ void k_lowscore(Blk B, Bat T, float thr) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= T.np) return;
    int qi = pair_qi(B, T, i), ri = pair_ri(B, T, i);
    int lq = B.qlen[qi], lr = B.rlen[ri];
    int ml = lq < lr ? lq : lr;
    if (T.grand[i] < __fmul_rn(thr, (float)ml)) T.flags[i] |= CONV_LOWTMSC;
}

void launch_lowscore(const Blk& B, const Bat& T, float thr, cudaStream_t st) {
    k_lowscore<<<(T.np + 255) / 256, 256, 0, st>>>(B, T, thr);
    GTB_LAUNCHED(T);
}

// ---------------------------------------------------------------------------
// alignment rows: MpDPHub.cpp:1919-2125.  The rows of a pair with an
// alignment are packed at an offset it reserves (atomically) once its column
// count is known; that count follows from the first and last aligned pairs:
// every aligned pair is one column, every skipped query residue between them
// one, and every skipped reference residue one unless --no-deletions.
//
// A warp per pair, a lane per aligned pair: its columns (itself and the skipped
// residues up to the next aligned pair) start at the running sum of the columns
// before.  (A thread per pair wrote its rows byte by byte: 0.39 ms for a pair of
// 1,200 residues, 1.5 ms for 5,000.)
__global__ void __launch_bounds__(128) k_alnstr(Blk B, Bat T) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (i >= T.np) return;
    if (T.flags[i] & CONV_LOWTMSC) {
        if (T.str && lane == 0) T.str_off[i] = -1;      // no alignment
        return;
    }
    int qi = pair_qi(B, T, i), ri = pair_ri(B, T, i);
    const unsigned* aln = T.aln + T.off_aln[i];
    const int n = T.naln[i];
    float t[12];
#pragma unroll
    for (int f = 0; f < 12; f++) t[f] = T.tfm_gr[i * 12 + f];
    const float4* q4 = B.q4 + B.q4off[qi];
    const float4* r4 = B.r4 + B.r4off[ri];
    const unsigned char* qa = B.qa + B.qoff[qi];
    const unsigned char* ra = B.ra + B.roff[ri];
    const char* qs = B.qs + B.qoff[qi];
    const char* rs = B.rs + B.roff[ri];
    char* dst = nullptr;
    int W = 1;
    unsigned wf = 0, wl = 0;                             // first and last aligned pairs
    if (n > 0) { wf = aln[n - 1]; wl = aln[0]; }
    if (T.str) {
        int ncol = 0;
        if (n > 0) {
            const int qf = (int)(wf >> 16), rf = (int)(wf & 0xffffu);
            const int ql = (int)(wl >> 16), rl = (int)(wl & 0xffffu);
            ncol = n + (ql - qf + 1 - n) + (B.nodeletions ? 0 : (rl - rf + 1 - n));
        }
        W = ncol + 1;
        unsigned long long o = 0;
        if (lane == 0) {
            o = atomicAdd(T.str_cnt, 5ull * (unsigned long long)W);
            T.str_off[i] = (long long)o;
        }
        dst = T.str + __shfl_sync(FULL, o, 0);
    }
    int col = 0, psts = 0, idts = 0;                     // col: columns so far (every lane)
    for (int k0 = 0; k0 < n; k0 += 32) {
        const int k = k0 + lane;
        int q = 0, r = 0, gq = 0, gr = 0, wid = 0;
        if (k < n) {
            const unsigned wv = aln[n - 1 - k];
            q = (int)(wv >> 16); r = (int)(wv & 0xffffu);
            wid = 1;
            if (k + 1 < n) {
                const unsigned w1 = aln[n - 2 - k];
                gq = (int)(w1 >> 16) - q - 1;
                gr = B.nodeletions ? 0 : (int)(w1 & 0xffffu) - r - 1;
                wid += gq + gr;
            }
        }
        int end = wid;                                   // inclusive sum
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(FULL, end, o);
            if (lane >= o) end += v;
        }
        int c = col + end - wid;
        col += __shfl_sync(FULL, end, 31);
        if (k < n) {
            const float4 u = __ldg(q4 + q), v = __ldg(r4 + r);
            const int eq = dist2_tf(t, u.x, u.y, u.z, v.x, v.y, v.z) < 25.0f;
            psts += eq;
            const char a = (char)qa[q], b = (char)ra[r];
            char mc = eq ? '+' : ' ';
            if (a != '-' && a == b) { idts++; mc = eq ? a : (char)(a | 32); }
            if (dst) {
                dst[c] = a; dst[2 * W + c] = b; dst[3 * W + c] = qs[q]; dst[4 * W + c] = rs[r]; dst[W + c] = mc;
                c++;
                for (int e = q + 1; e <= q + gq; e++, c++) {
                    dst[c] = (char)qa[e]; dst[3 * W + c] = qs[e]; dst[2 * W + c] = '-'; dst[4 * W + c] = ' '; dst[W + c] = ' ';
                }
                for (int e = r + 1; e <= r + gr; e++, c++) {
                    dst[2 * W + c] = (char)ra[e]; dst[4 * W + c] = rs[e]; dst[c] = '-'; dst[3 * W + c] = ' '; dst[W + c] = ' ';
                }
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        psts += __shfl_xor_sync(FULL, psts, o);
        idts += __shfl_xor_sync(FULL, idts, o);
    }
    if (lane != 0) return;
    if (dst) { dst[col] = 0; dst[W + col] = 0; dst[2 * W + col] = 0; dst[3 * W + col] = 0; dst[4 * W + col] = 0; }
    T.out[i * 16 + 2] = __uint_as_float(n > 0 ? ((wf & 0xffffu) + 1) << 16 | ((wf >> 16) + 1) : 0u);
    T.out[i * 16 + 3] = __uint_as_float(n > 0 ? ((wl & 0xffffu) + 1) << 16 | ((wl >> 16) + 1) : 0u);
    T.out[i * 16 + 4] = (float)col;
    T.out[i * 16 + 5] = (float)psts;
    T.out[i * 16 + 6] = (float)idts;
    T.out[i * 16 + 7] = (float)(col - n);
}

void launch_alnstr(const Blk& B, const Bat& T, cudaStream_t st) {
    k_alnstr<<<(T.np + 3) / 4, 128, 0, st>>>(B, T);
    GTB_LAUNCHED(T);
}

// ---------------------------------------------------------------------------
// FP64 recomputation of the reported TM-scores and RMSD, --referenced
//
// A warp per pair: 32 aligned pairs at a time, a lane each, their score terms and
// coordinates go to shared memory; then lane f adds the 32 terms of sum f in
// position order (25 sums: scores by both lengths, without helix mismatches, 9
// products, 6 coordinates, 6 squares).  (A thread per pair: 860 cycles a
// position, 0.54 ms for a pair of 1,200 residues.)
constexpr int FN_WARPS = 4;
__global__ void __launch_bounds__(FN_WARPS * 32) k_final(Blk B, Bat T, int referenced) {
    __shared__ float s_x[FN_WARPS][7][33];               // q xyz, r xyz, 1
    __shared__ double s_t[FN_WARPS][4][33];              // score terms
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int i = blockIdx.x * FN_WARPS + wp;
    if (i >= T.np) return;
    if (T.flags[i] & CONV_LOWTMSC) return;
    int qi = pair_qi(B, T, i), ri = pair_ri(B, T, i);
    int lq = B.qlen[qi], lr = B.rlen[ri];
    const unsigned* aln = T.aln + T.off_aln[i];
    int n = T.naln[i];
    float* t = T.tfm_gr + i * 12;
    float* out = T.out + i * 16;
    if (n > 0) {
        const float4* q4 = B.q4 + B.q4off[qi];
        const float4* r4 = B.r4 + B.r4off[ri];
        const char *qs = B.qs + B.qoff[qi], *rs = B.rs + B.roff[ri];
        double d0q = (double)B.t_d0fin[lq], d0r = (double)B.t_d0fin[lr];
        double d0q2 = __dmul_rn(d0q, d0q), d0r2 = __dmul_rn(d0r, d0r);
        double td[12];
#pragma unroll
        for (int f = 0; f < 12; f++) td[f] = (double)t[f];
        // this lane's sum (0..20: a product of two components, 21..24: a term)
        const int ca = lane < 9 ? lane / 3 : lane < 15 ? lane - 9 : lane < 21 ? lane - 15 : 0;
        const int cb = lane < 9 ? 3 + lane % 3 : lane < 15 ? 6 : lane < 21 ? lane - 15 : 0;
        const float* X = s_x[wp][ca];
        const float* Y = s_x[wp][cb];
        const double* Z = s_t[wp][lane >= 21 && lane < 25 ? lane - 21 : 0];
        s_x[wp][6][lane] = 1.f;
        double sum = 0.0;
        for (int k0 = 0; k0 < n; k0 += 32) {
            const int k = k0 + lane;
            __syncwarp();
            if (k < n) {
                const unsigned wv = aln[n - 1 - k];
                const int q = (int)(wv >> 16), r = (int)(wv & 0xffffu);
                const float4 u = __ldg(q4 + q), v = __ldg(r4 + r);
                s_x[wp][0][lane] = u.x; s_x[wp][1][lane] = u.y; s_x[wp][2][lane] = u.z;
                s_x[wp][3][lane] = v.x; s_x[wp][4][lane] = v.y; s_x[wp][5][lane] = v.z;
                double qq[3] = {(double)u.x, (double)u.y, (double)u.z};
                double rr[3] = {(double)v.x, (double)v.y, (double)v.z};
                double x = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(td[0], qq[0]), __dmul_rn(td[1], qq[1])), __dmul_rn(td[2], qq[2])), td[9]);
                double y = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(td[3], qq[0]), __dmul_rn(td[4], qq[1])), __dmul_rn(td[5], qq[2])), td[10]);
                double z = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(td[6], qq[0]), __dmul_rn(td[7], qq[1])), __dmul_rn(td[8], qq[2])), td[11]);
                double dx = __dsub_rn(x, rr[0]), dy = __dsub_rn(y, rr[1]), dz = __dsub_rn(z, rr[2]);
                double d = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
                const double sq = __ddiv_rn(d0q2, __dadd_rn(d0q2, d));
                const double sr = __ddiv_rn(d0r2, __dadd_rn(d0r2, d));
                // MpStageBase.h:825-856: a helix aligned to a non-helix residue is
                // left out of the --2tm-score sums
                bool in2 = false;
                if (B.twotm) {
                    const char a2 = qs[q], b2 = rs[r];
                    in2 = !((a2 == 'h' || b2 == 'h') && a2 != b2);
                }
                s_t[wp][0][lane] = sq; s_t[wp][1][lane] = sr;
                s_t[wp][2][lane] = in2 ? sq : 0.0; s_t[wp][3][lane] = in2 ? sr : 0.0;
            }
            __syncwarp();
            const int cnt = n - k0 < 32 ? n - k0 : 32;
            if (lane < 21) {
#pragma unroll 8
                for (int e = 0; e < cnt; e++) sum = __dadd_rn(sum, __dmul_rn((double)X[e], (double)Y[e]));
            } else {
#pragma unroll 8
                for (int e = 0; e < cnt; e++) sum = __dadd_rn(sum, Z[e]);
            }
        }
        double dv[21];
#pragma unroll
        for (int f = 0; f < 21; f++) dv[f] = __shfl_sync(FULL, sum, f);
        const double tq = __shfl_sync(FULL, sum, 21), tr = __shfl_sync(FULL, sum, 22);
        const double t2q = __shfl_sync(FULL, sum, 23), t2r = __shfl_sync(FULL, sum, 24);
        if (lane == 0) {
            double r64 = rmsd_from_sums(dv, (double)n);
            float r32 = T.rmsd32[i];
            if (r32 >= 0.f) {
                T.err[i * 4 + 2] = (float)fabs(__dsub_rn((double)r32, r64));
                out[8] = (float)r64;
            }
            if (out[9] > 0.f || out[10] > 0.f) {
                double tmq = __ddiv_rn(tq, (double)lq), tmr = __ddiv_rn(tr, (double)lr);
                T.err[i * 4 + 0] = (float)fabs(__dsub_rn((double)out[9], tmq));
                T.err[i * 4 + 1] = (float)fabs(__dsub_rn((double)out[10], tmr));
                out[9] = (float)tmq;
                out[10] = (float)tmr;
            }
            if (B.twotm) {
                // secondary TM-scores (MpStageFin.cpp:1723-1818), FP64 like the primary ones
                out[13] = (float)__ddiv_rn(t2q, (double)lq);
                out[14] = (float)__ddiv_rn(t2r, (double)lr);
            }
        }
    }
    if (referenced && lane == 0) {
        float R[9];
#pragma unroll
        for (int f = 0; f < 9; f++) R[f] = t[f];
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
            for (int b = 0; b < 3; b++) t[3 * a + b] = R[3 * b + a];
        float t0 = t[9], t1 = t[10], t2 = t[11];
        t[9] = -__fadd_rn(__fadd_rn(__fmul_rn(R[0], t0), __fmul_rn(R[3], t1)), __fmul_rn(R[6], t2));
        t[10] = -__fadd_rn(__fadd_rn(__fmul_rn(R[1], t0), __fmul_rn(R[4], t1)), __fmul_rn(R[7], t2));
        t[11] = -__fadd_rn(__fadd_rn(__fmul_rn(R[2], t0), __fmul_rn(R[5], t1)), __fmul_rn(R[8], t2));
    }
}

void launch_final(const Blk& B, const Bat& T, int referenced, cudaStream_t st) {
    k_final<<<(T.np + FN_WARPS - 1) / FN_WARPS, FN_WARPS * 32, 0, st>>>(B, T, referenced);
    GTB_LAUNCHED(T);
}

// ---------------------------------------------------------------------------
// Per-length constants; the FP32 formulas of stagecnsts.cuh:48-175 (host).
void make_tables(float* d0, float* d82, float* d0fin, int n) {
    for (int L = 0; L < n; L++) {
        float l = (float)L;
        float a = 0.168f;
        if (l > 19.f) a = 1.24f * cbrtf(l - 15.f) - 1.8f;
        d0[L] = a + 0.8f;
        float d8 = 1.5f * powf(l, 0.3f) + 3.5f;
        d82[L] = d8 * d8;
        float f = 0.5f;
        if (l > 21.f) f = 1.24f * cbrtf(l - 15.f) - 1.8f;
        if (f < 0.5f) f = 0.5f;
        d0fin[L] = f;
    }
}

// DPRefine (MpStage1.cpp:466-517): maxit rounds of DP, traceback, fragment
// refinement over the alignment and the convergence bookkeeping; the first
// DP uses the transform tfm1 (DP_TFM_IBEST, or DP_TFM_2ND after the detailed
// search, WRKMEMTM1)
void launch_dprefine(const Blk& B, const Bat& T, int gap0, int prescreen, int maxit,
                     float prescore, bool few, int tfm1, cudaStream_t st) {
    for (int dpi = 0; dpi < maxit; dpi++) {
        launch_dp(B, T, dpi == 0 ? tfm1 : DP_TFM_IBEST, gap0, gap0 ? 0.0f : -0.6f, 0, 0, 0, 0, st);
        launch_refine(RM_DP, B, T, st, few);
        launch_post(B, T, dpi, maxit, prescreen, prescore, st);
    }
}

// ---------------------------------------------------------------------------
// The stage sequence of one batch: CuBatch::ProcessBlock (CuBatch.cu:537-700)
// with the detailed search off.  ev (may be null): 5 events recorded at the
// stage boundaries.
void launch_stages(const Blk& B, const Bat& T, int refinement, int depth, int convergence,
                   float prescore, int referenced, float scorethld, cudaStream_t st,
                   cudaEvent_t* ev, int polish_steps) {
    auto mark = [&](int k) { if (ev) cudaEventRecord(ev[k], st); };
    // DPRefine: MpStage1.cpp:466-517
    // after the stage-1 --pre-score filter only a small share of pairs is left
    const bool few = 0.0f < prescore;
    auto dprefine = [&](int gap0, int prescreen, int maxit, bool fewp) {
        launch_dprefine(B, T, gap0, prescreen, maxit, prescore, fewp, DP_TFM_IBEST, st);
    };
    mark(0);
    launch_init(B, T, st);
    if (B.presim > 0.f) launch_presim(B, T, st);
    launch_findfrag(B, T, st);
    mark(1);
    launch_refine(RM_INIT, B, T, st, false);
    mark(2);
    dprefine(1, 1, 2, false);
    if (B.addss) {
        // --add-search-by-ss (custage_ssrr.cu:43-140, CuBatch.cu:583-600): the
        // alignment of the SS and residue-scored DP, fragment refinement over it,
        // DP refinement with the gap cost and without, 2 iterations each
        launch_dp(B, T, DP_TFM_GRAND, 0, -1.0f, DP_SC_SSRR, 0, 1, 0, st);
        launch_refine(RM_DP, B, T, st, few);
        dprefine(0, 0, 2, few);
        dprefine(1, 0, 2, few);
    }
    // the spatial-index detailed search (CuBatch.cu:612-623)
    if (B.f3) launch_frg3(B, T, st);
    // two stage-2 passes: MpStage2.h:63-83, CuBatch.cu:627-650
    for (int call = 0; call < 2; call++) {
        int gap0 = call == 1;
        launch_dp(B, T, DP_TFM_GRAND, gap0, gap0 ? 0.0f : -1.0f, !gap0, !gap0, 1, 0, st);
        launch_refine(RM_DP, B, T, st, few);
        dprefine(0, 0, 2, few);
        dprefine(1, 0, call == 0 ? 2 : convergence, few);
        if (call == 1 && 0.0f < scorethld) launch_lowscore(B, T, scorethld, st);
    }
    mark(3);
    // final stage: MpStageFin.h:63-96
    launch_dp(B, T, DP_TFM_GRAND, 1, 0.0f, 0, 0, 1, 0, st);
    launch_refine(RM_FIN1, B, T, st, few);
    if (!(depth == 3 || refinement == GTB_REFINEMENT_COARSE)) launch_refine(RM_FIN2, B, T, st, few);
    launch_dp(B, T, DP_TFM_GRAND, 1, 0.0f, 0, 0, 1, 1, st);
    launch_alnstr(B, T, st);
    launch_refine(RM_PROD1, B, T, st, few);
    if (refinement == GTB_REFINEMENT_LOG) {
        // MpStageFin.h:421-434: the log search, one launch per step
        Bat TL = T;
        for (int r = 0; r < PLOG_ROUNDS; r++) {
            TL.plog_round = r;
            launch_refine(RM_PLOG, B, TL, st, few);
        }
    } else {
        launch_refine(RM_PROD2, B, T, st, few);
    }
    launch_polish_final(B, T, polish_steps, st);
    launch_final(B, T, referenced, st);
    mark(4);
}

}  // namespace gtb
