// gtb_frg3.cu -- the spatial-index detailed search on sm_100a.
//
// The stage MpStageFrg3::Run (src/libmymp/mpstage1/MpStageFrg3.h:80-115,
// MpStageFrg3.cpp:35-469; GPU form custage1/custage_frg3.cu:54-560) between
// stage 1 and stage 2, for every pair that is not filtered out, each pair as
// if alone in its chunk:
//  1. a local alignment of the two structures by secondary structure, kept
//     as one score byte per cell (k_f3_localdp);
//  2. a grid of configurations (query position x reference position, steps
//     by length and --depth): those whose local score passes the --trigger
//     test are seeded by the local alignment through a cell of the
//     configuration (or by a gapless fragment, --seedrule 0), superposed, and
//     twice re-aligned by each residue's nearest neighbour in the other
//     structure's 3-d tree (first among residues of the same secondary
//     structure) and re-superposed; the final superposition's order-dependent
//     score goes to fragment slot (configuration count mod 32), which keeps
//     its best (k_f3_search, a cluster per pair);
//  3. each slot's transform is scored by a gap-0 DP (k_f3_dpscore), the
//     slots ordered by that score, and the best --nbranches refined by DP +
//     fragment refinement (the stage-1 kernels), keeping the best branch;
//  4. two DP refinements start from the best branch.
// Numeric form as elsewhere: FP32 with explicit FMAs, covariance sums over
// position slots in blocks of 32 reduced by xor-shuffle trees and folded into
// Neumaier totals, FP64 rotation solve.  Bit-identical to the oracle's
// frg3_stage.
#include <algorithm>
#include <cooperative_groups.h>
#include "gtb200.h"
#include "gtb_device.cuh"
#include "gtb_kernels.cuh"

namespace gtb {

namespace {

constexpr int F3_MAXVISIT = 64;     // CUSF_TBSP_INDEX_SCORE_MAXDEPTH
constexpr int F3_HASH = 512;        // CUSF_TBSP_INDEX_SCORE_POSLIMIT2
constexpr int F3_SIMROWS = 96;      // MPSF_TBSP_LOCAL_SIMILARITY_YDIM x 3
constexpr int F3_SIMCOLS = 128;     // MPSF_TBSP_LOCAL_SIMILARITY_XDIM
constexpr int F3_MAXSTACK = 17;
constexpr int F3_LENTHR = 150;      // MpStageFrg3.cpp:48: longer structures thin the sections
constexpr float F3_SSDST2 = 64.f;   // an SS-matched neighbour farther than 8 A is none
constexpr int F3_MAXWIN = 512;      // the largest --window
constexpr int F3_WARPS = 4;         // warps per CTA of the search
// CTAs per pair of the search (a cluster) by the pairs of the batch: 8, 4, else
// 2.  More spread a pair wider, fewer wait less for one another at a round's end.
// The stage's own kernels with 8, 4, 2 and 1: one query against 250, 1,000 and
// 4,000 references, 2 to 5% of them left by the score filter, 2.5, 4.1, 7.3, 13.9
// and 3.3, 5.0, 9.0, 16.2 and 8.4, 8.2, 9.7, 17.1 ms; all pairs searched, 100, 256,
// 1,600, 4,096 and 8,100 of them, 2.9, 2.9, 4.6, 8.0 and 5.6, 5.1, 5.6, 9.0 and 28.6, 26.6,
// 25.5, 26.5 and 73, 67, 61, 61 and 118, 105, 97, 96.  The lines lie between the two:
// the batch's pairs are known here, those left are not.
constexpr int F3_NP8 = 256, F3_NP4 = 4096;
constexpr int F3_GRID = 592;        // CTAs of the search at most (4 per SM)
constexpr int F3_ENT = 256;         // results of a round (configuration x fragment)
constexpr unsigned short F3_NONE = 0xffff;   // no residue (an index is below 65535)
struct F3Walk {                     // a warp's tree walks
    float diff[F3_MAXSTACK * 32];
    unsigned short node[F3_MAXSTACK * 32];
    unsigned char dim[F3_MAXSTACK * 32];
};
struct F3Chain {                    // a warp's chain score
    float max[F3_HASH], ndx[F3_HASH];
};
struct alignas(16) F3Smem {
    unsigned short pq[F3_WARPS][F3_MAXWIN], pr[F3_WARPS][F3_MAXWIN];
    union { F3Walk walk; F3Chain chain; } u[F3_WARPS];   // never both at once
    // in the cluster's first CTA: the next configuration of the round, per
    // entry scored (1) or not, and score and transform
    int next, slot;
    unsigned char got[F3_ENT];
    unsigned short list[F3_ENT];    // the scored entries, in order
    float res[F3_ENT * 13];
};

__device__ __forceinline__ int pair_q(const Blk& B, const Bat& T, int i) { return (int)((T.p0 + i) / B.nr); }
__device__ __forceinline__ int pair_r(const Blk& B, const Bat& T, int i) { return (int)((T.p0 + i) % B.nr); }

// ---------------------------------------------------------------------------
// 1. Local alignment by secondary structure (ExecDPSSLocal128xKernel,
// MpDPHub.cpp:1256-1480): +1 for equal, -1 for different SS, floored at 0
// (STOP), gap cost per step; the byte per cell is the truncated score
// rounded down to a multiple of 4 (mod 256) with the direction in its low
// two bits.  A CTA per pair; its warps run the strips of 32 rows (a row per
// lane) along anti-diagonals as a wavefront: strip s on warp s mod 4, 32 steps
// at a time, each chunk waiting (a bounded spin) until the previous strip has
// left the row values it reads in the pair's row buffer.  A chunk's bytes are
// kept in shared memory and written a row at a time; the columns' letters and
// the previous strip's row move from lane to lane.  What bounds it: the chain of
// steps.  (One warp a pair storing a byte per lane and row at each step, with the
// row buffer read in the chain: 4.3 ms for 2 x 3,000 references; now 1.1.)
__global__ void __launch_bounds__(F3_WARPS * 32) k_f3_localdp(Blk B, Bat T) {
    __shared__ volatile int s_prog[F3_WARPS];            // chunks done: strip * nchunks + chunk
    __shared__ unsigned char s_tile[F3_WARPS][32 * 36];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int slot = blockIdx.x;
    if (slot >= T.rhist[RL_NBUCKET]) return;             // the same for the whole CTA
    const int i = T.rlist[slot];
    const int qi = pair_q(B, T, i), ri = pair_r(B, T, i);
    const int lq = B.qlen[qi], lr = B.rlen[ri];
    const char* qs = B.qs + B.qoff[qi];
    const char* rs = B.rs + B.roff[ri];
    unsigned char* m = T.lsm + T.off_lsm[i];
    float* row = T.row + T.off_row[i];
    volatile int* err = T.dw_err;
    const float g = B.f3gapcost;
    const int nstrips = (lq + 31) >> 5, nchunks = (lr + 31 + 31) >> 5;
    if (threadIdx.x < F3_WARPS) s_prog[threadIdx.x] = 0;
    __syncthreads();
    unsigned char* tile = s_tile[w];
    for (int s = w; s < nstrips; s += F3_WARPS) {
        const int y = s * 32 + lane;
        const bool valid = y < lq;
        const char qss = valid ? qs[y] : 0;
        float h = 0.f;          // this lane's cell of the previous step: (y, j-1)
        float uplast = 0.f;     // (y-1, j-1)
        int css = 0;            // the letter of this lane's column
        for (int c = 0; c < nchunks; c++) {
            const int t0 = c * 32;
            if (s > 0) {
                // row[t0 .. t0+31] of strip s-1: written up to its step t0+62
                const int need = (s - 1) * nchunks + (c + 2 < nchunks ? c + 2 : nchunks);
                int ok = 1;
                if (lane == 0) {
                    long long it = 0;
                    while (s_prog[(w + F3_WARPS - 1) % F3_WARPS] < need) {
                        if (*err || ++it > T.dw_spin) { *err = 1; ok = 0; break; }
                        __nanosleep(32);
                    }
                }
                if (!__shfl_sync(FULL, ok, 0)) return;
                // lane 0's look at the counter before every lane's reads of the
                // row (a shuffle alone orders no memory)
                __syncwarp();
                __threadfence_block();
            }
            const int jj = t0 + lane;
            const float rb = s > 0 && jj < lr ? row[jj] : 0.f;
            const int cb = jj < lr ? rs[jj] : 0;
            __syncwarp();
#pragma unroll 8
            for (int u = 0; u < 32; u++) {
                const int j = t0 + u - lane;
                const float r0 = __shfl_sync(FULL, rb, u);
                const int c0 = __shfl_sync(FULL, cb, u);
                float up = __shfl_up_sync(FULL, h, 1);          // lane-1's (y-1, j)
                css = __shfl_up_sync(FULL, css, 1);
                if (lane == 0) { up = r0; css = c0; }
                if (0 <= j && j < lr) {
                    float v = __fadd_rn(__fsub_rn((float)((qss == (char)css) * 2), 1.0f), j > 0 ? uplast : 0.f);
                    int bk = BT_DIAG;
                    if (v < 0.f) { v = 0.f; bk = BT_STOP; }
                    const float l = __fadd_rn(j > 0 ? h : 0.f, g);
                    if (v < l) { v = l; bk = BT_LEFT; }
                    const float x = __fadd_rn(up, g);
                    if (v < x) { v = x; bk = BT_UP; }
                    h = v;
                    tile[lane * 36 + u] = (unsigned char)((((unsigned)v) & 0xfcu) | (unsigned)bk);
                    // lane 31's row is the next strip's "up"
                    if (lane == 31) row[j] = v;
                }
                uplast = up;
            }
            __syncwarp();
            // row r's bytes of this chunk: columns t0 - r ...
            const int nrow = lq - s * 32 < 32 ? lq - s * 32 : 32;
#pragma unroll 4
            for (int r = 0; r < nrow; r++) {
                const int j = t0 - r + lane;
                if (0 <= j && j < lr) m[(long long)(s * 32 + r) * lr + j] = tile[r * 36 + lane];
            }
            __syncwarp();
            if (lane == 31) {
                __threadfence_block();                   // the row values before the count
                s_prog[w] = s * nchunks + c + 1;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// 2. The configurations of a pair.

// fragment lengths (GetNAlnPoss_frg, covariancebase.h:93-110)
__device__ __forceinline__ int f3_fraglen(int lq, int lr, int fi, int seedrule) {
    const int minlen = lq < lr ? lq : lr;
    const int half = minlen >> 1;
    if (seedrule) return seedrule < half ? seedrule : half;
    if (fi == 0) {
        int leno3 = (int)__fmul_rn((float)minlen, 1.0f / 3.0f);
        if (leno3 < 1) leno3 = 1;
        return leno3 < 20 ? leno3 : 20;
    }
    return half < 100 ? half : 100;
}

// configuration position step (GetFragStepSize_frg_*, covariancebase.h:22-84)
__device__ __forceinline__ int f3_step(int depth, int len) {
    int leno3 = (int)__fmul_rn((float)len, 1.0f / 3.0f);
    if (leno3 < 1) leno3 = 1;
    const int small = leno3 < 15 ? leno3 : 15;
    if (depth == 0) return len > 150 ? 15 : small;
    if (depth == 1) return len > 150 ? 23 : small;
    const int med = len > 250 ? 45 : len > 200 ? 35 : len > 150 ? 25 : small;
    return depth == 2 ? med : 2 * med;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// the xor-shuffle tree sum of a warp (every lane gets it)
__device__ __forceinline__ float tree32(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// The local similarity test (CalcLocalSimilarity2_frg2,
// MpStageFrg3.h:327-415): the largest score byte over 96 rows from qrypos
// and up to 128 columns from rfnpos (rounded up to a multiple of 4) reaches
// the fragment length x the trigger fraction.
__device__ bool f3_similar(const unsigned char* m, int lq, int lr, int qrypos, int rfnpos, int fl,
                           float thr, int lane) {
    if (lq < qrypos + fl) fl = lq - qrypos;
    if (lr < rfnpos + fl) fl = lr - rfnpos;
    int pidelta = (lr - 3 - rfnpos) & ~3;
    if (pidelta > F3_SIMCOLS) pidelta = F3_SIMCOLS;
    const int pibeg = (rfnpos + 3) & ~3;
    unsigned mx = 0;
    for (int ii = 0; qrypos + ii < lq && ii < F3_SIMROWS; ii++) {
        const unsigned char* rowp = m + (long long)(qrypos + ii) * lr + pibeg;
        for (int c = lane; c < pidelta; c += 32) {
            const unsigned v = rowp[c] & 0xfcu;
            mx = v > mx ? v : mx;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned w = __shfl_xor_sync(0xffffffffu, mx, o);
        mx = w > mx ? w : mx;
    }
    return !(__fmul_rn((float)fl, thr) > (float)mx);
}

// Seed from the local alignment (CalcCCMatricesLocallyAligned_Complete,
// MpStage1.h:395-470), on lane 0: of 4 evenly spaced cells the first with
// the largest byte, the local alignment traced back from it inside the
// rectangle from (qrypos, rfnpos); the pairs go to pq/pr in increasing order.
// Returns their number (0: too few), the same on every lane.
__device__ int f3_seed_local(const unsigned char* m, int lq, int lr, int trig, int fraglen,
                             int qrypos, int rfnpos, unsigned short* pq,
                             unsigned short* pr, int lane) {
    int n = 0;
    if (lane == 0) {
        if (lq < qrypos + fraglen && lr < rfnpos + fraglen)
            fraglen = (lq - qrypos) > (lr - rfnpos) ? (lq - qrypos) : (lr - rfnpos);
        fraglen >>= 2;
        int y = qrypos, x = rfnpos;
        float vr = 0.f;
        for (int f = 0; f < 4; f++) {
            int yt = qrypos + (f + 1) * fraglen, xt = rfnpos + (f + 1) * fraglen;
            yt = yt < lq - 1 ? yt : lq - 1;
            xt = xt < lr - 1 ? xt : lr - 1;
            const float vrt = (float)(m[(long long)yt * lr + xt] & 0xfcu);
            if (vr < vrt) { vr = vrt; y = yt; x = xt; }
        }
        while (y >= qrypos && x >= rfnpos && n < F3_MAXWIN) {
            const int b = m[(long long)y * lr + x] & 3;
            if (b == BT_STOP) break;
            if (b == BT_UP) { y--; continue; }
            if (b == BT_LEFT) { x--; continue; }
            pq[n] = (unsigned short)y; pr[n] = (unsigned short)x; n++;
            x--; y--;
        }
        const int minf = fraglen < 16 ? fraglen : 16;
        if (n < 1 || (trig && n < minf)) n = 0;
        for (int a = 0, b = n - 1; a < b; a++, b--) {
            unsigned short t = pq[a]; pq[a] = pq[b]; pq[b] = t;
            t = pr[a]; pr[a] = pr[b]; pr[b] = t;
        }
    }
    __syncwarp();
    return __shfl_sync(0xffffffffu, n, 0);
}

// Covariance sums over position slots 0..n-1 (pq/pr; F3_NONE: no
// pair): lane k of block b takes slot 32b + k; each block's values are
// summed by the xor-shuffle tree and folded into Neumaier totals in block
// order.  Every lane gets the 16 values (15 sums and the count).
__device__ void f3_cov(const float* qx, const float* qy, const float* qz, const float* rx,
                       const float* ry, const float* rz, const unsigned short* pq,
                       const unsigned short* pr, int n, float* v, int lane) {
    float s[15], c[15];
#pragma unroll
    for (int f = 0; f < 15; f++) { s[f] = 0.f; c[f] = 0.f; }
    int cnt = 0;
    for (int b0 = 0; b0 < n; b0 += 32) {
        const int k = b0 + lane;
        const int a = k < n ? pq[k] : F3_NONE, b = k < n ? pr[k] : F3_NONE;
        const bool ok = a != F3_NONE && b != F3_NONE;
        const float x0 = ok ? qx[a] : 0.f, y0 = ok ? qy[a] : 0.f, z0 = ok ? qz[a] : 0.f;
        const float x1 = ok ? rx[b] : 0.f, y1 = ok ? ry[b] : 0.f, z1 = ok ? rz[b] : 0.f;
        float t[15] = {__fmul_rn(x0, x1), __fmul_rn(x0, y1), __fmul_rn(x0, z1),
                       __fmul_rn(y0, x1), __fmul_rn(y0, y1), __fmul_rn(y0, z1),
                       __fmul_rn(z0, x1), __fmul_rn(z0, y1), __fmul_rn(z0, z1),
                       x0, y0, z0, x1, y1, z1};
#pragma unroll
        for (int f = 0; f < 15; f++) {
            float bs = tree32(t[f]);
            nfold(s[f], c[f], bs);
        }
        cnt += __popc(__ballot_sync(0xffffffffu, ok));
    }
#pragma unroll
    for (int f = 0; f < 15; f++) v[f] = __fadd_rn(s[f], c[f]);
    v[15] = (float)cnt;
}

// Nearest neighbour in a structure's 3-d tree (NNByIndex*,
// MpStageFrg3.h:1270-1440): depth first with a bounded stack, at most 64
// nodes visited; with ssfilt only residues of secondary structure ss count
// and one farther than 8 A is none.  Returns the residue or -1.  Nodes are
// packed (k_pack_nodes): nd = (x, y, z, residue | SS << 16), nc = (left,
// right).  The stack is the lane's column of a shared-memory array (entry q
// at [q * 32]).
__device__ int f3_nn(const float4* nd, const int2* nc, int len, bool ssfilt, char ss, float px,
                     float py, float pz, int stacksize, unsigned short* stk_node, float* stk_diff,
                     unsigned char* stk_dim) {
    int sp = 0, nvisited = 0, best = -1, root = len >> 1, dim = 0;
    float bestd = 9.9e6f;
    while (0 < sp || 0 <= root) {
        if (0 <= root) {
            nvisited++;
            if (F3_MAXVISIT <= nvisited) break;
            const float4 n = __ldg(nd + root);
            const int2 ch = __ldg(nc + root);
            const int ow = __float_as_int(n.w);
            const int org = ow & 0xffff;
            const float dx = __fsub_rn(n.x, px), dy = __fsub_rn(n.y, py), dz = __fsub_rn(n.z, pz);
            const float d2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
            if ((best < 0 || d2 < bestd) && (!ssfilt || (char)(ow >> 16) == ss)) {
                bestd = d2;
                best = org;
            }
            if (bestd == 0.0f) break;
            const float diffc = dim == 0 ? dx : (dim == 1 ? dy : dz);
            if (2 < ++dim) dim = 0;
            if (sp < stacksize) {
                stk_node[sp * 32] = (unsigned short)root;    // a node index is below 65536
                stk_dim[sp * 32] = (unsigned char)dim;
                stk_diff[sp * 32] = diffc;
                sp++;
            }
            root = (0.0f < diffc) ? ch.x : ch.y;
        } else {
            bool cond = false;
            float diffc = 0.f;
            while (0 < sp && !cond) {
                sp--;
                root = stk_node[sp * 32]; dim = stk_dim[sp * 32]; diffc = stk_diff[sp * 32];
                cond = __fmul_rn(diffc, diffc) < bestd;
            }
            if (!cond) break;
            const int2 ch = __ldg(nc + root);
            root = (0.0f < diffc) ? ch.y : ch.x;
        }
    }
    if (ssfilt) return F3_SSDST2 < bestd ? -1 : best;
    return best;
}

// per-pair view of the search's inputs
struct F3Pair {
    int lq, lr;
    const float *qx, *qy, *qz, *rx, *ry, *rz;
    const char *qs, *rs;
    const float4 *qnd, *rnd;
    const int2 *qnc, *rnc;
};

// Neighbours over the window of the shorter structure
// (ProduceAlignmentUsingIndex2Reference/Query, MpStageFrg3.h:500-680), a
// window slot per lane per round; fills pq/pr (F3_NONE: empty), returns the
// window length.
__device__ int f3_window(const F3Pair& P, const float* tfm, bool ssfilt, int window, int qrypos,
                         int rfnpos, int stacksize, unsigned short* pq, unsigned short* pr, int lane,
                         unsigned short* sn, float* sd, unsigned char* sm) {
    const int lq = P.lq, lr = P.lr;
    int n;
    if (lq < lr) {
        const int fl = lr < window ? lr : window;
        int qp = qrypos - (fl >> 1); if (qp < 0) qp = 0;
        const int ql = qp + fl < lq ? qp + fl : lq;
        qp = ql - fl; if (qp < 0) qp = 0;
        n = ql - qp;
        for (int pi = lane; pi < n; pi += 32) {
            const int q = qp + pi;
            float x, y, z;
            xform(tfm, P.qx[q], P.qy[q], P.qz[q], x, y, z);
            const int r = f3_nn(P.rnd, P.rnc, lr, ssfilt, P.qs[q], x, y, z, stacksize, sn, sd, sm);
            pq[pi] = (unsigned short)q;
            pr[pi] = r > 0 ? (unsigned short)r : F3_NONE;
        }
    } else {
        const int fl = lq < window ? lq : window;
        int rp = rfnpos - (fl >> 1); if (rp < 0) rp = 0;
        const int rl = rp + fl < lr ? rp + fl : lr;
        rp = rl - fl; if (rp < 0) rp = 0;
        n = rl - rp;
        for (int pi = lane; pi < n; pi += 32) {
            const int r = rp + pi;
            float x, y, z;
            xform(tfm, P.rx[r], P.ry[r], P.rz[r], x, y, z);
            const int q = f3_nn(P.qnd, P.qnc, lq, ssfilt, P.rs[r], x, y, z, stacksize, sn, sd, sm);
            pq[pi] = q > 0 ? (unsigned short)q : F3_NONE;
            pr[pi] = (unsigned short)r;
        }
    }
    __syncwarp();
    return n;
}

// The order-dependent score (CalcScoresUnrl_SWFTscanProgressive_Complete,
// MpStageFrg3.h:760-850) over the first cnt window slots: each pair extends
// the best chain of earlier-partnered pairs kept in a 512-entry table hashed
// by partner index; lanes share the table scan, lane 0 updates it.
//
// When the partner structure has at most F3_HASH residues no two partners
// share an entry, so an entry only ever rises (to the larger chain score of
// its own partner) and the scan "best entry with a lower partner" is the
// running maximum of the entries below the partner's: the table is then
// kept as prefix maxima (pm[k] = max of entries 0..k), read with one load
// and raised by every lane for its own entries at or above the partner's.
__device__ float f3_progressive(const F3Pair& P, const float* tfm, float d02, const unsigned short* pq,
                                const unsigned short* pr, int cnt, bool partner_is_r, float* omax,
                                float* ondx, int lane) {
    if ((partner_is_r ? P.lr : P.lq) <= F3_HASH) {
        float* pm = omax;
        for (int k = lane; k < F3_HASH; k += 32) pm[k] = 0.f;
        __syncwarp();
        for (int pi = 0; pi < cnt; pi++) {
            const int a = pq[pi], b = pr[pi];
            if (a == F3_NONE || b == F3_NONE) continue;   // the same on every lane
            const float d = dist2_tf(tfm, P.qx[a], P.qy[a], P.qz[a], P.rx[b], P.ry[b], P.rz[b]);
            const float sco = tmterm(d02, d);
            if (!(0.f < sco)) continue;
            const int c = partner_is_r ? b : a;
            const float mx = c > 0 ? pm[c - 1] : 0.f;
            const float nsc = __fadd_rn(mx, sco);
            __syncwarp();
            for (int k = c + ((lane - c) & 31); k < F3_HASH; k += 32) pm[k] = fmaxf(pm[k], nsc);
            __syncwarp();
        }
        const float mx = pm[F3_HASH - 1];
        __syncwarp();
        return mx;
    }
    for (int k = lane; k < F3_HASH; k += 32) { omax[k] = 0.f; ondx[k] = -1.f; }
    __syncwarp();
    for (int pi = 0; pi < cnt; pi++) {
        const int a = pq[pi], b = pr[pi];
        if (a == F3_NONE || b == F3_NONE) continue;   // the same on every lane
        const float d = dist2_tf(tfm, P.qx[a], P.qy[a], P.qz[a], P.rx[b], P.ry[b], P.rz[b]);
        const float sco = tmterm(d02, d);
        if (!(0.f < sco)) continue;
        const float qnx = (float)(partner_is_r ? b : a);
        float mx = 0.f;
        for (int k = lane; k < F3_HASH; k += 32)
            if (ondx[k] < qnx && mx < omax[k]) mx = omax[k];
        mx = warp_max(mx);
        if (lane == 0) {
            const int c = (int)qnx & (F3_HASH - 1);
            const float st = ondx[c], ss = omax[c], nsc = __fadd_rn(mx, sco);
            const bool half2nd = pi > (cnt >> 1);
            if (st < 0.f || (st == qnx && ss < nsc) || ((half2nd && st < qnx) || (!half2nd && qnx < st))) {
                ondx[c] = qnx;
                omax[c] = nsc;
            }
        }
        __syncwarp();
    }
    float mx = 0.f;
    for (int k = lane; k < F3_HASH; k += 32) mx = mx < omax[k] ? omax[k] : mx;
    mx = warp_max(mx);
    __syncwarp();
    return mx;
}

__device__ __forceinline__ int f3_stacksize(int lq, int lr) {
    const int L = lq > lr ? lq : lr;
    int b = L > 1 ? 32 - __clz(L - 1) : 0;    // ceil(log2 L)
    b += 1;
    return b < F3_MAXSTACK ? b : F3_MAXSTACK;
}

__device__ __forceinline__ void f3_sync(cooperative_groups::cluster_group& cl, int C) {
    if (C > 1) cl.sync();
    else __syncthreads();
}

// A cluster of CTAs per listed pair (the grid's clusters walk the list,
// largest pairs first).  A round is F3_ENT consecutive entries (configuration
// x fragment); the cluster's warps draw the round's configurations one at a
// time and leave their results in the first CTA's shared memory.  A scored
// entry's slot is the pair's count of scored entries before it mod 32, and the
// slot keeps its best: after the round, lane j of one warp goes through the
// entries of slot j in order, as one warp going through all configurations
// would.  What bounds it: the latency of the tree walks.  With one CTA a pair
// and rounds of 16 configurations a launch lasted as long as its largest pair,
// SMs busy a fifth of the time: the stage's own kernels took 50 ms for 2 x 3,000
// references, now 20; for 2 x 8,000 68 ms, now 36 (with 3 CTAs a SM 66).
__global__ void __launch_bounds__(F3_WARPS * 32, 4) k_f3_search(Blk B, Bat T, int depth) {
    extern __shared__ __align__(16) unsigned char f3_smem[];
    F3Smem& S = *(F3Smem*)f3_smem;
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const int C = (int)cl.num_blocks(), crank = (int)cl.block_rank();
    F3Smem& S0 = *cl.map_shared_rank(&S, 0);       // the first CTA's
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned short* pq = S.pq[w];
    unsigned short* pr = S.pr[w];
    unsigned short* sn = S.u[w].walk.node + lane;
    float* sd = S.u[w].walk.diff + lane;
    unsigned char* sm = S.u[w].walk.dim + lane;
    const int nlist = T.rhist[RL_NBUCKET], ncl = (int)gridDim.x / C;
    int* ctr = T.rhist + RL_NBUCKET + 1;
    for (int slot = (int)blockIdx.x / C; slot < nlist;) {
        const int i = T.rlist[slot];
        const int qi = pair_q(B, T, i), ri = pair_r(B, T, i);
        F3Pair P;
        P.lq = B.qlen[qi]; P.lr = B.rlen[ri];
        const int qo = B.qoff[qi], ro = B.roff[ri];
        P.qx = B.qx + qo; P.qy = B.qy + qo; P.qz = B.qz + qo;
        P.rx = B.rx + ro; P.ry = B.ry + ro; P.rz = B.rz + ro;
        P.qs = B.qs + qo; P.rs = B.rs + ro;
        P.qnd = B.qnd + qo; P.qnc = B.qnc + qo;
        P.rnd = B.rnd + ro; P.rnc = B.rnc + ro;
        const int lq = P.lq, lr = P.lr;
        const int ml = lq < lr ? lq : lr;
        const float d0 = B.t_d0[ml];
        const float d02 = __fmul_rn(d0, d0);
        const unsigned char* m = T.lsm + T.off_lsm[i];
        const int nsec = B.f3nsec;
        float* slots = T.f3slot + (long long)i * nsec * F3_NTOP * 13;
        if (crank == 0)
            for (int k = threadIdx.x; k < nsec * F3_NTOP; k += blockDim.x) slots[k * 13] = 0.f;
        const float thr = __fdiv_rn((float)B.f3trigger, 100.0f);
        const int seedrule = B.f3seedrule;
        const int qstep = f3_step(depth, lq), rstep = f3_step(depth, lr);
        const int minn = depth == 3 ? 5 : 10;
        int nsy = lq / qstep + 1; if (nsy < minn) nsy = minn;
        int nsx = lr / rstep + 1; if (nsx < minn) nsx = minn;
        const int nconf = nsy * nsx;
        const int stacksize = f3_stacksize(lq, lr);
        const int f0 = f3_fraglen(lq, lr, 0, 0), f1 = f3_fraglen(lq, lr, 1, 0);
        const int nfr = seedrule ? 1 : 2;
        const int rconf = F3_ENT / nfr;               // configurations of a round
        int nscored = 0;                              // kept by the first CTA's first warp
        for (int c0 = 0; c0 < nconf; c0 += rconf) {
            const int nc = nconf - c0 < rconf ? nconf - c0 : rconf;
            if (crank == 0) {
                for (int k = threadIdx.x; k < F3_ENT; k += blockDim.x) S.got[k] = 0;
                if (threadIdx.x == 0) S.next = 0;
            }
            f3_sync(cl, C);
            for (;;) {
                int k = 0;
                if (lane == 0) k = atomicAdd(&S0.next, 1);
                k = __shfl_sync(FULL, k, 0);
                if (k >= nc) break;
                const int c = c0 + k;
                const int qrypos = (c / nsx) * qstep, rfnpos = (c % nsx) * rstep;
                bool go = !(lq < qrypos + f0 || lr < rfnpos + f0 || f0 < 1);
                const bool conv1 = (lq < qrypos + f1 || lr < rfnpos + f1 || f1 < 1);
                if (go && 0.0f < thr && !f3_similar(m, lq, lr, qrypos, rfnpos, f1, thr, lane)) go = false;
                for (int fi = 0; go && fi < nfr; fi++) {
                    if (fi == 1 && conv1) continue;
                    const int fraglen = fi == 0 ? f0 : f1;
                    if (lq < qrypos + fraglen || lr < rfnpos + fraglen) continue;
                    float v[16], tfm[12];
                    int n;
                    if (seedrule) {
                        n = f3_seed_local(m, lq, lr, B.f3trigger > 0, f3_fraglen(lq, lr, fi, seedrule),
                                          qrypos, rfnpos, pq, pr, lane);
                    } else {
                        for (int p = lane; p < fraglen; p += 32) { pq[p] = (unsigned short)(qrypos + p); pr[p] = (unsigned short)(rfnpos + p); }
                        __syncwarp();
                        n = fraglen;
                    }
                    if (n < 1) continue;
                    f3_cov(P.qx, P.qy, P.qz, P.rx, P.ry, P.rz, pq, pr, n, v, lane);
                    __syncwarp();
                    if (v[15] < 1.0f) continue;
                    solve_sums(v, lq < lr ? 0 : 2, tfm);
                    for (int it = 0; it < 2; it++) {
                        const int cw = f3_window(P, tfm, it == 0, B.f3window, qrypos, rfnpos, stacksize,
                                                 pq, pr, lane, sn, sd, sm);
                        f3_cov(P.qx, P.qy, P.qz, P.rx, P.ry, P.rz, pq, pr, cw, v, lane);
                        if (v[15] < 1.0f) { __syncwarp(); continue; }
                        solve_sums(v, it == 0 ? (lq < lr ? 0 : 2) : 0, tfm);
                        if (it == 0) { __syncwarp(); continue; }
                        const float sc = f3_progressive(P, tfm, d02, pq, pr, (int)v[15], lq < lr,
                                                        S.u[w].chain.max, S.u[w].chain.ndx, lane);
                        if (lane == 0) {
                            float* res = S0.res + (k * nfr + fi) * 13;
                            S0.got[k * nfr + fi] = 1;
                            res[0] = sc;
#pragma unroll
                            for (int f = 0; f < 12; f++) res[1 + f] = tfm[f];
                        }
                        __syncwarp();
                    }
                }
            }
            f3_sync(cl, C);
            if (crank == 0) {
                if (w == 0) {
                    int cnt = 0;
                    for (int e0 = 0; e0 < nc * nfr; e0 += 32) {
                        const bool g = e0 + lane < nc * nfr && S.got[e0 + lane];
                        const unsigned gm = __ballot_sync(FULL, g);
                        if (g) S.list[cnt + __popc(gm & ((1u << lane) - 1u))] = (unsigned short)(e0 + lane);
                        cnt += __popc(gm);
                    }
                    __syncwarp();
                    // the sections an entry feeds: section 0 all; at --depth 1 and
                    // 0 sections 1 and 2 the configurations on every second /
                    // third grid row and column of a structure longer than
                    // F3_LENTHR (sec2met, sec3met: MpStageFrg3.cpp:204-212)
                    float best[F3_NSEC];
                    int src[F3_NSEC];
#pragma unroll
                    for (int sec = 0; sec < F3_NSEC; sec++) {
                        best[sec] = sec < nsec ? slots[(sec * F3_NTOP + lane) * 13] : 0.f;
                        src[sec] = -1;
                    }
                    for (int e = (lane - nscored) & (F3_NTOP - 1); e < cnt; e += F3_NTOP) {
                        const int en = S.list[e];
                        const float sc = S.res[en * 13];
                        if (!(0.0f < sc)) continue;
                        const int cc = c0 + en / nfr, ys = cc / nsx, xs = cc % nsx;
                        const bool in[F3_NSEC] = {true,
                                                  (lq <= F3_LENTHR || (ys & 1) == 0) && (lr <= F3_LENTHR || (xs & 1) == 0),
                                                  (lq <= F3_LENTHR || ys % 3 == 0) && (lr <= F3_LENTHR || xs % 3 == 0)};
#pragma unroll
                        for (int sec = 0; sec < F3_NSEC; sec++)
                            if (sec < nsec && in[sec] && best[sec] < sc) { best[sec] = sc; src[sec] = en; }
                    }
                    nscored += cnt;
#pragma unroll
                    for (int sec = 0; sec < F3_NSEC; sec++)
                        if (src[sec] >= 0)
                            for (int f = 0; f < 13; f++)
                                slots[(sec * F3_NTOP + lane) * 13 + f] = S.res[src[sec] * 13 + f];
                }
                __syncthreads();
            }
        }
        // the first pair by position, the next ones as clusters come free
        if (crank == 0 && threadIdx.x == 0) S.slot = ncl + atomicAdd(ctr, 1);
        f3_sync(cl, C);
        slot = S0.slot;
    }
    f3_sync(cl, C);                    // the first CTA's shared memory is read until here
}

// ---------------------------------------------------------------------------
// 3. Per section, the slots by DP score (SortBestDPscoresAndTMsAmongDPswifts,
// MpStageFrg3.h:1150-1250), larger first, lower slot first on ties: the
// pair's flag becomes section 0's first slot's (SCOREDP when no slot scored),
// the first --nbranches of each section are its branches (branch index =
// section * nbranches + rank), and the next DP refinement skips refinement
// variant section * 32 + rank when that rank holds no score (section 0's
// rank 0 being the pair's flag).  A thread per pair.
__global__ void k_f3_select(Blk B, Bat T, int nbranches) {
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= T.rhist[RL_NBUCKET]) return;
    const int i = T.rlist[slot];
    const int nsec = B.f3nsec;
    for (int sec = 0; sec < F3_NSEC; sec++) {
        if (sec >= nsec) { T.vskip_mask[(long long)i * F3_NSEC + sec] = 0u; continue; }
        const float* dps = T.f3dps + ((long long)i * nsec + sec) * F3_NTOP;
        float d[F3_NTOP];
        int order[F3_NTOP];
        for (int k = 0; k < F3_NTOP; k++) { d[k] = dps[k]; order[k] = k; }
        for (int a = 1; a < F3_NTOP; a++) {
            const int k = order[a];
            int b = a - 1;
            while (b >= 0 && d[order[b]] < d[k]) { order[b + 1] = order[b]; b--; }
            order[b + 1] = k;
        }
        unsigned vs = 0u;
        for (int r = sec == 0 ? 1 : 0; r < F3_NTOP; r++)
            if (!(0.0f < d[order[r]])) vs |= 1u << r;
        T.vskip_mask[(long long)i * F3_NSEC + sec] = vs;
        if (sec == 0) T.flags[i] = 0.0f < d[order[0]] ? 0 : CONV_SCOREDP;
        for (int r = 0; r < nbranches; r++) {
            const int k = order[r];
            const bool ok = 0.0f < d[k];
            const long long br = (long long)i * T.f3br + sec * nbranches + r;
            T.f3ok[br] = ok ? 1 : 0;
            if (ok) {
                const float* src = T.f3slot + (((long long)i * nsec + sec) * F3_NTOP + k) * 13 + 1;
                float* dst = T.f3alt + br * 12;
                for (int f = 0; f < 12; f++) dst[f] = src[f];
            }
        }
    }
}

// The best branch so far (SaveBestScoreAndTMAmongBests with a secondary
// update, MpStageBase.h:1250-1310): after branch rci, its refinement result
// (score and iteration-best transform) replaces the kept one for the first
// branch, or when it scores higher.  A thread per listed pair.
__global__ void k_f3_second(Blk B, Bat T, int rci) {
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= T.rhist[RL_NBUCKET]) return;
    const int i = T.rlist[slot];
    const float b = T.best[i];
    if (rci == 0 || T.best2[i] < b) {
        T.best2[i] = b;
        for (int f = 0; f < 12; f++) T.tfm_2nd[i * 12 + f] = T.tfm_ib[i * 12 + f];
    }
}

}  // namespace

// The stage over a batch (the pairs not filtered out).  The pair list is
// built once; the stage-1 kernels (DP, traceback, refinement) build their
// own lists, so the frg3 list is rebuilt before each frg3 kernel that
// reads it.
void launch_frg3(const Blk& B, const Bat& T, cudaStream_t st) {
    auto plist = [&]() { launch_pair_list(B, T, CONV_LOWTMSC, st); };
    plist();
    const int nbr = B.f3nbranches < F3_NBMAX ? B.f3nbranches : F3_NBMAX;
    {
        KtScope kts(T, KF_FRG3, st);
        if (0 < B.f3trigger || B.f3seedrule) {
            k_f3_localdp<<<T.np, F3_WARPS * 32, 0, st>>>(B, T);
            if (T.launches) (*T.launches)++;
        }
        cudaFuncSetAttribute(k_f3_search, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(F3Smem));
        cudaLaunchConfig_t cfg{};
        const int C = T.np <= F3_NP8 ? 8 : T.np <= F3_NP4 ? 4 : 2;
        cfg.gridDim = dim3(std::min(T.np, F3_GRID / C) * C);
        cfg.blockDim = dim3(F3_WARPS * 32);
        cfg.dynamicSmemBytes = sizeof(F3Smem);
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = C;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        const cudaError_t e = cudaLaunchKernelEx(&cfg, k_f3_search, B, T, B.depth);
        if (e != cudaSuccess && T.lerr && *T.lerr == cudaSuccess) *T.lerr = e;
        if (T.launches) (*T.launches)++;
        launch_f3_dpscore(B, T, st);
        k_f3_select<<<(T.np + 255) / 256, 256, 0, st>>>(B, T, nbr);
        if (T.launches) (*T.launches)++;
    }
    // the branches, section by section (Refine_tfmaltconfig,
    // MpStageFrg3.cpp:425-467); at --depth 1 and 0 each branch's refinement
    // is followed by a DP under its iteration-best transform and a
    // refinement of that alignment (MpStageFrg3.cpp:452-466)
    for (int rci = 0; rci < B.f3nsec * nbr; rci++) {
        Bat TA = T;
        TA.alt_rci = rci;
        launch_dp(B, TA, DP_TFM_ALT, 1, 0.0f, 0, 0, 0, 0, st);
        launch_refine(RM_DP, B, T, st, true);
        plist();
        k_f3_second<<<(T.np + 255) / 256, 256, 0, st>>>(B, T, rci);
        if (T.launches) (*T.launches)++;
        if (B.depth <= 1) {
            launch_dp(B, T, DP_TFM_IBEST, 1, 0.0f, 0, 0, 0, 0, st);
            launch_refine(RM_DP, B, T, st, true);
            plist();
            k_f3_second<<<(T.np + 255) / 256, 256, 0, st>>>(B, T, rci);
            if (T.launches) (*T.launches)++;
        }
    }
    // DP refinement from the best branch, with a gap cost (its refinements
    // skipping the variants the slots rule out) and without
    // (MpStageFrg3.h:108-112)
    Bat TV = T;
    TV.vskip = T.vskip_mask;
    launch_dprefine(B, TV, 0, 0, 2, 0.0f, true, DP_TFM_2ND, st);
    launch_dprefine(B, T, 1, 0, 2, 0.0f, true, DP_TFM_IBEST, st);
}

}  // namespace gtb
