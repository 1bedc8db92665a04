// gtb_api.cu -- C ABI, device-memory plan and stage sequence of the search.
//
// The stage sequence is the reference's CuBatch::ProcessBlock with the
// detailed (spatial-index) search off: stage 1 (CuBatch.cu:537-556 ->
// custage1.cu:108-186), two stage-2 passes (CuBatch.cu:627-650 ->
// custage2.cu:46-165), final stage (custage_fin.cu:45-128).  A block of
// nq x nr pairs is processed in batches of consecutive pairs sized to the
// device-memory budget; every kernel of a stage covers the whole batch.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>
#include <algorithm>
#include <chrono>
#include <cuda_runtime.h>

#include "gtb200.h"
#include "gtb_kernels.cuh"

using namespace gtb;

struct gtb_handle {
    int dev = 0;
    size_t budget = 0;
    gtb_options opts{};
    cudaStream_t st = nullptr;
    float *t_d0 = nullptr, *t_d82 = nullptr, *t_d0fin = nullptr;
    char err[512] = {0};
    long long launches = 0;
    float timings[7] = {0};
    cudaEvent_t ev[8] = {};
    // sub-batches of a batch run concurrently on these streams (st first),
    // so the short, narrow launches at the end of one overlap the others
    static const int NSUB = 3;
    cudaStream_t sub[NSUB] = {};
    cudaStream_t aux[NSUB] = {};     // per sub-batch stream: a refinement's long pairs
    cudaEvent_t fork[NSUB] = {}, join[NSUB] = {};
    static const int NWAVE = 2;      // sub-batches per stream and batch
    cudaEvent_t sev[NWAVE * NSUB][8] = {};  // stage events per sub-batch
    int dw_cap = 0;                  // CTAs the wavefront DP keeps resident
    int* h_flag = nullptr;           // pinned: wavefront error flag per sub-batch
    long long wait_limit = gtb::DP_WAVE_SPIN_DEFAULT;  // spins of a wavefront wait
    unsigned long long* d_work = nullptr;  // device work counters of the last call
    unsigned long long work[gtb::WK_NKIND] = {0, 0, 0, 0};
    bool ktime = false;                    // per-family launch timing on
    gtb::KTimer kt;
    float kms[gtb::KF_N] = {0, 0, 0, 0};   // its times of the last call
    // launch shapes (gtb_set_tuning / gtb_autotune)
    gtb_tuning tn{gtb::FF_CHUNK, gtb::RLW_CTAS, gtb::DP_CTA_PAIRS, 16384};
};

static const int TBL = 65536;

#define CK(call)                                                                 \
    do {                                                                         \
        cudaError_t e_ = (call);                                                 \
        if (e_ != cudaSuccess) {                                                 \
            snprintf(h->err, sizeof(h->err), "%s: %s (%s:%d)", #call,            \
                     cudaGetErrorString(e_), __FILE__, __LINE__);                \
            return GTB_ERR_CUDA;                                                 \
        }                                                                        \
    } while (0)

extern "C" gtb_status gtb_create(int device, size_t mem_bytes, const gtb_options* opts,
                                 gtb_handle** out) {
    if (!out || !opts) return GTB_ERR_ARG;
    *out = nullptr;
    gtb_handle* h = new gtb_handle();
    h->dev = device;
    h->opts = *opts;
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) {
        snprintf(h->err, sizeof(h->err), "cudaSetDevice(%d): %s", device, cudaGetErrorString(e));
        *out = h;
        return GTB_ERR_CUDA;
    }
    size_t fr = 0, tot = 0;
    CK(cudaMemGetInfo(&fr, &tot));
    size_t avail = fr > ((size_t)256 << 20) ? fr - ((size_t)256 << 20) : fr / 2;
    h->budget = (mem_bytes == 0 || mem_bytes > avail) ? avail : mem_bytes;
    CK(cudaStreamCreateWithFlags(&h->st, cudaStreamNonBlocking));
    // keep freed batch memory in the device pool between calls instead of
    // unmapping it at every synchronisation (each block reuses similar sizes)
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess) {
        unsigned long long keep = ~0ull;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
    for (int k = 0; k < 8; k++) CK(cudaEventCreate(&h->ev[k]));
    h->dw_cap = dp_wave_capacity();
    configure_kernels();
    CK(cudaHostAlloc((void**)&h->h_flag, gtb_handle::NWAVE * gtb_handle::NSUB * sizeof(int),
                     cudaHostAllocDefault));
    CK(cudaMalloc(&h->d_work, gtb::WK_NKIND * gtb::WORK_SLOTS * sizeof(unsigned long long)));
    h->sub[0] = h->st;
    for (int j = 1; j < gtb_handle::NSUB; j++)
        CK(cudaStreamCreateWithFlags(&h->sub[j], cudaStreamNonBlocking));
    for (int j = 0; j < gtb_handle::NSUB; j++) {
        CK(cudaStreamCreateWithFlags(&h->aux[j], cudaStreamNonBlocking));
        CK(cudaEventCreateWithFlags(&h->fork[j], cudaEventDisableTiming));
        CK(cudaEventCreateWithFlags(&h->join[j], cudaEventDisableTiming));
    }
    for (int j = 0; j < gtb_handle::NWAVE * gtb_handle::NSUB; j++)
        for (int k = 0; k < 8; k++) CK(cudaEventCreate(&h->sev[j][k]));
    std::vector<float> a(TBL), b(TBL), c(TBL);
    make_tables(a.data(), b.data(), c.data(), TBL);
    CK(cudaMalloc(&h->t_d0, TBL * sizeof(float)));
    CK(cudaMalloc(&h->t_d82, TBL * sizeof(float)));
    CK(cudaMalloc(&h->t_d0fin, TBL * sizeof(float)));
    CK(cudaMemcpy(h->t_d0, a.data(), TBL * sizeof(float), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(h->t_d82, b.data(), TBL * sizeof(float), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(h->t_d0fin, c.data(), TBL * sizeof(float), cudaMemcpyHostToDevice));
    *out = h;
    return GTB_OK;
}

extern "C" void gtb_destroy(gtb_handle* h) {
    if (!h) return;
    cudaSetDevice(h->dev);
    if (h->t_d0) cudaFree(h->t_d0);
    if (h->t_d82) cudaFree(h->t_d82);
    if (h->t_d0fin) cudaFree(h->t_d0fin);
    if (h->d_work) cudaFree(h->d_work);
    for (int k = 0; k < 8; k++) if (h->ev[k]) cudaEventDestroy(h->ev[k]);
    for (int j = 0; j < gtb_handle::NWAVE * gtb_handle::NSUB; j++)
        for (int k = 0; k < 8; k++) if (h->sev[j][k]) cudaEventDestroy(h->sev[j][k]);
    for (int j = 1; j < gtb_handle::NSUB; j++)
        if (h->sub[j]) cudaStreamDestroy(h->sub[j]);
    for (int j = 0; j < gtb_handle::NSUB; j++) {
        if (h->aux[j]) cudaStreamDestroy(h->aux[j]);
        if (h->fork[j]) cudaEventDestroy(h->fork[j]);
        if (h->join[j]) cudaEventDestroy(h->join[j]);
    }
    if (h->st) cudaStreamDestroy(h->st);
    if (h->h_flag) cudaFreeHost(h->h_flag);
    delete h;
}

extern "C" const char* gtb_last_error(const gtb_handle* h) { return h ? h->err : "null handle"; }
extern "C" long long gtb_last_launch_count(const gtb_handle* h) { return h ? h->launches : -1; }
extern "C" gtb_status gtb_last_timings(const gtb_handle* h, float* ms7) {
    if (!h || !ms7) return GTB_ERR_ARG;
    memcpy(ms7, h->timings, sizeof(h->timings));
    return GTB_OK;
}
extern "C" gtb_status gtb_last_work(const gtb_handle* h, unsigned long long* w4) {
    if (!h || !w4) return GTB_ERR_ARG;
    memcpy(w4, h->work, sizeof(h->work));
    return GTB_OK;
}
extern "C" gtb_status gtb_set_kernel_timing(gtb_handle* h, int on) {
    if (!h) return GTB_ERR_ARG;
    h->ktime = on != 0;
    return GTB_OK;
}
extern "C" gtb_status gtb_last_kernel_ms(const gtb_handle* h, float* ms4) {
    if (!h || !ms4) return GTB_ERR_ARG;
    memcpy(ms4, h->kms, sizeof(h->kms));
    return GTB_OK;
}
extern "C" gtb_status gtb_set_wait_limit(gtb_handle* h, long long spins) {
    if (!h || spins < 0) return GTB_ERR_ARG;
    h->wait_limit = spins;
    return GTB_OK;
}

// ---------------------------------------------------------------------------
static gtb_status check_options(gtb_handle* h) {
    const gtb_options& o = h->opts;
    if (!o.nodetailedsearch) {
        if (o.trigger < 0 || o.trigger > 100 || o.nbranches < 1 || o.nbranches > F3_NBMAX ||
            o.gapcost < 0 || o.gapcost > 2 || o.seedrule < 0 || o.seedrule > 2 ||
            o.window < 256 || o.window > 512) {
            snprintf(h->err, sizeof(h->err), "detailed-search option out of range");
            return GTB_ERR_ARG;
        }
    }
    if (o.refinement < GTB_REFINEMENT_LOG || o.refinement > GTB_REFINEMENT_FULLA) {
        snprintf(h->err, sizeof(h->err), "--refinement %d out of -1..3", o.refinement);
        return GTB_ERR_ARG;
    }
    if (!(o.presimilarity >= 0.f && o.presimilarity < 1e6f)) {
        snprintf(h->err, sizeof(h->err), "--pre-similarity out of range");
        return GTB_ERR_ARG;
    }
    if (o.clsfilter < 0 || o.clsfilter > 1 ||
        (o.clsfilter && !(o.clscoverage > 0.f && o.clscoverage <= 1.f))) {
        snprintf(h->err, sizeof(h->err), "--cls-coverage out of (0,1]");
        return GTB_ERR_ARG;
    }
    if (o.polish_steps < 0 || o.polish_steps > 50) {
        snprintf(h->err, sizeof(h->err), "polish_steps %d out of 0..50", o.polish_steps);
        return GTB_ERR_ARG;
    }
    if (o.depth < 0 || o.depth > 3 || o.convergence < 1 || o.convergence > 30 ||
        !(o.prescore >= 0.f && o.prescore < 1.f)) {
        snprintf(h->err, sizeof(h->err), "option out of range");
        return GTB_ERR_ARG;
    }
    return GTB_OK;
}

// Device-resident block description (inputs) for run_block.
struct DevBlock {
    int nq, nr;
    const int *qlen, *rlen, *qoff, *roff, *qmol, *rmol;
    const float *qx, *qy, *qz, *rx, *ry, *rz;
    const float4 *q4, *r4;
    const unsigned char *qodd, *rodd;
    const unsigned char *qa, *ra;
    char *qs, *rs;
    // index trees (null: none)
    const float4 *qnd = nullptr, *rnd = nullptr;
    const int2 *qnc = nullptr, *rnc = nullptr;
    // clustering runs: the references' global indices and the end of the
    // query block's (qrysernrbeg + nqystrs, CuBatch.cu:492-494)
    const int* rtype = nullptr;
    int qtypeend = 0;
    std::vector<int> hqlen, hrlen;
};

// Results of one batch, device side.
struct BatchBufs {
    void* base = nullptr;
    size_t cap = 0;
};

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Bytes of device scratch one pair needs (f3: the detailed search's local
// score matrix, slots and branches).
static size_t pair_bytes(int lq, int lr, bool strings, bool f3 = false) {
    size_t b = (size_t)gtb::bt_words(lq, lr) * 4;     // traceback words
    if (f3) b += (size_t)gtb::f3_region_bytes(lq, lr, F3_NSEC) + (size_t)F3_NSEC * (F3_NTOP * 14 * 4 + F3_NBMAX * 13 * 4) +
                 13 * 4 + 8 + F3_NSEC * 4;
    b += (size_t)lr * 4;                               // DP row buffer
    b += (size_t)std::min(lq, lr) * 28;                // aligned pairs + coordinates
    if (strings) b += (size_t)5 * (lq + lr + 1);       // alignment rows
    b += 4 * 8 + 12 * 4 * 2 + 16 * 4 + 4 * 4 + 12 * 4 + 64 + 4 + 24;  // state, offsets, work lists
    // the refinement candidates of a long pair (RL_LONG); counted from 384 residues,
    // from where an earlier form had them: a budget (mem_bytes) splits and refuses
    // the blocks that it always has
    if (std::min(lq, lr) >= 384)
        b += (size_t)gtb::RLW_CTAS_MAX * gtb::RLW_CTA_WARPS * gtb::RLW_CAND * 4 + 12;
    return b;
}

// Destination of the alignment rows: the caller's buffer in the reference's
// layout (MpDPHub.cpp:1975-1981): for query qi, 5 rows of rowlen[qi] bytes
// starting at qbase[qi]; pair (qi, ri) at column roff[ri] + ri*(lq_i+1).
struct AlnSink {
    char* alns = nullptr;
    const float* rec = nullptr;      // the block's host records (alignment length at field 4)
    std::vector<long long> qbase, rowlen;
    std::vector<int> qlen, rlen, roff;
    int nr = 0;
    std::vector<long long> soff;     // staging: packed offsets of a sub-batch
    std::vector<char> sbytes;        // staging: its packed rows
    // copy the packed rows of pairs [p0, p0+np) to the reference layout; a
    // pair without an alignment gets empty rows
    void scatter(long long p0, int np) {
        for (int i = 0; i < np; i++) {
            long long p = p0 + i;
            int qi = (int)(p / nr), ri = (int)(p % nr);
            char* dst = alns + qbase[qi] + (long long)roff[ri] + (long long)ri * (qlen[qi] + 1);
            long long o = soff[i];
            if (o < 0) {
                for (int f = 0; f < 5; f++) dst[f * rowlen[qi]] = 0;
                continue;
            }
            // 5 rows of W bytes: the alignment's columns and the NUL
            const long long W = (long long)rec[p * GTB_NOUT + GTB_OUT_ALNLENGTH] + 1;
            for (int f = 0; f < 5; f++) memcpy(dst + f * rowlen[qi], sbytes.data() + o + f * W, (size_t)W);
        }
    }
};

// Runs the whole stage sequence over a device-resident block.
// Host outputs (may be null): alndata [nq*nr*16], tfm [nq*nr*12],
// numerr [nq*nr*4]; sink: alignment rows (null: none produced).
static gtb_status run_block(gtb_handle* h, const DevBlock& D, float scorethld,
                            float* h_alndata, float* h_tfm, float* h_err, AlnSink* sink) {
    const gtb_options& o = h->opts;
    const long long npairs = (long long)D.nq * D.nr;
    Blk B{};
    B.nq = D.nq; B.nr = D.nr;
    B.qlen = D.qlen; B.rlen = D.rlen; B.qoff = D.qoff; B.roff = D.roff;
    B.qx = D.qx; B.qy = D.qy; B.qz = D.qz; B.rx = D.rx; B.ry = D.ry; B.rz = D.rz;
    B.q4 = D.q4; B.r4 = D.r4; B.q4off = D.qoff; B.r4off = D.roff;
    B.qodd = D.qodd; B.rodd = D.rodd;
    B.qa = D.qa; B.ra = D.ra; B.qs = D.qs; B.rs = D.rs; B.qmol = D.qmol; B.rmol = D.rmol;
    B.qmax = *std::max_element(D.hqlen.begin(), D.hqlen.end());
    B.qmin = *std::min_element(D.hqlen.begin(), D.hqlen.end());
    B.rmax = *std::max_element(D.hrlen.begin(), D.hrlen.end());
    B.rmin = *std::min_element(D.hrlen.begin(), D.hrlen.end());
    B.t_d0 = h->t_d0; B.t_d82 = h->t_d82; B.t_d0fin = h->t_d0fin;
    B.stepinit = (o.depth == 3) ? 5 : 1;
    B.refinement = o.refinement; B.depth = o.depth; B.twotm = o.twotmscore ? 1 : 0;
    B.addss = o.addsearchbyss ? 1 : 0;
    // the screen runs when the block's longest structures exceed the edge
    // (CuBatch.cu:459-462)
    B.presim = (0.f < o.presimilarity && PRESIM_EDGE < B.qmax && PRESIM_EDGE < B.rmax) ? o.presimilarity : 0.f;
    B.symmetric = o.symmetric; B.nodeletions = o.nodeletions;
    B.cls = o.clsfilter ? 1 : 0;
    if (B.cls) {
        if (!D.rtype) { snprintf(h->err, sizeof(h->err), "a clustering run needs the type field"); return GTB_ERR_ARG; }
        B.rtype = D.rtype; B.clsqend = D.qtypeend; B.clscov = o.clscoverage;
    }
    B.f3 = o.nodetailedsearch ? 0 : 1;
    if (B.f3) {
        if (!D.qnd || !D.rnd) {
            snprintf(h->err, sizeof(h->err), "the detailed search needs the blocks' index trees");
            return GTB_ERR_ARG;
        }
        B.qnd = D.qnd; B.qnc = D.qnc; B.rnd = D.rnd; B.rnc = D.rnc;
        B.f3trigger = o.trigger; B.f3nbranches = o.nbranches;
        // configuration sections (MpStageFrg3.cpp:204-212, 403-404)
        B.f3nsec = o.depth <= 0 ? 3 : (o.depth <= 1 ? 2 : 1);
        B.f3gapcost = o.gapcost == 0 ? -0.8f : (o.gapcost == 1 ? -1.2f : -3.0f);
        B.f3seedrule = o.seedrule == 0 ? 0 : (o.seedrule == 1 ? 64 : 128);
        B.f3window = o.window;
    }
    const bool strings = sink != nullptr;

    size_t fr = 0, tot = 0;
    CK(cudaMemGetInfo(&fr, &tot));
    size_t budget = std::min(h->budget, fr > ((size_t)256 << 20) ? fr - ((size_t)256 << 20) : fr / 2);
    // keep batches moderate so the pair-level state stays L2-friendly
    const long long maxbatch = 1 << 20;

    float tsum[7] = {0, 0, 0, 0, 0, 0, 0};
    h->launches = 0;
    h->kt.used = 0;                     // pairs of an unfinished earlier call
    cudaError_t lerr = cudaSuccess;     // a launch that failed (cooperative DP)
    // work counters: cleared on the handle's stream, which the sub-batch
    // streams wait for below
    CK(cudaMemsetAsync(h->d_work, 0, gtb::WK_NKIND * gtb::WORK_SLOTS * sizeof(unsigned long long), h->st));
    // host offsets of the sub-batches in flight (kept until their copies ran)
    std::vector<long long> offv[gtb_handle::NSUB];
    std::vector<int> ffv[gtb_handle::NSUB], ffiv[gtb_handle::NSUB], dwvv[gtb_handle::NSUB];
    std::vector<long long> dwsv[gtb_handle::NSUB];
    // sub-batches whose packed alignment rows are read once the batch is done
    struct StrBat { char* base; long long p0; int np; long long* soff; unsigned long long* cnt; char* str; };
    std::vector<StrBat> strbat;

    // A copy to pageable host memory holds the host until it is done, and with
    // it the launches of the next sub-batch: such results are copied once all
    // sub-batches are launched (400 structures all against all 198 -> 113 ms).
    // Until then they have an allocation of their own (own), so that a
    // sub-batch's working memory goes to the next one on its stream.
    auto pageable = [](const void* p) {
        cudaPointerAttributes a{};
        if (!p) return false;
        if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return true; }
        return a.type == cudaMemoryTypeUnregistered;
    };
    const bool late = pageable(h_alndata) || pageable(h_tfm) || pageable(h_err);
    const bool own = late && !strings;
    struct LateBat { char* base; long long p0; int np; const float *out, *tfm, *err; cudaStream_t st; };
    std::vector<LateBat> latebat;
    auto copy_out = [&](long long q0, int np, const float* out, const float* tfm, const float* err,
                        cudaStream_t st) -> gtb_status {
        if (h_alndata)
            CK(cudaMemcpyAsync(h_alndata + q0 * 16, out, (size_t)np * 16 * sizeof(float), cudaMemcpyDefault, st));
        if (h_tfm)
            CK(cudaMemcpyAsync(h_tfm + q0 * 12, tfm, (size_t)np * 12 * sizeof(float), cudaMemcpyDefault, st));
        if (h_err)
            CK(cudaMemcpyAsync(h_err + q0 * 4, err, (size_t)np * 4 * sizeof(float), cudaMemcpyDefault, st));
        return GTB_OK;
    };
    // frees the memory kept past the launches: whole sub-batches with alignment
    // rows, else results
    auto drop_kept = [&](bool sync) {
        if (sync) for (int k = 0; k < gtb_handle::NSUB; k++) cudaStreamSynchronize(h->sub[k]);
        if (strings) for (const StrBat& sb : strbat) cudaFreeAsync(sb.base, h->st);
        else for (const LateBat& lb : latebat) cudaFreeAsync(lb.base, lb.st);
        strbat.clear();
        latebat.clear();
    };

    // One sub-batch [q0, q0 + np): plan, carve one allocation, upload the
    // offsets, launch the stage sequence and the result copies on stream st.
    auto launch_sub = [&](long long q0, int np, int j, int evset) -> gtb_status {
        cudaStream_t st = h->sub[j];
        std::vector<long long>& ov = offv[j];
        ov.assign((B.f3 ? 5 : 4) * (size_t)(np + 1), 0);
        long long* off_bt = ov.data();
        long long* off_row = off_bt + (np + 1);
        long long* off_aln = off_bt + 2 * (np + 1);
        long long* off_str = off_bt + 3 * (np + 1);
        long long* off_lsm = B.f3 ? off_bt + 4 * (np + 1) : nullptr;
        // seed work items: pairs with more offsets than one CTA takes are split
        std::vector<int>& ffn = ffv[j];
        ffn.assign(np, 1);
        long long nitems = 0;
        bool split = false;
        for (int i = 0; i < np; i++) {
            long long p = q0 + i;
            int lq = D.hqlen[p / D.nr], lr = D.hrlen[p % D.nr];
            off_bt[i + 1] = off_bt[i] + gtb::bt_words(lq, lr);
            off_row[i + 1] = off_row[i] + lr;
            off_aln[i + 1] = off_aln[i] + std::min(lq, lr);
            off_str[i + 1] = off_str[i] + (strings ? 5LL * (lq + lr + 1) : 0);
            if (off_lsm) off_lsm[i + 1] = off_lsm[i] + gtb::f3_region_bytes(lq, lr, B.f3nsec);
            int n1, silo, sihi, prv;
            gtb::seed_range(lq, lr, B.qmax, B.qmin, B.rmax, B.rmin, B.stepinit, n1, silo, sihi, prv);
            int cnt = sihi - silo + 1;
            const int chunk = h->tn.seed_chunk;
            int nch = cnt > chunk ? (cnt + chunk - 1) / chunk : 1;
            ffn[i] = nch;
            nitems += nch;
            split = split || nch > 1;
        }
        // long pairs: DP as a wavefront over several CTAs
        std::vector<int>& dwv = dwvv[j];
        dwv.clear();
        long long dnprog = 0;
        int nl = 0, nitw = 0;
        if (h->dw_cap > 0) {
            std::vector<int> lp;
            for (int i = 0; i < np; i++) {
                long long p = q0 + i;
                int lq = D.hqlen[p / D.nr], lr = D.hrlen[p % D.nr];
                if (gtb::dp_wave(lq, lr) && (int)lp.size() < h->dw_cap) lp.push_back(i);
            }
            nl = (int)lp.size();
            if (nl > 0) {
                // layout: items (slot, c) | pair | G | mark bytes (np) ; soff separately
                std::vector<int> G(nl), items;
                std::vector<long long>& so = dwsv[j];
                so.assign(nl, 0);
                for (int k = 0; k < nl; k++) {
                    long long p = q0 + lp[k];
                    int lq = D.hqlen[p / D.nr];
                    int ns = gtb::dp_strips(lq);
                    G[k] = std::min(ns, std::max(1, h->dw_cap / nl));
                    so[k] = dnprog;
                    dnprog += ns;
                    nitw += G[k];
                }
                dwv.assign(2 * (size_t)nitw + 2 * (size_t)nl + (np + 3) / 4, 0);
                int t = 0;
                for (int k = 0; k < nl; k++)
                    for (int c = 0; c < G[k]; c++, t++) { dwv[t] = k; dwv[nitw + t] = c; }
                for (int k = 0; k < nl; k++) { dwv[2 * nitw + k] = lp[k]; dwv[2 * nitw + nl + k] = G[k]; }
                unsigned char* mk = (unsigned char*)(dwv.data() + 2 * nitw + 2 * nl);
                for (int k = 0; k < nl; k++) mk[lp[k]] = 1;
            }
        }
        // pairs that may reach the refinement launches' length classes
        // (n <= min(lq, lr))
        int nml[4] = {np, 0, 0, 0};
        for (int i = 0; i < np; i++) {
            long long p = q0 + i;
            const int ml = std::min(D.hqlen[p / D.nr], D.hrlen[p % D.nr]);
            nml[1] += ml >= gtb::RC_N1;
            nml[2] += ml >= gtb::RC_N2;
            nml[3] += ml >= gtb::RL_LONG;
        }
        const int nlmax = nml[3];
        std::vector<int>& ffi = ffiv[j];
        if (split) {
            ffi.assign(2 * (size_t)nitems, 0);
            long long t = 0;
            for (int i = 0; i < np; i++)
                for (int c = 0; c < ffn[i]; c++, t++) { ffi[t] = i; ffi[nitems + t] = c; }
        }
        size_t sz = 0;
        auto carve = [&](size_t bytes) { size_t o2 = sz; sz += align256(bytes); return o2; };
        size_t o_ints = carve((size_t)np * 8 * sizeof(int));
        size_t o_flts = carve((size_t)np * 4 * sizeof(float));
        size_t o_tib = carve((size_t)np * 12 * sizeof(float));
        size_t o_tgr = carve((size_t)np * 12 * sizeof(float));
        size_t o_out = carve((size_t)np * 16 * sizeof(float));
        size_t o_err = carve((size_t)np * 4 * sizeof(float));
        const size_t nres = sz - o_tgr;         // the results' bytes
        if (own) sz = o_tgr;
        size_t o_offs = carve((size_t)(np + 1) * (B.f3 ? 5 : 4) * sizeof(long long));
        size_t o_bt = carve((size_t)off_bt[np] * sizeof(unsigned));
        size_t o_row = carve((size_t)off_row[np] * sizeof(float));
        size_t o_aln = carve((size_t)off_aln[np] * sizeof(unsigned));
        size_t o_str = carve((size_t)std::max<long long>(off_str[np], 1));
        size_t o_sto = strings ? carve((size_t)np * sizeof(long long) + sizeof(unsigned long long)) : 0;
        size_t o_alc = carve((size_t)off_aln[np] * 6 * sizeof(float));
        size_t o_rl = carve((size_t)np * sizeof(int));
        size_t o_rh = carve((size_t)gtb::RL_NHIST * sizeof(int));
        size_t o_ffi = split ? carve((size_t)nitems * 2 * sizeof(int)) : 0;
        size_t o_ffn = split ? carve((size_t)np * sizeof(int)) : 0;
        size_t o_ffk = split ? carve((size_t)np * sizeof(unsigned long long)) : 0;
        size_t o_dw = nl ? carve(dwv.size() * sizeof(int)) : 0;
        size_t o_dws = nl ? carve((size_t)nl * sizeof(long long)) : 0;
        size_t o_dwp = nl ? carve((size_t)dnprog * sizeof(int)) : 0;
        size_t o_dwe = carve(sizeof(int));      // wavefront error flag (multi-CTA and CTA waves)
        size_t o_rll = nlmax ? carve((size_t)(2 * nlmax + 1) * sizeof(int)) : 0;
        // CTAs per long pair (more when few pairs are long)
        const int ctasA = gtb::rlw_ctas_for(h->tn.refine_long_ctas, nlmax);
        size_t o_rlc = nlmax ? carve((size_t)nlmax * ctasA * gtb::RLW_CTA_WARPS * gtb::RLW_CAND * sizeof(float)) : 0;
        // detailed search: local score matrices, slots, DP scores, branches
        size_t o_lsm = B.f3 ? carve((size_t)std::max<long long>(off_lsm[np], 1)) : 0;
        const size_t nsl = (size_t)B.f3nsec * F3_NTOP, nbr = (size_t)B.f3nsec * F3_NBMAX;
        size_t o_f3s = B.f3 ? carve((size_t)np * nsl * 13 * sizeof(float)) : 0;
        size_t o_f3d = B.f3 ? carve((size_t)np * nsl * sizeof(float)) : 0;
        size_t o_f3a = B.f3 ? carve((size_t)np * nbr * 12 * sizeof(float)) : 0;
        size_t o_f3o = B.f3 ? carve((size_t)np * nbr) : 0;
        size_t o_f32 = B.f3 ? carve((size_t)np * 13 * sizeof(float)) : 0;
        size_t o_f3v = B.f3 ? carve((size_t)np * F3_NSEC * sizeof(unsigned)) : 0;
        char *base = nullptr, *res = nullptr;
        if (own) {
            CK(cudaMallocAsync((void**)&res, nres, st));
            latebat.push_back({res, q0, np, nullptr, nullptr, nullptr, st});
        }
        CK(cudaMallocAsync((void**)&base, sz, st));
        if (!own) res = base + o_tgr;
        Bat T{};
        T.p0 = q0; T.np = np;
        int* ints = (int*)(base + o_ints);
        T.flags = ints; T.seedq = ints + np; T.seedr = ints + 2 * np; T.naln = ints + 3 * np;
        T.sfndx = ints + 4 * np; T.sfpos = ints + 5 * np; T.sfndx_cur = ints + 6 * np; T.sfpos_cur = ints + 7 * np;
        float* fl = (float*)(base + o_flts);
        T.grand = fl; T.best = fl + np; T.best0 = fl + 2 * np; T.rmsd32 = fl + 3 * np;
        T.tfm_ib = (float*)(base + o_tib); T.tfm_gr = (float*)res;
        T.out = (float*)(res + (o_out - o_tgr)); T.err = (float*)(res + (o_err - o_tgr));
        long long* offs = (long long*)(base + o_offs);
        T.off_bt = offs; T.off_row = offs + (np + 1); T.off_aln = offs + 2 * (np + 1);
        T.bt = (unsigned*)(base + o_bt); T.row = (float*)(base + o_row);
        T.aln = (unsigned*)(base + o_aln); T.str = strings ? (base + o_str) : nullptr;
        T.str_off = strings ? (long long*)(base + o_sto) : nullptr;
        T.str_cnt = strings ? (unsigned long long*)(base + o_sto + (size_t)np * sizeof(long long)) : nullptr;
        if (strings) CK(cudaMemsetAsync(T.str_cnt, 0, sizeof(unsigned long long), st));
        T.alc = (float*)(base + o_alc);
        T.rlist = (int*)(base + o_rl); T.rhist = (int*)(base + o_rh);
        T.launches = &h->launches;
        T.lerr = &lerr;
        T.alt_rci = -1;
        T.vskip = nullptr;
        if (B.f3) {
            T.off_lsm = offs + 4 * (np + 1);
            T.lsm = (unsigned char*)(base + o_lsm);
            T.f3slot = (float*)(base + o_f3s);
            T.f3dps = (float*)(base + o_f3d);
            T.f3alt = (float*)(base + o_f3a);
            T.f3ok = (unsigned char*)(base + o_f3o);
            T.tfm_2nd = (float*)(base + o_f32);
            T.best2 = T.tfm_2nd + (size_t)np * 12;
            T.vskip_mask = (unsigned*)(base + o_f3v);
            T.f3br = (int)nbr;
        }
        T.work = h->d_work;
        T.kt = h->ktime ? &h->kt : nullptr;
        T.st2 = h->aux[j]; T.evfork = h->fork[j]; T.evjoin = h->join[j];
        T.dw_spin = h->wait_limit;
        T.nff = np; T.ff_pair = nullptr; T.ff_chunk = nullptr; T.ff_nch = nullptr; T.ff_key = nullptr;
        T.rl_nlmax = nlmax; T.rl_long = T.rl_count = T.rl_next = nullptr; T.rl_cand = nullptr;
        if (nlmax) {
            int* rl = (int*)(base + o_rll);
            T.rl_long = rl; T.rl_next = rl + nlmax; T.rl_count = rl + 2 * nlmax;
            T.rl_cand = (float*)(base + o_rlc);
        }
        for (int k = 0; k < 4; k++) T.nml[k] = nml[k];
        T.ndw = 0; T.dw_nprog = 0; T.dw_item = T.dw_pair = T.dw_G = nullptr; T.dw_soff = nullptr;
        T.dw_mark = nullptr; T.dw_prog = nullptr;
        T.dw_err = (int*)(base + o_dwe);
        T.dp_kc = h->tn.dp_cta_pairs;
        T.ff_span = h->tn.seed_chunk;
        T.rlw_ctas = ctasA;
        CK(cudaMemsetAsync(T.dw_err, 0, sizeof(int), st));
        h->h_flag[evset] = 0;
        if (nl) {
            int* dw = (int*)(base + o_dw);
            T.ndw = nitw; T.dw_nprog = dnprog;
            T.dw_item = dw; T.dw_pair = dw + 2 * nitw; T.dw_G = dw + 2 * nitw + nl;
            T.dw_mark = (const unsigned char*)(dw + 2 * nitw + 2 * nl);
            T.dw_soff = (const long long*)(base + o_dws);
            T.dw_prog = (int*)(base + o_dwp);
            CK(cudaMemcpyAsync(dw, dwv.data(), dwv.size() * sizeof(int), cudaMemcpyHostToDevice, st));
            CK(cudaMemcpyAsync(base + o_dws, dwsv[j].data(), (size_t)nl * sizeof(long long),
                               cudaMemcpyHostToDevice, st));
        }
        CK(cudaMemcpyAsync(offs, off_bt, (B.f3 ? 5 : 4) * (size_t)(np + 1) * sizeof(long long),
                           cudaMemcpyHostToDevice, st));
        if (split) {
            int* di = (int*)(base + o_ffi);
            int* dn = (int*)(base + o_ffn);
            T.nff = (int)nitems; T.ff_pair = di; T.ff_chunk = di + nitems; T.ff_nch = dn;
            T.ff_key = (unsigned long long*)(base + o_ffk);
            CK(cudaMemcpyAsync(di, ffi.data(), (size_t)nitems * 2 * sizeof(int), cudaMemcpyHostToDevice, st));
            CK(cudaMemcpyAsync(dn, ffn.data(), (size_t)np * sizeof(int), cudaMemcpyHostToDevice, st));
        }
        launch_stages(B, T, o.refinement, o.depth, o.convergence, o.prescore, o.referenced,
                      scorethld, st, h->sev[evset], o.polish_steps);
        CK(lerr);
        CK(cudaGetLastError());
        if (!late) {
            gtb_status s2 = copy_out(q0, np, T.out, T.tfm_gr, T.err, st);
            if (s2 != GTB_OK) return s2;
        }
        CK(cudaMemcpyAsync(h->h_flag + evset, T.dw_err, sizeof(int), cudaMemcpyDeviceToHost, st));
        if (strings) {
            // read after the batch: only the bytes the rows took
            strbat.push_back({base, q0, np, T.str_off, T.str_cnt, T.str});
            if (late) latebat.push_back({base, q0, np, T.out, T.tfm_gr, T.err, st});
            return GTB_OK;
        }
        if (own) latebat.back() = {res, q0, np, T.out, T.tfm_gr, T.err, st};
        CK(cudaFreeAsync(base, st));
        return GTB_OK;
    };

    // the sub-batch streams start after everything queued on the handle's
    // stream so far (block uploads, secondary structure, float4 copies)
    CK(cudaEventRecord(h->ev[7], h->st));
    for (int j = 1; j < gtb_handle::NSUB; j++) CK(cudaStreamWaitEvent(h->sub[j], h->ev[7], 0));

    auto add_times = [&](int j) -> gtb_status {
        cudaEvent_t* ev = h->sev[j];
        float ms = 0.f;
        CK(cudaEventElapsedTime(&ms, ev[0], ev[1])); tsum[0] += ms;
        CK(cudaEventElapsedTime(&ms, ev[1], ev[2])); tsum[1] += ms;
        CK(cudaEventElapsedTime(&ms, ev[2], ev[3])); tsum[2] += ms;
        CK(cudaEventElapsedTime(&ms, ev[3], ev[4])); tsum[5] += ms;
        CK(cudaEventElapsedTime(&ms, ev[0], ev[4])); tsum[6] += ms;
        return GTB_OK;
    };

    long long p0 = 0;
    while (p0 < npairs) {
        // choose the batch (fixed part: carve alignment and the work-list buckets)
        size_t used = 32768 * gtb_handle::NSUB;
        long long p1 = p0;
        while (p1 < npairs && p1 - p0 < maxbatch) {
            int lq = D.hqlen[p1 / D.nr], lr = D.hrlen[p1 % D.nr];
            size_t b = pair_bytes(lq, lr, strings, B.f3 != 0);
            if (used + b > budget && p1 > p0) break;
            used += b;
            p1++;
        }
        if (used > budget) {
            snprintf(h->err, sizeof(h->err), "pair (%lld) needs %zu bytes > budget %zu", p0, used, budget);
            return GTB_ERR_NOMEM;
        }
        // split into sub-batches of at least tn.sub_pairs pairs, in up to two waves
        // over the streams: the narrow stage-2 launches of the first wave
        // overlap the wide stage-1 launches of the second
        long long nb = p1 - p0;
        int nsub = (int)std::min<long long>(gtb_handle::NWAVE * gtb_handle::NSUB,
                                            std::max<long long>(1, nb / h->tn.sub_pairs));
        long long q0 = p0;
        for (int j = 0; j < nsub; j++) {
            long long q1 = p0 + nb * (j + 1) / nsub;
            gtb_status s = launch_sub(q0, (int)(q1 - q0), j % gtb_handle::NSUB, j);
            if (s != GTB_OK) {
                drop_kept(true);
                return s;
            }
            q0 = q1;
        }
        for (const LateBat& lb : latebat) {
            gtb_status s = copy_out(lb.p0, lb.np, lb.out, lb.tfm, lb.err, lb.st);
            if (s != GTB_OK) {
                drop_kept(true);
                return s;
            }
        }
        for (int j = 0; j < std::min(nsub, gtb_handle::NSUB); j++) CK(cudaStreamSynchronize(h->sub[j]));
        if (!strings) drop_kept(false);
        latebat.clear();
        if (!strbat.empty()) {
            gtb_status s2 = GTB_OK;
            for (const StrBat& sb : strbat) {
                unsigned long long used = 0;
                cudaError_t e = cudaMemcpy(&used, sb.cnt, sizeof(used), cudaMemcpyDeviceToHost);
                if (e == cudaSuccess) {
                    sink->soff.resize(sb.np);
                    e = cudaMemcpy(sink->soff.data(), sb.soff, (size_t)sb.np * sizeof(long long),
                                   cudaMemcpyDeviceToHost);
                }
                if (e == cudaSuccess) {
                    sink->sbytes.resize(used);
                    if (used) e = cudaMemcpy(sink->sbytes.data(), sb.str, used, cudaMemcpyDeviceToHost);
                }
                if (e != cudaSuccess && s2 == GTB_OK) {
                    snprintf(h->err, sizeof(h->err), "alignment rows: %s", cudaGetErrorString(e));
                    s2 = GTB_ERR_CUDA;
                }
                if (s2 == GTB_OK) sink->scatter(sb.p0, sb.np);
                cudaFreeAsync(sb.base, h->st);
            }
            strbat.clear();
            if (s2 != GTB_OK) return s2;
        }
        for (int j = 0; j < nsub; j++) {
            gtb_status s = add_times(j);
            if (s != GTB_OK) return s;
            if (h->h_flag[j]) {
                snprintf(h->err, sizeof(h->err), "a wavefront DP wait exceeded its limit (sub-batch %d)", j);
                return GTB_ERR_CUDA;
            }
        }
        p0 = p1;
    }
    memcpy(h->timings, tsum, sizeof(tsum));
    for (int k = 0; k < gtb::KF_N; k++) h->kms[k] = 0.f;
    if (h->ktime) CK(h->kt.collect(h->kms));
    {
        unsigned long long wk[gtb::WK_NKIND * gtb::WORK_SLOTS];
        CK(cudaMemcpy(wk, h->d_work, sizeof(wk), cudaMemcpyDeviceToHost));
        for (int k = 0; k < gtb::WK_NKIND; k++) {
            unsigned long long t = 0;
            for (int j = 0; j < gtb::WORK_SLOTS; j++) t += wk[k * gtb::WORK_SLOTS + j];
            h->work[k] = t;
        }
    }
    return GTB_OK;
}

// ---------------------------------------------------------------------------
// The reference's SoA batch, read from host field pointers.
struct HostSoA {
    int n = 0;
    long long npos = 0;
    const int* len = nullptr;
    const unsigned* dist = nullptr;
    const float *x = nullptr, *y = nullptr, *z = nullptr;
    const int* insch = nullptr;
    const char* rsd = nullptr;
    const int* type = nullptr;      // global indices of a clustering run (may be null)
    std::vector<int> mol, off;
};

static gtb_status parse_soa(gtb_handle* h, char* const* beg, char* const* end, HostSoA& S,
                            const char* what) {
    if (!beg || !end) { snprintf(h->err, sizeof(h->err), "%s: null field pointers", what); return GTB_ERR_ARG; }
    for (int f = 0; f < GTB_NFIELDS; f++)
        if ((f == GTB_FLD_LEN || f == GTB_FLD_DIST || f == GTB_FLD_X || f == GTB_FLD_Y ||
             f == GTB_FLD_Z || f == GTB_FLD_INSCHORD || f == GTB_FLD_RSD) && !beg[f]) {
            snprintf(h->err, sizeof(h->err), "%s: field %d is null", what, f);
            return GTB_ERR_ARG;
        }
    S.n = (int)((end[GTB_FLD_LEN] - beg[GTB_FLD_LEN]) / (long)sizeof(int));
    S.npos = (long long)(end[GTB_FLD_RSD] - beg[GTB_FLD_RSD]);
    if (S.n < 1 || S.npos < 1) { snprintf(h->err, sizeof(h->err), "%s: empty block", what); return GTB_ERR_ARG; }
    S.len = (const int*)beg[GTB_FLD_LEN];
    S.dist = (const unsigned*)beg[GTB_FLD_DIST];
    S.x = (const float*)beg[GTB_FLD_X]; S.y = (const float*)beg[GTB_FLD_Y]; S.z = (const float*)beg[GTB_FLD_Z];
    S.insch = (const int*)beg[GTB_FLD_INSCHORD];
    S.rsd = beg[GTB_FLD_RSD];
    S.type = (const int*)beg[GTB_FLD_TYPE];
    S.mol.resize(S.n); S.off.resize(S.n);
    for (int i = 0; i < S.n; i++) {
        int L = S.len[i];
        long long d = S.dist[i];
        if (L < 1 || d < 0 || d + L > S.npos) {
            snprintf(h->err, sizeof(h->err), "%s: structure %d has invalid length/offset", what, i);
            return GTB_ERR_ARG;
        }
        if (L > 65535) {
            snprintf(h->err, sizeof(h->err), "%s: structure %d longer than 65535", what, i);
            return GTB_ERR_TOO_LONG;
        }
        S.off[i] = (int)d;
        S.mol[i] = (S.insch[d] > 0) ? 1 : 0;   // GetMoleculeType, PM2DVectorFields.h:98-102
    }
    return GTB_OK;
}

// Pairs of two nucleic-acid structures need the reference's base-pairing
// secondary structure (sskna.cu, MpSecStr.cpp:140-200) and the nucleic-acid
// final d0 (GetD0finNA, stagecnsts.cuh:95-106), which this library does not
// have: blocks that would compare such a pair are refused rather than scored
// with the protein rules.  Protein/nucleic-acid pairs are skipped, as in the
// reference, except under --pre-similarity, which compares them too
// (custage1.cu:74-82), so there any nucleic-acid structure is refused.
static gtb_status check_na_pairs(gtb_handle* h, const std::vector<int>& qmol,
                                 const std::vector<int>& rmol) {
    const bool qna = std::find(qmol.begin(), qmol.end(), 1) != qmol.end();
    const bool rna = std::find(rmol.begin(), rmol.end(), 1) != rmol.end();
    if ((qna && rna) || (0.f < h->opts.presimilarity && (qna || rna))) {
        snprintf(h->err, sizeof(h->err),
                 "nucleic-acid structure pairs are not supported (protein rules would be applied)");
        return GTB_ERR_UNSUPPORTED;
    }
    return GTB_OK;
}

extern "C" size_t gtb_alns_size(char* const* qb, char* const* qe, char* const* rb, char* const* re) {
    if (!qb || !qe || !rb || !re) return 0;
    long long nq = (qe[GTB_FLD_LEN] - qb[GTB_FLD_LEN]) / (long)sizeof(int);
    long long nr = (re[GTB_FLD_LEN] - rb[GTB_FLD_LEN]) / (long)sizeof(int);
    long long Nr = re[GTB_FLD_RSD] - rb[GTB_FLD_RSD];
    const int* ql = (const int*)qb[GTB_FLD_LEN];
    size_t s = 0;
    for (long long i = 0; i < nq; i++) s += (size_t)5 * (Nr + nr * ((long long)ql[i] + 1));
    return s;
}

struct gtb_block {
    int n = 0;
    long long npos = 0;
    std::vector<int> len, off, mol;
    int typemin = 0;                 // smallest global index (clustering runs)
    char* dbase = nullptr;
    int *dlen = nullptr, *doff = nullptr, *dmol = nullptr, *dtype = nullptr;
    float *x = nullptr, *y = nullptr, *z = nullptr;
    float4* c4 = nullptr;
    cudaStream_t st = nullptr;       // stream of the allocation and of the free
    unsigned char* rsd = nullptr;
    unsigned char* odd = nullptr;    // per structure (Blk::qodd)
    char* ss = nullptr;
    // index trees (null: none): node x, y, z; left, right, residue
    float *nx = nullptr, *ny = nullptr, *nz = nullptr;
    int *nl = nullptr, *nr = nullptr, *no = nullptr;
    float4* nd = nullptr;            // the trees packed for the walks (launch_pack_nodes)
    int2* nc = nullptr;
};

// the detailed search needs the blocks' index trees
static bool needs_index(const gtb_handle* h) { return h->opts.nodetailedsearch == 0; }

// ndxbeg: the block's index fields (host), or null: built here when the
// detailed search needs them
static gtb_status upload_block(gtb_handle* h, const HostSoA& S, gtb_block* b,
                               char* const* ndxbeg = nullptr) {
    cudaStream_t st = h->st;
    const bool ndx = needs_index(h);
    std::vector<float> hf;
    std::vector<int> hi;
    const void* src[GTB_NNDXFIELDS] = {};
    if (ndx) {
        if (ndxbeg) {
            for (int f = 0; f < GTB_NNDXFIELDS; f++) {
                if (!ndxbeg[f]) { snprintf(h->err, sizeof(h->err), "null index field %d", f); return GTB_ERR_ARG; }
                src[f] = ndxbeg[f];
            }
            // a caller's trees are walked on the device: every child must be a
            // node of the same structure (or -1) and every residue its own
            const int* nl = (const int*)ndxbeg[GTB_NDX_LEFT];
            const int* nr = (const int*)ndxbeg[GTB_NDX_RIGHT];
            const int* no = (const int*)ndxbeg[GTB_NDX_ORGNDX];
            for (int si = 0; si < S.n; si++) {
                const long long a = S.off[si];
                const int L = S.len[si];
                for (int k = 0; k < L; k++) {
                    if (nl[a + k] < -1 || nl[a + k] >= L || nr[a + k] < -1 || nr[a + k] >= L ||
                        no[a + k] < 0 || no[a + k] >= L) {
                        snprintf(h->err, sizeof(h->err), "index tree of structure %d: node %d out of range", si, k);
                        return GTB_ERR_ARG;
                    }
                }
            }
        } else {
            hf.resize((size_t)3 * S.npos);
            hi.resize((size_t)3 * S.npos);
            if (!gtb::build_index_host(S.n, S.len, S.dist, S.x, S.y, S.z, S.npos, hf.data(),
                                       hf.data() + S.npos, hf.data() + 2 * S.npos, hi.data(),
                                       hi.data() + S.npos, hi.data() + 2 * S.npos)) {
                snprintf(h->err, sizeof(h->err), "inconsistent block for the index");
                return GTB_ERR_ARG;
            }
            for (int f = 0; f < 3; f++) { src[f] = hf.data() + f * S.npos; src[3 + f] = hi.data() + f * S.npos; }
        }
    }
    b->n = S.n; b->npos = S.npos;
    b->len.assign(S.len, S.len + S.n);
    b->off = S.off; b->mol = S.mol;
    // a clustering run's global indices (pps2DType; TdDataReader.cpp:736-745)
    const bool cls = h->opts.clsfilter != 0;
    if (cls && !S.type) { snprintf(h->err, sizeof(h->err), "a clustering run needs the type field"); return GTB_ERR_ARG; }
    if (cls) b->typemin = *std::min_element(S.type, S.type + S.n);
    size_t sz = 0;
    auto carve = [&](size_t bytes) { size_t o2 = sz; sz += align256(bytes); return o2; };
    size_t ol = carve(S.n * 4), oo = carve(S.n * 4), om = carve(S.n * 4);
    size_t ot = cls ? carve(S.n * 4) : 0;
    size_t ox = carve(S.npos * 4), oy = carve(S.npos * 4), oz = carve(S.npos * 4);
    size_t oa = carve(S.npos), os = carve(S.npos);
    size_t o4 = carve(S.npos * 16), od = carve(S.n);
    size_t on = ndx ? carve((size_t)S.npos * 4 * GTB_NNDXFIELDS) : 0;
    size_t ond = ndx ? carve((size_t)S.npos * 16) : 0;
    size_t onc = ndx ? carve((size_t)S.npos * 8) : 0;
    // from the device's memory pool (kept between calls), in stream order
    CK(cudaMallocAsync((void**)&b->dbase, sz, st));
    b->st = st;
    char* d = b->dbase;
    b->dlen = (int*)(d + ol); b->doff = (int*)(d + oo); b->dmol = (int*)(d + om);
    if (cls) {
        b->dtype = (int*)(d + ot);
        CK(cudaMemcpyAsync(b->dtype, S.type, S.n * 4, cudaMemcpyHostToDevice, st));
    }
    b->x = (float*)(d + ox); b->y = (float*)(d + oy); b->z = (float*)(d + oz);
    b->rsd = (unsigned char*)(d + oa); b->ss = d + os;
    b->c4 = (float4*)(d + o4); b->odd = (unsigned char*)(d + od);
    if (ndx) {
        float* nf = (float*)(d + on);
        int* ni = (int*)(nf + 3 * S.npos);
        b->nx = nf; b->ny = nf + S.npos; b->nz = nf + 2 * S.npos;
        b->nl = ni; b->nr = ni + S.npos; b->no = ni + 2 * S.npos;
        b->nd = (float4*)(d + ond); b->nc = (int2*)(d + onc);
        void* dst[GTB_NNDXFIELDS] = {b->nx, b->ny, b->nz, b->nl, b->nr, b->no};
        for (int f = 0; f < GTB_NNDXFIELDS; f++)
            CK(cudaMemcpyAsync(dst[f], src[f], (size_t)S.npos * 4, cudaMemcpyHostToDevice, st));
    }
    CK(cudaMemcpyAsync(b->dlen, S.len, S.n * 4, cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(b->doff, S.off.data(), S.n * 4, cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(b->dmol, S.mol.data(), S.n * 4, cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(b->x, S.x, S.npos * 4, cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(b->y, S.y, S.npos * 4, cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(b->z, S.z, S.npos * 4, cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(b->rsd, S.rsd, S.npos, cudaMemcpyHostToDevice, st));
    long long nl = 0;
    launch_pack4_structs(b->c4, b->odd, b->x, b->y, b->z, b->doff, b->dlen, b->doff, b->n, st);
    launch_secstr(b->ss, b->x, b->y, b->z, b->dlen, b->doff, b->dmol, b->n, st, &nl);
    if (ndx)
        launch_pack_nodes(b->nd, b->nc, b->nx, b->ny, b->nz, b->nl, b->nr, b->no, b->doff, b->dlen,
                          b->ss, S.npos, b->n, st);
    CK(cudaGetLastError());
    return GTB_OK;
}

static void free_block(gtb_block* b) {
    if (!b) return;
    if (b->dbase) cudaFreeAsync(b->dbase, b->st);
    delete b;
}

extern "C" gtb_status gtb_block_upload(gtb_handle* h, char* const* pmbeg, char* const* pmend,
                                       gtb_block** out) {
    return gtb_block_upload_ndx(h, pmbeg, pmend, nullptr, out);
}

extern "C" gtb_status gtb_block_upload_ndx(gtb_handle* h, char* const* pmbeg, char* const* pmend,
                                           char* const* ndxbeg, gtb_block** out) {
    if (!h || !out) return GTB_ERR_ARG;
    *out = nullptr;
    h->err[0] = 0;
    HostSoA S;
    gtb_status s = parse_soa(h, pmbeg, pmend, S, "block");
    if (s != GTB_OK) return s;
    CK(cudaSetDevice(h->dev));
    gtb_block* b = new gtb_block();
    s = upload_block(h, S, b, ndxbeg);
    if (s != GTB_OK) { cudaStreamSynchronize(h->st); free_block(b); return s; }
    CK(cudaStreamSynchronize(h->st));
    *out = b;
    return GTB_OK;
}

extern "C" void gtb_block_free(gtb_handle* h, gtb_block* b) {
    if (h) cudaSetDevice(h->dev);
    free_block(b);
}

static DevBlock make_devblock(const gtb_block* Q, const gtb_block* R) {
    DevBlock D;
    D.nq = Q->n; D.nr = R->n;
    D.qlen = Q->dlen; D.qoff = Q->doff; D.qmol = Q->dmol;
    D.rlen = R->dlen; D.roff = R->doff; D.rmol = R->dmol;
    D.qx = Q->x; D.qy = Q->y; D.qz = Q->z; D.rx = R->x; D.ry = R->y; D.rz = R->z;
    D.q4 = Q->c4; D.r4 = R->c4; D.qodd = Q->odd; D.rodd = R->odd;
    D.qa = Q->rsd; D.ra = R->rsd; D.qs = Q->ss; D.rs = R->ss;
    D.qnd = Q->nd; D.qnc = Q->nc; D.rnd = R->nd; D.rnc = R->nc;
    D.rtype = R->dtype; D.qtypeend = Q->typemin + Q->n;
    D.hqlen = Q->len; D.hrlen = R->len;
    return D;
}

extern "C" gtb_status gtb_process_resident(gtb_handle* h, float scorethld, const gtb_block* queries,
                                           const gtb_block* refs, float* d_alndata, float* d_tfm,
                                           float* d_numerr) {
    if (!h || !queries || !refs || !d_alndata || !d_tfm) return GTB_ERR_ARG;
    h->err[0] = 0;
    if (!(scorethld >= 0.f && scorethld < 1.f)) { snprintf(h->err, sizeof(h->err), "scorethld out of [0,1)"); return GTB_ERR_ARG; }
    gtb_status s = check_options(h);
    if (s != GTB_OK) return s;
    if ((s = check_na_pairs(h, queries->mol, refs->mol)) != GTB_OK) return s;
    CK(cudaSetDevice(h->dev));
    DevBlock D = make_devblock(queries, refs);
    return run_block(h, D, scorethld, d_alndata, d_tfm, d_numerr, nullptr);
}

// ---------------------------------------------------------------------------
// Launch shapes and their autotuner.

static bool tuning_ok(const gtb_tuning& t) {
    return t.seed_chunk >= 128 && t.seed_chunk <= 65536 && t.refine_long_ctas >= 1 &&
           t.refine_long_ctas <= gtb::RLW_CTAS && t.dp_cta_pairs >= 0 &&
           t.dp_cta_pairs <= 65536 && t.sub_pairs >= 1024 && t.sub_pairs <= (1 << 30);
}

extern "C" gtb_status gtb_get_tuning(const gtb_handle* h, gtb_tuning* t) {
    if (!h || !t) return GTB_ERR_ARG;
    *t = h->tn;
    return GTB_OK;
}

extern "C" gtb_status gtb_set_tuning(gtb_handle* h, const gtb_tuning* t) {
    if (!h || !t) return GTB_ERR_ARG;
    if (!tuning_ok(*t)) {
        snprintf(h->err, sizeof(h->err), "tuning field out of range");
        return GTB_ERR_ARG;
    }
    h->tn = *t;
    return GTB_OK;
}

extern "C" gtb_status gtb_autotune(gtb_handle* h, float scorethld, const gtb_block* queries,
                                   const gtb_block* refs, int trials, gtb_tuning* best,
                                   float* best_ms, gtb_tuning_trial* log, int nlog,
                                   int* nlogged) {
    if (!h) return GTB_ERR_ARG;
    h->err[0] = 0;
    if (nlogged) *nlogged = 0;
    if (!queries || !refs || trials < 1 || (nlog > 0 && !log) || !tuning_ok(h->tn)) {
        snprintf(h->err, sizeof(h->err), "autotune: bad arguments");
        return GTB_ERR_ARG;
    }
    const long long np = (long long)queries->n * refs->n;
    if (np <= 0) {
        snprintf(h->err, sizeof(h->err), "autotune: empty block");
        return GTB_ERR_ARG;
    }
    CK(cudaSetDevice(h->dev));
    // the calls' records go to scratch buffers freed on every return
    struct Scratch {
        float *rec = nullptr, *tfm = nullptr;
        ~Scratch() { if (rec) cudaFree(rec); if (tfm) cudaFree(tfm); }
    } sc;
    CK(cudaMalloc((void**)&sc.rec, (size_t)np * GTB_NOUT * sizeof(float)));
    CK(cudaMalloc((void**)&sc.tfm, (size_t)np * 12 * sizeof(float)));
    const gtb_tuning start = h->tn;
    int nl = 0;
    // the least time of `trials` calls under t, after one untimed call
    auto time_one = [&](const gtb_tuning& t, float& ms) -> gtb_status {
        h->tn = t;
        gtb_status s = gtb_process_resident(h, scorethld, queries, refs, sc.rec, sc.tfm, nullptr);
        ms = 3.0e38f;
        for (int k = 0; s == GTB_OK && k < trials; k++) {
            auto t0 = std::chrono::steady_clock::now();
            s = gtb_process_resident(h, scorethld, queries, refs, sc.rec, sc.tfm, nullptr);
            auto t1 = std::chrono::steady_clock::now();
            ms = std::min(ms, std::chrono::duration<float, std::milli>(t1 - t0).count());
        }
        if (s == GTB_OK && nl < nlog) log[nl++] = gtb_tuning_trial{t, ms};
        return s;
    };
    gtb_tuning cur = start;
    float curms = 0.f;
    // one more untimed call first: the device's clocks and memory pool settle
    // during the first calls, which would otherwise count against the start
    gtb_status s = gtb_process_resident(h, scorethld, queries, refs, sc.rec, sc.tfm, nullptr);
    if (s == GTB_OK) s = time_one(cur, curms);
    // one field at a time: its candidates with the others as they stand
    static const int c_seed[] = {256, 512, 1024, 2048};
    static const int c_rlw[] = {4, 8, 16};
    static const int c_dpk[] = {0, 296, 592, 1184};
    static const int c_sub[] = {8192, 16384, 32768};
    struct Field { int gtb_tuning::*f; const int* c; int n; };
    const Field fields[] = {{&gtb_tuning::seed_chunk, c_seed, 4},
                            {&gtb_tuning::refine_long_ctas, c_rlw, 3},
                            {&gtb_tuning::dp_cta_pairs, c_dpk, 4},
                            {&gtb_tuning::sub_pairs, c_sub, 3}};
    for (const Field& fd : fields) {
        const int v0 = cur.*(fd.f);
        for (int k = 0; s == GTB_OK && k < fd.n; k++) {
            if (fd.c[k] == v0) continue;
            gtb_tuning t = cur;
            t.*(fd.f) = fd.c[k];
            float ms = 0.f;
            s = time_one(t, ms);
            if (s == GTB_OK && ms < 0.98f * curms) { cur = t; curms = ms; }
        }
    }
    if (nlogged) *nlogged = nl;
    if (s != GTB_OK) {
        h->tn = start;
        return s;
    }
    h->tn = cur;
    if (best) *best = cur;
    if (best_ms) *best_ms = curms;
    return GTB_OK;
}

extern "C" gtb_status gtb_process_block(gtb_handle* h, float scorethld,
                                        char* const* querypmbeg, char* const* querypmend,
                                        char* const* bdbCpmbeg, char* const* bdbCpmend,
                                        gtb_results* out) {
    return gtb_process_block_ndx(h, scorethld, querypmbeg, querypmend, nullptr, bdbCpmbeg,
                                 bdbCpmend, nullptr, out);
}

extern "C" gtb_status gtb_process_block_ndx(gtb_handle* h, float scorethld,
                                            char* const* querypmbeg, char* const* querypmend,
                                            char* const* queryndxpmbeg,
                                            char* const* bdbCpmbeg, char* const* bdbCpmend,
                                            char* const* bdbCndxpmbeg, gtb_results* out) {
    if (!h) return GTB_ERR_ARG;
    h->err[0] = 0;
    if (!out || !out->alndata || !out->tfm) { snprintf(h->err, sizeof(h->err), "null result buffers"); return GTB_ERR_ARG; }
    if (!(scorethld >= 0.f && scorethld < 1.f)) { snprintf(h->err, sizeof(h->err), "scorethld out of [0,1)"); return GTB_ERR_ARG; }
    gtb_status s = check_options(h);
    if (s != GTB_OK) return s;
    HostSoA Q, R;
    if ((s = parse_soa(h, querypmbeg, querypmend, Q, "queries")) != GTB_OK) return s;
    if ((s = parse_soa(h, bdbCpmbeg, bdbCpmend, R, "references")) != GTB_OK) return s;
    if ((s = check_na_pairs(h, Q.mol, R.mol)) != GTB_OK) return s;
    CK(cudaSetDevice(h->dev));
    cudaStream_t st = h->st;
    gtb_block* qb = new gtb_block();
    gtb_block* rb = new gtb_block();
    s = upload_block(h, Q, qb, queryndxpmbeg);
    if (s == GTB_OK) s = upload_block(h, R, rb, bdbCndxpmbeg);
    if (s != GTB_OK) { cudaStreamSynchronize(st); free_block(qb); free_block(rb); return s; }
    DevBlock D = make_devblock(qb, rb);

    // alignment rows go straight from the packed device rows to the caller's
    // buffer in the reference layout
    AlnSink sink;
    if (out->alns) {
        sink.alns = out->alns;
        sink.rec = out->alndata;
        sink.nr = R.n;
        sink.qlen.assign(Q.len, Q.len + Q.n);
        sink.rlen.assign(R.len, R.len + R.n);
        sink.roff = R.off;
        long long base = 0;
        for (int qi = 0; qi < Q.n; qi++) {
            long long rowlen = R.npos + (long long)R.n * (Q.len[qi] + 1);
            sink.qbase.push_back(base);
            sink.rowlen.push_back(rowlen);
            base += 5 * rowlen;
        }
    }
    s = run_block(h, D, scorethld, out->alndata, out->tfm, out->numerr, out->alns ? &sink : nullptr);
    h->launches += 2;  // secondary-structure launches of the two uploads
    if (s == GTB_OK) {
        cudaError_t e1 = cudaSuccess;
        if (out->qss) e1 = cudaMemcpyAsync(out->qss, qb->ss, Q.npos, cudaMemcpyDeviceToHost, st);
        if (e1 == cudaSuccess && out->rss) e1 = cudaMemcpyAsync(out->rss, rb->ss, R.npos, cudaMemcpyDeviceToHost, st);
        if (e1 == cudaSuccess) e1 = cudaStreamSynchronize(st);
        if (e1 != cudaSuccess) {
            snprintf(h->err, sizeof(h->err), "result copy: %s", cudaGetErrorString(e1));
            s = GTB_ERR_CUDA;
        }
    }
    cudaStreamSynchronize(st);
    free_block(qb);
    free_block(rb);
    return s;
}
