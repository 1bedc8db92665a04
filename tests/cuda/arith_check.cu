// The arithmetic of gtb_device.cuh against CUDA's own: counts the operands for
// which a branch-free quotient, reciprocal or rotation solve differs in a bit
// from the IEEE division or from the solve written with IEEE divisions.
#include <cstring>
#include <cuda_runtime.h>
#include "gtb_device.cuh"

using namespace gtb;

namespace {

struct Rng {                                   // xorshift64* (Marsaglia, Vigna)
    unsigned long long s;
    __device__ unsigned long long next() {
        s ^= s >> 12; s ^= s << 25; s ^= s >> 27;
        return s * 0x2545F4914F6CDD1Dull;
    }
};

// a float with an exponent in [lo, hi]; one in four has a mantissa of all
// zeros or ones but for two low bits
__device__ float rnd32(Rng& g, int lo, int hi) {
    const unsigned long long u = g.next();
    unsigned m = (unsigned)u & 0x7fffffu;
    if ((u >> 24 & 3) == 0) m = (m & 3u) ^ (u >> 26 & 1 ? 0x7fffffu : 0u);
    const unsigned e = 127 + lo + (unsigned)((u >> 32) % (unsigned)(hi - lo + 1));
    return __uint_as_float(e << 23 | m);
}
__device__ double rnd64(Rng& g, int lo, int hi) {
    const unsigned long long u = g.next(), w = g.next();
    unsigned long long m = w >> 12;
    if ((u & 3) == 0) m = (m & 3) ^ (u >> 2 & 1 ? 0xfffffffffffffull : 0ull);
    const unsigned long long e = 1023 + lo + (u >> 32) % (unsigned)(hi - lo + 1);
    return __longlong_as_double((long long)(e << 52 | m));
}
__device__ bool same(float a, float b) {
    return __float_as_uint(a) == __float_as_uint(b) || (isnan(a) && isnan(b));
}
__device__ bool same(double a, double b) {
    return __double_as_longlong(a) == __double_as_longlong(b) || (isnan(a) && isnan(b));
}
__device__ bool all_ones(double b) {
    return ((unsigned long long)__double_as_longlong(b) & 0xfffffffffffffull) == 0xfffffffffffffull;
}

enum { TMTERM = 0, TMTERM_ENDS = 1, DIV_ORD = 2, DIV2_NEG = 3, RECIP64 = 4, DIV64 = 5, SOLVE = 6, MANTISSAS = 7 };

__device__ bool check(int what, long long i, Rng& g, double* op) {
    if (what == TMTERM || what == TMTERM_ENDS) {
        const float a = rnd32(g, -3, 12);
        float d = rnd32(g, -40, 127);
        if (what == TMTERM_ENDS) {
            const float ends[8] = {0.f, 1.17549435e-38f, 3.40282347e38f, 8.5070592e37f, 8.507058e37f,
                                   1e-45f, __int_as_float(0x7f800000), __int_as_float(0x7fc00000)};
            d = ends[i & 7];
        }
        op[0] = a; op[1] = d;
        return same(tmterm(a, d), __fdiv_rn(a, __fadd_rn(a, d)));
    }
    if (what == DIV_ORD) {
        const float a = rnd32(g, -3, 12), b = __fadd_rn(a, rnd32(g, -30, 120));
        op[0] = a; op[1] = b;
        return same(div_ord(a, b), __fdiv_rn(a, b));
    }
    if (what == DIV2_NEG) {
        const float a = rnd32(g, -3, 12), b0 = __fadd_rn(a, rnd32(g, -30, 120)),
                    b1 = __fadd_rn(a, rnd32(g, -30, 120));
        float x, y;
        unpack2(div2_neg(pack2(a, a), pack2(b0, b1), pack2(1.f, 1.f)), x, y);
        op[0] = a; op[1] = b0; op[2] = b1;
        return same(x, -__fdiv_rn(a, b0)) && same(y, -__fdiv_rn(a, b1));
    }
    if (what == MANTISSAS) {
        // every mantissa of the denominator against chosen ones of the numerator
        const unsigned mb = (unsigned)i & 0x7fffffu, k = (unsigned)(i >> 23) & 15u;
        const unsigned ma = k < 4 ? k : k < 8 ? 0x7fffffu - (k - 4) : k < 12 ? 1u << (k + 10) : (unsigned)(g.next() & 0x7fffffu);
        const float a = __uint_as_float(127u << 23 | ma), b = __uint_as_float(130u << 23 | mb);
        op[0] = a; op[1] = b;
        return same(div_ord(a, b), __fdiv_rn(a, b)) && same(div_pos(a, b), __fdiv_rn(a, b));
    }
    if (what == RECIP64 || what == DIV64) {
        const double b = rnd64(g, -400, 400), a = rnd64(g, -400, 400);
        op[0] = a; op[1] = b;
        if (all_ones(b)) return true;          // the one mantissa that is excepted
        const double y = div64_recip(b);
        return what == RECIP64 ? same(y, __drcp_rn(b)) : same(div64_by(a, b, y), __ddiv_rn(a, b));
    }
    // SOLVE: the sums of a few random points, some of them degenerate or out of range
    float v[16];
    for (int f = 0; f < 16; f++) v[f] = 0.f;
    const unsigned long long u = g.next();
    const int n = 1 + (int)(u & 31), kind = (int)(u >> 8 & 15);
    const float sc = kind == 0 ? 1e-24f : kind == 1 ? 1e17f : kind == 2 ? 1e9f : 20.f;
    for (int k = 0; k < n; k++) {
        float q[3], r[3];
        for (int c = 0; c < 3; c++) {
            q[c] = sc * (float)((long long)g.next() >> 32) * 0x1p-31f;
            r[c] = sc * (float)((long long)g.next() >> 32) * 0x1p-31f;
            if (kind == 3 && c > 0) q[c] = r[c] = q[0];            // on a line
            if (kind >= 8) r[c] = (c == 1 ? -q[c] : q[c]) + 0.02f * r[c];
            if (kind == 4) q[c] = r[c] = 3.f;                       // a point
        }
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++) v[3 * a + b] = __fmaf_rn(q[a], r[b], v[3 * a + b]);
        for (int c = 0; c < 3; c++) { v[9 + c] += q[c]; v[12 + c] += r[c]; }
    }
    v[15] = (float)n;
    if (kind == 5) v[(int)(u >> 16 & 7)] = __int_as_float(u >> 20 & 1 ? 0x7f800000 : 0x7fc00000);
    bool ok = true;
    for (int swap = 0; swap < 3; swap++) {
        float x[12], y[12];
        solve_sums(v, swap, x);
        solve_sums_any(v, swap, y);
        for (int f = 0; f < 12; f++) ok = ok && same(x[f], y[f]);
    }
    op[0] = kind; op[1] = n;
    return ok;
}

__global__ void k_check(int what, unsigned long long seed, long long n, unsigned long long* bad, double* first) {
    const long long step = (long long)gridDim.x * blockDim.x;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    Rng g{(seed + 1) * 0x9E3779B97F4A7C15ull ^ (unsigned long long)(i + 1) * 0xBF58476D1CE4E5B9ull};
    for (int k = 0; k < 4; k++) g.next();
    for (; i < n; i += step) {
        double op[3] = {0., 0., 0.};
        if (!check(what, i, g, op) && atomicAdd(bad, 1ull) == 0)
            for (int k = 0; k < 3; k++) first[k] = op[k];
    }
}

}  // namespace

// the number of differing operands among n, and the first one's values; returns a CUDA error code
extern "C" int arith_check(int what, unsigned long long seed, long long n, unsigned long long* bad, double* first) {
    unsigned long long* d = nullptr;
    cudaError_t e = cudaMalloc(&d, 4 * sizeof(double));
    if (e == cudaSuccess) e = cudaMemset(d, 0, 4 * sizeof(double));
    if (e == cudaSuccess) {
        k_check<<<148 * 8, 256>>>(what, seed, n, d, (double*)(d + 1));
        e = cudaGetLastError();
    }
    double h[4];
    if (e == cudaSuccess) e = cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) {
        memcpy(bad, h, sizeof(*bad));
        memcpy(first, h + 1, 3 * sizeof(double));
    }
    cudaFree(d);
    return (int)e;
}
