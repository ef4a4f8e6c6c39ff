// probe.cu -- FP64 fused multiply-add issue-rate probe (the FP64 roofline denominator),
// self-tests of the integer-pipe product and quotient and of the forms built on them
// (fp64ops.cuh, combine_cells.cuh) against the FP64 unit, and one of the bit-pattern MinMod
// and Superbee (common.cuh) against their fmin/fmax expressions.  Eight independent dependency chains per thread keep the FP64 pipe busy;
// every thread writes one result, so nothing is optimised away and every store is in bounds.
#include <cuda_runtime.h>

#include <cstring>
#include <vector>

#include "combine_cells.cuh"

namespace hgpu {
namespace {
constexpr int kIter = 4096;
__global__ void __launch_bounds__(256) dfmaProbe(double* out, double a, double b) {
    double x0 = threadIdx.x, x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3, x4 = x0 + 4, x5 = x0 + 5, x6 = x0 + 6, x7 = x0 + 7;
    for (int i = 0; i < kIter; ++i) {
        x0 = fma(x0, a, b); x1 = fma(x1, a, b); x2 = fma(x2, a, b); x3 = fma(x3, a, b);
        x4 = fma(x4, a, b); x5 = fma(x5, a, b); x6 = fma(x6, a, b); x7 = fma(x7, a, b);
    }
    out[(size_t)blockIdx.x * blockDim.x + threadIdx.x] = ((x0 + x1) + (x2 + x3)) + ((x4 + x5) + (x6 + x7));
}
__host__ __device__ __forceinline__ unsigned long long splitmix(unsigned long long z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// operand classes: any exponent (zeros, subnormals, Inf/NaN included), moderate
// exponents, short significands (exact products/quotients, powers of two), extremes,
// exact zeros / infinities / NaNs
__device__ double operand(unsigned long long s, int cls) {
    const unsigned long long r = splitmix(s), m = r & 0xFFFFFFFFFFFFFull, sg = (r >> 63) << 63;
    const unsigned long long t = splitmix(s ^ 0x5bd1e995ull);
    unsigned e;
    unsigned long long mm = m;
    if (cls == 0) e = (unsigned)(t % 2048);
    else if (cls == 1) e = 1023 - 60 + (unsigned)(t % 120);
    else if (cls == 2) { e = 1023 - 4 + (unsigned)(t % 8); mm = m & ~((1ull << (t >> 32) % 53) - 1); }
    else if (cls == 3) e = (t & 1) ? (unsigned)(t % 40) : 2047 - (unsigned)(t % 40);
    else { e = (t & 2) ? 0 : 2047; mm = (t & 4) ? 0 : (t & 8) ? mm : 1; }      // zeros, infinities, NaNs
    return fromBits((long long)(sg | ((unsigned long long)e << 52) | mm));
}

__global__ void selftestKernel(unsigned long long seed, long long cases, unsigned long long* bad) {
    unsigned long long nm = 0, nd = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < cases;
         i += (long long)gridDim.x * blockDim.x) {
        const unsigned long long s = splitmix(seed + (unsigned long long)i);
        const double x = operand(s, (int)(s % 5)), y = operand(s ^ 0xabcdefull, (int)((s >> 8) % 5));
        const double pm = x * y, qm = mulI(x, y), pd = x / y, qd = divI(x, y);
        if (bitsOf(pm) != bitsOf(qm) && !(pm != pm && qm != qm)) ++nm;
        if (bitsOf(pd) != bitsOf(qd) && !(pd != pd && qd != qd)) ++nd;
    }
    if (nm) atomicAdd(&bad[0], nm);
    if (nd) atomicAdd(&bad[1], nd);
}

__device__ __forceinline__ bool differ(double a, double b) { return bitsOf(a) != bitsOf(b) && !(a != a && b != b); }
__device__ __forceinline__ bool differ(float a, float b) {
    return __float_as_uint(a) != __float_as_uint(b) && !(a != a && b != b);
}
// a number of GroupPlain's window, [2^-480, 2^481)
__device__ double windowOperand(unsigned long long s) {
    const double x = operand(s, (int)(s % 3) == 2 ? 2 : 1);
    const unsigned e = 543u + (unsigned)(splitmix(s ^ 0x77ull) % 961);
    return fromBits((bitsOf(x) & (long long)0x800FFFFFFFFFFFFFull) | ((long long)e << 52));
}
__device__ __forceinline__ bool windowed(double x) { return fabs(x) >= 0x1p-480 && fabs(x) < 0x1p481; }

// floats for c - a b: any bits; c beside a b; c - a b beside a midpoint of two floats, by less
// than a double resolves; c a power of two; a b = (2^25 - 1) 2^103, the midpoint between the
// largest float and 2^128, or a huge product, beside a c of any size
__device__ void subOperands(unsigned long long s, float& c, float& a, float& b) {
    const unsigned long long r = splitmix(s), t = splitmix(s ^ 0x51ull);
    const unsigned sc = (unsigned)(t >> 60 & 1) << 31, sa = (unsigned)(t >> 61 & 1) << 31, sb = (unsigned)(t >> 62 & 1) << 31;
    const int cls = (int)(s % 5);
    if (cls == 0) {
        c = __uint_as_float((unsigned)r);
        a = __uint_as_float((unsigned)(r >> 32));
        b = __uint_as_float((unsigned)t);
        return;
    }
    if (cls == 4) {
        c = __uint_as_float(sc | (1u + (unsigned)(r % 254)) << 23 | ((unsigned)(r >> 16) & 0x7FFFFFu));
        a = __uint_as_float(sa | (unsigned)__float_as_int(18631.f * 0x1p60f));
        b = __uint_as_float(sb | (unsigned)__float_as_int(1801.f * 0x1p43f));
        if (t & 1) b = __uint_as_float(sb | 180u << 23 | ((unsigned)(t >> 8) & 0x7FFFFFu));
        return;
    }
    const unsigned ea = 100u + (unsigned)(r % 50), eb = 100u + (unsigned)(r >> 8) % 50;
    a = __uint_as_float(sa | ea << 23 | ((unsigned)(r >> 16) & 0x7FFFFFu));
    b = __uint_as_float(sb | eb << 23 | ((unsigned)(t >> 16) & 0x7FFFFFu));
    if (cls == 1) {
        c = a * b * (1.f + (float)((int)(t % 9) - 4) * 0x1p-23f);
        return;
    }
    // |a b| = 2^(ea + eb - 254) (1 - i^2 2^-46), half an ulp of c or next to it
    const unsigned i = 1u + (unsigned)(t >> 40) % 2000;
    a = __uint_as_float(sa | ea << 23 | i);
    b = __uint_as_float(sb | eb << 23) * (1.f - (float)i * 0x1p-23f);
    const unsigned ec = ea + eb - 127u + 24u - (unsigned)(r >> 40) % 2;
    c = __uint_as_float(sc | ec << 23 | (cls == 3 ? 0u : (unsigned)(r >> 41) & 0x7FFFFFu));
}

constexpr int kDivisors = 1 << 14;

// bad: sqrtI; quotients by a shared divisor (quotBy, quotPlain); the groups and CheckedOps;
// addEqual; subProduct
__global__ void arithSelftestKernel(unsigned long long seed, long long cases, const Divisor<double>* hostDivs,
                                    unsigned long long* bad) {
    unsigned long long n[5] = {};
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < cases;
         i += (long long)gridDim.x * blockDim.x) {
        const unsigned long long s = splitmix(seed + (unsigned long long)i);
        const double x = operand(s, (int)(s % 5)), y = operand(s ^ 0xabcdefull, (int)((s >> 8) % 5));
        n[0] += differ(sqrt(x), sqrtI(x)) + differ(sqrt(fabs(x)), sqrtI(fabs(x)));

        const Divisor<double> h = hostDivs[(s >> 16) % kDivisors];
        n[1] += differ(x / y, quotBy(x, divisorOf(y))) + differ(x / h.b, quotBy(x, h));
        const double wx = windowOperand(s ^ 0x33ull), wy = windowOperand(s ^ 0x44ull);
        n[1] += differ(wx / wy, quotPlain(wx, divisorOf(wy)));
        if (windowed(h.b)) n[1] += differ(wx / h.b, quotPlain(wx, h));

        n[2] += differ(wx * wy, GroupPlain::mul(wx, wy)) + differ(wx / wy, GroupPlain::div(wx, wy)) +
                differ(wx * wy * .5, GroupPlain::half(wx * wy));
        // zeros of either sign in the place of one operand, the other or both
        const double zx = (s >> 30 & 1) ? wx : fromBits(bitsOf(wx) & (long long)0x8000000000000000ull);
        const double zy = (s >> 31 & 1) ? wy : fromBits(bitsOf(wy) & (long long)0x8000000000000000ull);
        n[2] += differ(zx * zy, GroupZeros::mul(zx, zy)) + differ(zx / zy, GroupZeros::div(zx, zy)) +
                differ(zx * zy * .5, GroupZeros::half(zx * zy));
        // CheckedOps: `ok` exactly for operands of the window, and then the IEEE results
        const double ox = (s >> 32 & 1) ? x : wx, oy = (s >> 33 & 1) ? y : wy;
        const bool both = windowed(ox) && windowed(oy);
        CheckedOps m, d, q, r, f;
        const double om = m.mul(ox, oy), od = d.div(ox, oy), orr = r.root(ox), oh = f.half(ox);
        CheckedOps w;
        const double ow = w.twice(ox);
        const double oq = q.quot(ox, q.divisor(oy));
        n[2] += (m.ok != both) + (d.ok != both) + (q.ok != both) + (r.ok != (windowed(ox) && ox > 0.)) +
                (f.ok != windowed(ox)) + (w.ok != windowed(ox));
        if (m.ok) n[2] += differ(ox * oy, om);
        if (d.ok) n[2] += differ(ox / oy, od);
        if (q.ok) n[2] += differ(ox / oy, oq);
        if (r.ok) n[2] += differ(sqrt(ox), orr);
        if (f.ok) n[2] += differ(ox * .5, oh);
        if (w.ok) n[2] += differ(ox * 2., ow);

        // addEqual's operands: the same number, a zero beside a number that is not -0, or any
        const double e = bitsOf(x) == (long long)0x8000000000000000ull ? 0. : x;
        n[3] += differ(e + e, addEqual(e, e)) + differ(e + 0., addEqual(e, 0.)) + differ(e + -0., addEqual(e, -0.)) +
                differ(e + wy, addEqual(e, wy));

        float c, a, b;
        subOperands(s ^ 0x99ull, c, a, b);
        n[4] += differ(__double2float_rn(__dsub_rn((double)c, __dmul_rn((double)a, (double)b))), subProduct(c, a, b));
    }
    for (int k = 0; k < 5; ++k)
        if (n[k]) atomicAdd(&bad[k], n[k]);
}
// the limiters' res/SlopeLimiter.cl expressions with C-library fmin/fmax semantics
__device__ double minmodExpr(double r) { return fmaxLibm(0., fminLibm(r, 1.)); }
__device__ double superbeeExpr(double r) { return fmaxLibm(0., fmaxLibm(fminLibm(1., 2. * r), fminLibm(2., r))); }

// r: a seeded operand of any class, or a quotient of two (the ratios the flux forms)
__global__ void limiterSelftestKernel(unsigned long long seed, long long cases, unsigned long long* bad) {
    unsigned long long n = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < cases;
         i += (long long)gridDim.x * blockDim.x) {
        const unsigned long long s = splitmix(seed + (unsigned long long)i);
        double r = operand(s, (int)(s % 5));
        if ((s >> 40) & 1) r = r / operand(s ^ 0x1234567ull, (int)((s >> 8) % 5));
        if (bitsOf(minmodBits(r)) != bitsOf(minmodExpr(r))) ++n;
        if (bitsOf(superbeeBits(r)) != bitsOf(superbeeExpr(r))) ++n;
    }
    if (n) atomicAdd(bad, n);
}
}  // namespace

// mismatches (bit patterns, signs of zero included) of the bit-pattern MinMod and
// Superbee against their expressions over `cases` seeded ratios
int selftestLimiters(unsigned long long seed, long long cases, long long* bad) {
    unsigned long long* d = nullptr;
    if (cudaMalloc(&d, sizeof(unsigned long long)) != cudaSuccess) return -1;
    cudaMemset(d, 0, sizeof(unsigned long long));
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    limiterSelftestKernel<<<sms * 8, 256>>>(seed, cases, d);
    unsigned long long h = 0;
    cudaError_t e = cudaMemcpy(&h, d, sizeof h, cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) return -1;
    *bad = (long long)h;
    return 0;
}

// mismatches over `cases` seeded operands of arithSelftestKernel's five groups of forms
int selftestArith(unsigned long long seed, long long cases, long long* mismatches) {
    std::vector<Divisor<double>> divs(kDivisors);
    for (int i = 0; i < kDivisors; ++i) {
        // any bits, ordinary exponents, short significands and powers of two, subnormals
        unsigned long long u = splitmix(seed ^ splitmix((unsigned long long)i)), t = splitmix(u);
        if (i % 4) u = (u & 0x800FFFFFFFFFFFFFull) | ((963 + t % 120) << 52);
        if (i % 4 == 2) u &= ~((1ull << t % 53) - 1);
        if (i % 64 == 3) u &= 0x800FFFFFFFFFFFFFull;
        double b;
        std::memcpy(&b, &u, 8);
        hostDivisor(b, divs[i]);
    }
    Divisor<double>* d = nullptr;
    unsigned long long* bad = nullptr;
    if (cudaMalloc(&d, sizeof(Divisor<double>) * kDivisors) != cudaSuccess) return -1;
    if (cudaMalloc(&bad, 5 * sizeof(unsigned long long)) != cudaSuccess) {
        cudaFree(d);
        return -1;
    }
    cudaMemcpy(d, divs.data(), sizeof(Divisor<double>) * kDivisors, cudaMemcpyHostToDevice);
    cudaMemset(bad, 0, 5 * sizeof(unsigned long long));
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    arithSelftestKernel<<<sms * 8, 256>>>(seed, cases, d, bad);
    unsigned long long h[5] = {};
    const cudaError_t e = cudaMemcpy(h, bad, sizeof h, cudaMemcpyDeviceToHost);
    cudaFree(d);
    cudaFree(bad);
    if (e != cudaSuccess) return -1;
    for (int k = 0; k < 5; ++k) mismatches[k] = (long long)h[k];
    return 0;
}

// mismatches of mulI and divI against the FP64 unit over `cases` seeded operand pairs
int selftestFp64Ops(unsigned long long seed, long long cases, long long* mulBad, long long* divBad) {
    unsigned long long* bad = nullptr;
    if (cudaMalloc(&bad, 2 * sizeof(unsigned long long)) != cudaSuccess) return -1;
    cudaMemset(bad, 0, 2 * sizeof(unsigned long long));
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    selftestKernel<<<sms * 8, 256>>>(seed, cases, bad);
    unsigned long long h[2] = {0, 0};
    cudaError_t e = cudaMemcpy(h, bad, sizeof h, cudaMemcpyDeviceToHost);
    cudaFree(bad);
    if (e != cudaSuccess) return -1;
    *mulBad = (long long)h[0];
    *divBad = (long long)h[1];
    return 0;
}

// returns fma instructions per second over the whole device, or a negative value on error
double measureFp64FmaRate() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return -1;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -1;
    int blocks = sms * 8, threads = 256;
    double* out = nullptr;
    if (cudaMalloc(&out, sizeof(double) * (size_t)blocks * threads) != cudaSuccess) return -1;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    dfmaProbe<<<blocks, threads>>>(out, 0.999999, 1e-7);
    cudaEventRecord(e0);
    const int reps = 5;
    for (int r = 0; r < reps; ++r) dfmaProbe<<<blocks, threads>>>(out, 0.999999, 1e-7);
    cudaEventRecord(e1);
    cudaError_t err = cudaEventSynchronize(e1);
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(out);
    if (err != cudaSuccess || ms <= 0) return -1;
    double fmas = 8.0 * kIter * (double)blocks * threads * reps;
    return fmas / (ms * 1e-3);
}
}  // namespace hgpu
