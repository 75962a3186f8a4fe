// Counts where the operations of csrc/rounded.cuh differ from CUDA's rounded
// ones (__ddiv_rn, __drcp_rn, __dsqrt_rn), one line per operation and operand
// set: operation, set, exponents, operands tested, operands the check refuses,
// differences, differences of more than a unit in the last place.
//
// Operand sets: random significands; `near`, one rounding away from the middle m
// of two neighbouring doubles (a = b m, a = m m, b = 1 / m); `hard`, as near to it
// as exact arithmetic allows: for a quotient integers with A 2^j = B M + c (M of 54
// bits and odd, so M / 2^j is such a middle; M = -c / B modulo 2^j), for a root A 2^j
// = M M - c (M a square root of c modulo 2^j), c small; `ones`, significands next
// to all ones (the exception of Markstein's reciprocal) and to one.
#include <cstdio>
#include <cstdlib>
#include <cuda_runtime.h>

#include "rounded.cuh"

using namespace sphgpu;

__device__ unsigned long long mix(unsigned long long x)
{
    // SplitMix64 (G. Steele, D. Lea and C. Flood, 2014)
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

// 1 <= |x| < 2 times 2^(-span .. span)
__device__ double operand(unsigned long long bits, int span)
{
    const int e = (int)((bits >> 52) % (2 * span + 1)) - span;
    return __longlong_as_double((long long)((bits & 0xfffffffffffffull) | ((unsigned long long)(1023 + e) << 52)));
}

__device__ bool differ(double x, double y) { return __double_as_longlong(x) != __double_as_longlong(y); }

enum { DIV, OVER, INVERSE, ANY, ROOT, RSQRT, NOPS };
enum { RANDOM, NEAR, HARD, ONES };

// a / b next to a middle: false if this draw has none
__device__ bool hard_quotient(unsigned long long r0, unsigned long long r1, double& a, double& b)
{
    const unsigned long long B = (1ull << 52) | (r0 & 0xfffffffffffffull) | 1ull;
    const unsigned long long c = (unsigned long long)((long long)(r1 % 65) * 2 - 65);  // odd, -65 .. 63
    const int j = 53 + (int)((r1 >> 32) & 1u);
    unsigned long long inv = B;
    for(int k = 0; k < 6; ++k) inv *= 2ull - B * inv;
    unsigned long long M = (0ull - c) * inv & ((1ull << j) - 1ull);
    if(j == 53) M |= 1ull << 53;
    if(M < (1ull << 53)) return false;
    // (B M + c) / 2^j in 128 bits
    unsigned long long lo = B * M, hi = __umul64hi(B, M);
    const unsigned long long s = lo + c;
    hi += (s < lo ? 1ull : 0ull) - ((long long)c < 0 ? 1ull : 0ull);
    const unsigned long long A = (hi << (64 - j)) | (s >> j);
    if(A >= (1ull << 53) || (s & ((1ull << j) - 1ull)) != 0) return false;
    a = (double)A;
    b = (double)B;
    return true;
}

// sqrt(a) next to a middle
__device__ bool hard_root(unsigned long long r0, unsigned long long r1, double& a)
{
    const long long c = (long long)(r0 % (1ull << 24)) * 8 - (1ll << 26) + 1;  // 1 modulo 8: a square modulo 2^j
    const int j = 54 + (int)(r1 & 1u);
    unsigned long long M = 1;
    for(int k = 3; k < j; ++k) {  // M M = c modulo 2^k -> modulo 2^(k + 1)
        if(((M * M - (unsigned long long)c) >> k) & 1ull) M += 1ull << (k - 1);
    }
    if((r1 >> 1) & 1u) M = 0ull - M;
    if((r1 >> 2) & 1u) M += 1ull << (j - 1);
    M &= (1ull << j) - 1ull;
    if(M < (1ull << 53) || M >= (1ull << 54)) return false;
    const unsigned long long lo = M * M, hi = __umul64hi(M, M), s = lo - (unsigned long long)c;
    const unsigned long long h = hi - (c > 0 ? (lo < (unsigned long long)c ? 1ull : 0ull) : 0ull)
        + (c < 0 ? (s < lo ? 1ull : 0ull) : 0ull);
    if((s & ((1ull << j) - 1ull)) != 0) return false;
    const unsigned long long A = (h << (64 - j)) | (s >> j);
    if(A >= (1ull << 53)) return false;
    a = (double)A * (j & 1 ? 2.0 : 1.0);
    return true;
}

__global__ void k_compare(int op, int set, int span, unsigned long long seed, long long n, unsigned long long* out)
{
    unsigned long long tested = 0, refused = 0, wrong = 0, far = 0;
    for(long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const unsigned long long r0 = mix(seed + 2 * (unsigned long long)i), r1 = mix(seed + 2 * (unsigned long long)i + 1);
        double b = operand(r0, span), a = operand(r1, span);
        if(set == NEAR) {
            const double x = operand(r1, span / 2), half = 0x1p-53 * operand(r1 & ~0xfffffffffffffull, span / 2);
            if(op == DIV || op == OVER) {
                b = operand(r0, span / 2);
                a = __fma_rn(b, x, b * half);
            } else if(op == ROOT) {
                a = __fma_rn(x, x, 2.0 * x * half);
            } else {
                a = b = 1.0 / x;
            }
        } else if(set == HARD) {
            if(op == DIV || op == OVER ? !hard_quotient(r0, r1, a, b) : !hard_root(r0, r1, a)) continue;
        }
        if(set == ONES) {
            // significands within 8 of all ones, or of one; for a root, of their squares
            const long long one = 0x3ff0000000000000ll + (((long long)(r0 >> 40) % (2 * span + 1) - span) << 52);
            b = __longlong_as_double(one + (long long)(r0 % 17) - 8);
            if(op == ROOT || op == RSQRT) {
                a = r1 >> 63 ? __dmul_rn(b, b) : b;
                a = __longlong_as_double(__double_as_longlong(a) + (long long)(r1 % 9) - 4);
            }
            else a = r1 >> 60 ? operand(r1, span / 2) : 1.0;
        }
        ++tested;
        Quick q;
        double got, want;
        if(op == DIV) {
            got = q.div(a, b);
            want = __ddiv_rn(a, b);
        } else if(op == OVER) {
            got = q.over(a, b, q.inverse(b));
            want = __ddiv_rn(a, b);
        } else if(op == INVERSE) {
            got = q.inverse(b);
            want = __drcp_rn(b);
        } else if(op == ANY) {
            // from a y a few units off, as the walk's cube has it
            const double y = __longlong_as_double(__double_as_longlong(recip_rn(b)) + (long long)(r1 >> 61) - 3);
            got = q.check(recip_any(b, y));
            want = __drcp_rn(b);
        } else if(op == ROOT) {
            got = q.root(a);
            want = __dsqrt_rn(a);
        } else {
            // the gravity walk's monopole
            const double y = rsqrt_near(a);
            got = q.check(recip_rn(root_rn(a, y), y));
            q.bad = q.bad || !root_not_ones(a);
            want = __drcp_rn(__dsqrt_rn(a));
        }
        if(q.bad) ++refused;
        else if(differ(got, want)) {
            ++wrong;
            const long long d = __double_as_longlong(got) - __double_as_longlong(want);
            if(d > 1 || d < -1) ++far;
        }
    }
    atomicAdd(&out[0], tested);
    atomicAdd(&out[1], refused);
    atomicAdd(&out[2], wrong);
    atomicAdd(&out[3], far);
}

int main(int argc, char** argv)
{
    const long long n = argc > 1 ? atoll(argv[1]) : 1ll << 26;
    const char* names[NOPS] = {"div", "over", "inverse", "any", "root", "rsqrt"};
    const char* sets[4] = {"random", "near", "hard", "ones"};
    unsigned long long* d = nullptr;
    if(cudaMalloc(&d, 4 * sizeof(*d)) != cudaSuccess) return 1;
    for(int op = 0; op < NOPS; ++op) {
        for(int set = 0; set < 4; ++set) {
            if(set == HARD && (op == INVERSE || op == ANY)) continue;
            for(int span : {290, 1}) {
                unsigned long long h[4] = {0, 0, 0, 0};
                cudaMemset(d, 0, sizeof(h));
                k_compare<<<148 * 8, 256>>>(op, set, span, 0x1234567ull * (2 * set + (span > 1) + 1), n, d);
                if(cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
                std::printf("%s %s %d %llu %llu %llu %llu\n", names[op], sets[set], span, h[0], h[1], h[2], h[3]);
                if(set == HARD) break;
            }
        }
    }
    cudaFree(d);
    return 0;
}
