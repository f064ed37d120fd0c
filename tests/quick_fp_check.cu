// Bit-for-bit comparison of quick_fp.cuh's reciprocal, quotient, square root and arc
// cosine with the plain operators. Prints one line per form: name, values compared,
// values whose range check refused them, mismatches.
#include "quick_fp.cuh"
#include <cstdio>

using namespace sc;

__device__ unsigned long long g_n, g_out, g_bad;
__device__ unsigned g_first[2];

// a thread's counts, added to the totals when it is done
struct Tally
{
    unsigned long long n = 0, out = 0, bad = 0;
    // operands in range (`inside`) must be accepted, accepted ones must agree
    __device__ void check(float got, float want, const QuickRange& g, bool inside, float x, float y)
    {
        if (!g.ok()) { out++; bad += inside; return; }
        n++;
        if (__float_as_uint(got) != __float_as_uint(want) && !(isnan(got) && isnan(want)))
        {
            if (bad++ == 0) { g_first[0] = __float_as_uint(x); g_first[1] = __float_as_uint(y); }
        }
    }
    __device__ ~Tally() { atomicAdd(&g_n, n); atomicAdd(&g_out, out); atomicAdd(&g_bad, bad); }
};

__device__ unsigned hash(unsigned long long i, unsigned k)
{
    return mix32((unsigned)i ^ mix32((unsigned)(i >> 32) + 0x9e3779b9u * k));
}
__device__ float scaled(unsigned mantissa, int e) { return __uint_as_float((unsigned)(127 + e) << 23 | (mantissa & 0x7fffffu)); }

// every mantissa, both signs, at five exponents; 2^-60 and 2^59 are the range's ends
__global__ void k_recip()
{
    Tally t;
    const int ex[5] = {0, 1, -60, 59, -17};
    for (unsigned m = blockIdx.x * blockDim.x + threadIdx.x; m < 1u << 23; m += gridDim.x * blockDim.x)
        for (int e : ex)
            for (int s = 0; s < 2; s++)
            {
                QuickRange g;
                const float b = s ? -scaled(m, e) : scaled(m, e);
                t.check(quick_recip(b, g).r, 1.f / b, g, true, b, 0.f);
            }
}

// every mantissa at both parities of the exponent and at the range's ends
__global__ void k_sqrt()
{
    Tally t;
    const int ex[6] = {0, 1, -60, -59, 58, 59};
    for (unsigned m = blockIdx.x * blockDim.x + threadIdx.x; m < 1u << 23; m += gridDim.x * blockDim.x)
        for (int e : ex)
        {
            QuickRange g;
            const float x = scaled(m, e);
            t.check(quick_sqrt(x, g), sqrtf(x), g, true, x, 0.f);
        }
}

__device__ void quotient(Tally& t, float a, float b, bool inside)
{
    QuickRange g, h;
    t.check(quick_quot(a, quick_recip(b, g), g), a / b, g, inside, a, b);
    t.check(quick_quot0(a, quick_recip(b, h), h), a / b, h, inside, a, b);
}

// random mantissas and signs, exponents over the whole range
__global__ void k_quot_random(unsigned long long n)
{
    Tally t;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n; i += (unsigned long long)gridDim.x * blockDim.x)
    {
        const unsigned r = hash(i, 3);
        float a = scaled(hash(i, 1), (int)(r % 120u) - 60), b = scaled(hash(i, 2), (int)(r / 120u % 120u) - 60);
        if (r >> 31) a = -a;
        if (r >> 30 & 1u) b = -b;
        quotient(t, a, b, true);
    }
}

// quotients next to a midpoint between two floats: a = b (q + half an ulp) rounded, and its neighbours
__global__ void k_quot_midpoint(unsigned long long n)
{
    Tally t;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n; i += (unsigned long long)gridDim.x * blockDim.x)
    {
        const float b = scaled(hash(i, 4), 0), q = scaled(hash(i, 5), (int)(hash(i, 6) % 5u) - 2);
        const double mid = (double)q + 0.5 * ((double)__uint_as_float(__float_as_uint(q) + 1u) - (double)q);
        const float a = (float)((double)b * mid);
        for (int k = -1; k <= 1; k++) quotient(t, __uint_as_float(__float_as_uint(a) + k), b, true);
    }
}

// divisors at the ends of the binade (1 + k ulp, 2 - k ulp) under every dividend mantissa
__global__ void k_quot_ends()
{
    Tally t;
    for (unsigned m = blockIdx.x * blockDim.x + threadIdx.x; m < 1u << 23; m += gridDim.x * blockDim.x)
        for (unsigned k = 0; k < 8; k++)
        {
            quotient(t, scaled(m, 0), scaled(k, 0), true);
            quotient(t, scaled(m, 0), scaled(0x7fffffu - k, 0), true);
            quotient(t, scaled(m, 59), scaled(0x7fffffu - k, -60), true);
            quotient(t, scaled(m, -60), scaled(0x7fffffu - k, 59), true);
        }
}

// zero dividends (quick_quot0 alone takes them), and operands outside the range: refused
__global__ void k_special()
{
    Tally t;
    const float zero[2] = {0.f, -0.f}, b[4] = {3.f, -3.f, 1e-10f, 1e10f};
    for (float a : zero)
        for (float d : b)
        {
            QuickRange g;
            t.check(quick_quot0(a, quick_recip(d, g), g), a / d, g, true, a, d);
        }
    const float out[8] = {0.f, -0.f, 1e-38f, 1e-45f, -1e-19f, 2e18f, -3e38f, __int_as_float(0x7f800000)};
    for (float x : out)
    {
        QuickRange g, h, r;
        quick_recip(x, g);
        quick_quot(x, quick_recip(1.f, h), h);
        quick_sqrt(fabsf(x), r);
        if (g.ok() || h.ok() || r.ok()) t.bad++;
        QuickRange z;
        quick_quot0(x, quick_recip(1.f, z), z);
        if (z.ok() != (x == 0.f)) t.bad++;
    }
}

// every float of [-1, 1]; |x| so near 1 that 0.5 (1 - |x|) is 0 leaves the range
__global__ void k_acos()
{
    Tally t;
    for (unsigned u = blockIdx.x * blockDim.x + threadIdx.x; u <= 0x3f800000u; u += gridDim.x * blockDim.x)
        for (unsigned s = 0; s < 2; s++)
        {
            QuickRange g;
            const float x = __uint_as_float(u | s << 31);
            t.check(quick_acos(x, g), portable_acos(x), g, u < 0x3f800000u, x, 0.f);
        }
}

static int report(const char* name)
{
    cudaError_t e = cudaDeviceSynchronize();
    unsigned long long n = 0, out = 0, bad = 0, zero = 0;
    unsigned first[2] = {0, 0};
    if (e == cudaSuccess) e = cudaMemcpyFromSymbol(&n, g_n, 8);
    if (e == cudaSuccess) e = cudaMemcpyFromSymbol(&out, g_out, 8);
    if (e == cudaSuccess) e = cudaMemcpyFromSymbol(&bad, g_bad, 8);
    if (e == cudaSuccess) e = cudaMemcpyFromSymbol(first, g_first, 8);
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_n, &zero, 8);
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_out, &zero, 8);
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_bad, &zero, 8);
    if (e != cudaSuccess) { printf("%s error: %s\n", name, cudaGetErrorString(e)); return 1; }
    printf("%s %llu %llu %llu", name, n, out, bad);
    if (bad) printf(" first %08x %08x", first[0], first[1]);
    printf("\n");
    return bad != 0;
}

int main()
{
    int bad = 0;
    const int grid = 148 * 8, block = 256;
    k_recip<<<grid, block>>>(); bad |= report("recip");
    k_sqrt<<<grid, block>>>(); bad |= report("sqrt");
    k_quot_random<<<grid, block>>>(1ull << 30); bad |= report("quot_random");
    k_quot_midpoint<<<grid, block>>>(1ull << 28); bad |= report("quot_midpoint");
    k_quot_ends<<<grid, block>>>(); bad |= report("quot_ends");
    k_special<<<1, 1>>>(); bad |= report("special");
    k_acos<<<grid, block>>>(); bad |= report("acos");
    return bad;
}
