// Words that the CTAs of one cooperative launch hand each other without a
// barrier: 16 bytes, three floats and the tag of the exchange they belong to,
// stored and loaded as one relaxed 128-bit access.  A reader polls the words it
// needs until their tags match; a writer may overwrite a word once it knows
// its readers to be done.  Used by the frame kernel (frame.cu) and the
// conjugate-gradient solve (cg.cu).
#pragma once
#include "chunk_tets.cuh"
#include "pass_math.cuh"

namespace pbs {

// A wait that has not ended in two seconds means a CTA is gone (a fault
// elsewhere) or the launch was not co-resident: the kernel records it (*err;
// its call ends with PBS_E_DEVICE_TIMEOUT) and every CTA returns instead of
// spinning on.
constexpr unsigned long long EXCHANGE_WAIT_NS = 2000000000ull;

// A word of the exchange: three floats and a tag, one 128-bit access.  A caller
// uses all four: a load of which a part goes unused may be compiled into
// narrower ones, and a tag loaded by itself says nothing about the value.
__device__ __forceinline__ uint4 ld_word(const float4 *p) {
    uint4 v;
    asm volatile(
        "{\n\t.reg .b128 v;\n\t.reg .b64 a, b;\n\tld.relaxed.gpu.global.b128 v, [%4];\n\tmov.b128 {a, b}, v;\n\t"
        "mov.b64 {%0, %1}, a;\n\tmov.b64 {%2, %3}, b;\n\t}"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
        : "l"(p)
        : "memory");
    return v;
}
__device__ __forceinline__ void st_word(float4 *p, unsigned x, unsigned y, unsigned z, unsigned tag) {
    asm volatile(
        "{\n\t.reg .b128 v;\n\t.reg .b64 a, b;\n\tmov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
        "mov.b128 v, {a, b};\n\tst.relaxed.gpu.global.b128 [%0], v;\n\t}" ::"l"(p),
        "r"(x), "r"(y), "r"(z), "r"(tag)
        : "memory");
}
__device__ __forceinline__ void st_word(float4 *p, const float3 &v, unsigned tag) {
    st_word(p, __float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), tag);
}
__device__ __forceinline__ float4 word_f4(const uint4 &v) {
    return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), 0.f);
}
// The bound of a polling loop: every 1024 polls, whether to give up (the wait
// ran out, or any CTA's did).
struct Spin {
    unsigned n = 0;
    unsigned long long t0 = 0;
    __device__ __forceinline__ bool expired(int *err) {
        if (++n & 1023u) return false;
        const unsigned long long t = globaltimer_ns();
        if (t0 == 0) t0 = t;
        if (*(volatile int *)err == 0 && t - t0 <= EXCHANGE_WAIT_NS) return false;
        atomicExch(err, 1);
        return true;
    }
};

// Polls N words at consecutive places (n of them; the others read as zero)
// until their tags are `tag`; false when the wait gave up.
template <int N>
__device__ __forceinline__ bool poll_words(const float4 *p, int n, unsigned tag, float4 (&out)[N], int *err) {
    uint4 v[N];
#pragma unroll
    for (int q = 0; q < N; ++q) v[q] = q < n ? ld_word(p + q) : make_uint4(0u, 0u, 0u, tag);
    Spin spin;
    for (;;) {
        bool ready = true;
#pragma unroll
        for (int q = 0; q < N; ++q) ready &= v[q].w == tag;
        if (ready) break;
        if (spin.expired(err)) return false;
#pragma unroll
        for (int q = 0; q < N; ++q)
            if (v[q].w != tag) v[q] = ld_word(p + q);
    }
#pragma unroll
    for (int q = 0; q < N; ++q) out[q] = word_f4(v[q]);
    return true;
}

__device__ __forceinline__ DFloat warp_sum_df(DFloat v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v = df_add(v, DFloat{__shfl_down_sync(0xffffffffu, v.hi, o), __shfl_down_sync(0xffffffffu, v.lo, o)});
    return v;
}
__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

}  // namespace pbs
