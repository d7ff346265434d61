/*
 * rsc_popgen.cuh -- RS_populate's random draws on the device.
 *
 * RS_populate draws from the C library's rand(), an additive lagged Fibonacci
 * generator, r[i] = r[i - 3] + r[i - 31] (mod 2^32), whose outputs are
 * r[i] >> 1.  The recurrence is linear, so
 *   - the 31 words before any draw are a linear combination of the first 31,
 *     with the coefficients of x^n mod (x^31 - x^28 - 1): the host forms the
 *     words at the start of every chunk of draws (rscpop::chunk_states);
 *   - with S the shift by one, 1 = S^3 + S^31, hence 1 = (S^3 + S^31)^P =
 *     sum_t C(P, t) S^(3 P + 28 t): 3 P words at once from the 31 P before
 *     them.  A warp doubles P as its history grows, to P = 16: a word per
 *     lane and step.
 * One warp per chunk, its history in a ring in shared memory.  The values are
 * the reference's, draw for draw.
 *
 * One thread of the host made 38 M scatterers a second and its blocks were
 * copied from page-locked buffers made for the call: 1,000,003 drops and
 * 3 x 1000 debris in 26.2 ms, now in 0.45; 33,554,432 in 973 ms, now in 4.2
 * (the stores of 48 bytes a scatterer, and the fills of the arrays that are
 * constant, take 0.6 at the copy bandwidth; the serial steps of a chunk, one
 * trip to shared memory each, the rest).
 */
#ifndef SIMRADAR_GB300_RSC_POPGEN_CUH
#define SIMRADAR_GB300_RSC_POPGEN_CUH

#include <cuda_runtime.h>
#include <stdint.h>

namespace rsc {

constexpr unsigned kPopWarps = 4;         /* per block */
constexpr unsigned kPopRing = 1024;       /* words of history: 496 are needed, plus those not yet drawn */
constexpr unsigned kPopWords = 31;

struct PopArgs {
    const uint32_t *states;               /* 31 words before each chunk's first draw */
    unsigned long long total;             /* scatterers */
    unsigned per_chunk, chunks;           /* scatterers per chunk */
    float4 *pos, *aux;
    uint4 *rnd;
    float origin[3], size[3];
    /* drop sizes */
    const float *dsd_r, *dsd_cdf;
    unsigned dsd_count;
    int uniform;
    unsigned *pop;                        /* scatterers per size */
};

/* Words i0 .. i0 + 3 P - 1 (at most 32) of the ring from the 31 P before. */
template <int P>
__device__ __forceinline__ unsigned pop_generate(uint32_t *ring, unsigned i0, unsigned lane) {
    constexpr unsigned kNew = 3 * P < 32 ? 3 * P : 32;
    uint32_t v = 0;
    uint32_t c = 1;   /* C(P, t) */
    if (lane < kNew) {
        const unsigned i = i0 + lane - 3 * P;
#pragma unroll
        for (int t = 0; t <= P; t++) {
            v += c * ring[(i - 28u * t) & (kPopRing - 1)];
            c = c * (uint32_t)(P - t) / (uint32_t)(t + 1);
        }
    }
    __syncwarp();
    if (lane < kNew) ring[(i0 + lane) & (kPopRing - 1)] = v;
    __syncwarp();
    return i0 + kNew;
}

/* The draws of one chunk: `emit(first, word)` for 32 at a time, lane l the
 * draw first + l. */
template <class Emit>
__device__ __forceinline__ void pop_chunk(uint32_t *ring, const uint32_t *state, unsigned long long draws, unsigned lane,
                                          Emit emit) {
    if (lane < kPopWords) ring[lane] = state[lane];
    __syncwarp();
    unsigned made = kPopWords;            /* words so far (a chunk holds below 2^32) */
    unsigned long long done = 0;          /* draws emitted */
    unsigned at = kPopWords;              /* the word of the next one */
    while (done < draws) {
        if (made >= 496) made = pop_generate<16>(ring, made, lane);   /* 31 P words of history */
        else if (made >= 248) made = pop_generate<8>(ring, made, lane);
        else if (made >= 124) made = pop_generate<4>(ring, made, lane);
        else if (made >= 62) made = pop_generate<2>(ring, made, lane);
        else made = pop_generate<1>(ring, made, lane);
        while (made - at >= 32u && done < draws) {
            emit(done, ring[(at + lane) & (kPopRing - 1)]);
            at += 32u;
            done += 32u;
        }
        __syncwarp();
    }
}

/* (float)rand() / RAND_MAX: the divisor rounds to 2^31 */
__device__ __forceinline__ float pop_unit(uint32_t word) { return (float)(int)(word >> 1) * 0x1p-31f; }

/* x, y, z, age and the four respawn seeds of every scatterer, eight draws in
 * a row; radius and size class 0. */
__global__ void __launch_bounds__(32 * kPopWarps) k_pop_scatterers(const PopArgs a) {
    __shared__ uint32_t rings[kPopWarps][kPopRing];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const unsigned chunk = blockIdx.x * kPopWarps + warp;
    if (chunk >= a.chunks) return;
    const unsigned long long first = (unsigned long long)chunk * a.per_chunk;
    const unsigned long long n = min((unsigned long long)a.per_chunk, a.total - first);
    const unsigned c = lane & 7u;
    const float size = c < 2 ? a.size[c] : 10.0f, origin = c < 3 ? a.origin[c] : 0.0f;
    pop_chunk(rings[warp], a.states + (size_t)chunk * kPopWords, 8ull * n, lane, [&](unsigned long long d, uint32_t word) {
        const unsigned long long s = (d + lane) >> 3;
        if (s >= n) return;
        const size_t i = (size_t)(first + s);
        if (c < 3) {
            const float t = pop_unit(word) * size;   /* two roundings */
            float *o = reinterpret_cast<float *>(a.pos + i) + c;
            if (c == 2) *reinterpret_cast<float2 *>(o) = make_float2(t + origin, 0.0f);
            else *o = t + origin;
        } else if (c == 3) {
            a.aux[i] = make_float4(0.0f, pop_unit(word), 0.0f, 1.0f);
        } else {
            reinterpret_cast<uint32_t *>(a.rnd + i)[c - 4] = word >> 1;
        }
    });
}

/* The drop size of every background scatterer, one draw each from the second
 * sequence; after k_pop_scatterers. */
__global__ void __launch_bounds__(32 * kPopWarps) k_pop_sizes(const PopArgs a) {
    __shared__ uint32_t rings[kPopWarps][kPopRing];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const unsigned chunk = blockIdx.x * kPopWarps + warp;
    if (chunk >= a.chunks) return;
    const unsigned long long first = (unsigned long long)chunk * a.per_chunk;
    const unsigned long long n = min((unsigned long long)a.per_chunk, a.total - first);
    pop_chunk(rings[warp], a.states + (size_t)chunk * kPopWords, n, lane, [&](unsigned long long d, uint32_t word) {
        const bool in = d + lane < n;
        const float u = pop_unit(word);
        unsigned bin = 0;
        if (a.uniform) {
            bin = min((unsigned)(u * (float)a.dsd_count), a.dsd_count - 1u);
        } else {
            for (int k = (int)a.dsd_count - 1; k >= 0; k--) {
                if (u >= __ldg(a.dsd_cdf + k)) {
                    bin = (unsigned)k;
                    break;
                }
            }
        }
        if (in) {
            const size_t i = (size_t)(first + d + lane);
            reinterpret_cast<float *>(a.pos + i)[3] = __ldg(a.dsd_r + bin);
            reinterpret_cast<float *>(a.aux + i)[2] = ((float)bin + 0.5f) / (float)a.dsd_count;
        }
        /* one count per size and warp */
        const unsigned peers = __match_any_sync(0xffffffffu, in ? bin : 0xffffffffu);
        if (in && lane == (unsigned)(__ffs(peers) - 1)) atomicAdd(a.pop + bin, (unsigned)__popc(peers));
    });
}

}  // namespace rsc

#endif
