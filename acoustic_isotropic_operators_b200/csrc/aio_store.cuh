// Stored-wavefield precision of the interval steppers: the FP16 units of a coarse slice, quantization of
// staged slices, the 16-bit source field of tomo / WEMVA (d2/dt2), and the grid dependency of overlapped
// launches.
#pragma once
#include <cuda_bf16.h>

#include "aio_common.cuh"
#include "aio_tb.cuh"

namespace aio {

constexpr int KT_T = 4;        // fine steps per launch
// Programmatic dependent launch: a launch made with programmatic stream serialization may start
// while the previous kernel of its stream still runs. kt_grid_wait returns once that kernel has
// finished and its writes are visible (at once when there is no such dependency); before it a
// kernel reads only what the host uploaded ahead of the pass and writes only shared memory.
// kt_grid_release lets the next launch of the stream start its own prologue.
__device__ __forceinline__ void kt_grid_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void kt_grid_release() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
template <int WPREC>
__device__ __forceinline__ void kt_wstore4(void* W, long long idx, const float v[4]) {
    if (WPREC == TBW_F32) {
        *reinterpret_cast<float4*>((float*)W + idx) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
        const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]);
        const __nv_bfloat162 b = __floats2bfloat162_rn(v[2], v[3]);
        uint2 r;
        r.x = *reinterpret_cast<const unsigned*>(&a);
        r.y = *reinterpret_cast<const unsigned*>(&b);
        *reinterpret_cast<uint2*>((__nv_bfloat16*)W + idx) = r;
    }
}

// FP16 unit of a slice whose max |W| is m (0 for an all-zero slice): m / 2^15
__device__ __forceinline__ float kt_f16_scale(unsigned maxBits) {
    const float m = __uint_as_float(maxBits);
    return m > 0.f ? m * (1.f / 32768.f) : 1.f;
}
// Speculative FP16 unit of slice t from the finished slice t-1 (max bits prevBits): the power of
// two 2^(e - 11) for a previous max in [2^e, 2^(e+1)), which maps that max into [2^11, 2^12).
// FP16 keeps 11 significant bits over its whole normal range, so this scale loses no precision
// against the exact one; it leaves headroom for slice t to grow 16x (up to 65504) before an
// overflow, which the source pass flags so the pass is run again with exact scales. Usable when
// the previous max is a normal float of at least 2^-115 (then the unit is a normal float too).
__host__ __device__ __forceinline__ bool kt_f16_spec_ok(unsigned prevBits) {
    const unsigned e = (prevBits >> 23) & 0xffu;
    return e >= 12u && e < 255u;
}
__device__ __forceinline__ float kt_f16_spec_scale(unsigned prevBits) {
    return __uint_as_float((((prevBits >> 23) & 0xffu) - 11u) << 23);
}
// slice t of a source pass was stored directly with the speculative scale (else staged in FP32
// and quantized with its exact max); slice 0 and the last slice are always staged
__device__ __forceinline__ bool kt_f16_spec_slice(const unsigned* wmax, int t, int nts, int spec) {
    return spec && t >= 1 && t <= nts - 2 && kt_f16_spec_ok(wmax[t - 1]);
}
// quantize four FP32 samples to FP16 units of `sc`
__device__ __forceinline__ uint2 kt_f16_pack(const float4& v, float sc) {
    const float inv = 1.f / sc;
    const __half2 a = __floats2half2_rn(v.x * inv, v.y * inv);
    const __half2 b = __floats2half2_rn(v.z * inv, v.w * inv);
    uint2 r;
    r.x = *reinterpret_cast<const unsigned*>(&a);
    r.y = *reinterpret_cast<const unsigned*>(&b);
    return r;
}

// FP16 stored wavefield: quantize the finished FP32 slice t (staging buffer) over the
// region [z0, z1) x [x0, x1) (z0 multiple of 4) with its exact scale.
__device__ __forceinline__ void kt_f16_quantize(const TBShot& sh, long long wStride, int ip, int t, int z0, int z1,
                                                int x0, int x1, int tid, int nthr) {
    const float sc = kt_f16_scale(sh.wmax[t]);
    const float* src = sh.wstage + (long long)(t & 1) * wStride;
    unsigned short* dst = (unsigned short*)sh.W + (long long)t * wStride;
    const int nq = (z1 - z0 + 3) / 4, n = nq * (x1 - x0);
    for (int i = tid; i < n; i += nthr) {
        const int x = x0 + i / nq, z = z0 + 4 * (i % nq);
        const long long idx = (long long)x * ip + z;
        *reinterpret_cast<uint2*>(dst + idx) = kt_f16_pack(*reinterpret_cast<const float4*>(src + idx), sc);
    }
}

#ifndef AIO_MARCH_UNIT
// Finishes the last two slices (nts-2, nts-1) of an FP16 source pass (those staged in FP32) and
// records every slice's scale: the speculative one where the slice was stored directly.
__global__ void k_f16_finish(const TBShot* shots, long long wStride, int ip, int nzi, int nxi, int nts, int spec) {
    const TBShot sh = shots[blockIdx.y];
    const int nthr = gridDim.x * blockDim.x, tid = blockIdx.x * blockDim.x + threadIdx.x;
    for (int t = nts - 2; t < nts; t++)
        if (!kt_f16_spec_slice(sh.wmax, t, nts, spec)) kt_f16_quantize(sh, wStride, ip, t, 0, nzi, 0, nxi, tid, nthr);
    if (tid == 0)
        for (int t = 0; t < nts; t++)
            sh.wscale[t] = kt_f16_spec_slice(sh.wmax, t, nts, spec) ? kt_f16_spec_scale(sh.wmax[t - 1])
                                                                    : kt_f16_scale(sh.wmax[t]);
}

#endif
__device__ __forceinline__ void kt_st4(float* p, const float v[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
#ifndef AIO_MARCH_UNIT
// 16-bit source field of tomo / WEMVA: coarse d2/dt2 (srcWfldSecondTimeDerivative,
// F/src/kernelsGpu.cu:188-197, k_dt2's expression) of the slices [t0, t1] (at most KT_DT2_B) of a
// source wavefield held in an FP32 ring of `ring` slices (slice t in slot t % ring; zero outside
// [0, nts)). BF16 stores the result; FP16 stages it in FP32 (slot t - t0 of `stage`) and folds
// each slice's max |d| into wmax[t] (one atomic per warp and slice) for k_dt2_f16_pack. Four
// points per thread (interior slices are whole float4s: isz % 32 == 0).
constexpr int KT_DT2_B = 32;
template <int WP>
__global__ void k_dt2_block(const float* __restrict__ ring, long long ringSt, int ringLen, void* out, long long outSt,
                            float* stage, long long stageSt, unsigned* wmax, int nts, long long isz, int t0, int t1,
                            float cSide, float cCenter) {
    const int b = blockIdx.y;
    ring += b * ringSt;
    float mx[KT_DT2_B];
#pragma unroll
    for (int k = 0; k < KT_DT2_B; k++) mx[k] = 0.f;
    const long long n4 = isz / 4;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n4; q += (long long)gridDim.x * blockDim.x) {
        const long long i = 4 * q;
        const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
        float4 prev = t0 > 0 ? *reinterpret_cast<const float4*>(ring + (long long)((t0 - 1) % ringLen) * isz + i) : z4;
        float4 c = *reinterpret_cast<const float4*>(ring + (long long)(t0 % ringLen) * isz + i);
#pragma unroll
        for (int k = 0; k < KT_DT2_B; k++) {
            const int t = t0 + k;
            if (t > t1) break;
            const float4 nx =
                t + 1 < nts ? *reinterpret_cast<const float4*>(ring + (long long)((t + 1) % ringLen) * isz + i) : z4;
            float d[4] = {cSide * (prev.x + nx.x) + cCenter * c.x, cSide * (prev.y + nx.y) + cCenter * c.y,
                          cSide * (prev.z + nx.z) + cCenter * c.z, cSide * (prev.w + nx.w) + cCenter * c.w};
            if (WP == TBW_BF16) {
                kt_wstore4<TBW_BF16>((unsigned short*)out + b * outSt + (long long)t * isz, i, d);
            } else {
                kt_st4(stage + b * stageSt + (long long)k * isz + i, d);
                mx[k] = fmaxf(mx[k], fmaxf(fmaxf(fabsf(d[0]), fabsf(d[1])), fmaxf(fabsf(d[2]), fabsf(d[3]))));
            }
            prev = c;
            c = nx;
        }
    }
    if (WP == TBW_F16) {
        // non-negative floats order like their bit patterns: one warp max, one atomic per warp
#pragma unroll
        for (int k = 0; k < KT_DT2_B; k++) {
            const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(mx[k]));
            if ((threadIdx.x & 31) == 0 && m && t0 + k <= t1) atomicMax(wmax + (long long)b * nts + t0 + k, m);
        }
    }
}
// FP16: slices [t0, t1] staged by k_dt2_block, quantized with each slice's exact unit (max / 2^15,
// kt_f16_scale), and the units recorded in wscale.
__global__ void k_dt2_f16_pack(const float* __restrict__ stage, long long stageSt, void* out, long long outSt,
                               const unsigned* __restrict__ wmax, float* wscale, int nts, long long isz, int t0,
                               int t1) {
    const int b = blockIdx.y;
    const long long n4 = isz / 4, tot = (long long)(t1 - t0 + 1) * n4;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < tot; q += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(q / n4);
        const long long i = 4 * (q - k * n4);
        const float sc = kt_f16_scale(wmax[(long long)b * nts + t0 + k]);
        const float4 v = *reinterpret_cast<const float4*>(stage + b * stageSt + (long long)k * isz + i);
        *reinterpret_cast<uint2*>((unsigned short*)out + b * outSt + (long long)(t0 + k) * isz + i) = kt_f16_pack(v, sc);
        if (i == 0) wscale[(long long)b * nts + t0 + k] = sc;
    }
}

#endif
__host__ __device__ constexpr bool kt_adj(int mode) {
    return mode == TB_ADJ || mode == TB_ADJG || mode == TB_ADJR || mode == TB_ADJX || mode == TB_NLA;
}

}  // namespace aio
