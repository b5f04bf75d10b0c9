// Marching interval stepper: one launch advances every shot of a wave by T = 4 fine steps, one time level
// per warp.
//
// A CTA owns an interior z-strip (HZ output rows and 20 recomputed halo rows towards each neighbouring
// strip) and an x-chunk of LX output columns, and marches along x in blocks of 3 columns. Each warp
// computes one time level t = 1..4 of 32 row quads: at iteration n level t is at column xs - 8t + n
// (xs = x0 - 20), 8 columns behind level t-1. A thread keeps the last columns of its quad of level t-1 in
// registers (13 float4, shifted by 3 per block): the x-stencil and the centre cost one shared load per
// column, that of the newest neighbour. The z-neighbours (two quads above, two below), the old level t-2
// and, at level 4, the level-1 and level-2 samples of the outputs come from shared rings. All of these were
// written at least one block earlier, so one barrier per block orders everything, and the levels run in
// parallel.
//
// Shared memory holds, per row quad, KM_SLOTS consecutive float4 slots: rings of 24 / 27 / 21 / 12
// columns of levels 0..3 (the distance to their last reader, 16 / 24 / 16 / 8 columns, in whole blocks and
// for level 0 one block that is landing), the raw secondary sources of the scattered modes, and the
// image operands of ADJ. The odd stride makes every 128-bit access of a warp conflict-free, and a
// neighbour quad or another column of a block is a constant offset away.
//
// What bounds it (source pass, 32 shots of 512 x 1312, 9 chunks of 146 columns, one B200): 226 us per launch
// against 413 for the sliding-block stepper (aio_slide.cuh) that it replaced there, 381 G output updates/s;
// 139 instructions per warp and column of 128 points (256 at 2 per update before), issue slots 49 % busy,
// shared-memory pipe 57 %, DRAM traffic 649 MB (2.9 TB/s). 16 warps per SM (128 registers, 1360 bytes of shared
// memory per row quad) wait for one another at the barrier of each block 26 % of the time. Unrolling the columns
// instead of shifting the queue (24 KB of code) costs instruction-cache misses; a thread marching all four
// levels (53 KB) ran at a third of the rate.
//
// The scheme per fine step is the reference's (F/src/kernelsGpu.cu:202-219, 513-552):
// S_t = D * (v2 * L(S_{t-1}) + 2 S_{t-1} - D * S_{t-2} + injection), with the second damping of p_cur
// applied when the level is used as p_old, D = taper[min(dist_z, dist_x)] = min(Dz, Dx) (monotone taper)
// and D = 0 outside the interior so the zero boundary stays zero. Adjoint passes use the same recursion on
// U = v2 * S (stepAdjGpu, :574-610, multiplied by v2 point-wise). Per-interval products (the coarse
// source-wavefield sample, receiver data, the imaging condition) are formed from the four levels of each
// output point when level 4 is computed.
#pragma once
#include "aio_store.cuh"

namespace aio {

constexpr int KM_B = 3;           // columns per block (and barrier)
constexpr int KM_LAG = 8;         // columns between consecutive levels: 5 + KM_B
constexpr int KM_Q = 10 + KM_B;   // register queue: x-window of a block
constexpr int KM_L0 = 0, KM_L1 = 24, KM_L2 = 51, KM_L3 = 72, KM_END = 84;  // first slot of each ring
constexpr int KM_SSLEN = 33;      // secondary sources (two fields): level 4 is 24 columns behind level 1, and
                                  // two blocks are landing
__host__ __device__ constexpr int km_fields(int mode) { return mode == TB_SCATG ? 3 : 2; }  // secondary-source slices
__host__ __device__ constexpr int km_slots(int mode) {
    const int n = KM_END + (tb_scatlike(mode)                      ? km_fields(mode) * KM_SSLEN
                            : (mode == TB_ADJ || mode == TB_ADJG) ? 4 * KM_B
                                                                   : 0);
    return n | 1;
}
// Copies into shared memory are issued by the warps of the levels with the least other work (level 1 reads
// the old level, level 4 writes the outputs): level 0 by level 3's, secondary sources by level 2's.
constexpr int KM_TIN = 3, KM_TSS = 2;
constexpr int KM_PADQ = 2;        // zero row quads above and below the strip
constexpr int KM_FILL = 10 * KT_T + 3 * KT_T;  // iterations of level 4 beyond the LX output columns
// zero columns around the v^2 slice: level t reads columns xs - 8t .. xs - 8t + n + 5, n < LX + KM_FILL + 3
constexpr int KM_GUARD = 20 + KM_LAG * KT_T + 8;
constexpr int KM_MAXT = 512;      // threads per CTA: 4 levels x 128 row quads

struct KMArgs {
    Geom g;
    Coefs c;
    const float* v2;
    const float* taper;
    const float* dm;       // SCAT (and SCATW / ADJX when set): scaled model perturbation (interior slice)
    const TBShot* shots;
    // Fine steps f0 .. f0 + 3 of the pass's F (levels past the end carry zero weights). Coarse samples
    // c0, c0 + 1, c0 + 2 (adjoint passes: c0, c0 - 1, c0 - 2) take w[k][l] of level l + 1; the secondary
    // sources of slice k enter level l + 1 by hs[k][l].
    int its;               // coarse interval of f0
    int f0, F, c0;
    int nK;                // samples that the launch adds to
    int nfin;              // sub > 4: sample c0 is finished
    int last;              // last launch of the pass: the sample after it is finished too
    float w[3][KT_T], hs[3][KT_T];
    float h[2 * (SUB_MAX + 1)];
    int HZ, LX, nStrips, nChunks;
    int NQ;                // row quads of a CTA
    int maxInj, maxRec;    // shared capacity: injection slots, recordings,
    int recWarps;          // level-4 warps that record
    long long wStride;     // elements per stored coarse slice (= isz)
    int rSlot, rSlot0;     // ADJR: ring slots of R(its+1) and (its == 0) R(0);
                           // SCATX / SCATW / ADJX: slices of W holding the sources at its, its+1
    int oA, oB;            // SCATW / ADJX: slices receiving the samples its, its+1
    int f16spec;           // FP16 source pass: store slices with the speculative scale where allowed
    int wRing;             // SRC: W is a ring of wRing FP32 slices (slice t in slot t % wRing); 0: all nts
    int imgF32;            // ADJ: image in FP32 or FP64
    int relEarly;          // 1: the stream's next launch may begin its set-up right after the dependency
                           // wait; 0: once this CTA's last group of columns begins
    // per-shot arrays: base, and elements per shot
    const float* cur;      // levels read (current, old) and written, 4 isz per shot
    const float* old;
    float* ncur;
    float* nold;
    const float* part;     // partial coarse sum of sample c0 read / written, partShot per shot; sub > 4: that
    float* partOut;        // of the next sample 2 isz behind it
    long long partShot;
    void* W;               // stored wavefield or secondary sources, wShot elements per shot
    long long wShot;
    float* out;            // coarse samples written (ADJR, SCATW, ADJX)
    long long outShot;
    void* img;             // image (ADJ), isz per shot, FP32 or FP64
    float* wstage;         // FP16: 2 isz per shot
};

__host__ __device__ constexpr int km_warps(int NQ) { return (NQ + 31) / 32; }  // per level
__host__ __device__ constexpr int km_threads(int NQ) { return 4 * 32 * km_warps(NQ); }
// Recording modes: values staged per quad and column (partial sums of up to three coarse samples, or the
// four levels of the nonlinear adjoint).
__host__ __device__ constexpr int km_stage(int mode) {
    return mode == TB_NLA ? 4 : (mode == TB_NL || mode == TB_SCATG ? 3 : (mode == TB_SCAT || mode == TB_SCATX ? 2 : 0));
}
// quads of shared slots: the strip's with their pads, and one that idle lanes write to
__host__ __device__ constexpr int km_quads(int NQ) { return NQ + 2 * KM_PADQ + (NQ % 32 ? 1 : 0); }
__host__ __device__ constexpr size_t km_smem_bytes(int mode, int NQ, int LX, int maxInj, int maxRec,
                                                          int recWarps) {
    return (size_t)km_quads(NQ) * km_slots(mode) * 16 + (size_t)maxInj * (KT_T * 16 + 4) + (size_t)maxRec * 8 +
           4 + 4 * ((size_t)LX + 2 * KM_FILL) + 4 * (size_t)NQ + 4 * (size_t)(km_warps(NQ) + 1) +
           (size_t)km_stage(mode) * KM_B * 512 * recWarps;
}

// (state, partial sums, stored slices: plain loads, which stay behind the grid dependency wait)
__device__ __forceinline__ float4 km_ld(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void km_st(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void km_cp16(float4* s, const float* g, bool ok) {  // zero-filled when !ok
    const unsigned sa = (unsigned)__cvta_generic_to_shared(s);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(g), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void km_cp8(float4* s, const void* g, bool ok) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(s);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(g), "r"(ok ? 8 : 0) : "memory");
}
// four stored-wavefield samples at element idx, raw, into a slot
template <int WPREC>
__device__ __forceinline__ void km_cpw(float4* s, const void* W, int idx, bool ok) {
    if (WPREC == TBW_F32) km_cp16(s, (const float*)W + idx, ok);
    else km_cp8(s, (const unsigned short*)W + idx, ok);
}
__device__ __forceinline__ float2 km_lo(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 km_hi(const float4& v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float4 km_join(float2 a, float2 b) { return make_float4(a.x, a.y, b.x, b.y); }
__device__ __forceinline__ float2 km_dup(float v) { return make_float2(v, v); }
__device__ __forceinline__ float4 km_fma(float4 a, float b, float4 c) {
    return km_join(__ffma2_rn(km_lo(a), km_dup(b), km_lo(c)), __ffma2_rn(km_hi(a), km_dup(b), km_hi(c)));
}
__device__ __forceinline__ float4 km_mul(float4 a, float4 b) {
    return km_join(__fmul2_rn(km_lo(a), km_lo(b)), __fmul2_rn(km_hi(a), km_hi(b)));
}
__device__ __forceinline__ float km_el(const float4& v, int i) {
    return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w));
}
__device__ __forceinline__ float km_max(const float4& v) {
    return fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
}

// four stored-wavefield samples from a slot (FP32: 16 bytes, BF16 / FP16: the first 8), or at element idx
template <int WPREC>
__device__ __forceinline__ float4 km_wfrom(const float4& slot, float sc) {
    if (WPREC == TBW_F32) return slot;
    const uint2 r = *reinterpret_cast<const uint2*>(&slot);
    if (WPREC == TBW_BF16)
        return km_join(__bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.x)),
                       __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.y)));
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&r.x));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&r.y));
    return make_float4(a.x * sc, a.y * sc, b.x * sc, b.y * sc);
}
template <int WPREC>
__device__ __forceinline__ float4 km_wload(const void* W, int idx, float sc) {
    if (WPREC == TBW_F32) return km_ld((const float*)W + idx);
    const uint2 r = *reinterpret_cast<const uint2*>((const unsigned short*)W + idx);
    return km_wfrom<WPREC>(make_float4(__uint_as_float(r.x), __uint_as_float(r.y), 0.f, 0.f), sc);
}

// One fine step of a row quad before injection and the last damping. w: the previous level at the columns
// -5..5 of the quad; m2, m1, p1, p2: the quads above and below it; ol: the old level; fsq: free surface, 0
// or 1 for the quads of rows 0-3 and 4-7, else -1.
template <bool ADJ, bool FS>
__device__ __forceinline__ float4 km_point(const Coefs& co, const float4* w, float4 m2, float4 m1, const float4 p1,
                                           const float4 p2, float4 ol, const float4 v2, const float4 D, int fsq) {
    float4 ctr = w[5];
    const float* zc = co.zc;
    const float* xc = co.xc;
    if (FS && !ADJ) {
        // setFsConditionFwdGpu (F/src/kernelsGpu.cu:555-567): the stencil sees row 0 as zero and rows
        // -1..-5 as minus rows 1..5; row 0 of the old level is zero too
        if (fsq == 0) {
            ctr.x = 0.f;
            ol.x = 0.f;
            m1 = make_float4(-p1.x, -ctr.w, -ctr.z, -ctr.y);
            m2.w = -p1.y;
        } else if (fsq == 1) {  // rows 4..7: m1 holds rows 0..3, m2 rows -4..-1
            m1.x = 0.f;
            m2.w = -m1.y;
        }
    }
    float2 lzA = __fmul2_rn(km_dup(zc[0]), km_lo(ctr)), lzB = __fmul2_rn(km_dup(zc[0]), km_hi(ctr));
    lzA = __ffma2_rn(km_dup(zc[1]), make_float2(ctr.y + m1.w, ctr.z + ctr.x), lzA);
    lzB = __ffma2_rn(km_dup(zc[1]), make_float2(ctr.w + ctr.y, p1.x + ctr.z), lzB);
    lzA = __ffma2_rn(km_dup(zc[2]), __fadd2_rn(km_hi(ctr), km_hi(m1)), lzA);
    lzB = __ffma2_rn(km_dup(zc[2]), __fadd2_rn(km_lo(p1), km_lo(ctr)), lzB);
    lzA = __ffma2_rn(km_dup(zc[3]), make_float2(ctr.w + m1.y, p1.x + m1.z), lzA);
    lzB = __ffma2_rn(km_dup(zc[3]), make_float2(p1.y + m1.w, p1.z + ctr.x), lzB);
    lzA = __ffma2_rn(km_dup(zc[4]), __fadd2_rn(km_lo(p1), km_lo(m1)), lzA);
    lzB = __ffma2_rn(km_dup(zc[4]), __fadd2_rn(km_hi(p1), km_hi(m1)), lzB);
    lzA = __ffma2_rn(km_dup(zc[5]), make_float2(p1.y + m2.w, p1.z + m1.x), lzA);
    lzB = __ffma2_rn(km_dup(zc[5]), make_float2(p1.w + m1.y, p2.x + m1.z), lzB);
    if (FS && ADJ) {
        // stepAdjFsGpu (F/src/kernelsGpu.cu:613-740), U-form: row z = 1..4 drops the mirror terms
        // sum_{k = z+1..5} zc[k] U(k - z)
        if (fsq == 0) {
            const float u[4] = {ctr.y, ctr.z, ctr.w, p1.x};  // rows 1..4
#pragma unroll
            for (int k = 2; k <= 5; k++) lzA.y = fmaf(-zc[k], u[k - 2], lzA.y);
#pragma unroll
            for (int k = 3; k <= 5; k++) lzB.x = fmaf(-zc[k], u[k - 3], lzB.x);
#pragma unroll
            for (int k = 4; k <= 5; k++) lzB.y = fmaf(-zc[k], u[k - 4], lzB.y);
        } else if (fsq == 1) {
            lzA.x = fmaf(-zc[5], m1.y, lzA.x);
        }
    }
    float2 lxA = __fmul2_rn(km_dup(xc[0]), km_lo(ctr)), lxB = __fmul2_rn(km_dup(xc[0]), km_hi(ctr));
#pragma unroll
    for (int k = 1; k <= 5; k++) {
        const float4 r = w[5 + k], l = w[5 - k];
        float2 sA = __fadd2_rn(km_lo(r), km_lo(l));
        if (FS && !ADJ && fsq == 0) sA.x = 0.f;
        lxA = __ffma2_rn(km_dup(xc[k]), sA, lxA);
        lxB = __ffma2_rn(km_dup(xc[k]), __fadd2_rn(km_hi(r), km_hi(l)), lxB);
    }
    float2 nA = __ffma2_rn(km_lo(v2), __fadd2_rn(lzA, lxA), km_lo(ctr));
    float2 nB = __ffma2_rn(km_hi(v2), __fadd2_rn(lzB, lxB), km_hi(ctr));
    nA = __ffma2_rn(make_float2(-D.x, -D.y), km_lo(ol), __fadd2_rn(nA, km_lo(ctr)));
    nB = __ffma2_rn(make_float2(-D.z, -D.w), km_hi(ol), __fadd2_rn(nB, km_hi(ctr)));
    if (FS && ADJ && fsq == 0) nA.x = D.x * ol.x;  // the top row keeps the old level
    return km_join(nA, nB);
}

// value that device dev injects at level l
template <bool ADJ>
__device__ __forceinline__ float km_injected(const KMArgs& a, const TBShot& sh, int dev, int l) {
    const Geom& g = a.g;
    const float* tr = sh.injSig + (long long)dev * sh.injLd;
    const int f = a.f0 + l - 1;
    if (f >= a.F) return 0.f;
    if (!ADJ) return tr[f];
    const int iv = f / g.sub, it = g.nts - 2 - iv, it2 = g.sub - 1 - (f - iv * g.sub);
    // (this rounding: a dot-product test sees the last bit of the injected data, which the two-step
    // recursion integrates twice)
    return __fmaf_rn(tr[it], a.h[it2 + 1], __fmul_rn(tr[it + 1], a.h[g.H + it2 + 1]));
}
// Value of the point of entry e at level l into its injection slot. Devices of one point are next to one
// another in list order, and the first one's thread adds them up in that order: the same sum in every CTA that
// holds the point, and in every run.
template <bool ADJ>
__device__ __forceinline__ void km_slot_value(const KMArgs& a, const TBShot& sh, const KMEnt* ent, int e, const KMEnt& en, int l,
                                              float4* sV) {
    if (!(en.slot & KM_FIRST)) return;
    float v = km_injected<ADJ>(a, sh, en.dev, l);
#pragma unroll 1
    for (int more = en.slot & KM_MORE; more;) {
        const KMEnt next = ent[++e];
        v += km_injected<ADJ>(a, sh, next.dev, l);
        more = next.slot & KM_MORE;
    }
    reinterpret_cast<float*>(sV + (en.slot >> KM_SLOT) * KT_T + l - 1)[en.slot & 3] = v;
}
// adds injected values to a quad before its last damping (adjoint recursion: times v^2, product and sum
// rounded separately but in the nonlinear adjoint)
template <int MODE>
__device__ __forceinline__ float4 km_inject(const float4 n, float4 v, const float4 v2) {
    if (MODE == TB_NLA)
        return make_float4(fmaf(v2.x, v.x, n.x), fmaf(v2.y, v.y, n.y), fmaf(v2.z, v.z, n.z), fmaf(v2.w, v.w, n.w));
    if (kt_adj(MODE))
        v = make_float4(__fmul_rn(v2.x, v.x), __fmul_rn(v2.y, v.y), __fmul_rn(v2.z, v.z), __fmul_rn(v2.w, v.w));
    return make_float4(__fadd_rn(n.x, v.x), __fadd_rn(n.y, v.y), __fadd_rn(n.z, v.z), __fadd_rn(n.w, v.w));
}

// adds the secondary sources of one level: slices sa, sb (and sc) by their weights
__device__ __forceinline__ float4 km_add_sources(const float4 n, const float4 sa, const float4 sb, float hA, float hB, bool three,
                                                 const float4 sc, float hC) {
    float2 lo = __ffma2_rn(km_lo(sb), km_dup(hB), __fmul2_rn(km_lo(sa), km_dup(hA)));
    float2 hi = __ffma2_rn(km_hi(sb), km_dup(hB), __fmul2_rn(km_hi(sa), km_dup(hA)));
    if (three) {
        lo = __ffma2_rn(km_lo(sc), km_dup(hC), lo);
        hi = __ffma2_rn(km_hi(sc), km_dup(hC), hi);
    }
    return km_join(__fadd2_rn(km_lo(n), lo), __fadd2_rn(km_hi(n), hi));
}

// Output stage of one shot, shared by the two steppers.
template <int MODE, int WPREC>
struct KMOut {
    const KMArgs& a;
    float *ncur, *nold, *partOut, *outA, *outB;
    void *W, *img;
    float* wstage;
    unsigned* wover;
    const void *wA, *wB, *wC;  // stored-wavefield slices read by this launch
    float scA, scB, sc0, f16Sc;
    bool f16Spec;
    float wmaxA, wmaxB;        // FP16: max |W| of this thread's points in the slices written

    static constexpr bool GEN = tb_gen(MODE);
    static constexpr bool SRC = MODE == TB_SRC || MODE == TB_SRCG, ADJ = MODE == TB_ADJ || MODE == TB_ADJG;
    static constexpr bool PART = SRC || ADJ || MODE == TB_ADJR || tb_dense_out(MODE);
    static constexpr bool DM = MODE == TB_SCAT || MODE == TB_SCATG || tb_dense_out(MODE);

    // (after the grid dependency wait) z0, z1, x0, x1: the CTA's output region
    __device__ __forceinline__ KMOut(const KMArgs& a_, const TBShot& sh, int z0, int z1, int x0, int x1) : a(a_) {
        const Geom& g = a.g;
        const long long shot = blockIdx.z, isz = g.isz;
        const int its = a.its;
        constexpr bool SCAT = MODE == TB_SCAT || MODE == TB_SCATG, H = WPREC == TBW_F16;
        scA = H && MODE == TB_SCAT ? sh.wscale[its] : (H && MODE == TB_SCATW ? sh.wscale[a.rSlot] : 1.f);
        scB = H && (MODE == TB_SCAT || MODE == TB_ADJ) ? sh.wscale[its + 1]
                                                       : (H && MODE == TB_SCATW ? sh.wscale[a.rSlot0] : 1.f);
        sc0 = H && MODE == TB_ADJ ? sh.wscale[0] : 1.f;
        // FP16 source pass: slice its is stored directly with the speculative scale of slice its-1's max when
        // that max allows it (the same decision in every CTA), else staged in FP32; a staged slice its-1 is
        // complete now and quantized here with its exact max
        f16Spec = H && MODE == TB_SRC && kt_f16_spec_slice(sh.wmax, its, g.nts, a.f16spec);
        f16Sc = f16Spec ? kt_f16_spec_scale(sh.wmax[its - 1]) : 1.f;
        if (H && MODE == TB_SRC && its > 0 && !kt_f16_spec_slice(sh.wmax, its - 1, g.nts, a.f16spec))
            kt_f16_quantize(sh, a.wStride, g.ip, its - 1, z0, z1, x0, x1, threadIdx.x, blockDim.x);
        W = (char*)a.W + shot * a.wShot * (WPREC == TBW_F32 ? 4 : 2);
        wA = tb_scatlike(MODE) ? tb_wslice<WPREC>(W, a.wStride, SCAT ? a.c0 : a.rSlot) : nullptr;
        wB = tb_scatlike(MODE) ? tb_wslice<WPREC>(W, a.wStride, SCAT ? a.c0 + 1 : a.rSlot0)
             : ADJ             ? tb_wslice<WPREC>(W, a.wStride, a.c0)
                               : nullptr;
        wC = MODE == TB_SCATG ? tb_wslice<WPREC>(W, a.wStride, a.c0 + 2) : nullptr;  // read when nK > 2
        ncur = a.ncur + shot * 4 * isz;
        nold = a.nold + shot * 4 * isz;
        partOut = a.partOut + shot * a.partShot;
        float* const out = a.out + shot * a.outShot;
        outA = out + (long long)(MODE == TB_ADJR ? a.rSlot0 : a.oA) * a.wStride;
        outB = out + (long long)(MODE == TB_ADJR ? a.rSlot : a.oB) * a.wStride;
        img = a.imgF32 ? (void*)((float*)a.img + shot * isz) : (void*)((double*)a.img + shot * isz);
        wstage = a.wstage + shot * 2 * isz;
        wover = sh.wover;
        wmaxA = wmaxB = 0.f;
    }
    // FP16: folds the maxima into the slices'
    __device__ __forceinline__ void finish(const TBShot& sh) const {
        if (WPREC != TBW_F16 || MODE != TB_SRC) return;
        // non-negative floats order like their bit patterns: one warp max, one atomic per warp
        const unsigned ma = __reduce_max_sync(0xffffffffu, __float_as_uint(wmaxA));
        const unsigned mb = __reduce_max_sync(0xffffffffu, __float_as_uint(wmaxB));
        if ((threadIdx.x & 31) == 0) {
            if (ma) atomicMax(sh.wmax + a.its, ma);
            if (mb) atomicMax(sh.wmax + a.its + 1, mb);
        }
    }
    __device__ __forceinline__ void store_w(int slice, int idx, float4 v) const {
        void* p = tb_wslice<WPREC>(W, a.wStride, slice);
        if (WPREC == TBW_F32) {
            km_st((float*)p + idx, v);
        } else {
            const __nv_bfloat162 x = __floats2bfloat162_rn(v.x, v.y), y = __floats2bfloat162_rn(v.z, v.w);
            *reinterpret_cast<uint2*>((__nv_bfloat16*)p + idx) =
                make_uint2(*reinterpret_cast<const unsigned*>(&x), *reinterpret_cast<const unsigned*>(&y));
        }
    }

    // one coarse sample of the source / receiver wavefield
    __device__ __forceinline__ void emit_image(const float4 w, const float4 r, float4& acc) const {
        // imagingAdjGpu (F/src/kernelsGpu.cu:318-325): model += W * R
        acc = km_join(__ffma2_rn(km_lo(w), km_lo(r), km_lo(acc)), __ffma2_rn(km_hi(w), km_hi(r), km_hi(acc)));
    }
    __device__ __forceinline__ void emit_source(int t0, int idx, const float4 wa, bool next) {
        if (WPREC == TBW_F16) {
            // slice its: FP16 with the speculative scale, or FP32 into the staging buffer (the next launch
            // or k_f16_finish quantizes it with the slice's exact max); the pass's last slice is always staged
            const float m = km_max(wa);
            if (f16Spec && !next) {
                *reinterpret_cast<uint2*>((unsigned short*)W + (long long)t0 * a.wStride + idx) = kt_f16_pack(wa, f16Sc);
                if (m >= 65504.f * f16Sc) atomicOr(wover, 1u);  // FP16 overflow: redo exactly
            } else {
                km_st(wstage + (long long)(t0 & 1) * a.wStride + idx, wa);
            }
            if (next) wmaxB = fmaxf(wmaxB, m);
            else wmaxA = fmaxf(wmaxA, m);
        } else {
            store_w(a.wRing ? t0 % a.wRing : t0, idx, wa);
        }
    }

    // Output of the quad at idx: its levels 1..4, the partial sums carried in, and (ADJ) the stored wavefield
    // and the FP32 image.
    __device__ __forceinline__ void write(int idx, const float4 S1, const float4 S2, const float4 S3, const float4 S4,
                                          const float4 part, const float4 partB, const float4 w, const float4 oldImg) {
        km_st(ncur + idx, S4);
        km_st(nold + idx, S3);
        const float4 S[4] = {S1, S2, S3, S4};
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        if (PART) {
            // interpFineToCoarseSlice (F/src/kernelsGpu.cu:166-182) and its adjoint: samples c0 and the next
            float4 sa = part, sb = GEN ? partB : zero, sc = zero;
#pragma unroll
            for (int l = 0; l < KT_T; l++) {
                sa = km_fma(S[l], a.w[0][l], sa);
                sb = km_fma(S[l], a.w[1][l], sb);
                if (GEN) sc = km_fma(S[l], a.w[2][l], sc);
            }
            const bool fin = !GEN || a.nfin;
            km_st(partOut + idx, fin ? sb : sa);
            if (GEN) km_st(partOut + 2 * a.g.isz + idx, fin ? sc : sb);
            if (fin && SRC) {
                emit_source(a.c0, idx, sa, false);
                if (a.last) emit_source(a.c0 + 1, idx, sb, true);
            } else if (fin && ADJ) {
                // R(c0) here and R(0) after it at the end, as the reference's loop
                float4 w0 = zero;
                if (a.last) w0 = km_wload<WPREC>(tb_wslice<WPREC>(W, a.wStride, 0), idx, sc0);
                if (a.imgF32) {
                    float4 acc = oldImg;
                    emit_image(w, sa, acc);
                    if (a.last) emit_image(w0, sb, acc);
                    km_st((float*)img + idx, acc);
                } else {
                    double* p = (double*)img + idx;
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        double acc = p[i] + (double)(km_el(w, i) * km_el(sa, i));
                        if (a.last) acc += (double)(km_el(w0, i) * km_el(sb, i));
                        p[i] = acc;
                    }
                }
            } else if (MODE == TB_SCATW) {
                km_st(outA + idx, sa);
                if (a.last) km_st(outB + idx, sb);
            } else if (MODE == TB_ADJR || MODE == TB_ADJX) {
                km_st(outB + idx, sa);              // R(its+1)
                if (a.last) km_st(outA + idx, sb);  // R(0)
            }
        }
    }
};

// next block of a ring
__device__ __forceinline__ float4* km_next(float4* p, float4* first, int slots) {
    p += KM_B;
    return p == first + slots ? first : p;
}

template <int MODE, int WPREC, bool FS>
struct KM : KMOut<MODE, WPREC> {
    using Out = KMOut<MODE, WPREC>;
    using Out::a;
    using Out::wA;
    using Out::wB;
    using Out::wC;
    using Out::img;
    using Out::scA;
    using Out::scB;
    const int t;           // this warp's level
    float4* const sm;      // the quad's slots
    float4* const smw;     // the same, for writing (idle lanes read the last quad and write a dummy)
    const float* const dx; // column damping, indexed by column - xs
    // sparse entries of the thread's quad
    const int *const sKey, *const rKey, *const rDev;
    const float4* const sV;
    const bool sparse;     // any injection entry in this warp
    float4* const stg;     // level 4: this warp's staged recordings [column][value][lane], null: none to record
    const int crEnd;       // end of this warp's recordings
    const int zw;          // first row of the warp's quads
    const int key0;
    const float4 Dz;
    const int fsq;         // free surface: quad 0 or 1 of the top strip, else -1
    const int nEnd;        // iterations of this level: [13 t, nEnd)
    const int xs, x0, lxE, ip, zq, nxE;
    const float *cur, *dmp;
    float* recSig;
    int recLd;

    float4 q[KM_Q];        // level t-1 at the columns + 5 of iterations n - 10 .. n + 2
    float4 opA[KM_B];      // v^2 of a block's columns
    float4 opB[KM_B];      // old level (t = 1) or partial sum (t = 4) of a block's columns
    float4 opC[KM_B];      // scattered modes: model perturbation of a block's columns; sub > 4, t = 4: partial
                           // sum of the next sample
    const float *pA, *pB;  // v^2 / old level or partial sum at the column of the next fetch
    int cu;                // cursors into the quad's injection entries
    int cr;                // and (level 4) the warp's recordings

    static constexpr int SL = km_slots(MODE);
    static constexpr bool GEN = Out::GEN, ADJ = Out::ADJ, PART = Out::PART, DM = Out::DM;

    __device__ __forceinline__ KM(const Out& o, int t_, float4* sm_, float4* smw_, const float* dx_, const int* sKey_,
                                  const int* rKey_, const int* rDev_, const float4* sV_, bool sparse_, float4* stg_, int crEnd_,
                                  int zw_, int key0_, float4 Dz_, int fsq_, int nEnd_, int xs_, int x0_, int lxE_, int ip_,
                                  int zq_, int nxE_, const float* cur_, const float* dmp_, float* recSig_, int recLd_)
        : Out(o), t(t_), sm(sm_), smw(smw_), dx(dx_), sKey(sKey_), rKey(rKey_), rDev(rDev_), sV(sV_), sparse(sparse_),
          stg(stg_), crEnd(crEnd_), zw(zw_), key0(key0_), Dz(Dz_), fsq(fsq_), nEnd(nEnd_), xs(xs_), x0(x0_), lxE(lxE_),
          ip(ip_), zq(zq_), nxE(nxE_), cur(cur_), dmp(dmp_), recSig(recSig_), recLd(recLd_) {}

    // operands of the block of iteration n
    __device__ __forceinline__ void fetch(int n) {
        const int c = xs - KM_LAG * t + n;
#pragma unroll
        for (int j = 0; j < KM_B; j++) {
            const bool ok = (unsigned)(c + j) < (unsigned)nxE;
            // (v^2 has KM_GUARD zero columns on each side of the grid)
            opA[j] = __ldg(reinterpret_cast<const float4*>(pA));
            if (ok && (t == 1 || (PART && t == 4))) opB[j] = km_ld(pB);
            if (GEN && PART && ok && t == 4) opC[j] = km_ld(pB + 2 * a.g.isz);
            if (DM && ok && dmp) opC[j] = __ldg(reinterpret_cast<const float4*>(dmp + ((c + j) * ip + zq)));
            pA += ip;
            pB += ip;
        }
    }
    // level 0 of iterations n .. n + 2 into block l0 of its ring
    __device__ __forceinline__ void load_input(int n, float4* l0) const {
#pragma unroll
        for (int j = 0; j < KM_B; j++) {
            const int c = xs + n + j;
            const bool ok = (unsigned)c < (unsigned)nxE;
            km_cp16(l0 + j, cur + (ok ? c * ip + zq : 0), ok);
        }
    }
    // raw secondary-source slices at level 1's columns of iterations n .. n + 2
    __device__ __forceinline__ void load_sources(int n, int e) const {
#pragma unroll
        for (int j = 0; j < KM_B; j++) {
            const int c = xs - KM_LAG + n + j;
            const bool ok = (unsigned)c < (unsigned)nxE;
            const int idx = ok ? c * ip + zq : 0;
            float4* s = smw + KM_END + e + j;
            km_cpw<WPREC>(s, wA, idx, ok);
            km_cpw<WPREC>(s + KM_SSLEN, wB, idx, ok);
            if (MODE == TB_SCATG && a.nK > 2) km_cpw<WPREC>(s + 2 * KM_SSLEN, wC, idx, ok);
        }
    }
    // ADJ: stored wavefield and FP32 image at level 4's columns of iterations n .. n + 2
    __device__ __forceinline__ void load_image(int n, float4* s) const {
#pragma unroll
        for (int j = 0; j < KM_B; j++) {
            const int rel = n + j - KM_FILL;
            if ((unsigned)rel < (unsigned)lxE) {
                const int idx = (x0 + rel) * ip + zq;
                km_cpw<WPREC>(s + j, wB, idx, true);
                if (a.imgF32) km_cp16(s + KM_B + j, (const float*)img + idx, true);
            }
        }
    }
    // Recording, level 4 of a block of columns from iteration n on: every lane stages what its quad could
    // record, then the warp's devices in these columns are taken one per lane.
    __device__ __forceinline__ void stage(int j, const float4 S1, const float4 S2, const float4 S3, const float4 S4) const {
        constexpr int K = km_stage(MODE);
        const int lane = threadIdx.x & 31;
        const float4 S[4] = {S1, S2, S3, S4};
#pragma unroll
        for (int k = 0; k < K; k++) {
            float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
            if (MODE == TB_NLA) r = S[k];
            else
#pragma unroll
                for (int l = 0; l < KT_T; l++) r = km_fma(S[l], a.w[k][l], r);
            stg[(j * K + k) * 32 + lane] = r;
        }
    }
    __device__ __forceinline__ void record(int n) {
        constexpr int K = km_stage(MODE);
        const int lane = threadIdx.x & 31, rel0 = n - KM_LAG * KT_T;
        __syncwarp();
        unsigned m;
        do {
            const int e = cr + lane;
            const int rel = e < crEnd ? (rKey[e] & 0xffff) : 0x7fffffff;
            const bool mine = rel < rel0 + KM_B;
            m = __ballot_sync(0xffffffffu, mine);
            if (mine) {
                const int d = rDev[e], row = d & 3, dev = d >> 7;
                const float* v = reinterpret_cast<const float*>(stg + (rel - rel0) * K * 32 + ((d >> 2) & 31)) + row;
                float* tr = recSig + (long long)dev * recLd;
                if (MODE == TB_NLA) {
                    // fine step f of the pass is trace sample F - 1 - f; the recursion holds v2 * S
                    const float v2 = __ldg(a.v2 + ((xs + rel) * ip + zw + 4 * ((d >> 2) & 31) + row));
                    tr += a.F - 1 - a.f0;
#pragma unroll
                    for (int l = 0; l < KT_T; l++)
                        if (a.f0 + l < a.F) tr[-l] = v[l * 128] / v2;
                } else {
                    // one thread owns each receiver: the atomics are plain read-free adds
                    atomicAdd(tr + a.c0, v[0]);
                    atomicAdd(tr + a.c0 + 1, v[128]);
                    if (K > 2 && a.nK > 2) atomicAdd(tr + a.c0 + 2, v[256]);
                }
            }
            cr += __popc(m);
        } while (m == 0xffffffffu);
        __syncwarp();
    }

    __device__ __forceinline__ float4 damping(int rel) const {
        const float Dx = dx[rel];
        return make_float4(fminf(Dz.x, Dx), fminf(Dz.y, Dx), fminf(Dz.z, Dx), fminf(Dz.w, Dx));
    }

    // Level t of iteration n + j, before injection and the last damping: z: the quad's slot of level t-1
    // at its column, ol: the old level, v2.
    __device__ __forceinline__ float4 stencil(int j, int n, const float4* z, float4 ol, const float4 v2) const {
        return km_point<kt_adj(MODE), FS>(a.c, q + j, z[-2 * SL], z[-SL], z[SL], z[2 * SL], ol, v2,
                                          damping(n + j - KM_LAG * t), fsq);
    }

    __device__ __forceinline__ void march(int blocks) {
        // rings of levels t-1, t-2 and t; X: level 0's (its loads) or level 1's (outputs of level 4)
        const int rB = t == 1 ? KM_L0 : (t == 2 ? KM_L1 : (t == 3 ? KM_L2 : KM_L3));
        const int rN = t == 1 ? 24 : (t == 2 ? 27 : (t == 3 ? 21 : 12));
        const int oB = t == 2 ? KM_L0 : (t == 3 ? KM_L1 : KM_L2), oN = t == 2 ? 24 : (t == 3 ? 27 : 21);
        const int wB = t == 1 ? KM_L1 : (t == 2 ? KM_L2 : KM_L3), wN = t == 1 ? 27 : (t == 2 ? 21 : 12);
        const int xB = t == KM_TIN ? KM_L0 : KM_L1, xN = t == KM_TIN ? 24 : 27;
        float4 *const r0 = sm + rB, *const o0 = sm + oB, *const w0 = smw + wB, *const x0p = (t == KM_TIN ? smw : sm) + xB;
        // blocks of iterations n-3, n-6, n-9 (level t-1), n-15, n-18 (level t-2), n (level t), n+3 (level 0)
        // or n-24 (level 1)
        float4 *r3 = r0 + rN - 3, *r6 = r0 + rN - 6, *r9 = r0 + rN - 9;
        float4 *o15 = o0 + (oN - 15), *o18 = o0 + oN - 18, *w = w0, *x = x0p + 3;
        int e = 2 * KM_B;                     // level 1: slot of the sources two blocks ahead
        int eR = (2 * KM_SSLEN - KM_LAG * (t - 1)) % KM_SSLEN;  // slot of this level's sources
        if (t == KM_TIN) load_input(0, x0p);
        if (tb_scatlike(MODE) && t == KM_TSS) {
            load_sources(0, 0);
            load_sources(KM_B, KM_B);
        }
        if (t == KM_TIN || t == KM_TSS) asm volatile("cp.async.commit_group;\n" ::: "memory");
        fetch(0);
        for (int b = 0; b < blocks; b++) {
            const int n = KM_B * b;
            if (b == blocks - 4 && !a.relEarly) kt_grid_release();
            if (t == KM_TIN) load_input(n + KM_B, x);
            if (tb_scatlike(MODE) && t == KM_TSS) {
                load_sources(n + 2 * KM_B, e);
                e = e + KM_B == KM_SSLEN ? 0 : e + KM_B;
            }
            if (t == KM_TIN || t == KM_TSS) asm volatile("cp.async.commit_group;\n" ::: "memory");
            if (ADJ && t == KT_T) {
                if (!GEN || a.nfin) load_image(n + KM_B, sm + KM_END + ((b + 1) & 1) * 2 * KM_B);
                asm volatile("cp.async.commit_group;\n" ::: "memory");
            }
#pragma unroll
            for (int j = 0; j < KM_B; j++) q[10 + j] = r3[j];
            if (n + KM_B > 13 * t && n < nEnd) {
                float4 S[KM_B];
#pragma unroll
                for (int j = 0; j < KM_B; j++) {
                    const float4* z = j < 2 ? r9 + 1 + j : r6;
                    const float4 ol = t == 1 ? opB[j] : (j == 0 ? o18[2] : o15[j - 1]);
                    S[j] = stencil(j, n, z, ol, opA[j]);
                }
                if (tb_scatlike(MODE)) {
                    // imagingFwdGpu (F/src/kernelsGpu.cu:309-316): dm * W, or the slices as they are;
                    // injectSecondarySource (:102-107): forward fine step it2 = t weighs ss(its), ss(its+1)
                    // by h[it2-1], h[H+it2-1]; adjoint step it2 = T-t by h[it2+1], h[H+it2+1]
#pragma unroll
                    for (int j = 0; j < KM_B; j++) {
                        const int k = eR + j < KM_SSLEN ? eR + j : eR + j - KM_SSLEN;
                        float4 sa = km_wfrom<WPREC>(sm[KM_END + k], scA);
                        float4 sb = km_wfrom<WPREC>(sm[KM_END + KM_SSLEN + k], scB);
                        if (DM && dmp) {
                            sa = km_mul(opC[j], sa);
                            sb = km_mul(opC[j], sb);
                        }
                        float4 sc = sa;
                        const bool three = MODE == TB_SCATG && a.nK > 2;
                        if (three) {
                            sc = km_wfrom<WPREC>(sm[KM_END + 2 * KM_SSLEN + k], 1.f);
                            if (dmp) sc = km_mul(opC[j], sc);
                        }
                        S[j] = km_add_sources(S[j], sa, sb, a.hs[0][t - 1], a.hs[1][t - 1], three, sc, a.hs[2][t - 1]);
                    }
                } else if (sparse) {
#pragma unroll
                    for (int j = 0; j < KM_B; j++) {
                        if (sKey[cu] == (key0 | (n + j - KM_LAG * t))) {
                            S[j] = km_inject<MODE>(S[j], sV[cu * KT_T + t - 1], opA[j]);
                            cu++;
                        }
                    }
                }
#pragma unroll
                for (int j = 0; j < KM_B; j++) S[j] = km_mul(S[j], damping(n + j - KM_LAG * t));
                if (t < KT_T) {
#pragma unroll
                    for (int j = 0; j < KM_B; j++) w[j] = S[j];
                } else {
                    if (ADJ) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
#pragma unroll
                    for (int j = 0; j < KM_B; j++) {
                        const int rel = n + j - KM_FILL;  // output column - x0
                        if ((unsigned)rel < (unsigned)lxE) {
                            const float4* im = sm + KM_END + (b & 1) * 2 * KM_B + j;
                            const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
                            this->write((x0 + rel) * ip + zq, x[j], j == 0 ? o18[2] : o15[j - 1], q[5 + j], S[j], opB[j],
                                        opC[j], ADJ ? km_wfrom<WPREC>(im[0], scB) : zero, ADJ ? im[KM_B] : zero);
                        }
                    }
                    if (km_stage(MODE) > 0 && stg) {
#pragma unroll
                        for (int j = 0; j < KM_B; j++) stage(j, x[j], j == 0 ? o18[2] : o15[j - 1], q[5 + j], S[j]);
                        record(n);
                    }
                }
            }
            fetch(n + KM_B);
#pragma unroll
            for (int k = 0; k < 10; k++) q[k] = q[k + KM_B];
            r9 = r6;
            r6 = r3;
            r3 = km_next(r3, r0, rN);
            o18 = o15;
            o15 = km_next(o15, o0, oN);
            w = km_next(w, w0, wN);
            x = km_next(x, x0p, xN);
            if (tb_scatlike(MODE)) eR = eR + KM_B >= KM_SSLEN ? eR + KM_B - KM_SSLEN : eR + KM_B;
            if (t == KM_TIN || t == KM_TSS) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            asm volatile("bar.sync 0;\n" ::: "memory");
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
};

template <int MODE, int WPREC, bool FS>
__global__ void __launch_bounds__(KM_MAXT, 1) k_march(const KMArgs a) {
    constexpr int T = KT_T;
    extern __shared__ float4 km_smem4[];
    const int nthr = blockDim.x, tid = threadIdx.x, NQ = a.NQ;
    const Geom& g = a.g;
    const TBShot sh = a.shots[blockIdx.z];
    constexpr int SL = km_slots(MODE);
    float4* smAll = km_smem4;
    float4* sV = smAll + km_quads(NQ) * SL;              // [maxInj][T] injected values of a quad
    float4* stgAll = sV + a.maxInj * T;                        // staged recordings of the level-4 warps
    int* rDev = reinterpret_cast<int*>(stgAll + km_stage(MODE) * KM_B * 32 * a.recWarps);
                                                               // [maxRec] trace << 7 | lane << 2 | row of the quad
    int* rKey = rDev + a.maxRec;                               // recordings: warp of level 4 << 16 | column - xs
    int* sKey = rKey + a.maxRec;                               // injection keys, -1
    float* dxt = reinterpret_cast<float*>(sKey + a.maxInj + 1);
    int* first = reinterpret_cast<int*>(dxt + a.LX + 2 * KM_FILL);  // first injection slot of a quad
    int* firstRec = first + NQ;                                     // first recording of a warp of level 4, end
    const int strip = blockIdx.x, chunk = blockIdx.y;
    const int z0 = strip * a.HZ, zb = max(0, z0 - 5 * T), x0 = chunk * a.LX, xs = x0 - 5 * T;
    const int x1 = min(x0 + a.LX, g.nxi);
    // warp: level, and 32 quads; consecutive groups of four warps rotate the levels, so that each
    // scheduler of the SM gets every level
    const int wrp = __shfl_sync(0xffffffffu, tid >> 5, 0), t = 1 + ((wrp + (wrp >> 2)) & 3);
    const int qi = (wrp >> 2) * 32 + (tid & 31);
    const bool act = qi < NQ;
    const int qa = act ? qi : NQ - 1, zq = zb + 4 * qa;
    const int qw = act ? KM_PADQ + qi : NQ + 2 * KM_PADQ;  // the shared quad that the thread writes

    // ---- set-up that reads only what the host uploaded ahead of the pass
    for (int k = tid; k < KM_PADQ * SL; k += nthr) smAll[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = tid; k < KM_PADQ * SL; k += nthr) smAll[(KM_PADQ + NQ) * SL + k] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = tid; k < a.LX + 2 * KM_FILL; k += nthr) {  // columns xs - KM_B ...
        const int c = xs - KM_B + k;
        float d = 0.f;
        if (c >= 0 && c < g.nxi) {
            const int dd = min(c, g.nxi - 1 - c);
            d = dd < g.minPad ? __ldg(a.taper + dd) : 1.f;
        }
        dxt[k] = d;
    }
    const int4 se = sh.entStart[strip * a.nChunks + chunk];
    const int nInj = se.y - se.x, nRec = se.w - se.z;
    const int nSlots = nInj > 0 ? (sh.ent[se.y - 1].slot >> KM_SLOT) + 1 : 0;
    for (int k = tid; k < NQ; k += nthr) first[k] = nSlots;
    for (int k = tid; k <= km_warps(NQ); k += nthr) firstRec[k] = nRec;
    for (int k = tid; k < nSlots * T; k += nthr) sV[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    float Dz[4];
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const int z = zq + r, dd = FS ? g.nzi - 1 - z : min(z, g.nzi - 1 - z);  // free surface: no top taper
        Dz[r] = dd < 0 ? 0.f : (dd < g.minPad ? __ldg(a.taper + dd) : 1.f);
    }
    __syncthreads();
    for (int e = tid; e < nInj; e += nthr) {
        const KMEnt en = sh.ent[se.x + e];
        sKey[en.slot >> KM_SLOT] = en.key;
        if (e == 0 || (sh.ent[se.x + e - 1].key >> 16) != (en.key >> 16)) first[en.key >> 16] = en.slot >> KM_SLOT;
    }
    for (int e = tid; e < nRec; e += nthr) {
        const KMEnt en = sh.ent[se.z + e];
        rKey[e] = en.key;
        rDev[e] = en.dev << 7 | en.slot;
        // (the entries are sorted by warp: the first of each, and of the warps before it that have none)
        for (int k = e == 0 ? 0 : (sh.ent[se.z + e - 1].key >> 16) + 1; k <= en.key >> 16; k++) firstRec[k] = e;
    }
    if (tid == 0) sKey[nSlots] = -1;
    KMEnt mine = {};  // the first entry that this thread injects
    if (!tb_scatlike(MODE) && tid < nInj * T) mine = sh.ent[se.x + tid / T];
    // ---- everything below reads what the previous launch of the stream wrote
    kt_grid_wait();
    if (a.relEarly) kt_grid_release();
    if (!tb_scatlike(MODE)) {
#pragma unroll 1
        for (int k = tid; k < nInj * T; k += nthr) {
            const int e = k / T, l = k - e * T + 1;
            const KMEnt en = k == tid ? mine : sh.ent[se.x + e];
            km_slot_value<kt_adj(MODE)>(a, sh, sh.ent + se.x, e, en, l, sV);
        }
    }
    const bool zIn = act && zq < g.nzi;
    const bool zOut = zIn && zq >= z0 && zq < z0 + a.HZ;
    const KMOut<MODE, WPREC> out(a, sh, z0, min(z0 + a.HZ, g.nzi), x0, x1);
    const long long shot = blockIdx.z, isz = g.isz;
    __syncthreads();
    // level t starts at column xs + 5t: its cursor starts at the quad's first entry from there on
    int cu = act ? first[qa] : nSlots;
    const int cr = firstRec[wrp >> 2], crEnd = firstRec[(wrp >> 2) + 1];
    const bool recs = km_stage(MODE) > 0 && t == T && cr < crEnd;
    int rank = 0;  // among the CTA's recording warps
    for (int k = 0; recs && k < wrp >> 2; k++) rank += firstRec[k] < firstRec[k + 1];
    while ((sKey[cu] >> 16) == qa && (sKey[cu] & 0xffff) < 5 * t) cu++;
    const bool sparse = __any_sync(0xffffffffu, act && cu < nSlots && (sKey[cu] >> 16) == qa);
    const long long st4 = shot * 4 * isz;
    const float* old = a.old + st4;
    const float* part = a.part + shot * a.partShot;
    const long long c3 = (long long)(xs - KM_LAG * t) * g.ip + zq;  // column of iteration 0
    KM<MODE, WPREC, FS> m(out, t, smAll + (KM_PADQ + qa) * SL, smAll + qw * SL, dxt + KM_B, sKey, rKey, rDev, sV, sparse,
                          recs ? stgAll + rank * km_stage(MODE) * KM_B * 32 : nullptr, crEnd, zb + 128 * (wrp >> 2),
                          act ? qa << 16 : 0x7fff0000, make_float4(Dz[0], Dz[1], Dz[2], Dz[3]),
                          FS && strip == 0 && act && qa < 2 ? qa : -1, x1 - x0 + 10 * T + 3 * t, xs, x0,
                          zOut ? x1 - x0 : 0, g.ip, zq, zIn ? g.nxi : 0, a.cur + st4, a.dm, sh.recSig, sh.recLd);
#pragma unroll
    for (int j = 0; j < KM_Q; j++) m.q[j] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < KM_B; j++) m.opB[j] = m.opC[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    m.pA = a.v2 + c3;
    m.pB = (t == 1 ? old : part) + c3;
    m.cu = cu;
    m.cr = cr;
    m.march((x1 - x0 + KM_FILL + KM_B - 1) / KM_B);
    if (t == T) m.finish(sh);
}

// Tile interval stepper for waves too small to fill the GPU with marching CTAs: a CTA holds
// its (HZ + 40) x (LX + 40) input tile in shared memory and computes the four levels one after the other,
// each on a region 5 points smaller on every side, all threads on one level, a row quad x 4 columns per
// thread. A launch is one load, four dependent levels and one store; the march instead walks its LX + 52
// columns with a few warps. It recomputes more (2.1 updates per output update at 44 x 32 points) and is bound by
// latency: 9.3 us per launch for one shot of 304 x 512 points (16.4 with the sliding-block stepper, 16.8 with the
// march), 7.5 for one of 96 x 160 (19.6, 13.7). Plans of both kinds are timed for waves of up to 12000 points
// per SM; beyond that the march's smaller recomputation always won.
constexpr int KB_C = 4;           // columns per thread and level
constexpr int KB_MAXT = 512;
__host__ __device__ constexpr int kb_threads(int NQ, int LX) {
    const int n = (NQ - 2) * ((LX + 30 + KB_C - 1) / KB_C);
    return n >= KB_MAXT ? KB_MAXT : (n + 31) / 32 * 32;
}
__host__ __device__ constexpr int kb_quads(int NQ, int LX) { return (NQ + 2 * KM_PADQ) * (LX + 40 + KB_C); }  // one array
__host__ __device__ constexpr int kb_arrays(int mode) { return tb_scatlike(mode) ? 7 : 5; }
__host__ __device__ constexpr size_t kb_smem_bytes(int mode, int NQ, int LX, int maxInj) {
    return (size_t)kb_arrays(mode) * kb_quads(NQ, LX) * 16 + (size_t)maxInj * KT_T * 16 + (size_t)NQ * 16 + 4 * (size_t)(LX + 40 + KB_C) +
           2 * (size_t)NQ * (LX + 40 + KB_C);
}

template <int MODE, int WPREC, bool FS>
__global__ void __launch_bounds__(KB_MAXT, 1) k_block(const KMArgs a) {
    constexpr int T = KT_T;
    using Out = KMOut<MODE, WPREC>;
    constexpr bool UADJ = kt_adj(MODE), SCATL = tb_scatlike(MODE);
    extern __shared__ float4 km_smem4[];
    const int nthr = blockDim.x, tid = threadIdx.x, NQ = a.NQ, PQ = NQ + 2 * KM_PADQ, C = a.LX + 40, CA = C + KB_C;
    const Geom& g = a.g;
    const TBShot sh = a.shots[blockIdx.z];
    const int asz = PQ * CA;
    // levels 0..3 (the old level first in level 3's place, level 4 at last in level 0's) and v^2: quad q of
    // column i at (i * PQ + KM_PADQ + q)
    float4* const A = km_smem4;
    float4* const V = A + 4 * asz;
    float4* const E = V + asz;                                     // raw secondary sources: two slices
    float4* const sV = A + kb_arrays(MODE) * asz;                  // [maxInj][T] injected values of a quad
    float4* const dzt = sV + a.maxInj * T;                         // row damping of a quad
    float* const dxt = reinterpret_cast<float*>(dzt + NQ);         // column damping
    short* const slotAt = reinterpret_cast<short*>(dxt + CA);      // [NQ][CA] injection slot, or -1
    const int strip = blockIdx.x, chunk = blockIdx.y;
    const int z0 = strip * a.HZ, zb = z0 - 5 * T, x0 = chunk * a.LX, xs = x0 - 5 * T, x1 = min(x0 + a.LX, g.nxi);
    const int ip = g.ip;

    // ---- set-up that reads only what the host uploaded ahead of the pass
    // each thread's quads of the tile: (column i, quad q), then dI columns and dQ quads further on
    const int dI = nthr / NQ, dQ = nthr - dI * NQ, i00 = tid / NQ, q00 = tid - i00 * NQ;
    auto each = [&](auto&& f) {
        for (int i = i00, q = q00; i < C;) {
            const int c = xs + i, z = zb + 4 * q;
            const bool ok = (unsigned)c < (unsigned)g.nxi && (unsigned)z < (unsigned)g.nzi;
            f(i * PQ + KM_PADQ + q, ok ? c * ip + z : 0, ok);
            i += dI;
            q += dQ;
            if (q >= NQ) {
                q -= NQ;
                i++;
            }
        }
    };
    const int4 se = sh.entStart[strip * a.nChunks + chunk];
    const int nInj = se.y - se.x, nRec = se.w - se.z;
    if (nInj > 0)
        for (int k = tid; k < NQ * CA; k += nthr) slotAt[k] = -1;
    for (int k = tid; k < CA; k += nthr) {
        const int c = xs + k, dd = min(c, g.nxi - 1 - c);
        dxt[k] = dd < 0 ? 0.f : (dd < g.minPad ? __ldg(a.taper + dd) : 1.f);
    }
    for (int k = tid; k < 4 * NQ; k += nthr) {
        const int z = zb + k, dd = z < 0 ? -1 : (FS ? g.nzi - 1 - z : min(z, g.nzi - 1 - z));  // free surface: no top taper
        reinterpret_cast<float*>(dzt)[k] = dd < 0 ? 0.f : (dd < g.minPad ? __ldg(a.taper + dd) : 1.f);
    }
    const int nSlots = nInj > 0 ? (sh.ent[se.y - 1].slot >> KM_SLOT) + 1 : 0;
    for (int k = tid; k < nSlots * T; k += nthr) sV[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    // ---- everything below reads what the previous launch of the stream wrote
    kt_grid_wait();
    if (a.relEarly) kt_grid_release();
    const long long st4 = (long long)blockIdx.z * 4 * g.isz;
    const float *cur = a.cur + st4, *old = a.old + st4;
    Out out(a, sh, z0, min(z0 + a.HZ, g.nzi), x0, x1);
    each([&](int at, int idx, bool ok) {
        km_cp16(A + at, cur + idx, ok);
        km_cp16(A + 3 * asz + at, old + idx, ok);
        km_cp16(V + at, a.v2 + idx, ok);
        if (SCATL) {
            km_cpw<WPREC>(E + at, out.wA, idx, ok);
            km_cpw<WPREC>(E + asz + at, out.wB, idx, ok);
        }
    });
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    for (int k = tid; k < nInj * T; k += nthr) {
        const int e = k / T, l = k - e * T + 1;
        const KMEnt en = sh.ent[se.x + e];
        km_slot_value<UADJ>(a, sh, sh.ent + se.x, e, en, l, sV);
        if (l == 1) slotAt[(en.key >> 16) * CA + (en.key & 0xffff)] = (short)(en.slot >> KM_SLOT);
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    const float* const part = a.part + (long long)blockIdx.z * a.partShot;
#pragma unroll 1
    for (int l = 1; l <= T; l++) {
        const float4* src = A + (l - 1) * asz;
        const float4* oldp = A + ((l + 2) & 3) * asz;
        float4* dst = A + (l & 3) * asz;
        const int qlo = 5 * l / 4, nq = NQ - 2 * qlo, clo = 5 * l, items = nq * ((C - 10 * l + KB_C - 1) / KB_C);
        for (int it = tid; it < items; it += nthr) {
            const int gi = it / nq, q = qlo + it - gi * nq, i0 = clo + KB_C * gi;
            const float4* p = src + i0 * PQ + KM_PADQ + q;
            const int fsq = !FS ? -1 : (zb + 4 * q == 0 ? 0 : (zb + 4 * q == 4 ? 1 : -1));
            const float4 Dz = dzt[q];
            float4 w[10 + KB_C], S[KB_C];
#pragma unroll
            for (int k = 0; k < 10 + KB_C; k++) w[k] = p[(k - 5) * PQ];
#pragma unroll
            for (int j = 0; j < KB_C; j++) {
                const float4* z = p + j * PQ;
                const int at = (i0 + j) * PQ + KM_PADQ + q;
                const float Dx = dxt[i0 + j];
                const float4 D = make_float4(fminf(Dz.x, Dx), fminf(Dz.y, Dx), fminf(Dz.z, Dx), fminf(Dz.w, Dx));
                const float4 v2 = V[at];
                S[j] = km_point<UADJ, FS>(a.c, w + j, z[-2], z[-1], z[1], z[2], oldp[at], v2, D, fsq);
                if (SCATL) {
                    float4 sa = km_wfrom<WPREC>(E[at], out.scA), sb = km_wfrom<WPREC>(E[asz + at], out.scB);
                    const int c = min(max(xs + i0 + j, 0), g.nxi - 1), z4 = min(max(zb + 4 * q, 0), ip - 4);
                    float4 d = make_float4(1.f, 1.f, 1.f, 1.f);
                    if (Out::DM && a.dm) {
                        d = __ldg(reinterpret_cast<const float4*>(a.dm + c * ip + z4));
                        sa = km_mul(d, sa);
                        sb = km_mul(d, sb);
                    }
                    S[j] = km_add_sources(S[j], sa, sb, a.hs[0][l - 1], a.hs[1][l - 1], MODE == TB_SCATG && a.nK > 2,
                                          MODE == TB_SCATG && a.nK > 2 ? km_mul(d, km_wload<WPREC>(out.wC, c * ip + z4, 1.f)) : sa,
                                          a.hs[2][l - 1]);
                } else if (nSlots > 0) {
                    const int e = slotAt[q * CA + i0 + j];
                    if (e >= 0) S[j] = km_inject<MODE>(S[j], sV[e * T + l - 1], v2);
                }
                S[j] = km_mul(S[j], D);
            }
            if (l < T || nRec > 0) {
#pragma unroll
                for (int j = 0; j < KB_C; j++) dst[(i0 + j) * PQ + KM_PADQ + q] = S[j];
            }
            const int z = zb + 4 * q;
            if (l == T && z >= z0 && z < z0 + a.HZ && z < g.nzi) {
#pragma unroll
                for (int j = 0; j < KB_C; j++) {
                    const int c = xs + i0 + j;
                    if (c >= x0 && c < x1) {
                        const int idx = c * ip + z, at = (i0 + j) * PQ + KM_PADQ + q;
                        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
                        const bool fin = !Out::GEN || a.nfin;
                        out.write(idx, A[asz + at], A[2 * asz + at], w[5 + j], S[j], Out::PART ? km_ld(part + idx) : zero,
                                  Out::GEN && Out::PART ? km_ld(part + 2 * g.isz + idx) : zero,
                                  Out::ADJ && fin ? km_wload<WPREC>(out.wB, idx, out.scB) : zero,
                                  Out::ADJ && fin && a.imgF32 ? km_ld((const float*)out.img + idx) : zero);
                    }
                }
            }
        }
        __syncthreads();
    }
    if (!a.relEarly) kt_grid_release();
    out.finish(sh);
    for (int e = tid; e < nRec; e += nthr) {
        const KMEnt en = sh.ent[se.z + e];
        const int at = (en.key & 0xffff) * PQ + KM_PADQ + (en.key >> 16) * 32 + (en.slot >> 2), row = en.slot & 3;
        float S[T];
#pragma unroll
        for (int l = 1; l <= T; l++) S[l - 1] = reinterpret_cast<const float*>(A + (l & 3) * asz + at)[row];
        float* tr = sh.recSig + (long long)en.dev * sh.recLd;
        if (MODE == TB_NLA) {
            const float v2 = reinterpret_cast<const float*>(V + at)[row];
            tr += a.F - 1 - a.f0;
#pragma unroll
            for (int l = 0; l < T; l++)
                if (a.f0 + l < a.F) tr[-l] = S[l] / v2;
        } else {
#pragma unroll
            for (int k = 0; k < 3; k++) {
                float r = 0.f;
#pragma unroll
                for (int l = 0; l < T; l++) r = fmaf(S[l], a.w[k][l], r);
                if (k < a.nK) atomicAdd(tr + a.c0 + k, r);
            }
        }
    }
}

// Every instantiation, each compiled from aio_march.cu into an object of its own.
#define AIO_MARCH_BOTH(X, M, W) X(M, W, false) X(M, W, true)
#define AIO_MARCH_ALL(X)                                                                                              \
    AIO_MARCH_BOTH(X, TB_SRC, TBW_F32) AIO_MARCH_BOTH(X, TB_SRC, TBW_BF16) AIO_MARCH_BOTH(X, TB_SRC, TBW_F16)         \
    AIO_MARCH_BOTH(X, TB_SCAT, TBW_F32) AIO_MARCH_BOTH(X, TB_SCAT, TBW_BF16) AIO_MARCH_BOTH(X, TB_SCAT, TBW_F16)      \
    AIO_MARCH_BOTH(X, TB_ADJ, TBW_F32) AIO_MARCH_BOTH(X, TB_ADJ, TBW_BF16) AIO_MARCH_BOTH(X, TB_ADJ, TBW_F16)         \
    AIO_MARCH_BOTH(X, TB_SCATW, TBW_F32) AIO_MARCH_BOTH(X, TB_SCATW, TBW_BF16) AIO_MARCH_BOTH(X, TB_SCATW, TBW_F16)   \
    AIO_MARCH_BOTH(X, TB_NL, TBW_F32) AIO_MARCH_BOTH(X, TB_ADJR, TBW_F32) AIO_MARCH_BOTH(X, TB_SCATX, TBW_F32)        \
    AIO_MARCH_BOTH(X, TB_ADJX, TBW_F32) AIO_MARCH_BOTH(X, TB_NLA, TBW_F32) AIO_MARCH_BOTH(X, TB_SRCG, TBW_F32)        \
    AIO_MARCH_BOTH(X, TB_SCATG, TBW_F32) AIO_MARCH_BOTH(X, TB_ADJG, TBW_F32)
#ifndef AIO_MARCH_UNIT
#define AIO_MARCH_EXTERN(M, W, F)                                        \
    extern template __global__ void k_march<M, W, F>(const KMArgs); \
    extern template __global__ void k_block<M, W, F>(const KMArgs);
AIO_MARCH_ALL(AIO_MARCH_EXTERN)
#undef AIO_MARCH_EXTERN
#endif

}  // namespace aio
