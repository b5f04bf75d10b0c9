// Sliding-block interval stepper for the dense-source passes (TB_SCAT, TB_SCATX, TB_SCATW, TB_ADJX): one
// launch advances every shot of a wave by one coarse interval (T = sub = 4 fine steps).
//
// Each CTA owns an interior z-strip of HZ output rows (recomputing 5*T halo rows on each side: NQ = HZ/4 + 10
// row quads) and an x-chunk of LX output columns, and marches along x in blocks of BX = 16 columns. At
// iteration k the input block starts at column B = xs + 16k and time level t (t = 1..T) is computed on the
// columns [B - 5t, B - 5t + 16) by all threads: the blocks of consecutive levels are skewed by the stencil
// half-width, so level t only needs level t-1 columns that are already in shared memory. Levels 1..T-1 live
// in shared rings of KS_CB = 32 columns, level 0 in one of 64; one barrier separates the levels. A thread
// owns a 4 (z) x 2 (x) micro-tile and reads 22 quads per level from the rings. The secondary sources are
// formed once per column, at level 1, and kept in two rings of 32 columns.
//
// The marching stepper (aio_march.cuh) needs fewer instructions and barriers per update, but its dense-source
// modes hold 33 columns of both source slices for every row: at most 384 rows per SM, so strips that do
// not fill its warps (32 row quads) leave them idle, and its 52 columns of filling weigh on narrow chunks.
// Measured on one B200, whole calls with the dense passes on this stepper, and on the marching one: tomo adjoint,
// one shot of 912 x 3104 points, nts = 100: 35.7 and 44.2 ms; 21 shots of 78 x 569, nts = 200: 33.3 and 42.9;
// Born forward, 11 shots of 386 x 267, nts = 400: 26.0 and 31.2; 32 shots of 512 x 1312, nts = 100: 70.5 and
// 77.7 (0.40 and 0.47 ms per scattering launch). The plan is chosen by timing. Same bits either way.
#pragma once
#include "aio_march.cuh"

namespace aio {

constexpr int KS_BX = 16;      // block columns per iteration
constexpr int KS_CB = 32;      // ring depth in columns of levels 1..T-1 (>= BX + 5T - 5 + 1 for the output reads)
constexpr int KS_CB0 = 64;     // ring depth of level 0: the next input block lands while the current one is read
constexpr int KS_RINGCOLS = KS_CB0 + (KT_T - 1) * KS_CB + 2 * KS_CB;  // levels 0..T-1 and both source slices
constexpr int KS_PADQ = 2;     // zero quads above and below every ring column
constexpr int KS_MAXQ = 42;    // row quads per strip (HZ <= 128)
constexpr int KS_MAXQ_S = 26;  // short-strip variant (HZ <= 64): two CTAs per SM fit
__host__ __device__ constexpr int ks_rs(int maxq) { return (maxq + 2 * KS_PADQ) * 4; }  // floats per ring column
__host__ __device__ constexpr int ks_threads(int NQ) { return (8 * NQ + 31) / 32 * 32; }  // 8 column pairs per quad
__host__ __device__ constexpr int ks_iters(int LX) { return (LX + 10 * KT_T + KS_BX - 1) / KS_BX; }
static_assert(KS_CB >= KS_BX + 5 * KT_T - 5 + 1, "output stage reads level 1 5(T-1) columns behind its block");
// staging slots per thread (old level, v^2, sources at its and its+1), filled by asynchronous copies
constexpr int KS_SLOTS = 8;
// (the free surface runs on the large variant only)
inline size_t ks_smem_bytes(int NQ, int LX, int maxRec, bool fs) {
    return (size_t)KS_RINGCOLS * ks_rs(NQ <= KS_MAXQ_S && !fs ? KS_MAXQ_S : KS_MAXQ) * 4 + (size_t)KS_SLOTS * ks_threads(NQ) * 16 +
           ((size_t)ks_iters(LX) * (KS_BX + 1) + 64 + 2) * 4 + (size_t)maxRec * sizeof(KMEnt);
}

// Recordings: entries sorted by column (key: interior column, slot: interior row).
template <int MODE, int WPREC, int MAXQ, bool FS>
__global__ void __launch_bounds__(ks_threads(MAXQ), MAXQ == KS_MAXQ ? 1 : 2) k_slide(const KMArgs a) {
    constexpr int T = KT_T, RS = ks_rs(MAXQ);
    using Out = KMOut<MODE, WPREC>;
    extern __shared__ float4 km_smem4[];
    const int NQ = a.NQ, bd = blockDim.x, tid = threadIdx.x, iters = ks_iters(a.LX);
    float* ring = reinterpret_cast<float*>(km_smem4);
    float4* stg = reinterpret_cast<float4*>(ring + KS_RINGCOLS * RS);  // [KS_SLOTS][blockDim.x]
    float* dxt = reinterpret_cast<float*>(stg + KS_SLOTS * bd);        // column damping, columns xs-32 ...
    const int nDx = iters * KS_BX + 64;
    int* recFirst = reinterpret_cast<int*>(dxt + nDx);                 // first recording of an iteration's output columns
    KMEnt* sEnt = reinterpret_cast<KMEnt*>(recFirst + iters + 2);

    const Geom& g = a.g;
    const TBShot sh = a.shots[blockIdx.z];
    const int strip = blockIdx.x, chunk = blockIdx.y;
    const int ip = g.ip, nxi = g.nxi, nzi = g.nzi;
    const int cp = tid / NQ;              // column pair 0..7 (>= 8: idle thread)
    const int q = tid - cp * NQ;          // row quad
    const bool act = cp < KS_BX / 2;
    const int z0 = strip * a.HZ;
    const int zq = z0 - 5 * T + 4 * q;    // first row of the quad (multiple of 4)
    const int x0 = chunk * a.LX, x1 = min(x0 + a.LX, nxi), xs = x0 - 5 * T;
    const long long st4 = (long long)blockIdx.z * 4 * g.isz;
    const float *cur = a.cur + st4, *old = a.old + st4, *part = a.part + (long long)blockIdx.z * a.partShot;

    float4 Dz;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int z = zq + i, dd = z < 0 ? -1 : (FS ? nzi - 1 - z : min(z, nzi - 1 - z));  // free surface: no top taper
        (&Dz.x)[i] = dd < 0 ? 0.f : (dd < g.minPad ? __ldg(a.taper + dd) : 1.f);
    }
    const bool zLoad = act && zq >= 0 && zq < nzi;        // quad holds interior rows
    const int zv = min(max(zq, 0), ip - 4);               // clamped quad for v2 / operand reads
    const bool zOut = act && q >= 5 * T / 4 && q < 5 * T / 4 + a.HZ / 4 && zq < nzi;
    const int fsq = !FS ? -1 : (zq == 0 ? 0 : (zq == 4 ? 1 : -1));
    float* const ringQ = ring + (KS_PADQ + q) * 4;        // quad q of ring column 0, level 0
    auto col = [&](int t, int c) -> float4* {
        return reinterpret_cast<float4*>(t == 0 ? ringQ + (c & (KS_CB0 - 1)) * RS
                                                : ringQ + (KS_CB0 + (t - 1) * KS_CB + (c & (KS_CB - 1))) * RS);
    };
    // secondary-source rings (s = 0: slice its, 1: its+1; times dm)
    auto ssCol = [&](int s, int c) -> float4* {
        return reinterpret_cast<float4*>(ringQ + (KS_CB0 + (T - 1 + s) * KS_CB + (c & (KS_CB - 1))) * RS);
    };
    float4* const mySlot = stg + tid;     // slot i of this thread: mySlot[i * bd]

    // ---- shared set-up: zero rings, column damping table, recordings
    for (int i = tid; i < KS_RINGCOLS * (RS / 4); i += bd) km_smem4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i = tid; i < nDx; i += bd) {
        const int c = xs - 32 + i, dd = min(c, nxi - 1 - c);
        dxt[i] = dd < 0 ? 0.f : (dd < g.minPad ? __ldg(a.taper + dd) : 1.f);
    }
    const int4 se = sh.entStart[strip * a.nChunks + chunk];
    const int nRec = min(se.w - se.z, a.maxRec);
    for (int i = tid; i < nRec; i += bd) sEnt[i] = sh.ent[se.z + i];
    for (int i = tid; i <= iters; i += bd) recFirst[i] = nRec;
    // everything below reads what the previous launch of the stream wrote
    kt_grid_wait();
    if (a.relEarly) kt_grid_release();
    Out out(a, sh, z0, min(z0 + a.HZ, nzi), x0, x1);
    __syncthreads();

    // Input of iteration k, issued one iteration ahead: the level-0 block [B, B+16) into its ring slots,
    // and the level-1 operands into this thread's staging slots.
    auto issue_input = [&](int k) {
        if (!act) return;
        const int B = xs + KS_BX * k;
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int c = B + 2 * cp + j;
            const bool okc = zLoad && c >= 0 && c < nxi;
            km_cp16(col(0, c), cur + (okc ? c * ip + zq : 0), okc);
            const int co = c - 5;
            const bool oko = zLoad && co >= 0 && co < nxi;
            km_cp16(mySlot + j * bd, old + (oko ? co * ip + zq : 0), oko);
            const int ic = min(max(co, 0), nxi - 1) * ip + zv;
            km_cp16(mySlot + (2 + j) * bd, a.v2 + ic, true);
            km_cpw<WPREC>(mySlot + (4 + j) * bd, out.wA, ic, true);
            km_cpw<WPREC>(mySlot + (6 + j) * bd, out.wB, ic, true);
        }
    };
    issue_input(0);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    for (int e = tid; e < nRec; e += bd) {  // (sorted by column; iteration k puts out columns xs + 16 k - 20 ..)
        const int k = (sEnt[e].key - xs + 5 * T) / KS_BX;
        for (int i = e == 0 ? 0 : (sEnt[e - 1].key - xs + 5 * T) / KS_BX + 1; i <= k; i++) recFirst[i] = e;
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();

    for (int k = 0; k < iters; k++) {
        const int B = xs + KS_BX * k;
        if (k == iters - 1 && !a.relEarly) kt_grid_release();
        float4 ST[2];  // level T at the output columns (T-1 .. 1 from the rings)
#pragma unroll
        for (int t = 1; t <= T; t++) {
            const int c0 = B - 5 * t + 2 * cp;
            // level t is valid on columns >= xs + 5t and needed up to x1 - 1 + 5(T - t)
            const bool need = act && q >= (5 * t) / 4 && q < NQ - (5 * t) / 4 && c0 + 1 >= xs + 5 * t &&
                              c0 <= x1 - 1 + 5 * (T - t);
            ST[0] = ST[1] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (need) {
                float4 w[12];  // columns c0-5 .. c0+6
#pragma unroll
                for (int d = 0; d < 12; d++) w[d] = *col(t - 1, c0 - 5 + d);
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const int c = c0 + j;
                    const float4* z = col(t - 1, c);
                    const float4 ol = t == 1 ? mySlot[j * bd] : *col(t - 2, c);
                    const int ic = min(max(c, 0), nxi - 1) * ip + zv;
                    // level 1: prefetched with the input; otherwise read through L1
                    const float4 v2 = t == 1 ? mySlot[(2 + j) * bd] : __ldg(reinterpret_cast<const float4*>(a.v2 + ic));
                    const float Dx = dxt[c - xs + 32];
                    const float4 D = make_float4(fminf(Dz.x, Dx), fminf(Dz.y, Dx), fminf(Dz.z, Dx), fminf(Dz.w, Dx));
                    float4 n = km_point<kt_adj(MODE), FS>(a.c, w + j, z[-2], z[-1], z[1], z[2], ol, v2, D, fsq);
                    float4 sa, sb;
                    if (t == 1) {
                        // imagingFwdGpu (F/src/kernelsGpu.cu:309-316): dm * W, or the slices as they are
                        sa = km_wfrom<WPREC>(mySlot[(4 + j) * bd], out.scA);
                        sb = km_wfrom<WPREC>(mySlot[(6 + j) * bd], out.scB);
                        if (Out::DM && a.dm) {
                            const float4 dm = __ldg(reinterpret_cast<const float4*>(a.dm + ic));
                            sa = km_mul(dm, sa);
                            sb = km_mul(dm, sb);
                        }
                        *ssCol(0, c) = sa;
                        *ssCol(1, c) = sb;
                    } else {
                        sa = *ssCol(0, c);
                        sb = *ssCol(1, c);
                    }
                    n = km_add_sources(n, sa, sb, a.hs[0][t - 1], a.hs[1][t - 1], false, sa, 0.f);
                    ST[j] = km_mul(n, D);
                    if (t < T) *col(t, c) = ST[j];
                }
            }
            if (t == 1) {
                issue_input(k + 1);  // level-1 operands of this iteration are consumed
                asm volatile("cp.async.commit_group;\n" ::: "memory");
            }
            if (t < T) __syncthreads();  // level t complete before level t+1 (and the outputs) read it
        }
        // ---- outputs at the level-T columns [B - 5T, B - 5T + 16)
        {
            const int c0 = B - 5 * T + 2 * cp;
            const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const int c = c0 + j;
                if (!(zOut && c >= x0 && c < x1)) continue;
                const int idx = c * ip + zq;
                const float4 S[4] = {*col(1, c), *col(2, c), *col(3, c), ST[j]};
                out.write(idx, S[0], S[1], S[2], S[3], Out::PART ? km_ld(part + idx) : zero, zero, zero, zero);
                // (level 0 of these columns is done with: its ring keeps level T for the recordings)
                if (!Out::PART && nRec > 0) *col(0, c) = ST[j];
            }
        }
        if (!Out::PART && nRec > 0) {
            // the devices of these columns, one per thread
            __syncthreads();
            for (int e = recFirst[k] + tid; e < recFirst[k + 1]; e += bd) {
                const int c = sEnt[e].key, row = sEnt[e].slot - (z0 - 5 * T);
                const float* p = ring + KS_PADQ * 4 + row;
                float ra = 0.f, rb = 0.f;
#pragma unroll
                for (int l = 0; l < T; l++) {
                    const float v = p[(l + 1 < T ? KS_CB0 + l * KS_CB + (c & (KS_CB - 1)) : (c & (KS_CB0 - 1))) * RS];
                    ra = fmaf(v, a.w[0][l], ra);
                    rb = fmaf(v, a.w[1][l], rb);
                }
                // one thread owns each receiver: the atomics are plain read-free adds
                float* tr = sh.recSig + (long long)sEnt[e].dev * sh.recLd + a.c0;
                atomicAdd(tr, ra);
                atomicAdd(tr + 1, rb);
            }
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");  // the next input block and level-1 operands
        __syncthreads();  // ... for every thread; outputs done before level 1 reuses ring slots
    }
}

#ifndef AIO_MARCH_UNIT
#define AIO_SLIDE_EXTERN(M, W)                                                      \
    extern template __global__ void k_slide<M, W, KS_MAXQ_S, false>(const KMArgs); \
    extern template __global__ void k_slide<M, W, KS_MAXQ, false>(const KMArgs);   \
    extern template __global__ void k_slide<M, W, KS_MAXQ, true>(const KMArgs);
AIO_SLIDE_EXTERN(TB_SCAT, TBW_F32) AIO_SLIDE_EXTERN(TB_SCAT, TBW_BF16) AIO_SLIDE_EXTERN(TB_SCAT, TBW_F16)
AIO_SLIDE_EXTERN(TB_SCATW, TBW_F32) AIO_SLIDE_EXTERN(TB_SCATW, TBW_BF16) AIO_SLIDE_EXTERN(TB_SCATW, TBW_F16)
AIO_SLIDE_EXTERN(TB_SCATX, TBW_F32) AIO_SLIDE_EXTERN(TB_ADJX, TBW_F32)
#undef AIO_SLIDE_EXTERN
#endif

}  // namespace aio
