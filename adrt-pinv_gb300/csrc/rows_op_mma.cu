// Row operators on the tensor cores (FP32 rows, N = 256 and 512; the operators and their real centro-symmetric form are
// described in rows_op.cu): per frequency e = T_e E, o = T_o O, real H x H matrices, H = N/2, on 64 real columns at a
// time (32 complex row vectors), tcgen05.mma kind::f16 with every operand split into two FP16 numbers (22 significant
// bits, as a TF32 split has, at half its bytes and twice its rate): lo.hi + hi.lo into one accumulator, hi.hi into a
// second, added in FP32 by the epilogue, so the chain of truncating accumulations on full-size partial sums is H/16
// long. FP16's range is kept by exact power-of-two scales: one per frequency for the matrices (at build time), one per
// vector from its largest |E|, |O| (found while it is loaded), undone in the epilogue; what falls below 2^-38 of a
// vector's largest value is lost.
//
// Persistent CTAs, one per SM, warp-specialised, over units of (frequency, 32 vectors); the units of a frequency run on
// neighbouring CTAs, which share its matrices through L2:
//   warps 8-15  load a unit's rows (coalesced, LPV = H/8 lanes per vector), apply the phases, fold E and O,
//               scale, split and store both as K-major core matrices. K runs in the order the lanes hold the values
//               (slot 8 l + 2 q + r is column 2 l + 2 LPV q + r; the matrices are stored in the same order), so each
//               lane writes 16-byte pieces; core matrices lie 144 bytes apart, which makes those stores conflict-free.
//               N = 256: two buffers, so the next unit loads while this one multiplies; N = 512: one.
//   warp 0      streams the matrices, 16 KB (128 rows x 32 columns, hi and lo) per bulk copy, through a ring of four
//   warp 1      issues the MMAs: M = 128 outputs, N = 64 columns, K = 16
//   warps 4-7   read the accumulators (two sets, so they overlap the next unit's MMAs), combine e and o, undo scales and
//               phases and write the rows in place (the unit's rows were all read before its MMAs began).
// Bounded by HBM and L2 traffic of the rows (N = 256: 16 bytes per value and pass) once the batch is large, by the
// matrices (34 MB at N = 256, 269 MB at N = 512) when it is small; figures at the dispatch in the host code below.
#include <cuda_fp16.h>

#include "common.cuh"
#include "launch.h"
#include "rows_op.cuh"
#include "tcgen05.cuh"

namespace adrt {

template <int n> struct OmCfg {
    static constexpr int N = 1 << n, H = N / 2, L = 2 * N;
    static constexpr int VT = 32;             // vectors per unit
    static constexpr int LPV = H / 8;         // loader lanes per vector
    static constexpr int MT = H / 128;        // blocks of 128 outputs
    static constexpr int KC = 32;             // K per matrix chunk
    static constexpr int NKC = H / KC;
    static constexpr int CHUNK = 2 * 128 * KC;  // halves per chunk: hi tile, lo tile
    static constexpr int CHUNKS = MT * 2 * NKC;  // per unit
    static constexpr int RING = 4;
    static constexpr int LBO = 144;           // bytes between core matrices along K (B operand)
    static constexpr int SBO = (H / 8) * LBO;  // between groups of 8 columns
    static constexpr int BT = (2 * VT / 8) * SBO;  // bytes of one B tile (parity, hi or lo)
    static constexpr int NB = n == 8 ? 2 : 1;  // B buffers
    static constexpr int ACC = 256;           // TMEM columns per accumulator set: parity x {lo terms, hi.hi} x 2 VT
    static constexpr size_t smem = (size_t)RING * CHUNK * 2 + (size_t)NB * 4 * BT + 1024;
};
constexpr int OM_THREADS = 512;

// column of T that K slot s multiplies
template <int n> __host__ __device__ constexpr int om_col(int s) {
    return 2 * (s / 8) + 2 * OmCfg<n>::LPV * ((s % 8) / 2) + (s & 1);
}

// FP32 operators T (N+1 x 2 x H x H, [j][c]) -> FP16 hi / lo tiles scaled by scale[k], in the order the kernel streams them
template <int n>
__global__ void rows_op_split_kernel(long long total, const float* __restrict__ T, const float* __restrict__ scale,
                                     __half* __restrict__ Ts) {
    using W = OmCfg<n>;
    constexpr int H = W::H;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
        const int o = (int)(e % H), s = (int)(e / H % H), par = (int)(e / H / H % 2);
        const long long k = e / H / H / 2;
        const float v = T[((k * 2 + par) * H + om_col<n>(s)) * H + o] * scale[k];
        const __half hi = __float2half_rn(v), lo = __float2half_rn(v - __half2float(hi));
        const int mt = o / 128, om = o % 128, kc = s / W::KC, ks = s % W::KC;
        __half* t = Ts + (((k * W::MT + mt) * 2 + par) * W::NKC + kc) * W::CHUNK + ((om / 8) * (W::KC / 8) + ks / 8) * 64 +
                    (om % 8) * 8 + ks % 8;
        t[0] = hi;
        t[128 * W::KC] = lo;
    }
}

__device__ __forceinline__ uint32_t half2_bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }

// eight values times s as FP16 hi and lo, 16 bytes each
__device__ __forceinline__ void split8(const float (&v)[8], float s, uint4& hi, uint4& lo) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float a = v[2 * q] * s, b = v[2 * q + 1] * s;
        const __half2 hh = __floats2half2_rn(a, b);
        const float2 f = __half22float2(hh);
        h[q] = half2_bits(hh);
        l[q] = half2_bits(__floats2half2_rn(a - f.x, b - f.y));
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}

__device__ __forceinline__ void tmem_ld8(uint32_t addr, float (&v)[8]) {
    uint32_t t[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(t[0]), "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7])
                 : "r"(addr));
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = __uint_as_float(t[q]);
}

template <int n>
__global__ void __launch_bounds__(OM_THREADS, 1)
    rows_op_mma_kernel(int nimg, int tiles, const __half* __restrict__ Ts, const float* __restrict__ tinv, float2* Y,
                       long long img_stride, const float2* __restrict__ roots, bool bp, int* __restrict__ err) {
    using W = OmCfg<n>;
    constexpr int N = W::N, L = W::L, VT = W::VT, LPV = W::LPV;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* ring = smem_raw;
    unsigned char* bbuf = smem_raw + (size_t)W::RING * W::CHUNK * 2;
    float* inv = reinterpret_cast<float*>(bbuf + (size_t)W::NB * 4 * W::BT);  // [4][VT]
    uint64_t* a_full = reinterpret_cast<uint64_t*>(inv + 4 * VT);
    uint64_t* a_free = a_full + W::RING;
    uint64_t* b_full = a_free + W::RING;
    uint64_t* b_free = b_full + 2;
    uint64_t* acc_full = b_free + 2;
    uint64_t* acc_free = acc_full + 2;
    uint64_t* drain = acc_free + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* s_issued = abort_flag + 1;
    volatile int* s_consumed = abort_flag + 2;
    static_assert(4 * VT * 4 + (2 * W::RING + 9) * 8 + 16 <= 1024, "barrier area");

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int total = (N + 1) * tiles;
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 0) {
        for (int q = 0; q < W::RING; ++q) {
            mbar_init(&a_full[q], 1);
            mbar_init(&a_free[q], 1);
        }
        for (int q = 0; q < 2; ++q) {
            mbar_init(&b_full[q], 8);  // one arrival per loader warp
            mbar_init(&b_free[q], 1);
            mbar_init(&acc_full[q], 1);
            mbar_init(&acc_free[q], 4);  // one per epilogue warp
        }
        mbar_init(drain, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        *abort_flag = 0;
        *s_issued = 0;
        *s_consumed = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    // the units of this CTA: frequency and first vector; every role walks the same list
    auto vectors = [&](int k) { return nimg * ((k == 0 || k == N) ? 2 : 4); };

    if (warp == 0) {  // matrices
        int ch = 0;
        bool ok = true;
        for (int u = blockIdx.x; ok && u < total; u += gridDim.x) {
            const int k = u / tiles;
            if ((u % tiles) * VT >= vectors(k)) continue;
            const __half* src = Ts + (size_t)k * W::CHUNKS * W::CHUNK;
            for (int q = 0; q < W::CHUNKS; ++q, ++ch) {
                const int s = ch % W::RING, r = ch / W::RING;
                if (r > 0 && !warp_wait(smem_addr(&a_free[s]), (uint32_t)((r - 1) & 1), abort_flag)) {
                    if (lane == 0) *abort_flag = 1;
                    ok = false;
                    break;
                }
                if (lane == 0) {
                    mbar_expect_bulk(smem_addr(&a_full[s]), smem_addr(ring + (size_t)s * W::CHUNK * 2),
                                     src + (size_t)q * W::CHUNK, W::CHUNK * 2);
                    *s_issued = ch + 1;
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {  // MMAs
        // D f32 (bit 4), A and B f16, K-major, N >> 3 at bits 17-22, M >> 4 at bits 24-28
        constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(2 * VT >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        int ch = 0, un = 0, ac = 0;
        bool ok = true;
        for (int u = blockIdx.x; ok && u < total; u += gridDim.x) {
            if ((u % tiles) * VT >= vectors(u / tiles)) continue;
            const int bi = un % W::NB, br = un / W::NB;
            if (!warp_wait(smem_addr(&b_full[bi]), (uint32_t)(br & 1), abort_flag)) ok = false;
            const uint32_t b0 = smem_addr(bbuf + (size_t)bi * 4 * W::BT);
            for (int mt = 0; ok && mt < W::MT; ++mt, ++ac) {
                const int ai = ac & 1, ar = ac >> 1;
                if (ar > 0 && !warp_wait(smem_addr(&acc_free[ai]), (uint32_t)((ar - 1) & 1), abort_flag)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int pk = 0; pk < 2 * W::NKC; ++pk, ++ch) {
                    const int par = pk / W::NKC, kc = pk % W::NKC, s = ch % W::RING;
                    if (!warp_wait(smem_addr(&a_full[s]), (uint32_t)((ch / W::RING) & 1), abort_flag)) {
                        ok = false;
                        break;
                    }
                    if (lane == 0) {
                        *s_consumed = ch + 1;
                        const uint32_t dl = tmem + (uint32_t)(ai * W::ACC + par * 4 * VT), dh = dl + 2 * VT;
                        const uint32_t a0 = smem_addr(ring + (size_t)s * W::CHUNK * 2);
                        const uint32_t bt = b0 + (uint32_t)(par * 2 * W::BT);
#pragma unroll
                        for (int ks = 0; ks < W::KC / 16; ++ks) {
                            const int kk = kc * (W::KC / 16) + ks;
                            const uint64_t ah = desc_kmajor(a0 + ks * 256, 128, (W::KC / 8) * 128);
                            const uint64_t al = desc_kmajor(a0 + 128 * W::KC * 2 + ks * 256, 128, (W::KC / 8) * 128);
                            const uint64_t bh = desc_kmajor(bt + kk * 2 * W::LBO, W::LBO, W::SBO);
                            const uint64_t bl = desc_kmajor(bt + W::BT + kk * 2 * W::LBO, W::LBO, W::SBO);
                            mma_f16(dl, al, bh, idesc, kk > 0 ? 1u : 0u);
                            mma_f16(dl, ah, bl, idesc, 1u);
                            mma_f16(dh, ah, bh, idesc, kk > 0 ? 1u : 0u);
                        }
                        tc_commit(&a_free[s]);
                    }
                    __syncwarp();
                }
                if (ok && lane == 0) {
                    if (mt == W::MT - 1) tc_commit(&b_free[bi]);
                    tc_commit(&acc_full[ai]);  // last: once the epilogue has seen it, no arrival is outstanding
                }
                __syncwarp();
            }
            ++un;
        }
        if (!ok && lane == 0) *abort_flag = 1;
    } else if (warp >= 4 && warp < 8) {  // epilogue: TMEM lanes 32 (warp % 4) .., one output c per lane
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        int un = 0, ac = 0;
        bool ok = true;
        for (int u = blockIdx.x; ok && u < total; u += gridDim.x) {
            const int k = u / tiles, v0 = (u % tiles) * VT, nv = vectors(k);
            if (v0 >= nv) continue;
            const bool self = (k == 0 || k == N);
            const float ti = tinv[k];
            const float* iv = inv + (un & 3) * VT;
            for (int mt = 0; mt < W::MT; ++mt, ++ac) {
                const int ai = ac & 1, c = mt * 128 + (warp & 3) * 32 + lane;
                const float2 pa = roots[op_phase_out<n>(k, c)], pb = roots[op_phase_out<n>(k, N - 1 - c)];
                if (!warp_wait(smem_addr(&acc_full[ai]), (uint32_t)((ac >> 1) & 1), abort_flag)) {
                    if (lane == 0) *abort_flag = 1;
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d = tmem + lane_base + (uint32_t)(ai * W::ACC);
#pragma unroll 1
                for (int vb = 0; vb < VT; vb += 8) {
                    if (v0 + vb >= nv) break;
                    float er[8], ei[8], orr[8], oi[8], t0[8], t1[8], t2[8], t3[8];
                    tmem_ld8(d + vb, er);
                    tmem_ld8(d + VT + vb, ei);
                    tmem_ld8(d + 2 * VT + vb, t0);
                    tmem_ld8(d + 3 * VT + vb, t1);
                    tmem_ld8(d + 4 * VT + vb, orr);
                    tmem_ld8(d + 5 * VT + vb, oi);
                    tmem_ld8(d + 6 * VT + vb, t2);
                    tmem_ld8(d + 7 * VT + vb, t3);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const int v = v0 + vb + q;
                        if (v >= nv) break;
                        const float sc = iv[vb + q] * ti;
                        const float e_r = er[q] + t0[q], e_i = ei[q] + t1[q], o_r = orr[q] + t2[q], o_i = oi[q] + t3[q];
                        float2 za = make_float2((e_r + o_r) * sc, (e_i + o_i) * sc);
                        float2 zb = make_float2((e_r - o_r) * sc, (e_i - o_i) * sc);
                        za = cmulc(pa, za);
                        zb = cmulc(pb, zb);
                        const bool neg = !self && (v & 2);
                        if (neg) {
                            za.y = -za.y;
                            zb.y = -zb.y;
                        }
                        const int img = self ? v >> 1 : v >> 2, row = (v & 1) * L + (neg ? L - k : k);
                        float2* y = Y + (long long)img * img_stride + (long long)row * N;
                        y[c] = za;
                        y[N - 1 - c] = zb;
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_addr(&acc_free[ai]));
            }
            ++un;
        }
    } else if (warp >= 8) {  // rows of the unit -> E and O, split, in shared memory
        constexpr int VPW = 32 / LPV;  // vectors per warp and step
        const int l = lane % LPV, vs = lane / LPV;
        int un = 0;
        bool ok = true;
        for (int u = blockIdx.x; ok && u < total; u += gridDim.x) {
            const int k = u / tiles, v0 = (u % tiles) * VT, nv = vectors(k);
            if (v0 >= nv) continue;
            const bool self = (k == 0 || k == N);
            const int bi = un % W::NB, br = un / W::NB;
            unsigned char* B0 = bbuf + (size_t)bi * 4 * W::BT;
            float* iv = inv + (un & 3) * VT;
            float2 pa[8], pb[8];  // phases of entries c = 2 l + 2 LPV q + r and N - 1 - c
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int c = 2 * l + 2 * LPV * q + r;
                    pa[2 * q + r] = roots[op_phase_in<n>(k, c, bp)];
                    pb[2 * q + r] = roots[op_phase_in<n>(k, N - 1 - c, bp)];
                }
            bool waited = br == 0;
            for (int vb = (warp - 8) * VPW; vb < VT; vb += 8 * VPW) {
                const int v = v0 + vb + vs;
                float er[8], ei[8], orr[8], oi[8], m = 0.f;
                if (v < nv) {
                    const bool neg = !self && (v & 2);
                    const int img = self ? v >> 1 : v >> 2, row = (v & 1) * L + (neg ? L - k : k);
                    const float2* y = Y + (long long)img * img_stride + (long long)row * N;
                    const float sg = neg ? -1.f : 1.f;  // the row of -k enters conjugated
                    float4 ya[4], yb[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int c = 2 * l + 2 * LPV * q;
                        ya[q] = *reinterpret_cast<const float4*>(y + c);
                        yb[q] = *reinterpret_cast<const float4*>(y + (N - 2 - c));
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q)
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            const int i = 2 * q + r;
                            const float2 a = cmul(pa[i], r ? make_float2(ya[q].z, sg * ya[q].w) : make_float2(ya[q].x, sg * ya[q].y));
                            const float2 b = cmul(pb[i], r ? make_float2(yb[q].x, sg * yb[q].y) : make_float2(yb[q].z, sg * yb[q].w));
                            er[i] = a.x + b.x;
                            ei[i] = a.y + b.y;
                            orr[i] = bp ? a.y - b.y : a.x - b.x;
                            oi[i] = bp ? b.x - a.x : a.y - b.y;
                            m = fmaxf(m, fmaxf(fmaxf(fabsf(er[i]), fabsf(ei[i])), fmaxf(fabsf(orr[i]), fabsf(oi[i]))));
                        }
                }
#pragma unroll
                for (int o = LPV / 2; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
                if (!waited) {  // the buffer's previous unit must have been multiplied
                    waited = true;
                    if (!warp_wait(smem_addr(&b_free[bi]), (uint32_t)((br - 1) & 1), abort_flag)) {
                        if (lane == 0) *abort_flag = 1;
                        ok = false;
                        break;
                    }
                }
                if (v < nv) {
                    // 2^(13 - floor(log2 m)): the largest value lands in [2^13, 2^14)
                    int ex = (int)(__float_as_uint(m) >> 23) - 127;
                    ex = ex < -113 ? -113 : ex;
                    const float s = __uint_as_float((uint32_t)(127 + 13 - ex) << 23);
                    if (l == 0) iv[vb + vs] = __uint_as_float((uint32_t)(127 - 13 + ex) << 23);
                    const int vr = vb + vs;
                    unsigned char* re = B0 + (size_t)(vr / 8) * W::SBO + l * W::LBO + (vr % 8) * 16;
                    unsigned char* im = re + (size_t)(VT / 8) * W::SBO;
                    uint4 hi, lo;
                    split8(er, s, hi, lo);
                    *reinterpret_cast<uint4*>(re) = hi;
                    *reinterpret_cast<uint4*>(re + W::BT) = lo;
                    split8(ei, s, hi, lo);
                    *reinterpret_cast<uint4*>(im) = hi;
                    *reinterpret_cast<uint4*>(im + W::BT) = lo;
                    split8(orr, s, hi, lo);
                    *reinterpret_cast<uint4*>(re + 2 * W::BT) = hi;
                    *reinterpret_cast<uint4*>(re + 3 * W::BT) = lo;
                    split8(oi, s, hi, lo);
                    *reinterpret_cast<uint4*>(im + 2 * W::BT) = hi;
                    *reinterpret_cast<uint4*>(im + 3 * W::BT) = lo;
                }
            }
            if (!ok) break;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_addr(&b_full[bi]));
            ++un;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*abort_flag && threadIdx.x == 32) {
        // a wait gave up: every MMA and every matrix copy that was issued must have completed before the tensor memory is
        // freed and the CTA leaves (bounded). Flag 1: this launch's rows are not all written; 2: even the drain ran out
        tc_commit(drain);
        bool drained = mbar_wait(smem_addr(drain), 0u);
        for (int ch = *s_consumed; ch < *s_issued; ++ch)  // at most RING outstanding copies, in distinct stages
            drained = mbar_wait(smem_addr(&a_full[ch % W::RING]), (uint32_t)((ch / W::RING) & 1)) && drained;
        atomicMax(err, drained ? 1 : 2);
    }
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

template <int n>
static int launch_mma(int nimg, const void* Ts, const float* tinv, void* Y, long long img_stride, const void* roots, bool bp,
                      int* err, cudaStream_t st) {
    using W = OmCfg<n>;
    static_assert(W::smem <= 227 * 1024, "shared memory");
    auto kern = rows_op_mma_kernel<n>;
    if (int rc = ensure_smem((const void*)kern, W::smem)) return rc;
    const int tiles = (4 * nimg + W::VT - 1) / W::VT;
    const int total = (W::N + 1) * tiles, sms = device_sm_count();
    kern<<<total < sms ? total : sms, OM_THREADS, W::smem, st>>>(
        nimg, tiles, reinterpret_cast<const __half*>(Ts), tinv, reinterpret_cast<float2*>(Y), img_stride,
        reinterpret_cast<const float2*>(roots), bp, err);
    return launch_status("rows_op_mma_kernel");
}

}  // namespace adrt

using namespace adrt;

extern "C" int adrt_rows_operator_split(int n, const void* T, const float* scale, void* Ts, void* stream) {
    if (n < 8 || n > 9 || !T || !scale || !Ts) {
        set_error("rows_operator_split: bad arguments (n=%d; n must be 8 or 9)", n);
        return ADRT_EINVAL;
    }
    const long long N = 1ll << n, total = (N + 1) * N * N / 2;
    const int grid = 152 * 32;
    const float* t = reinterpret_cast<const float*>(T);
    __half* ts = reinterpret_cast<__half*>(Ts);
    if (n == 8) rows_op_split_kernel<8><<<grid, 256, 0, as_stream(stream)>>>(total, t, scale, ts);
    else rows_op_split_kernel<9><<<grid, 256, 0, as_stream(stream)>>>(total, t, scale, ts);
    return launch_status("rows_op_split_kernel");
}

extern "C" int adrt_rows_operator_mma(int n, int nimg, int kind, const void* Ts, const float* inv_scale, void* Y,
                                      long long img_stride, const void* roots8, int32_t* err, void* stream) {
    if (n < 8 || n > 9 || nimg < 0 || nimg > 65535 || (kind != 0 && kind != 1) ||
        (nimg && (!Ts || !inv_scale || !Y || !roots8 || !err))) {
        set_error("rows_operator_mma: bad arguments (n=%d nimg=%d kind=%d; n must be 8 or 9)", n, nimg, kind);
        return ADRT_EINVAL;
    }
    if ((reinterpret_cast<uintptr_t>(Y) & 15) || (reinterpret_cast<uintptr_t>(Ts) & 15) || (img_stride & 1)) {
        set_error("rows_operator_mma: Ts and Y must be 16-byte aligned with an even image stride");
        return ADRT_EINVAL;
    }
    if (!nimg) return ADRT_OK;
    cudaStream_t st = as_stream(stream);
    if (n == 8) return launch_mma<8>(nimg, Ts, inv_scale, Y, img_stride, roots8, kind == 1, err, st);
    return launch_mma<9>(nimg, Ts, inv_scale, Y, img_stride, roots8, kind == 1, err, st);
}
