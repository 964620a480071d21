// The learned far-field closure (no counterpart in the reference): per-particle
// features from the order-1 local expansion, the MLP correction on the
// 5th-generation tensor cores (tcgen05.mma, BF16 operands in shared memory,
// FP32 accumulators in tensor memory), the sampled FP64 judge with fallback
// to the uncorrected forces, and the training kernels (forward on the tensor
// cores with mma.sync m16n8k16, backward and Adam in FP32).
//
// Features of particle i in leaf u (half width h, depth d), with the leaf's
// field L and field gradient G after the order-1 downward pass:
//   s = |L| + h |G|_F
//   x = (L / s, G h / s [xx yy zz xy xz yz], (x_i - c_u) / h, d / 10, 0, 0, 0)
// and the correction is dF_i = m_i s kMlpOutScale MLP(x).
//
// Bounds: the MLP is ~2 x 9.9K flop per particle on the BF16 tensor pipe and
// reads ~80 B per particle; the judge is 4096 x N FP64 pair terms.
#include <algorithm>
#include <cfloat>
#include <cuda_bf16.h>

#include "psg_closure.cuh"
#include "psg_common.cuh"
#include "psg_kernels.h"

namespace psg {

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}

__device__ __forceinline__ float bf16_bits_to_float(uint16_t h) {
    return __uint_as_float((uint32_t)h << 16);
}

__device__ __forceinline__ uint16_t float_to_bf16_bits(float f) {
    __nv_bfloat16 b = __float2bfloat16_rn(f);
    return *reinterpret_cast<uint16_t*>(&b);
}

// D += A (16x16, row) . B (16x8, col), BF16 in, FP32 accumulate
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                         uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// GELU, tanh form: 0.5 x (1 + tanh(sqrt(2/pi) (x + 0.044715 x^3))), and its
// derivative
__device__ __forceinline__ float gelu(float x, float& grad) {
    const float x2 = x * x;
    const float u = 0.7978845608028654f * fmaf(0.044715f * x, x2, x);
    const float th = tanhf(u);
    grad = fmaf(0.5f * x * (1.0f - th * th) * 0.7978845608028654f, fmaf(0.134145f, x2, 1.0f),
                0.5f * (1.0f + th));
    return 0.5f * x * (1.0f + th);
}

// features of sorted particle i; returns m_i s kMlpOutScale
__device__ __forceinline__ float closure_features(const TreeView& tv,
                                                  const uint32_t* __restrict__ leaf_of,
                                                  const float4* __restrict__ xyzm, size_t i,
                                                  float* x) {
    const uint32_t u = leaf_of[i];
    if (u >= tv.lvl_base[kLevels]) {  // no leaf recorded: no features, no correction
        for (int k = 0; k < 16; ++k) x[k] = 0.f;
        return 0.f;
    }
    const float4 L = tv.lt[u];
    const float4 g0 = tv.lg0[u];
    const float2 g1 = tv.lg1[u];
    const float4 c = tv.geo[u];
    const float4 p = xyzm[i];
    int depth = 0;
#pragma unroll
    for (int d = 1; d <= kMaxDepth; ++d) depth += u >= tv.lvl_base[d] ? 1 : 0;
    const float h = c.w;
    const float gn = sqrtf(g0.x * g0.x + g0.y * g0.y + g0.z * g0.z +
                           2.0f * (g0.w * g0.w + g1.x * g1.x + g1.y * g1.y));
    const float s = sqrtf(L.y * L.y + L.z * L.z + L.w * L.w) + h * gn + 1e-30f;
    const float is = 1.0f / s;
    const float gh = h * is;
    const float ih = 1.0f / h;
    x[0] = L.y * is;
    x[1] = L.z * is;
    x[2] = L.w * is;
    x[3] = g0.x * gh;
    x[4] = g0.y * gh;
    x[5] = g0.z * gh;
    x[6] = g0.w * gh;
    x[7] = g1.x * gh;
    x[8] = g1.y * gh;
    x[9] = (p.x - c.x) * ih;
    x[10] = (p.y - c.y) * ih;
    x[11] = (p.z - c.z) * ih;
    x[12] = 0.1f * (float)depth;
    x[13] = x[14] = x[15] = 0.f;
    return p.w * s * kMlpOutScale;
}

__device__ __forceinline__ void load_packed(MlpPacked& dst, const MlpPacked* src) {
    const uint4* s = reinterpret_cast<const uint4*>(src);
    uint4* d = reinterpret_cast<uint4*>(&dst);
    for (int i = threadIdx.x; i < (int)(sizeof(MlpPacked) / 16); i += blockDim.x) d[i] = s[i];
}

// ---- inference on the 5th-generation tensor cores (tcgen05, TMEM) ----------
// CTAs of 128 threads (4 per SM) take tiles of 128 particles; thread t owns
// row t.  Each layer is D[128 x N] = A[128 x K] . Wt^T (K x N) by
// tcgen05.mma (kind::f16: BF16 operands from shared memory, FP32
// accumulator in tensor memory), issued by one thread, its completion
// signalled on an mbarrier; every thread then reads its row of D from
// tensor memory (tcgen05.ld), adds the bias, applies GELU and writes the
// BF16 row as the next layer's A.  Shared-memory operands are in the
// no-swizzle K-major layout: 8-row x 16-byte core matrices, 128 B apart
// along the rows (the descriptor's stride offset) and R/8 x 128 B apart
// along K (its leading offset) for a matrix of R rows.
constexpr int kTcRows = 128;       // the MMA's M, one particle per row
constexpr uint32_t kTcCols = 64;   // tensor-memory columns: one 128 x 64 FP32 accumulator
constexpr long long kTcWaitCycles = 1ll << 31;  // ~1 s: the bound on an MMA's completion
// CTAs per SM: while one waits on its MMA, the others compute features and
// activations (41 KB of shared memory and 64 tensor-memory columns each)
constexpr int kTcBlocksPerSm = 4;

struct __align__(128) TcSmem {
    uint8_t a0[kTcRows * kMlpIn * 2];   // features, 128 x 16
    uint8_t h[kTcRows * kMlpHid * 2];   // hidden activations, 128 x 64
    uint8_t w1[kMlpHid * kMlpIn * 2];   // Wt1: N = 64 rows x K = 16
    uint8_t w2[kMlpHid * kMlpHid * 2];  // Wt2: 64 x 64
    uint8_t w3[kMlpHid * kMlpHid * 2];  // Wt3: 64 x 64
    uint8_t w4[16 * kMlpHid * 2];       // Wt4: N = 16 rows (8 .. 15 zero) x K = 64
    float b1[kMlpHid], b2[kMlpHid], b3[kMlpHid], b4[16];
    uint64_t mbar;
    uint32_t tmem;
};

// byte offset of element (row, k) of a K-major BF16 operand of `rows` rows
__device__ __forceinline__ uint32_t kmaj_off(uint32_t row, uint32_t k, uint32_t rows) {
    return ((k >> 3) * (rows >> 3) + (row >> 3)) * 128u + (row & 7u) * 16u + (k & 7u) * 2u;
}

// shared-memory matrix descriptor of a K-major operand at shared address
// saddr (no swizzle; leading offset = rows/8 x 128 B between the two 8-wide
// K chunks of one MMA, stride offset = 128 B between 8-row groups; version 1)
__device__ __forceinline__ uint64_t kmaj_desc(uint32_t saddr, uint32_t rows) {
    const uint64_t lbo = (uint64_t)(rows >> 3) * 128u, sbo = 128u;
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((lbo >> 4) << 16) | ((sbo >> 4) << 32) |
           (1ull << 46);
}

// instruction descriptor: BF16 A and B (K-major), FP32 D, M = 128, N = n
__host__ __device__ constexpr uint32_t tc_idesc(uint32_t n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) |
           ((uint32_t)(kTcRows >> 4) << 24);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// one thread: D (+)= A . B over `ksteps` K-steps of 16, then the commit that
// arrives on the mbarrier when they are done
__device__ __forceinline__ void tc_layer(uint32_t tmem, uint32_t a_addr, uint32_t a_rows,
                                         uint32_t b_addr, uint32_t b_rows, uint32_t idesc,
                                         int ksteps, uint32_t mbar) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    for (int s = 0; s < ksteps; ++s) {
        const uint64_t ad = kmaj_desc(a_addr + (uint32_t)s * 2u * (a_rows >> 3) * 128u, a_rows);
        const uint64_t bd = kmaj_desc(b_addr + (uint32_t)s * 2u * (b_rows >> 3) * 128u, b_rows);
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
            "l"(ad), "l"(bd), "r"(idesc), "r"(s));
    }
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
        : "memory");
}

// wait for the mbarrier's phase `ph` to complete, at most kTcWaitCycles
__device__ __forceinline__ bool tc_wait(uint32_t mbar, uint32_t ph) {
    const long long t0 = clock64();
    for (;;) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(mbar), "r"(ph)
            : "memory");
        if (done) return true;
        if (clock64() - t0 > kTcWaitCycles) return false;
    }
}

// this thread's row of the accumulator, columns [c0, c0 + 16)
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
        "%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = __uint_as_float(r[k]);
}

// GELU with the hardware's approximate tanh (PTX tanh.approx.f32, relative
// error below 2^-10.9): far below the BF16 rounding every activation gets
// next, and a quarter of the closure network's time against tanhf
__device__ __forceinline__ float gelu_hw(float x) {
    const float u = 0.7978845608028654f * fmaf(0.044715f * x, x * x, x);
    float th;
    asm("tanh.approx.f32 %0, %1;" : "=f"(th) : "f"(u));
    return 0.5f * x * (1.0f + th);
}

// z = D[t] + b; GELU(z) rounded to BF16 into row t of the activations
__device__ __forceinline__ void tc_act(TcSmem& sm, uint32_t trow, const float* bias, uint32_t t) {
#pragma unroll
    for (int c0 = 0; c0 < kMlpHid; c0 += 16) {
        float v[16];
        tc_ld16(trow + (uint32_t)c0, v);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            uint4 q;
            uint32_t* qq = reinterpret_cast<uint32_t*>(&q);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int k = c0 + half * 8 + 2 * j;
                qq[j] = pack_bf16x2(gelu_hw(v[half * 8 + 2 * j] + bias[k]),
                                    gelu_hw(v[half * 8 + 2 * j + 1] + bias[k + 1]));
            }
            *reinterpret_cast<uint4*>(sm.h + kmaj_off(t, (uint32_t)(c0 + half * 8), kTcRows)) = q;
        }
    }
}

__device__ __forceinline__ void tc_sync() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
}

// FEAT: features from the tree (the closure's correction dF = s y); else
// given inputs x[n][16] -> y[n][8] (the checks of the tensor-core path)
template <bool FEAT>
__global__ void __launch_bounds__(kTcRows, kTcBlocksPerSm)
    k_mlp_tc(TreeView tv, const uint32_t* leaf_of, const float4* __restrict__ xyzm,
             const float* __restrict__ xin, size_t n, const MlpPacked* __restrict__ wts,
             float4* __restrict__ dF, float* __restrict__ yout, uint32_t* err) {
    __shared__ TcSmem sm;
    const uint32_t t = threadIdx.x, w = t >> 5;
    const uint32_t mbar = smem_u32(&sm.mbar);
    if (t == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (w == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&sm.tmem)),
                     "r"(kTcCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // weights (transposed, BF16) and biases into the operand layout
    for (uint32_t e = t; e < (uint32_t)(kMlpHid * kMlpIn); e += kTcRows) {
        const uint32_t r = e / kMlpIn, k = e % kMlpIn;
        *reinterpret_cast<uint16_t*>(sm.w1 + kmaj_off(r, k, kMlpHid)) = wts->wt1[r * kLd1 + k];
    }
    for (uint32_t e = t; e < (uint32_t)(kMlpHid * kMlpHid); e += kTcRows) {
        const uint32_t r = e / kMlpHid, k = e % kMlpHid;
        *reinterpret_cast<uint16_t*>(sm.w2 + kmaj_off(r, k, kMlpHid)) = wts->wt2[r * kLdH + k];
        *reinterpret_cast<uint16_t*>(sm.w3 + kmaj_off(r, k, kMlpHid)) = wts->wt3[r * kLdH + k];
    }
    for (uint32_t e = t; e < 16u * kMlpHid; e += kTcRows) {
        const uint32_t r = e / kMlpHid, k = e % kMlpHid;
        *reinterpret_cast<uint16_t*>(sm.w4 + kmaj_off(r, k, 16)) =
            r < (uint32_t)kMlpOut ? wts->wt4[r * kLdH + k] : (uint16_t)0;
    }
    if (t < (uint32_t)kMlpHid) {
        sm.b1[t] = wts->b1[t];
        sm.b2[t] = wts->b2[t];
        sm.b3[t] = wts->b3[t];
    }
    if (t < 16) sm.b4[t] = t < (uint32_t)kMlpOut ? wts->b4[t] : 0.f;
    tc_sync();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sm.tmem;
    const uint32_t trow = tmem + ((w * 32u) << 16);  // this warp's 32 lanes
    const uint32_t a0 = smem_u32(sm.a0), hh = smem_u32(sm.h);
    const uint32_t w1 = smem_u32(sm.w1), w2 = smem_u32(sm.w2), w3 = smem_u32(sm.w3),
                   w4 = smem_u32(sm.w4);
    uint32_t ph = 0;
    bool ok = true;
    const size_t tiles = (n + kTcRows - 1) / kTcRows;
    for (size_t tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        const size_t i = tile * kTcRows + t;
        float x[16];
        float sc = 0.f;
        if (i < n) {
            if constexpr (FEAT) {
                sc = closure_features(tv, leaf_of, xyzm, i, x);
            } else {
#pragma unroll
                for (int k = 0; k < 16; ++k) x[k] = xin[i * 16 + k];
            }
        } else {
#pragma unroll
            for (int k = 0; k < 16; ++k) x[k] = 0.f;
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            uint4 q;
            q.x = pack_bf16x2(x[8 * c + 0], x[8 * c + 1]);
            q.y = pack_bf16x2(x[8 * c + 2], x[8 * c + 3]);
            q.z = pack_bf16x2(x[8 * c + 4], x[8 * c + 5]);
            q.w = pack_bf16x2(x[8 * c + 6], x[8 * c + 7]);
            *reinterpret_cast<uint4*>(sm.a0 + kmaj_off(t, (uint32_t)(8 * c), kTcRows)) = q;
        }
        // layers 1 .. 3 (64 wide), then the output layer (16 wide, 8 used)
        const uint32_t a_addr[4] = {a0, hh, hh, hh};
        const uint32_t b_addr[4] = {w1, w2, w3, w4};
        const float* bias[3] = {sm.b1, sm.b2, sm.b3};
        for (int l = 0; l < 4 && ok; ++l) {
            tc_sync();
            if (t == 0)
                tc_layer(tmem, a_addr[l], kTcRows, b_addr[l], l < 3 ? kMlpHid : 16,
                         tc_idesc(l < 3 ? kMlpHid : 16), l == 0 ? 1 : 4, mbar);
            const bool done = tc_wait(mbar, ph);
            ph ^= 1u;
            ok = !__syncthreads_or(!done);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (l < 3) {
                tc_act(sm, trow, bias[l], t);
            } else {
                float y[16];
                tc_ld16(trow, y);
                if (i < n) {
                    if constexpr (FEAT) {
                        dF[i] = make_float4(sc * (y[0] + sm.b4[0]), sc * (y[1] + sm.b4[1]),
                                            sc * (y[2] + sm.b4[2]), 0.f);
                    } else {
#pragma unroll
                        for (int o = 0; o < kMlpOut; ++o) yout[i * kMlpOut + o] = y[o] + sm.b4[o];
                    }
                }
            }
        }
    }
    if (!ok) {
        // an MMA that did not complete in time: report it, give the last
        // commit one more bounded wait, then release the tensor memory
        if (t == 0) atomicOr(err, PSG_ERR_TC_TIMEOUT);
        tc_wait(mbar, ph ^ 1u);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (w == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(kTcCols)
                     : "memory");
}

// features (and scale) of selected particles, for building training data
__global__ void __launch_bounds__(256) k_closure_features(TreeView tv, const uint32_t* leaf_of,
                                                          const float4* __restrict__ xyzm,
                                                          size_t n, const uint32_t* idx,
                                                          size_t k, float* __restrict__ x_out,
                                                          float* __restrict__ scale_out) {
    const size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= k) return;
    const uint32_t i = idx[j];
    float x[16];
    float sc = 0.f;
    if (i < n) {
        sc = closure_features(tv, leaf_of, xyzm, i, x);
    } else {
        for (int q = 0; q < 16; ++q) x[q] = 0.f;
    }
    for (int q = 0; q < 16; ++q) x_out[j * 16 + q] = x[q];
    scale_out[j] = sc;
}

// ---- judge ----------------------------------------------------------------
__global__ void k_judge_sample(uint32_t* tg, int s, size_t n, uint32_t tick) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= s) return;
    const size_t stride = n / (size_t)s;
    const size_t off = stride > 1 ? ((size_t)tick * 7919u) % stride : 0;
    size_t i = (size_t)k * n / (size_t)s + off;
    tg[k] = (uint32_t)(i < n ? i : n - 1);
}

// medians of the per-sample relative errors with and without the correction;
// the correction is used only when its median is lower
__global__ void __launch_bounds__(1024) k_judge_decide(const uint32_t* tg, int s,
                                                       const double* f64, const float* fx,
                                                       const float* fy, const float* fz,
                                                       const float4* dF, int allow,
                                                       JudgeOut* out) {
    __shared__ float e0[kJudgeSamples], e1[kJudgeSamples];
    // the sort runs over the smallest power of two >= s, padded with FLT_MAX
    int s2 = 2;
    while (s2 < s && s2 < kJudgeSamples) s2 <<= 1;
    for (int k = threadIdx.x; k < s2; k += blockDim.x) {
        float a = FLT_MAX, b = FLT_MAX;
        if (k < s) {
            const uint32_t i = tg[k];
            const double rx = f64[3 * k], ry = f64[3 * k + 1], rz = f64[3 * k + 2];
            const double nr = sqrt(rx * rx + ry * ry + rz * rz);
            const double bx = (double)fx[i] - rx, by = (double)fy[i] - ry, bz = (double)fz[i] - rz;
            const float4 d = dF[i];
            const double cx = bx + d.x, cy = by + d.y, cz = bz + d.z;
            const double den = nr > 1e-300 ? nr : 1e-300;
            a = (float)(sqrt(bx * bx + by * by + bz * bz) / den);
            b = (float)(sqrt(cx * cx + cy * cy + cz * cz) / den);
        }
        e0[k] = a;
        e1[k] = b;
    }
    __syncthreads();
    // bitonic sort, ascending, both arrays
    for (int size = 2; size <= s2; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = threadIdx.x; i < s2; i += blockDim.x) {
                const int j = i ^ stride;
                if (j > i) {
                    const bool up = (i & size) == 0;
                    float x = e0[i], y = e0[j];
                    if ((x > y) == up) {
                        e0[i] = y;
                        e0[j] = x;
                    }
                    x = e1[i];
                    y = e1[j];
                    if ((x > y) == up) {
                        e1[i] = y;
                        e1[j] = x;
                    }
                }
            }
            __syncthreads();
        }
    }
    if (threadIdx.x == 0) {
        double m0 = 0.0, m1 = 0.0;
        if (s > 0) {
            if (s & 1) {
                m0 = e0[s / 2];
                m1 = e1[s / 2];
            } else {
                m0 = 0.5 * ((double)e0[s / 2 - 1] + (double)e0[s / 2]);
                m1 = 0.5 * ((double)e1[s / 2 - 1] + (double)e1[s / 2]);
            }
        }
        out->median_base = m0;
        out->median_mlp = m1;
        out->use_mlp = (allow && s > 0 && m1 < m0) ? 1 : 0;
        out->samples = s;
    }
}

__global__ void __launch_bounds__(256) k_closure_apply(float* fx, float* fy, float* fz,
                                                       const float4* __restrict__ dF, size_t n,
                                                       const JudgeOut* j) {
    if (!j->use_mlp) return;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const float4 d = dF[i];
        fx[i] += d.x;
        fy[i] += d.y;
        fz[i] += d.z;
    }
}

// ---- parameters -------------------------------------------------------------
// FP32 parameter vector -> BF16 transposed weights + FP32 biases
__global__ void k_mlp_pack(const float* __restrict__ p, MlpPacked* __restrict__ out) {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int stride = gridDim.x * blockDim.x;
    for (int e = tid; e < kMlpHid * kLd1; e += stride) {
        const int o = e / kLd1, i = e % kLd1;
        out->wt1[e] = float_to_bf16_bits(i < kMlpIn ? p[kOffW1 + i * kMlpHid + o] : 0.f);
    }
    for (int e = tid; e < kMlpHid * kLdH; e += stride) {
        const int o = e / kLdH, i = e % kLdH;
        out->wt2[e] = float_to_bf16_bits(i < kMlpHid ? p[kOffW2 + i * kMlpHid + o] : 0.f);
        out->wt3[e] = float_to_bf16_bits(i < kMlpHid ? p[kOffW3 + i * kMlpHid + o] : 0.f);
    }
    for (int e = tid; e < kMlpOut * kLdH; e += stride) {
        const int o = e / kLdH, i = e % kLdH;
        out->wt4[e] = float_to_bf16_bits(i < kMlpHid ? p[kOffW4 + i * kMlpOut + o] : 0.f);
    }
    for (int e = tid; e < kMlpHid; e += stride) {
        out->b1[e] = p[kOffB1 + e];
        out->b2[e] = p[kOffB2 + e];
        out->b3[e] = p[kOffB3 + e];
    }
    for (int e = tid; e < kMlpOut; e += stride) out->b4[e] = p[kOffB4 + e];
}

// ---- training ---------------------------------------------------------------
constexpr int kTrainRows = 32;      // samples per block: 128 blocks a batch of 4096
constexpr int kTrainThreads = 256;  // 8 warps: 2 row tiles of 16 x 4 column groups of 16
constexpr int kTrLd0 = kLd1;        // row strides in shared memory, padded against
constexpr int kTrLdH = kLdH;        // bank conflicts
constexpr int kTrLdF = kMlpHid + 4;

struct TrainSmem {
    MlpPacked w;
    uint16_t h0[kTrainRows * kTrLd0];  // BF16 inputs
    uint16_t h[3][kTrainRows * kTrLdH];  // BF16 activations
    float dact[3][kTrainRows * kTrLdF];  // GELU' at the pre-activations
    float da[kTrainRows * kTrLdF];       // gradients, ping-pong
    float db[kTrainRows * kTrLdF];
    float dy[kTrainRows * kMlpOut];
};

size_t mlp_train_smem_bytes() { return sizeof(TrainSmem); }

// this warp's tiles of C[32 x 8 NT] = A[32 x 16 KC] . W: row tile rt, the NT
// n-tiles from nt0, A as BF16 rows (stride LDA), W as Wt[out][in] (stride LDW)
template <int KC, int NT, int LDA, int LDW>
__device__ __forceinline__ void train_layer(const uint16_t* a, const uint16_t* wt, int rt, int nt0,
                                            float (&c)[NT][4]) {
    const uint32_t lane = lane_id(), g = lane >> 2, t = lane & 3;
    uint32_t f[KC][4];
    const uint16_t* row = a + (rt * 16 + g) * LDA + 2 * t;
#pragma unroll
    for (int kc = 0; kc < KC; ++kc) {
        f[kc][0] = *reinterpret_cast<const uint32_t*>(row + kc * 16);
        f[kc][1] = *reinterpret_cast<const uint32_t*>(row + 8 * LDA + kc * 16);
        f[kc][2] = *reinterpret_cast<const uint32_t*>(row + kc * 16 + 8);
        f[kc][3] = *reinterpret_cast<const uint32_t*>(row + 8 * LDA + kc * 16 + 8);
    }
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        c[j][0] = c[j][1] = c[j][2] = c[j][3] = 0.f;
        const uint16_t* wr = wt + ((nt0 + j) * 8 + g) * LDW + 2 * t;
#pragma unroll
        for (int kc = 0; kc < KC; ++kc) {
            const uint32_t b0 = *reinterpret_cast<const uint32_t*>(wr + kc * 16);
            const uint32_t b1 = *reinterpret_cast<const uint32_t*>(wr + kc * 16 + 8);
            mma_bf16(c[j], f[kc], b0, b1);
        }
    }
}

// z = c + b; GELU(z) rounded to BF16 and GELU'(z) to shared memory
__device__ __forceinline__ void train_act(const float (&c)[2][4], const float* bias, int rt,
                                          int nt0, uint16_t* h, float* dact) {
    const uint32_t lane = lane_id(), g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int col = (nt0 + j) * 8 + 2 * t;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int r = rt * 16 + half * 8 + g;
            float g0, g1;
            const float a0 = gelu(c[j][2 * half] + bias[col], g0);
            const float a1 = gelu(c[j][2 * half + 1] + bias[col + 1], g1);
            *reinterpret_cast<uint32_t*>(h + r * kTrLdH + col) = pack_bf16x2(a0, a1);
            *reinterpret_cast<float2*>(dact + r * kTrLdF + col) = make_float2(g0, g1);
        }
    }
}

__device__ __forceinline__ float4 bf16x4_to_float4(uint2 v) {
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xFFFF0000u),
                       __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xFFFF0000u));
}

// dW[k][n] += sum_b h[b][k] d[b][n] over 64 columns n and K = 64 or 16 rows k:
// each thread a tile of K / 16 x 4
template <int K, int LDH>
__device__ __forceinline__ void accum_dw(const uint16_t* h, const float* d, float* gW) {
    constexpr int R = K / 16;
    const int k0 = (threadIdx.x >> 4) * R, n0 = (threadIdx.x & 15) * 4;
    float4 acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int b = 0; b < kTrainRows; ++b) {
        const float4 v = *reinterpret_cast<const float4*>(d + b * kTrLdF + n0);
        float hk[R];
        if constexpr (R == 4) {
            const float4 q =
                bf16x4_to_float4(*reinterpret_cast<const uint2*>(h + b * LDH + k0));
            hk[0] = q.x;
            hk[1] = q.y;
            hk[2] = q.z;
            hk[3] = q.w;
        } else {
            hk[0] = bf16_bits_to_float(h[b * LDH + k0]);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            acc[r].x = fmaf(hk[r], v.x, acc[r].x);
            acc[r].y = fmaf(hk[r], v.y, acc[r].y);
            acc[r].z = fmaf(hk[r], v.z, acc[r].z);
            acc[r].w = fmaf(hk[r], v.w, acc[r].w);
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
        atomicAdd(reinterpret_cast<float4*>(gW + (k0 + r) * kMlpHid + n0), acc[r]);
}

// db[n] += sum_b d[b][n] over 64 columns
__device__ __forceinline__ void accum_db(const float* d, float* gB) {
    if (threadIdx.x < (unsigned)kMlpHid) {
        float sum = 0.f;
#pragma unroll 8
        for (int b = 0; b < kTrainRows; ++b) sum += d[b * kTrLdF + threadIdx.x];
        atomicAdd(gB + threadIdx.x, sum);
    }
}

// dnext[b][k] = (sum_n d[b][n] W[k][n]) * GELU'(z[b][k]), W[k][n] = Wt[n][k]:
// each thread 2 rows x 4 columns
template <int N, int LDD>
__device__ __forceinline__ void back_act(const float* d, const uint16_t* wt, const float* dact,
                                         float* dnext) {
    const int b0 = (threadIdx.x >> 4) * 2, k0 = (threadIdx.x & 15) * 4;
    float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int n = 0; n < N; ++n) {
        const float4 w = bf16x4_to_float4(*reinterpret_cast<const uint2*>(wt + n * kLdH + k0));
        const float d0 = d[b0 * LDD + n], d1 = d[(b0 + 1) * LDD + n];
        s0[0] = fmaf(d0, w.x, s0[0]);
        s0[1] = fmaf(d0, w.y, s0[1]);
        s0[2] = fmaf(d0, w.z, s0[2]);
        s0[3] = fmaf(d0, w.w, s0[3]);
        s1[0] = fmaf(d1, w.x, s1[0]);
        s1[1] = fmaf(d1, w.y, s1[1]);
        s1[2] = fmaf(d1, w.z, s1[2]);
        s1[3] = fmaf(d1, w.w, s1[3]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        dnext[b0 * kTrLdF + k0 + j] = s0[j] * dact[b0 * kTrLdF + k0 + j];
        dnext[(b0 + 1) * kTrLdF + k0 + j] = s1[j] * dact[(b0 + 1) * kTrLdF + k0 + j];
    }
}

// Loss sum_{samples, outputs 0..2} (y - t)^2 and its gradient, scaled by
// inv_norm, accumulated into grad (FP32 parameter layout) and loss_sum.
// Forward on the tensor cores (mma.sync, BF16 with FP32 accumulation), backward
// in FP32 with register tiles: a batch of 4096 is 164 MFLOP of FP32, so the
// kernel is bound by the chain of small phases and their barriers, not by a
// pipe; 32 rows a block spread a batch over 128 SMs.  Measured: a batch of 4096
// 62 us (64 rows a block, one thread per output, one shared-memory load per
// FMA) -> 17 us.
__global__ void __launch_bounds__(kTrainThreads) k_mlp_grad(const float* __restrict__ X,
                                                  const float* __restrict__ T,
                                                  const uint32_t* __restrict__ perm, size_t b0,
                                                  size_t count, const MlpPacked* __restrict__ wts,
                                                  float inv_norm, float* __restrict__ grad,
                                                  float* __restrict__ loss_sum) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TrainSmem& S = *reinterpret_cast<TrainSmem*>(smem_raw);
    const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
    const int rt = (int)w >> 2, nt0 = ((int)w & 3) * 2;
    const size_t r_blk = (size_t)blockIdx.x * kTrainRows;
    load_packed(S.w, wts);
    // inputs, rounded to BF16 (zeros past the batch)
    for (int e = threadIdx.x; e < kTrainRows * kMlpIn; e += kTrainThreads) {
        const int r = e / kMlpIn, k = e % kMlpIn;
        const bool valid = r_blk + r < count;
        const size_t src = valid ? (perm ? perm[b0 + r_blk + r] : b0 + r_blk + r) : 0;
        S.h0[r * kTrLd0 + k] = float_to_bf16_bits(valid ? X[src * kMlpIn + k] : 0.f);
    }
    __syncthreads();
    float c[2][4];
    train_layer<1, 2, kTrLd0, kLd1>(S.h0, S.w.wt1, rt, nt0, c);
    train_act(c, S.w.b1, rt, nt0, S.h[0], S.dact[0]);
    __syncthreads();
    train_layer<4, 2, kTrLdH, kLdH>(S.h[0], S.w.wt2, rt, nt0, c);
    train_act(c, S.w.b2, rt, nt0, S.h[1], S.dact[1]);
    __syncthreads();
    train_layer<4, 2, kTrLdH, kLdH>(S.h[1], S.w.wt3, rt, nt0, c);
    train_act(c, S.w.b3, rt, nt0, S.h[2], S.dact[2]);
    __syncthreads();
    if (nt0 == 0) {  // the output layer: one warp per row tile
        float o[1][4];
        train_layer<4, 1, kTrLdH, kLdH>(S.h[2], S.w.wt4, rt, 0, o);
        const uint32_t g = lane >> 2, t = lane & 3;
        float lsum = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = rt * 16 + (j >> 1) * 8 + (int)g, col = 2 * (int)t + (j & 1);
            const bool valid = r_blk + r < count;
            float d = 0.f;
            if (valid && col < kMlpOutUsed) {
                const size_t src = perm ? perm[b0 + r_blk + r] : b0 + r_blk + r;
                const float e = o[0][j] + S.w.b4[col] - T[src * kMlpOutUsed + col];
                lsum = fmaf(e, e, lsum);
                d = 2.0f * e * inv_norm;
            }
            S.dy[r * kMlpOut + col] = d;
        }
        lsum = warp_sum(lsum);
        if (lane == 0 && lsum != 0.f) atomicAdd(loss_sum, lsum);
    }
    __syncthreads();
    // layer 4: 64 x 8 weights, 2 per thread
    {
        const int k = threadIdx.x >> 2, n = (threadIdx.x & 3) * 2;
        float s0 = 0.f, s1 = 0.f;
#pragma unroll 8
        for (int b = 0; b < kTrainRows; ++b) {
            const float hk = bf16_bits_to_float(S.h[2][b * kTrLdH + k]);
            const float2 v = *reinterpret_cast<const float2*>(S.dy + b * kMlpOut + n);
            s0 = fmaf(hk, v.x, s0);
            s1 = fmaf(hk, v.y, s1);
        }
        atomicAdd(reinterpret_cast<float2*>(grad + kOffW4 + k * kMlpOut + n), make_float2(s0, s1));
    }
    if (threadIdx.x < (unsigned)kMlpOut) {
        float sum = 0.f;
        for (int b = 0; b < kTrainRows; ++b) sum += S.dy[b * kMlpOut + threadIdx.x];
        atomicAdd(grad + kOffB4 + threadIdx.x, sum);
    }
    back_act<kMlpOut, kMlpOut>(S.dy, S.w.wt4, S.dact[2], S.da);
    __syncthreads();
    // layer 3
    accum_dw<kMlpHid, kTrLdH>(S.h[1], S.da, grad + kOffW3);
    accum_db(S.da, grad + kOffB3);
    back_act<kMlpHid, kTrLdF>(S.da, S.w.wt3, S.dact[1], S.db);
    __syncthreads();
    // layer 2
    accum_dw<kMlpHid, kTrLdH>(S.h[0], S.db, grad + kOffW2);
    accum_db(S.db, grad + kOffB2);
    back_act<kMlpHid, kTrLdF>(S.db, S.w.wt2, S.dact[0], S.da);
    __syncthreads();
    // layer 1
    accum_dw<kMlpIn, kTrLd0>(S.h0, S.da, grad + kOffW1);
    accum_db(S.da, grad + kOffB1);
}

// the BF16 weight or FP32 bias of parameter i in the kernels' packed copy
__device__ __forceinline__ void pack_param(MlpPacked* out, int i, float p) {
    const uint16_t w = float_to_bf16_bits(p);
    if (i < kOffB1) out->wt1[(i % kMlpHid) * kLd1 + i / kMlpHid] = w;
    else if (i < kOffW2) out->b1[i - kOffB1] = p;
    else if (i < kOffB2) out->wt2[((i - kOffW2) % kMlpHid) * kLdH + (i - kOffW2) / kMlpHid] = w;
    else if (i < kOffW3) out->b2[i - kOffB2] = p;
    else if (i < kOffB3) out->wt3[((i - kOffW3) % kMlpHid) * kLdH + (i - kOffW3) / kMlpHid] = w;
    else if (i < kOffW4) out->b3[i - kOffB3] = p;
    else if (i < kOffB4) out->wt4[((i - kOffW4) % kMlpOut) * kLdH + (i - kOffW4) / kMlpOut] = w;
    else out->b4[i - kOffB4] = p;
}

// Adam (Kingma & Ba 2015) on the FP32 master parameters; the next step's packed
// weights and zeroed gradient too (launches of their own took 5 us each)
__global__ void k_mlp_adam(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v,
                           float* __restrict__ g, MlpPacked* __restrict__ packed, int n, float lr,
                           float beta1, float beta2, float eps, float bc1, float bc2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    g[i] = 0.f;
    const float mi = fmaf(beta1, m[i], (1.0f - beta1) * gi);
    const float vi = fmaf(beta2, v[i], (1.0f - beta2) * gi * gi);
    m[i] = mi;
    v[i] = vi;
    const float pi = p[i] - lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    p[i] = pi;
    pack_param(packed, i, pi);
}

// ---- launchers ------------------------------------------------------------------
void launch_closure_mlp(const TreeView& tv, const uint32_t* leaf_of, const float4* xyzm, size_t n,
                        const MlpPacked* w, float4* dF, int sms, uint32_t* err, cudaStream_t st) {
    const size_t tiles = (n + kTcRows - 1) / kTcRows;
    const size_t grid =
        std::max<size_t>(1, std::min<size_t>(tiles, (size_t)sms * kTcBlocksPerSm));
    k_mlp_tc<true><<<(unsigned)grid, kTcRows, 0, st>>>(tv, leaf_of, xyzm, nullptr, n, w, dF,
                                                       nullptr, err);
}

void launch_mlp_forward(const float* x, size_t n, const MlpPacked* w, float* y, int sms,
                        uint32_t* err, cudaStream_t st) {
    const size_t tiles = (n + kTcRows - 1) / kTcRows;
    const size_t grid =
        std::max<size_t>(1, std::min<size_t>(tiles, (size_t)sms * kTcBlocksPerSm));
    k_mlp_tc<false><<<(unsigned)grid, kTcRows, 0, st>>>(TreeView{}, nullptr, nullptr, x, n, w,
                                                        nullptr, y, err);
}

void launch_closure_features(const TreeView& tv, const uint32_t* leaf_of, const float4* xyzm,
                             size_t n, const uint32_t* idx, size_t k, float* x_out,
                             float* scale_out, cudaStream_t st) {
    if (k == 0) return;
    k_closure_features<<<(unsigned)((k + 255) / 256), 256, 0, st>>>(tv, leaf_of, xyzm, n, idx, k,
                                                                    x_out, scale_out);
}

void launch_judge_direct(const float4* xyzm, size_t n, uint32_t* tg, int s, double* f64,
                         uint32_t tick, int blocks, cudaStream_t st, double* part,
                         size_t part_doubles) {
    k_judge_sample<<<(s + 255) / 256, 256, 0, st>>>(tg, s, n, tick);
    launch_direct_f64(xyzm, n, tg, (size_t)s, f64, blocks, st, part, part_doubles);
}

void launch_judge_decide(const uint32_t* tg, int s, const double* f64, const float* fx,
                         const float* fy, const float* fz, const float4* dF, int allow,
                         JudgeOut* out, cudaStream_t st) {
    k_judge_decide<<<1, 1024, 0, st>>>(tg, s, f64, fx, fy, fz, dF, allow, out);
}

void launch_closure_apply(float* fx, float* fy, float* fz, const float4* dF, size_t n,
                          const JudgeOut* j, int sms, cudaStream_t st) {
    size_t grid = (n + 255) / 256;
    const size_t cap = (size_t)sms * 8;
    if (grid > cap) grid = cap;
    if (grid < 1) grid = 1;
    k_closure_apply<<<(unsigned)grid, 256, 0, st>>>(fx, fy, fz, dF, n, j);
}

void launch_mlp_pack(const float* params, MlpPacked* out, cudaStream_t st) {
    k_mlp_pack<<<16, 256, 0, st>>>(params, out);
}

cudaError_t prepare_mlp_grad_kernel() {
    return cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)sizeof(TrainSmem));
}

void launch_mlp_grad(const float* X, const float* T, const uint32_t* perm, size_t b0,
                     size_t count, const MlpPacked* w, float inv_norm, float* grad,
                     float* loss_sum, cudaStream_t st) {
    if (count == 0) return;
    const unsigned grid = (unsigned)((count + kTrainRows - 1) / kTrainRows);
    k_mlp_grad<<<grid, kTrainThreads, sizeof(TrainSmem), st>>>(X, T, perm, b0, count, w, inv_norm,
                                                               grad, loss_sum);
}

void launch_mlp_adam(float* p, float* m, float* v, float* g, MlpPacked* packed, int n, float lr,
                     float beta1, float beta2, float eps, float bc1, float bc2, cudaStream_t st) {
    k_mlp_adam<<<(n + 127) / 128, 128, 0, st>>>(p, m, v, g, packed, n, lr, beta1, beta2, eps, bc1,
                                                bc2);
}

}  // namespace psg
