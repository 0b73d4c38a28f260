// colo_mlp.cu -- the learned cost model: a 24 -> 64 -> 64 -> 1 ReLU MLP with
// BF16 weights and activations and FP32 accumulation, trained and evaluated
// by hand-written tensor-core kernels (mma.sync.m16n8k16 BF16 -> FP32).
//
// It predicts log1p(instance-table rows) of a candidate from cell-aggregate
// statistics and only presizes output buffers / orders work; results never
// depend on it.
//
// Rounding points (mirrored by the CPU reference in the oracle): inputs,
// weights, H1, H2, dZ2 and dZ1 are rounded to BF16 before they enter a
// product; every product accumulates in FP32; biases, losses and updates
// stay FP32.
//
// Parameter layout (FP32 master copy, kMlpParams floats):
//   W1[32][64] (rows 24..31 zero), b1[64], W2[64][64], b2[64], W3[64], b3
#include <cuda_bf16.h>

#include <cstddef>

#include "colo_internal.h"
#include "colo_mlp.h"

namespace colo {
namespace {

constexpr int IN = kMlpIn, INP = 32, H = 64;
constexpr int OFF_W1 = 0, OFF_B1 = INP * H, OFF_W2 = OFF_B1 + H, OFF_B2 = OFF_W2 + H * H, OFF_W3 = OFF_B2 + H,
              OFF_B3 = OFF_W3 + H;
constexpr int kRowsPerWarp = 16, kWarps = 8, kRowsPerBlock = kRowsPerWarp * kWarps;

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float bf16r(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

__device__ __forceinline__ void mma16816(float* d, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Shared weights: BF16, both orientations for the hidden layer.  Rows are padded by 16 bytes: the
// eight rows that a B fragment is read from then lie in different banks.
struct SmemW {
    __nv_bfloat16 w1t[H][INP + 8];   // [out][in]  (B operand of X.W1)
    __nv_bfloat16 w2t[H][H + 8];     // [out][in]  (B operand of H1.W2)
    __nv_bfloat16 w2[H][H + 8];      // [in][out]  (B operand of dZ2.W2^T)
    float b1[H], b2[H], w3[H];
    float b3;
};

__device__ void load_weights(SmemW& s, const float* __restrict__ P) {
    for (int i = threadIdx.x; i < INP * H; i += blockDim.x) {
        int in = i / H, o = i % H;
        s.w1t[o][in] = __float2bfloat16_rn(P[OFF_W1 + i]);
    }
    for (int i = threadIdx.x; i < H * H; i += blockDim.x) {
        int in = i / H, o = i % H;
        __nv_bfloat16 v = __float2bfloat16_rn(P[OFF_W2 + i]);
        s.w2t[o][in] = v;
        s.w2[in][o] = v;
    }
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        s.b1[i] = P[OFF_B1 + i];
        s.b2[i] = P[OFF_B2 + i];
        s.w3[i] = bf16r(P[OFF_W3 + i]);
    }
    if (threadIdx.x == 0) s.b3 = P[OFF_B3];
}

// B fragment of a [N][K] row-major BF16 matrix for n-tile nt, k-tile kt.
template <int LD>
__device__ __forceinline__ void bfrag(const __nv_bfloat16 (*m)[LD], int nt, int kt, int gid, int tig, uint32_t& b0,
                                      uint32_t& b1) {
    const __nv_bfloat16* r = m[nt * 8 + gid] + kt * 16 + tig * 2;
    b0 = *reinterpret_cast<const uint32_t*>(r);
    b1 = *reinterpret_cast<const uint32_t*>(r + 8);
}

// Forward pass of one warp's 16 rows.  Outputs pre-activations (z1, z2) in
// accumulator layout and the prediction y for rows gid and gid+8.
__device__ __forceinline__ void forward16(const SmemW& s, const float* __restrict__ X,
                                          const uint32_t* __restrict__ idx, uint64_t row0, uint64_t n, int gid,
                                          int tig, float z1[8][4], float z2[8][4], float& y_lo, float& y_hi,
                                          uint32_t xa[2][4]) {
    // X tile -> A fragments (K = 32, 2 k-tiles)
    const uint64_t r_lo = row0 + gid, r_hi = row0 + gid + 8;
    const uint64_t x_lo = r_lo < n ? (idx ? idx[r_lo] : r_lo) : 0, x_hi = r_hi < n ? (idx ? idx[r_hi] : r_hi) : 0;
    for (int kt = 0; kt < 2; ++kt) {
        float v[8];
        for (int q = 0; q < 8; ++q) {
            int col = kt * 16 + (q >= 4 ? 8 : 0) + tig * 2 + (q & 1);
            uint64_t rr = (q & 2) ? r_hi : r_lo;
            uint64_t xr = (q & 2) ? x_hi : x_lo;
            v[q] = (col < IN && rr < n) ? X[xr * IN + col] : 0.0f;
        }
        xa[kt][0] = pack_bf16(v[0], v[1]);   // row gid,   cols tig*2..
        xa[kt][1] = pack_bf16(v[2], v[3]);   // row gid+8
        xa[kt][2] = pack_bf16(v[4], v[5]);   // row gid,   cols 8+tig*2..
        xa[kt][3] = pack_bf16(v[6], v[7]);   // row gid+8
    }
    for (int nt = 0; nt < 8; ++nt) {
        float bb0 = s.b1[nt * 8 + tig * 2], bb1 = s.b1[nt * 8 + tig * 2 + 1];
        z1[nt][0] = bb0;
        z1[nt][1] = bb1;
        z1[nt][2] = bb0;
        z1[nt][3] = bb1;
        for (int kt = 0; kt < 2; ++kt) {
            uint32_t b0, b1;
            bfrag(s.w1t, nt, kt, gid, tig, b0, b1);
            mma16816(z1[nt], xa[kt], b0, b1);
        }
    }
    // H1 = relu(z1) -> A fragments (K = 64, 4 k-tiles)
    uint32_t ha[4][4];
    for (int kt = 0; kt < 4; ++kt) {
        const float* c0 = z1[2 * kt];
        const float* c1 = z1[2 * kt + 1];
        ha[kt][0] = pack_bf16(fmaxf(c0[0], 0.f), fmaxf(c0[1], 0.f));
        ha[kt][1] = pack_bf16(fmaxf(c0[2], 0.f), fmaxf(c0[3], 0.f));
        ha[kt][2] = pack_bf16(fmaxf(c1[0], 0.f), fmaxf(c1[1], 0.f));
        ha[kt][3] = pack_bf16(fmaxf(c1[2], 0.f), fmaxf(c1[3], 0.f));
    }
    for (int nt = 0; nt < 8; ++nt) {
        float bb0 = s.b2[nt * 8 + tig * 2], bb1 = s.b2[nt * 8 + tig * 2 + 1];
        z2[nt][0] = bb0;
        z2[nt][1] = bb1;
        z2[nt][2] = bb0;
        z2[nt][3] = bb1;
        for (int kt = 0; kt < 4; ++kt) {
            uint32_t b0, b1;
            bfrag(s.w2t, nt, kt, gid, tig, b0, b1);
            mma16816(z2[nt], ha[kt], b0, b1);
        }
    }
    // y = bf16(relu(z2)) . w3 + b3, reduced over the 4 lanes of a row quad
    float plo = 0.f, phi = 0.f;
    for (int nt = 0; nt < 8; ++nt)
        for (int e = 0; e < 2; ++e) {
            int col = nt * 8 + tig * 2 + e;
            plo += bf16r(fmaxf(z2[nt][e], 0.f)) * s.w3[col];
            phi += bf16r(fmaxf(z2[nt][2 + e], 0.f)) * s.w3[col];
        }
    plo += __shfl_xor_sync(0xffffffffu, plo, 1);
    plo += __shfl_xor_sync(0xffffffffu, plo, 2);
    phi += __shfl_xor_sync(0xffffffffu, phi, 1);
    phi += __shfl_xor_sync(0xffffffffu, phi, 2);
    y_lo = plo + s.b3;
    y_hi = phi + s.b3;
}

__global__ void __launch_bounds__(256) k_mlp_forward(const float* __restrict__ P, const float* __restrict__ X,
                                                     uint64_t n, float* __restrict__ y) {
    __shared__ SmemW s;
    load_weights(s, P);
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, gid = lane >> 2, tig = lane & 3;
    for (uint64_t row0 = ((uint64_t)blockIdx.x * kWarps + w) * kRowsPerWarp; row0 < n;
         row0 += (uint64_t)gridDim.x * kRowsPerBlock) {
        float z1[8][4], z2[8][4], ylo, yhi;
        uint32_t xa[2][4];
        forward16(s, X, nullptr, row0, n, gid, tig, z1, z2, ylo, yhi, xa);
        if (tig == 0) {
            if (row0 + gid < n) y[row0 + gid] = ylo;
            if (row0 + gid + 8 < n) y[row0 + gid + 8] = yhi;
        }
    }
}

// Shared memory of the gradient kernel (dynamic): the weights and, for the tile's 128 rows, the
// BF16 operands of the weight gradients.  Rows are padded by 16 bytes: the eight rows of an
// ldmatrix then lie in different banks.
struct GradSmem {
    SmemW w;
    alignas(16) __nv_bfloat16 h1[kRowsPerBlock][H + 8];
    alignas(16) __nv_bfloat16 dz2[kRowsPerBlock][H + 8];
    alignas(16) __nv_bfloat16 dz1[kRowsPerBlock][H + 8];
    alignas(16) __nv_bfloat16 x[kRowsPerBlock][INP + 8];
    float col[3][H], gb3, lsum;   // the block's sums at the end: b1, b2, W3
};
// ldmatrix reads 16-byte rows at 16-byte addresses
static_assert(offsetof(GradSmem, h1) % 16 == 0 && offsetof(GradSmem, dz2) % 16 == 0 && offsetof(GradSmem, dz1) % 16 == 0 &&
                  offsetof(GradSmem, x) % 16 == 0 && sizeof(__nv_bfloat16) * (H + 8) % 16 == 0 &&
                  sizeof(__nv_bfloat16) * (INP + 8) % 16 == 0 && alignof(GradSmem) == 16,
              "alignment");

// A fragment (16 x 16) of S^T, S[k][m] in shared memory: rows m0.., columns (S's rows) k0...
template <int LD>
__device__ __forceinline__ void frag_a_t(const __nv_bfloat16 (*S)[LD], int k0, int m0, int lane, uint32_t (&a)[4]) {
    const int t = lane >> 3;   // 8x8 tile: m half t & 1, k half t >> 1
    const __nv_bfloat16* p = &S[k0 + (t >> 1) * 8 + (lane & 7)][m0 + (t & 1) * 8];
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p)));
}

// B fragments (16 x 8) of two neighbouring column tiles of S[k][n]: columns n0.. and n0 + 8...
template <int LD>
__device__ __forceinline__ void frag_b2(const __nv_bfloat16 (*S)[LD], int k0, int n0, int lane, uint32_t (&b)[4]) {
    const int t = lane >> 3;   // k half t & 1, column tile t >> 1
    const __nv_bfloat16* p = &S[k0 + (t & 1) * 8 + (lane & 7)][n0 + (t >> 1) * 8];
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p)));
}

__device__ __forceinline__ float quad_sum(float v) {   // sum over the 8 lanes sharing tig
    for (int o = 4; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Forward + backward of a mini-batch; gradients of the mean of 0.5*(y-t)^2
// over `n` rows (rows idx[r], or r when idx is null) accumulate (FP32
// atomics) into G (kMlpParams floats).
//
// A block takes 128 rows at a time.  Each warp runs 16 of them forward and back
// and leaves the operands of the weight gradients in shared memory; the warps
// then split dW2 (64 x 64) and dW1 (32 x 64) between them, 128 rows deep, and
// keep their parts, and the bias and W3 sums of their rows, in registers over
// all of the block's rows: one round of atomics per block at the end.  (Summing
// each 16-row product into shared memory, 6,144 FP32 atomics a warp and tile,
// took 387 us for 205,545 rows; this takes 55 us.)  A call on host arrays is then bound by
// their copy over the link: 20 MB of rows, 115 us of its 238.
__global__ void __launch_bounds__(256, 1) k_mlp_grad(const float* __restrict__ P, const float* __restrict__ X,
                                                     const float* __restrict__ T, const uint32_t* __restrict__ idx,
                                                     uint64_t n, float inv_n, float* __restrict__ G,
                                                     float* __restrict__ loss) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    GradSmem& S = *reinterpret_cast<GradSmem*>(smem_raw);
    const SmemW& s = S.w;
    load_weights(S.w, P);
    for (int i = threadIdx.x; i < H; i += blockDim.x) S.col[0][i] = S.col[1][i] = S.col[2][i] = 0.f;
    if (threadIdx.x == 0) S.gb3 = S.lsum = 0.f;
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, gid = lane >> 2, tig = lane & 3;
    // this warp's parts: dW2 rows (in) 16 (w / 2).., columns 32 (w % 2)..; dW1 rows 16 (w % 2).., columns 16 (w / 2)..
    const int m2 = (w >> 1) * 16, n2 = (w & 1) * 32, m1 = (w & 1) * 16, n1 = (w >> 1) * 16;
    float gw2[4][4], gw1[2][4], gb1[16], gb2[16], gw3[16], gb3 = 0.f, lsum = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        gw2[i >> 2][i & 3] = gb1[i] = gb2[i] = gw3[i] = 0.f;
        if (i < 8) gw1[i >> 2][i & 3] = 0.f;
    }
    for (uint64_t tile0 = (uint64_t)blockIdx.x * kRowsPerBlock; tile0 < n; tile0 += (uint64_t)gridDim.x * kRowsPerBlock) {
        const uint64_t row0 = tile0 + (uint64_t)w * kRowsPerWarp;
        const int r_lo = w * kRowsPerWarp + gid, r_hi = r_lo + 8;
        float z1[8][4], z2[8][4], ylo, yhi;
        uint32_t xa[2][4];
        forward16(s, X, idx, row0, n, gid, tig, z1, z2, ylo, yhi, xa);   // rows past n read as zeros
        const bool vlo = row0 + gid < n, vhi = row0 + gid + 8 < n;
        const float tlo = vlo ? T[idx ? idx[row0 + gid] : row0 + gid] : 0.f;
        const float thi = vhi ? T[idx ? idx[row0 + gid + 8] : row0 + gid + 8] : 0.f;
        const float dlo = vlo ? (ylo - tlo) * inv_n : 0.f;
        const float dhi = vhi ? (yhi - thi) * inv_n : 0.f;
        if (tig == 0) {   // one lane per row pair
            lsum += ((vlo ? 0.5f * (ylo - tlo) * (ylo - tlo) : 0.f) + (vhi ? 0.5f * (yhi - thi) * (yhi - thi) : 0.f)) * inv_n;
            gb3 += dlo + dhi;
        }
        __syncthreads();   // the last tile's operands have been read
        // layer 3: dW3 = H2b^T dy; dZ2 = dy * w3 * (z2 > 0), summed for db2 and left in BF16
        uint32_t da[4][4], on1 = 0;   // dZ2b as the A operand; bit 4 nt + i: z1[nt][i] > 0
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            float lo[2], hi[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int col = nt * 8 + tig * 2 + e;
                gw3[nt * 2 + e] += bf16r(fmaxf(z2[nt][e], 0.f)) * dlo + bf16r(fmaxf(z2[nt][2 + e], 0.f)) * dhi;
                lo[e] = z2[nt][e] > 0.f ? dlo * s.w3[col] : 0.f;
                hi[e] = z2[nt][2 + e] > 0.f ? dhi * s.w3[col] : 0.f;
                gb2[nt * 2 + e] += lo[e] + hi[e];
                on1 |= (z1[nt][e] > 0.f ? 1u : 0u) << (nt * 4 + e) | (z1[nt][2 + e] > 0.f ? 1u : 0u) << (nt * 4 + 2 + e);
            }
            const int c = nt * 8 + tig * 2;
            const uint32_t plo = pack_bf16(lo[0], lo[1]), phi = pack_bf16(hi[0], hi[1]);
            da[nt >> 1][(nt & 1) * 2] = plo;
            da[nt >> 1][(nt & 1) * 2 + 1] = phi;
            *reinterpret_cast<uint32_t*>(&S.dz2[r_lo][c]) = plo;
            *reinterpret_cast<uint32_t*>(&S.dz2[r_hi][c]) = phi;
            *reinterpret_cast<uint32_t*>(&S.h1[r_lo][c]) = pack_bf16(fmaxf(z1[nt][0], 0.f), fmaxf(z1[nt][1], 0.f));
            *reinterpret_cast<uint32_t*>(&S.h1[r_hi][c]) = pack_bf16(fmaxf(z1[nt][2], 0.f), fmaxf(z1[nt][3], 0.f));
        }
#pragma unroll
        for (int kt = 0; kt < 2; ++kt) {
            *reinterpret_cast<uint32_t*>(&S.x[r_lo][kt * 16 + tig * 2]) = xa[kt][0];
            *reinterpret_cast<uint32_t*>(&S.x[r_hi][kt * 16 + tig * 2]) = xa[kt][1];
            *reinterpret_cast<uint32_t*>(&S.x[r_lo][kt * 16 + 8 + tig * 2]) = xa[kt][2];
            *reinterpret_cast<uint32_t*>(&S.x[r_hi][kt * 16 + 8 + tig * 2]) = xa[kt][3];
        }
        // dH1 = dZ2b . W2^T; dZ1 = dH1 * (z1 > 0), summed for db1 and left in BF16
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int kt = 0; kt < 4; ++kt) {
                uint32_t b0, b1;
                bfrag(s.w2, nt, kt, gid, tig, b0, b1);
                mma16816(acc, da[kt], b0, b1);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i] = on1 >> (nt * 4 + i) & 1u ? acc[i] : 0.f;
            gb1[nt * 2] += acc[0] + acc[2];
            gb1[nt * 2 + 1] += acc[1] + acc[3];
            const int c = nt * 8 + tig * 2;
            *reinterpret_cast<uint32_t*>(&S.dz1[r_lo][c]) = pack_bf16(acc[0], acc[1]);
            *reinterpret_cast<uint32_t*>(&S.dz1[r_hi][c]) = pack_bf16(acc[2], acc[3]);
        }
        __syncthreads();
        // dW2[in][out] += sum_r H1b[r][in] dZ2b[r][out]; dW1[in][out] += sum_r Xb[r][in] dZ1b[r][out]
#pragma unroll
        for (int k0 = 0; k0 < kRowsPerBlock; k0 += 16) {
            uint32_t a[4], b[4];
            frag_a_t(S.h1, k0, m2, lane, a);
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                frag_b2(S.dz2, k0, n2 + t * 16, lane, b);
                mma16816(gw2[t * 2], a, b[0], b[1]);
                mma16816(gw2[t * 2 + 1], a, b[2], b[3]);
            }
            frag_a_t(S.x, k0, m1, lane, a);
            frag_b2(S.dz1, k0, n1, lane, b);
            mma16816(gw1[0], a, b[0], b[1]);
            mma16816(gw1[1], a, b[2], b[3]);
        }
    }
    // the block's sums, one atomic per parameter
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i)
            atomicAdd(&G[OFF_W2 + (m2 + gid + (i >> 1) * 8) * H + n2 + t * 8 + tig * 2 + (i & 1)], gw2[t][i]);
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int in = m1 + gid + (i >> 1) * 8;
            if (in < IN) atomicAdd(&G[OFF_W1 + in * H + n1 + t * 8 + tig * 2 + (i & 1)], gw1[t][i]);   // rows >= 24 stay 0
        }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int col = (i >> 1) * 8 + tig * 2 + (i & 1);
        const float v1 = quad_sum(gb1[i]), v2 = quad_sum(gb2[i]), v3 = quad_sum(gw3[i]);
        if (gid == 0) {
            atomicAdd(&S.col[0][col], v1);
            atomicAdd(&S.col[1][col], v2);
            atomicAdd(&S.col[2][col], v3);
        }
    }
    for (int o = 1; o < 32; o <<= 1) {
        lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
        gb3 += __shfl_xor_sync(0xffffffffu, gb3, o);
    }
    if (lane == 0) {
        atomicAdd(&S.lsum, lsum);
        atomicAdd(&S.gb3, gb3);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        atomicAdd(&G[OFF_B1 + i], S.col[0][i]);
        atomicAdd(&G[OFF_B2 + i], S.col[1][i]);
        atomicAdd(&G[OFF_W3 + i], S.col[2][i]);
    }
    if (threadIdx.x == 0) {
        atomicAdd(&G[OFF_B3], S.gb3);
        atomicAdd(loss, S.lsum);
    }
}

__global__ void k_adam(float* __restrict__ P, float* __restrict__ G, float* __restrict__ m1, float* __restrict__ m2,
                       int n, float lr, float b1, float b2, float eps, float c1, float c2) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float g = G[i];
    G[i] = 0.f;
    float a = m1[i] = b1 * m1[i] + (1.f - b1) * g;
    float v = m2[i] = b2 * m2[i] + (1.f - b2) * g * g;
    P[i] -= lr * (a / c1) / (sqrtf(v / c2) + eps);
}

__global__ void k_zero_pad_rows(float* P) {
    int i = threadIdx.x;
    for (int r = IN; r < INP; ++r)
        if (i < H) P[OFF_W1 + r * H + i] = 0.f;
}

// Cost-model features of level-k candidates (the layout colo_result_features
// documents), from the filter's bounds and quad statistics on the device.
__global__ void k_features(uint64_t ncand, uint32_t k, const uint32_t* __restrict__ cand,
                           const uint32_t* __restrict__ ub, const unsigned long long* __restrict__ fstats,
                           const uint32_t* __restrict__ fcount, const uint64_t* __restrict__ prow,
                           float* __restrict__ X) {
    const uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncand) return;
    const uint32_t* mem = cand + c * k;
    const uint32_t m = k < 8 ? k : 8;
    float x[IN];
    for (int i = 0; i < IN; ++i) x[i] = 0.f;
    x[0] = (float)k / 8.0f;
    float minn = INFINITY, minub = INFINITY;
    for (uint32_t j = 0; j < k; ++j) minn = fminf(minn, (float)fcount[mem[j]]);
    for (uint32_t j = 0; j < m; ++j) {
        const float u = (float)ub[c * k + j];
        x[1 + j] = log1pf((float)fcount[mem[j]]);
        x[9 + j] = log1pf(u);
        minub = fminf(minub, u);
    }
    const float lnl = log1pf((float)fcount[mem[k - 1]]), lpr = log1pf((float)prow[c]);
    x[17] = lpr;
    x[18] = log1pf(fstats ? (float)fstats[c * 2 + 1] : 0.f);
    x[19] = log1pf(fstats ? (float)fstats[c * 2] : 0.f);
    x[20] = log1pf(minn);
    x[21] = log1pf(minub);
    x[22] = lpr - lnl;
    x[23] = k <= 8 ? log1pf((float)ub[c * k + k - 1]) - lnl : 0.f;
    for (int i = 0; i < IN; ++i) X[c * IN + i] = x[i];
}

}  // namespace

void mlp_features(uint64_t ncand, uint32_t k, const uint32_t* d_cand, const uint32_t* d_ub,
                  const unsigned long long* d_fstats, const uint32_t* d_fcount, const uint64_t* d_prow, float* d_x,
                  cudaStream_t s) {
    if (ncand == 0) return;
    KScope ks("mlp_features");
    k_features<<<(unsigned)((ncand + 127) / 128), 128, 0, s>>>(ncand, k, d_cand, d_ub, d_fstats, d_fcount, d_prow,
                                                               d_x);
    COLO_LAUNCH_CHECK();
    count_launch();
}

void mlp_forward(const float* d_params, const float* d_x, uint64_t n, float* d_y, cudaStream_t s) {
    if (n == 0) return;
    uint64_t blocks = (n + kRowsPerBlock - 1) / kRowsPerBlock;
    if (blocks > 4096) blocks = 4096;
    KScope ks("mlp_forward");
    k_mlp_forward<<<(unsigned)blocks, 256, 0, s>>>(d_params, d_x, n, d_y);
    COLO_LAUNCH_CHECK();
    count_launch();
}

void mlp_grad(const float* d_params, const float* d_x, const float* d_t, const uint32_t* d_idx, uint64_t n,
              float* d_grad, float* d_loss, cudaStream_t s) {
    if (n == 0) return;
    static thread_local int attr_dev = -1;
    int dev = 0;
    COLO_CUDA(cudaGetDevice(&dev));
    if (attr_dev != dev) {
        COLO_CUDA(cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GradSmem)));
        attr_dev = dev;
    }
    uint64_t blocks = (n + kRowsPerBlock - 1) / kRowsPerBlock;
    int sms = 0;
    COLO_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (blocks > (uint64_t)sms) blocks = (uint64_t)sms;   // one resident block an SM (255 registers)
    KScope ks("mlp_grad");
    k_mlp_grad<<<(unsigned)blocks, 256, sizeof(GradSmem), s>>>(d_params, d_x, d_t, d_idx, n, 1.0f / (float)n, d_grad,
                                                                d_loss);
    COLO_LAUNCH_CHECK();
    count_launch();
}

void mlp_adam(float* d_params, float* d_grad, float* d_m1, float* d_m2, int step, float lr, cudaStream_t s) {
    const float b1 = 0.9f, b2 = 0.999f;
    float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    KScope ks("mlp_adam");
    k_adam<<<(kMlpParams + 255) / 256, 256, 0, s>>>(d_params, d_grad, d_m1, d_m2, kMlpParams, lr, b1, b2, 1e-8f, c1, c2);
    COLO_LAUNCH_CHECK();
    k_zero_pad_rows<<<1, 64, 0, s>>>(d_params);
    COLO_LAUNCH_CHECK();
    count_launch(2);
}

}  // namespace colo
