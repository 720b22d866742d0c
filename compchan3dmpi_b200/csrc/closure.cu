// closure.cu -- tensor-core (tcgen05) kernels of the learned subgrid closure.
//
// This translation unit holds the BF16 tensor-core GEMM path the closure's
// MLP runs on, and a self-test entry point that checks it against a host
// product through the C ABI.
#include "chanrhs.h"
#include "chan_internal.h"
#include "host_copy.h"
#include "phase_bits.h"
#include "umma.cuh"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

namespace {

// mbarrier polls before a kernel gives up waiting for its own MMAs, records
// an error and frees its tensor memory (a few seconds at most)
constexpr uint32_t kWaitLimit = 1u << 24;

std::string g_cl_error;

// D[128][N] = A[128][K] * B[N][K]^T on the tensor cores; one CTA of 128 threads
__global__ void __launch_bounds__(128, 1)
    k_umma_selftest(const __nv_bfloat16 *A, const __nv_bfloat16 *B, float *D, int K, int N, int *err)
{
    extern __shared__ __align__(128) unsigned char sm[];
    unsigned char *sA = sm;                       // 128 x K
    unsigned char *sB = sm + 128 * K * 2;         // N x K
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tbase;
    const int tid = threadIdx.x, warp = tid >> 5;
    for (int e = tid; e < 128 * K; e += 128)
        *(__nv_bfloat16 *)(sA + umma::kmaj_off(e / K, e % K, K)) = A[e];
    for (int e = tid; e < N * K; e += 128)
        *(__nv_bfloat16 *)(sB + umma::kmaj_off(e / K, e % K, K)) = B[e];
    if (warp == 0) umma::tmem_alloc(&tbase, 256);
    if (tid == 0) umma::mbar_init(&mbar, 1);
    umma::fence_async_smem();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tb = tbase;
    if (tid == 0) {
        umma::gemm_kmajor(tb, sA, sB, K, N, false);
        umma::commit(&mbar);
    }
    const bool ok = umma::mbar_wait(&mbar, 0, kWaitLimit);
    if (!ok) {
        // give the MMA one more bounded wait before its tensor memory is freed
        if (tid == 0) {
            atomicExch(err, 1);
            umma::mbar_wait(&mbar, 0, kWaitLimit);
        }
    } else {
        umma::fence_after_sync();
        for (int c = 0; c < N; c += 16) {
            float v[16];
            umma::tmem_ld16(umma::lane_addr(tb, warp, c), v);
#pragma unroll
            for (int i = 0; i < 16; i++) D[(size_t)tid * N + c + i] = v[i];
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_free(tb, 256);
}

// ---------------------------------------------------------------------------
// The closure MLP: 13 inputs (padded to 16) -> 64 -> 64 -> 9 outputs (padded
// to 16), GELU activations, BF16 weights and activations on the tensor cores,
// F32 accumulation in tensor memory, F32 biases, F32 master weights.
constexpr int kIn = 13, kInP = 16, kHid = 64, kOut = 9, kOutP = 16, kTile = 128;

// BF16 weight images in the shared-memory layout (K-major core matrices):
// W1 [64][16], W2 [64][64], W3 [16][64] (rows 9..15 zero), and the
// transposes used by the backward pass W2t [64][64], W3t [64][16].
struct WImages {
    static constexpr int w1 = 0, w2 = w1 + kHid * kInP * 2, w3 = w2 + kHid * kHid * 2, w2t = w3 + kOutP * kHid * 2,
                         w3t = w2t + kHid * kHid * 2, bytes = w3t + kHid * kOutP * 2;
};

struct MlpParams {
    const unsigned char *wimg;   // WImages::bytes of BF16 images
    const float *b1, *b2, *b3;   // biases (64, 64, 9)
    const float *X;              // inputs (raw): X[row * xr + f * xc]
    const float *T;              // [n][9] targets (raw), training only
    const float *xmu, *xsd;      // input normalisation (13 each)
    const float *ymu, *ysd;      // output normalisation (9 each)
    long long n;                 // samples
    long long perm_a, perm_b;    // sample of batch row r: (perm_a * (row0 + r) + perm_b) mod n
    long long row0, rows;        // batch rows [row0, row0 + rows)
    float *Y;                    // outputs (raw units), inference only: Y[row * yr + o * yc]
    long long xr, xc, yr, yc;    // element strides of X and Y (rows, columns)
    float *part;                 // gradient sums of each CTA, [CTA][kPartStride] (training)
    float *loss;                 // sum of squared normalised errors (training)
    float inv_count;             // 2 / (9 * rows): d loss / d y factor
    float out_limit;             // inference: |normalised output| above this sets *flag
    int *flag;
    int *err;
};

// GELU in its tanh form, 0.5 z (1 + tanh(sqrt(2/pi) (z + 0.044715 z^3))), on
// the hardware tanh approximation (tanh.approx.f32), and its derivative
__device__ __forceinline__ float tanh_hw(float x)
{
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
constexpr float kGeluA = 0.7978845608028654f, kGeluB = 0.044715f;
__device__ __forceinline__ float gelu(float z)
{
    const float t = tanh_hw(kGeluA * (z + kGeluB * z * z * z));
    return 0.5f * z * (1.0f + t);
}
__device__ __forceinline__ float gelu_d(float z)
{
    const float t = tanh_hw(kGeluA * (z + kGeluB * z * z * z));
    return 0.5f * (1.0f + t) + 0.5f * z * (1.0f - t * t) * kGeluA * (1.0f + 3.0f * kGeluB * z * z);
}

__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ void st_bf16(unsigned char *base, uint32_t off, float v)
{
    *(__nv_bfloat16 *)(base + off) = __float2bfloat16_rn(v);
}

// 8 consecutive K elements of one row as one 16-byte store
__device__ __forceinline__ void st_bf16x8(unsigned char *base, uint32_t off, const float *v)
{
    __nv_bfloat162 h[4];
#pragma unroll
    for (int i = 0; i < 4; i++) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    *(uint4 *)(base + off) = *(uint4 *)h;
}

// ---------------------------------------------------------------------------
// Training kernel: forward and backward pass over the batch rows, 128 per tile.
//
// A tile is a chain of five dependent tensor-core steps with an epilogue between
// each two, far too little work to fill the tensor cores: the chain's latency and the
// epilogues' GELUs bound it.  So a CTA (one per SM) runs two tiles at a time, each by
// a group of 256 threads (two per row, 32 columns each), and one more warp issues every
// MMA, the two groups' steps in turn; one group's epilogue covers the other's products.  Groups
// and issuer meet on mbarriers (ready: the group's operands are written; done: the
// step's MMAs are complete), never on a CTA barrier.
//   step 0: dW1 += dZ1^T X of the previous tile; Z1 = X W1^T
//   step 1: Z2 = H1 W2^T        step 2: Y = H2 W3^T
//   step 3: dH2 = dY W3;  dW3^T += H2^T dY
//   step 4: dH1 = dZ2 W2; dW2 += dZ2^T H1
// Tensor memory: Z1, Z2 and dH (Y, dH2, dH1 in turn) per group, the weight-gradient
// sums shared: the one issuing thread's MMAs on them run in order.  The weight
// gradients read the tiles MN-major, so there are no transposed copies; bias
// gradients are reduced across the warp by halving exchanges, 31 shuffles for 32
// columns, into one register per thread and layer.  The sample of a row needs no division: the
// permutation is affine, so a group's next tile is a fixed step further.
// 65,536 rows: 197 us in the earlier form (one tile per CTA, transposed copies, 128-bit
// sample indices, a five-shuffle sum and an atomic per bias column), 45 now.
constexpr int kGroups = 2, kGroupThreads = 2 * kTile, kTrainThreads = kGroups * kGroupThreads + 32;
struct TrainSmem {
    static constexpr int x = 0;                                      // X   [2][128][16], alternating by tile
    static constexpr int h1 = x + 2 * kTile * kInP * 2;              // H1  [128][64]
    static constexpr int h2 = h1 + kTile * kHid * 2;                 // H2  [128][64]
    static constexpr int dz = h2 + kTile * kHid * 2;                 // dZ2, then dZ1 [128][64]
    static constexpr int dy = dz + kTile * kHid * 2;                 // dY  [128][16]
    static constexpr int group = dy + kTile * kOutP * 2;             // bytes of one group's tiles
    static constexpr int w = kGroups * group;                        // weight images
    static constexpr int fl = w + WImages::bytes;                    // floats: b1 b2 b3, norm, db1 db2 db3, loss
    static constexpr int bytes = fl + (64 + 64 + 16 + 44 + 64 + 64 + 16 + 4) * 4;
};
constexpr int cZ1 = 0, cZ2 = 64, cdH = 128, cGroup = 192, cdW2 = kGroups * cGroup, cdW1 = cdW2 + 64, cdW3 = cdW1 + 16;

// One CTA's gradient sums: W1 and W2 by input column, 64 outputs each (the lanes that
// hold a column write it in one go), then W3, b1, b2, b3 as in the parameter vector.
constexpr int kPartW2 = kIn * kHid, kPartW3 = kPartW2 + kHid * kHid, kPartB1 = kPartW3 + kOut * kHid,
              kPartB2 = kPartB1 + kHid, kPartB3 = kPartB2 + kHid, kPartN = kPartB3 + kOut,
              kPartStride = (kPartN + 31) / 32 * 32;

// v[i] of every lane summed over the warp; lane l gets the sum of v[l]
__device__ __forceinline__ float warp_colsum32(float v[32], int lane)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < o; i++) {
            const float keep = up ? v[i + o] : v[i], give = up ? v[i] : v[i + o];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    return v[0];
}

__global__ void __launch_bounds__(kTrainThreads, 1) k_mlp_train(const MlpParams P)
{
    using S = TrainSmem;
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ __align__(8) uint64_t ready[kGroups], done[kGroups];
    __shared__ uint32_t tbase;
    __shared__ int sfail;
    __shared__ CommitBits slog;   // the issuer's commits
    __shared__ float wloss[2][kGroups][4];   // loss sums of a tile's warps, by tile parity and group
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float *fb1 = (float *)(sm + S::fl), *fb2 = fb1 + 64, *fb3 = fb2 + 64, *nrm = fb3 + 16;
    float *db1 = nrm + 44, *db2 = db1 + 64, *db3 = db2 + 64, *sloss = db3 + 16;
    unsigned char *sW = sm + S::w;
    grid_dep_launch();
    if (warp == 0) umma::tmem_alloc(&tbase, 512);
    if (tid == 0) {
        for (int g = 0; g < kGroups; g++) { umma::mbar_init(&ready[g], kGroupThreads); umma::mbar_init(&done[g], 1); }
        sloss[0] = 0.f;
        sfail = 0;
    }
    if (tid < 44) nrm[tid] = P.xmu[tid];   // xmu, xsd, ymu, ysd in one array
    if (tid < 64) { db1[tid] = 0.f; db2[tid] = 0.f; }
    if (tid < 16) db3[tid] = 0.f;
    grid_dep_wait();   // the optimiser step before: weight images and biases
    {
        const uint4 *src = (const uint4 *)P.wimg;
        uint4 *dst = (uint4 *)sW;
        for (int e = tid; e < WImages::bytes / 16; e += kTrainThreads) dst[e] = src[e];
        if (tid < 64) { fb1[tid] = P.b1[tid]; fb2[tid] = P.b2[tid]; }
        if (tid < 16) fb3[tid] = tid < kOut ? P.b3[tid] : 0.f;
    }
    umma::fence_async_smem();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tb = tbase;
    const int ntiles = (int)((P.rows + kTile - 1) / kTile), grid = (int)gridDim.x;
    // tiles of group g: blockIdx.x + grid * (g + kGroups * it)
    auto count = [&](int g) {
        const int t0 = (int)blockIdx.x + grid * g;
        return t0 < ntiles ? (ntiles - t0 + grid * kGroups - 1) / (grid * kGroups) : 0;
    };
    if (warp == kTrainThreads / 32 - 1) {
        // ---- the issuing warp: the groups' steps in turn, group 0 first (it has as many
        // tiles as group 1 or one more); a group's last step 0 only ends its last tile
        if (lane == 0) {
            const int n0 = count(0), n1 = count(1);
            uint32_t ph[kGroups] = {0, 0};
            CommitBits log{};
            bool acc2 = false, acc1 = false, acc3 = false, ok = true;
            // the CTA's tiles and their warps are added in order; the CTAs' sums, and a CTA's
            // bias sums, by float atomics in the order of arrival
            float loss = 0.f;
            for (int it = 0; it <= n0 && ok; it++)
                for (int step = 0; step < 5 && ok; step++)
                    for (int g = 0; g < kGroups && ok; g++) {
                        const int n = g == 0 ? n0 : n1;
                        if (it > n || n == 0 || (it == n && step > 0)) continue;
                        ok = umma::mbar_wait(&ready[g], ph[g], kWaitLimit);
                        if (!ok) break;
                        ph[g] ^= 1u;
                        umma::fence_after_sync();
                        unsigned char *T = sm + g * S::group;
                        unsigned char *X = T + S::x, *H1 = T + S::h1, *H2 = T + S::h2, *dZ = T + S::dz, *dY = T + S::dy;
                        const uint32_t tz = tb + g * cGroup;
                        constexpr int xb = kTile * kInP * 2;
                        if (step == 0) {
                            if (it > 0) {
#pragma unroll
                                for (int q = 0; q < 4; q++) loss += wloss[(it - 1) & 1][g][q];
                                umma::gemm_mnmajor(tb + cdW1, dZ, kHid, X + ((it - 1) & 1) * xb, kInP, kTile, acc1);
                                acc1 = true;
                            }
                            if (it < n) umma::gemm_kmajor(tz + cZ1, X + (it & 1) * xb, sW + WImages::w1, kInP, kHid, false);
                        } else if (step == 1) {
                            umma::gemm_kmajor(tz + cZ2, H1, sW + WImages::w2, kHid, kHid, false);
                        } else if (step == 2) {
                            umma::gemm_kmajor(tz + cdH, H2, sW + WImages::w3, kHid, kOutP, false);
                        } else if (step == 3) {
                            umma::gemm_kmajor(tz + cdH, dY, sW + WImages::w3t, kOutP, kHid, false);
                            umma::gemm_mnmajor(tb + cdW3, H2, kHid, dY, kOutP, kTile, acc3);
                            acc3 = true;
                        } else {
                            umma::gemm_kmajor(tz + cdH, dZ, sW + WImages::w2t, kHid, kHid, false);
                            umma::gemm_mnmajor(tb + cdW2, dZ, kHid, H1, kHid, kTile, acc2);
                            acc2 = true;
                        }
                        umma::commit(&done[g]);
                        log.committed(g);
                    }
            if (!ok) atomicExch(&sfail, 1);
            slog = log;
            sloss[0] = loss;
        }
    } else {
        // thread: row r of the group's tile, columns 32*half .. 32*half + 31 of each layer
        const int g = warp >> 3, half = (warp >> 2) & 1, wq = warp & 3, r = wq * 32 + lane, c0 = 32 * half;
        unsigned char *T = sm + g * S::group;
        unsigned char *sH1 = T + S::h1, *sH2 = T + S::h2, *sdZ = T + S::dz, *sdY = T + S::dy;
        const uint32_t tz = umma::lane_addr(tb + g * cGroup, wq, 0);
        const int n = count(g);
        uint32_t ph = 0;
        bool ok = true;
        float sb1 = 0.f, sb2 = 0.f, sb3 = 0.f;
        auto signal = [&]() {   // this thread's operands of the next step are written, its reads of TMEM done
            umma::fence_async_smem();
            umma::fence_before_sync();
            umma::mbar_arrive(&ready[g]);
        };
        auto wait = [&]() {   // one verdict per warp, which meets again for the loads from TMEM
            ok = __all_sync(0xffffffffu, ok && umma::mbar_wait(&done[g], ph, kWaitLimit));
            ph ^= 1u;
            umma::fence_after_sync();
        };
        // 32 values of this row as BF16 into columns c0.. of a [128][64] tile
        auto put32 = [&](unsigned char *t, const float *v) {
#pragma unroll
            for (int c = 0; c < 32; c += 8) st_bf16x8(t, umma::kmaj_off(r, c0 + c, kHid), v + c);
        };
        // h = gelu(z + b) of this thread's columns of a layer
        auto forward = [&](int cz, const float *b, unsigned char *t) {
            uint32_t z[32];
            float h[32];
            umma::tmem_ld32(tz + cz + c0, z);
            umma::tmem_wait(z);
#pragma unroll
            for (int i = 0; i < 32; i++) h[i] = gelu(__uint_as_float(z[i]) + b[c0 + i]);
            put32(t, h);
        };
        // d = dH gelu'(z + b) of this thread's columns into dZ
        auto backward = [&](int cz, const float *b, bool live, float d[32]) {
            uint32_t q[32], z[32];
            umma::tmem_ld32(tz + cdH + c0, q);
            umma::tmem_ld32(tz + cz + c0, z);
            umma::tmem_wait(q);
            umma::tmem_wait(z);
#pragma unroll
            for (int i = 0; i < 32; i++)
                d[i] = live ? __uint_as_float(q[i]) * gelu_d(__uint_as_float(z[i]) + b[c0 + i]) : 0.f;
            put32(sdZ, d);
        };
        // sample of this thread's row, and the step to the group's next tile (mod n samples;
        // all factors are below 2^32, the products below 2^64)
        const unsigned long long ns = (unsigned long long)P.n, pa = (unsigned long long)P.perm_a;
        const long long row0 = ((long long)blockIdx.x + (long long)grid * g) * kTile + r;
        unsigned long long smp = (pa * ((unsigned long long)(P.row0 + row0) % ns) + (unsigned long long)P.perm_b) % ns;
        const unsigned long long sstep = (pa * ((unsigned long long)grid * kGroups * kTile % ns)) % ns;
        long long row = row0;
        // raw inputs 8*half .. and (half 0) targets of the coming tile
        float xr[8], tr[kOut];
        auto fetch = [&]() {
#pragma unroll
            for (int f = 0; f < 8; f++) xr[f] = row < P.rows && 8 * half + f < kIn ? P.X[smp * kIn + 8 * half + f] : 0.f;
#pragma unroll
            for (int o = 0; o < kOut; o++) tr[o] = row < P.rows && half == 0 ? P.T[smp * kOut + o] : 0.f;
        };
        if (n > 0) fetch();
        for (int it = 0; it < n; it++) {
            const bool live = row < P.rows;
            float tgt[kOut];
            {
                float xin[8];
#pragma unroll
                for (int f = 0; f < 8; f++) {
                    const int i = 8 * half + f;
                    xin[f] = live && i < kIn ? (xr[f] - nrm[min(i, kIn - 1)]) / nrm[13 + min(i, kIn - 1)] : 0.f;
                }
                st_bf16x8(T + S::x + (it & 1) * (kTile * kInP * 2), umma::kmaj_off(r, 8 * half, kInP), xin);
            }
            signal();
#pragma unroll
            for (int o = 0; o < kOut; o++) tgt[o] = live ? (tr[o] - nrm[26 + o]) / nrm[35 + o] : 0.f;
            row += (long long)grid * kGroups * kTile;
            smp += sstep;
            if (smp >= ns) smp -= ns;
            if (it + 1 < n) fetch();
            wait();
            forward(cZ1, fb1, sH1);
            signal();
            wait();
            forward(cZ2, fb2, sH2);
            signal();
            // ---- loss and dY = 2 (y - t) / (9 rows), by the first half
            wait();
            if (half == 0) {
                float y[16], dy[32], l = 0.f;
                umma::tmem_ld16(tz + cdH, y);
#pragma unroll
                for (int o = 0; o < 32; o++) dy[o] = 0.f;
#pragma unroll
                for (int o = 0; o < kOut; o++) {
                    const float e = live ? (y[o] + fb3[o]) - tgt[o] : 0.f;
                    l += e * e;
                    dy[o] = e * P.inv_count;
                }
                l = warp_sum(l);
                if (lane == 0) wloss[it & 1][g][wq] = l;
                st_bf16x8(sdY, umma::kmaj_off(r, 0, kOutP), dy);
                st_bf16x8(sdY, umma::kmaj_off(r, 8, kOutP), dy + 8);
                signal();
                sb3 += warp_colsum32(dy, lane);
            } else {
                signal();
            }
            float d[32];
            wait();
            backward(cZ2, fb2, live, d);
            signal();
            sb2 += warp_colsum32(d, lane);
            // ---- dZ1 over dZ2; its product joins the next step 0
            wait();
            backward(cZ1, fb1, live, d);
            sb1 += warp_colsum32(d, lane);
            if (!ok) break;
        }
        if (n > 0 && ok) {
            signal();
            wait();
        }
        if (!ok) atomicExch(&sfail, 1);
        // bias gradients and loss of the CTA
        atomicAdd(&db1[c0 + lane], sb1);
        atomicAdd(&db2[c0 + lane], sb2);
        if (half == 0 && lane < kOut) atomicAdd(&db3[lane], sb3);
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    if (!sfail) {
        // weight-gradient sums out of tensor memory (lanes 0..63 hold rows): dW2 row o, 16
        // columns per four warps; dW1 row o; dW3^T row = feature.  Each CTA writes its own
        // sums, which the optimiser adds up: as atomics on one array the CTAs' 835,000
        // took 15 of 53 us
        float *out = P.part + (size_t)blockIdx.x * kPartStride;
        const int part = warp >> 2, wq = warp & 3, o = wq * 32 + lane;
        if (part < 4 && wq < 2) {
            float v[16];
            umma::tmem_ld16(umma::lane_addr(tb, wq, cdW2 + 16 * part), v);
#pragma unroll
            for (int i = 0; i < 16; i++) out[kPartW2 + (16 * part + i) * kHid + o] = v[i];
            if (part < 2) {
                umma::tmem_ld16(umma::lane_addr(tb, wq, part == 0 ? cdW1 : cdW3), v);
                if (part == 0) {
#pragma unroll
                    for (int i = 0; i < kIn; i++) out[i * kHid + o] = v[i];
                } else {
#pragma unroll
                    for (int i = 0; i < kOut; i++) out[kPartW3 + i * kHid + o] = v[i];
                }
            }
        }
        if (tid < 64) { out[kPartB1 + tid] = db1[tid]; out[kPartB2 + tid] = db2[tid]; }
        else if (tid < 64 + kOut) out[kPartB3 + tid - 64] = db3[tid - 64];
        else if (tid == 96) atomicAdd(P.loss, sloss[0]);
    }
    if (sfail && tid == 0) {
        // an MMA did not signal completion: give each group's last commit one more bounded
        // wait before the tensor memory it writes is released
        for (int g = 0; g < kGroups; g++)
            if (slog.some(g)) umma::mbar_wait(&done[g], slog.last(g), kWaitLimit);
        atomicExch(P.err, 1);
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_free(tb, 512);
}

// ---------------------------------------------------------------------------
// Inference: forward only, 128 rows per tile, one CTA of 128 threads per tile in turn.
// Three dependent products and two GELU epilogues per tile; what hides their latency
// is other CTAs, so everything is sized for six per SM: 64 tensor-memory columns (Z1,
// Z2 and Y in turn) and 34 KB of shared memory (H2 over H1).
struct InferSmem {
    static constexpr int wbytes = WImages::w2t;                      // W1, W2, W3 images
    static constexpr int x = wbytes;
    static constexpr int h = x + kTile * kInP * 2;                   // H1, then H2 [128][64]
    static constexpr int fl = h + kTile * kHid * 2;                  // floats: b1 b2 b3, norm
    static constexpr int bytes = fl + (64 + 64 + 16 + 44) * 4;
};
constexpr int kInferCtas = 6;

__global__ void __launch_bounds__(kTile, kInferCtas) k_mlp_infer(const MlpParams P)
{
    using S = InferSmem;
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tbase;
    const int tid = threadIdx.x, warp = tid >> 5;
    float *fb1 = (float *)(sm + S::fl), *fb2 = fb1 + 64, *fb3 = fb2 + 64, *nrm = fb3 + 16;
    grid_dep_enter();
    {   // weight images, biases, normalisation
        const uint4 *src = (const uint4 *)P.wimg;
        uint4 *dst = (uint4 *)sm;
        for (int e = tid; e < S::wbytes / 16; e += kTile) dst[e] = src[e];
        if (tid < 64) { fb1[tid] = P.b1[tid]; fb2[tid] = P.b2[tid]; }
        if (tid < 16) fb3[tid] = tid < kOut ? P.b3[tid] : 0.f;
        if (tid < 44) nrm[tid] = P.xmu[tid];   // xmu, xsd, ymu, ysd in one array
    }
    if (warp == 0) umma::tmem_alloc(&tbase, 64);
    if (tid == 0) umma::mbar_init(&mbar, 1);
    umma::fence_async_smem();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tb = tbase;
    unsigned char *sX = sm + S::x, *sH = sm + S::h;
    uint32_t phase = 0;
    bool ok = true;
    // issue by thread 0 after the smem writes of every thread; then wait
    auto sync_issue_wait = [&](auto &&issue) {
        umma::fence_async_smem();
        umma::fence_before_sync();
        __syncthreads();
        if (tid == 0 && ok) {
            umma::fence_after_sync();
            issue();
            umma::commit(&mbar);
        }
        if (ok) {
            ok = umma::mbar_wait(&mbar, phase, kWaitLimit);
            if (ok) phase ^= 1u;
        }
        ok = __syncthreads_and(ok) != 0;   // one verdict for the whole CTA
        umma::fence_after_sync();
    };
    const long long ntiles = (P.rows + kTile - 1) / kTile;
    auto layer = [&](const float *b) {
#pragma unroll 1
        for (int c = 0; c < kHid; c += 32) {
            uint32_t z[32];
            float h[32];
            umma::tmem_ld32(umma::lane_addr(tb, warp, c), z);
            umma::tmem_wait(z);
#pragma unroll
            for (int i = 0; i < 32; i++) h[i] = gelu(__uint_as_float(z[i]) + b[c + i]);
#pragma unroll
            for (int i = 0; i < 32; i += 8) st_bf16x8(sH, umma::kmaj_off(tid, c + i, kHid), h + i);
        }
    };
    for (long long tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
        const long long row = tile * kTile + tid;
        const bool live = row < P.rows;
        float xin[kInP];
#pragma unroll
        for (int f = 0; f < kInP; f++)
            xin[f] = (live && f < kIn) ? (P.X[row * P.xr + f * P.xc] - nrm[f < kIn ? f : 0]) / nrm[13 + (f < kIn ? f : 0)] : 0.f;
        st_bf16x8(sX, umma::kmaj_off(tid, 0, kInP), xin);
        st_bf16x8(sX, umma::kmaj_off(tid, 8, kInP), xin + 8);
        sync_issue_wait([&] { umma::gemm_kmajor(tb, sX, sm + WImages::w1, kInP, kHid, false); });
        if (!ok) break;
        layer(fb1);
        sync_issue_wait([&] { umma::gemm_kmajor(tb, sH, sm + WImages::w2, kHid, kHid, false); });
        if (!ok) break;
        layer(fb2);
        sync_issue_wait([&] { umma::gemm_kmajor(tb, sH, sm + WImages::w3, kHid, kOutP, false); });
        if (!ok) break;
        float y[16];
        umma::tmem_ld16(umma::lane_addr(tb, warp, 0), y);
        if (live) {
            bool big = false;
#pragma unroll
            for (int o = 0; o < kOut; o++) {
                const float v = y[o] + fb3[o];
                big = big || !(fabsf(v) <= P.out_limit);
                P.Y[row * P.yr + o * P.yc] = v * nrm[35 + o] + nrm[26 + o];
            }
            if (big && P.flag) atomicOr(P.flag, 1);
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (!ok) {
        // an MMA did not signal completion: give it one more bounded wait
        // before the tensor memory it writes is released
        if (tid == 0) {
            umma::mbar_wait(&mbar, phase, kWaitLimit);
            atomicExch(P.err, 1);
        }
        __syncthreads();
    }
    if (warp == 0) umma::tmem_free(tb, 64);
}

// Adam on the F32 master parameters, with the BF16 weight images.
// Parameter vector: W1[64][13] b1[64] W2[64][64] b2[64] W3[9][64] b3[9].
constexpr int kNW1 = kHid * kIn, kNW2 = kHid * kHid, kNW3 = kOut * kHid;
constexpr int kOffB1 = kNW1, kOffW2 = kOffB1 + kHid, kOffB2 = kOffW2 + kNW2, kOffW3 = kOffB2 + kHid,
              kOffB3 = kOffW3 + kNW3, kNParam = kOffB3 + kOut,
              kPStride = (kNParam + 31) / 32 * 32;   // each of w, m, v, g starts on a 128-byte boundary

// BF16 images of parameter i of the F32 master weights (padding stays zero from the memset)
__device__ __forceinline__ void put_images(int i, float x, unsigned char *img)
{
    if (i < kNW1) {
        st_bf16(img + WImages::w1, umma::kmaj_off(i / kIn, i % kIn, kInP), x);
    } else if (i >= kOffW2 && i < kOffW2 + kNW2) {
        const int j = i - kOffW2, o = j / kHid, f = j % kHid;
        st_bf16(img + WImages::w2, umma::kmaj_off(o, f, kHid), x);
        st_bf16(img + WImages::w2t, umma::kmaj_off(f, o, kHid), x);
    } else if (i >= kOffW3 && i < kOffW3 + kNW3) {
        const int j = i - kOffW3, o = j / kHid, f = j % kHid;
        st_bf16(img + WImages::w3, umma::kmaj_off(o, f, kHid), x);
        st_bf16(img + WImages::w3t, umma::kmaj_off(f, o, kOutP), x);
    }
}

// parameter of entry q of a CTA's sums
__host__ __device__ __forceinline__ int part_param(int q)
{
    if (q < kPartW2) return (q % kHid) * kIn + q / kHid;
    if (q < kPartW3) return kOffW2 + ((q - kPartW2) % kHid) * kHid + (q - kPartW2) / kHid;
    if (q < kPartB1) return kOffW3 + (q - kPartW3);
    if (q < kPartB2) return kOffB1 + (q - kPartB1);
    if (q < kPartB3) return kOffB2 + (q - kPartB2);
    return kOffB3 + (q - kPartB3);
}

// gradient of 32 parameters (partial-layout indices 32*blockIdx.x ..) from the CTAs'
// sums: eight warps add a share of the CTAs each, warp 0 adds those.  Returns the
// parameter index of warp 0's lane, or -1.
constexpr int kSumThreads = 256;
__device__ __forceinline__ int sum_parts(const float *part, int nparts, float (&acc)[kSumThreads / 32][32], float &g)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (q < kPartN) {
#pragma unroll 8
        for (int p = warp; p < nparts; p += kSumThreads / 32) s += part[(size_t)p * kPartStride + q];
    }
    acc[warp][lane] = s;
    __syncthreads();
    if (warp != 0 || q >= kPartN) return -1;
    g = 0.f;
#pragma unroll
    for (int w = 0; w < kSumThreads / 32; w++) g += acc[w][lane];
    return part_param(q);
}
constexpr int kSumBlocks = (kPartN + 31) / 32;

// one Adam step of every parameter, with its BF16 images; none after a training kernel
// that gave up (*err), whose sums are not all there
__global__ void __launch_bounds__(kSumThreads) k_adam(float *w, float *m, float *v, const float *part, int nparts,
                                                      unsigned char *img, const int *err, float lr, float b1, float b2,
                                                      float eps, float c1, float c2)
{
    __shared__ float acc[kSumThreads / 32][32];
    grid_dep_enter();   // the training kernel's sums
    float gi;
    const int i = sum_parts(part, nparts, acc, gi);
    if (i < 0) return;
    const int failed = *err;
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    const float x = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    if (failed) return;   // after the loads, beside which its own costs nothing
    m[i] = mi;
    v[i] = vi;
    w[i] = x;
    put_images(i, x, img);
}

// the gradient itself, in the parameter vector's order
__global__ void __launch_bounds__(kSumThreads) k_grad_sum(const float *part, int nparts, float *g)
{
    __shared__ float acc[kSumThreads / 32][32];
    float gi;
    const int i = sum_parts(part, nparts, acc, gi);
    if (i >= 0) g[i] = gi;
}

__global__ void k_weight_images(const float *w, unsigned char *img)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kNParam) put_images(i, w[i], img);
}

// column sums and sums of squares of an [n][NCOL] array (double atomics, one per block
// and sum; one per warp, and a run-time NCOL that put the sums in local memory, took 88 us
// for 127,000 rows of 13)
template <int NCOL>
__global__ void __launch_bounds__(256) k_colstats(const float *A, long long n, double *sum, double *sumsq)
{
    __shared__ double red[8][2 * NCOL];
    double s[NCOL], s2[NCOL];
#pragma unroll
    for (int c = 0; c < NCOL; c++) s[c] = s2[c] = 0.0;
    for (long long r = blockIdx.x * 256LL + threadIdx.x; r < n; r += gridDim.x * 256LL)
#pragma unroll
        for (int c = 0; c < NCOL; c++) {
            const double v = A[r * NCOL + c];
            s[c] += v;
            s2[c] += v * v;
        }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < NCOL; c++) {
        for (int o = 16; o > 0; o >>= 1) {
            s[c] += __shfl_xor_sync(0xffffffffu, s[c], o);
            s2[c] += __shfl_xor_sync(0xffffffffu, s2[c], o);
        }
        if (lane == 0) { red[warp][c] = s[c]; red[warp][NCOL + c] = s2[c]; }
    }
    __syncthreads();
    if (threadIdx.x < 2 * NCOL) {
        double t = 0.0;
        for (int w = 0; w < 8; w++) t += red[w][threadIdx.x];
        atomicAdd(threadIdx.x < NCOL ? &sum[threadIdx.x] : &sumsq[threadIdx.x - NCOL], t);
    }
}

uint64_t splitmix(uint64_t &x)
{
    uint64_t z = (x += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

long long gcd_ll(long long a, long long b)
{
    while (b) { const long long t = a % b; a = b; b = t; }
    return a;
}

}  // namespace

// Dataset, parameters, optimiser state and weight images of one closure.
struct chan_closure {
    int dev = 0;
    cudaStream_t stream = nullptr;
    float *X = nullptr, *T = nullptr;       // [cap][13], [cap][9] samples (one allocation)
    unsigned char *block = nullptr;         // what acc, w, img, norm, loss and err point into
    double *acc = nullptr;                  // column sums [44]
    long long cap = 0, count = 0;
    float *w = nullptr, *m = nullptr, *v = nullptr, *g = nullptr;   // kNParam each
    unsigned char *img = nullptr;           // BF16 weight images
    float *part = nullptr;                  // gradient sums of the training kernel's CTAs, [sms][kPartStride]
    bool part_own = true;                   // its own allocation
    float *norm = nullptr;                  // xmu[13] xsd[13] ymu[9] ysd[9]
    float *loss = nullptr;
    int *err = nullptr;
    long long adam_t = 0;
    float out_limit = 50.f;
    int sms = 148;
    float *ws = nullptr;                    // rows of infer and grad calls (Batch)
    size_t ws_bytes = 0;
    std::mutex ws_mu;
    std::mutex acc_mu;                      // one call at a time uses acc
    std::mutex sum_mu;                      // one call at a time uses part, g, loss and err
    std::shared_ptr<HostCopy> hc;           // staged copies (host_copy.h), from the first large one on
    std::string msg;
};

namespace {

int cfail(chan_closure *m, const char *what, cudaError_t e)
{
    if (m) m->msg = std::string(what) + ": " + cudaGetErrorString(e);
    else g_cl_error = std::string(what) + ": " + cudaGetErrorString(e);
    return CHAN_ECUDA;
}

#define CLK(m, call)                                    \
    do {                                                \
        cudaError_t e_ = (call);                        \
        if (e_ != cudaSuccess) return cfail((m), #call, e_); \
    } while (0)

MlpParams base_params(chan_closure *m)
{
    MlpParams P{};
    P.wimg = m->img;
    P.b1 = m->w + kOffB1; P.b2 = m->w + kOffB2; P.b3 = m->w + kOffB3;
    P.xmu = m->norm; P.xsd = m->norm + 13; P.ymu = m->norm + 26; P.ysd = m->norm + 35;
    P.part = m->part;
    P.loss = m->loss;
    P.err = m->err;
    P.out_limit = m->out_limit;
    P.perm_a = 1; P.perm_b = 0;
    P.xr = kIn; P.xc = 1; P.yr = kOut; P.yc = 1;
    return P;
}

int refresh_images(chan_closure *m)
{
    k_weight_images<<<(kNParam + 255) / 256, 256, 0, m->stream>>>(m->w, m->img);
    CLK(m, cudaGetLastError());
    return CHAN_OK;
}

int launch_infer(chan_closure *m, const MlpParams &P, cudaStream_t st, bool early)
{
    const long long ntiles = (P.rows + kTile - 1) / kTile, slots = (long long)m->sms * kInferCtas;
    const int grid = (int)(ntiles < slots ? ntiles : slots);
    if (grid < 1) return CHAN_OK;
    CLK(m, launch_kernel(early, k_mlp_infer, grid, kTile, InferSmem::bytes, st, P));
    return CHAN_OK;
}

// CTAs of a training launch (one per SM, which is also how many sums m->part holds)
int train_grid(const chan_closure *m, long long rows)
{
    const long long ntiles = (rows + kTile - 1) / kTile;
    return (int)(ntiles < m->sms ? ntiles : m->sms);
}

// the gradient sums' array, unless it came with the samples
cudaError_t ensure_part(chan_closure *m)
{
    return m->part ? cudaSuccess : cudaMalloc((void **)&m->part, (size_t)m->sms * kPartStride * sizeof(float));
}

// a copy to or from the host on the closure's stream, complete on return
cudaError_t host_copy(chan_closure *m, void *dst, const void *src, size_t n, cudaMemcpyKind kind)
{
    const cudaError_t e = HostCopy::copy(m->hc, m->dev, dst, src, n, kind, m->stream);
    return e == cudaSuccess ? cudaStreamSynchronize(m->stream) : e;
}

// device arrays of one call's rows, X [n][13] and Y [n][9]: the closure's workspace, which
// grows to kBatchKeep rows and stays (allocating and freeing both took 1.1 of the 1.6 ms of
// 50,001 rows' inference); for more rows, or while another thread has it, the call's own
// allocation
constexpr long long kBatchKeep = 1 << 20;   // 92 MB
struct Batch {
    float *X = nullptr, *Y = nullptr, *own = nullptr;
    int *err = nullptr;   // the call's own error word, behind Y
    cudaError_t e = cudaSuccess;
    std::unique_lock<std::mutex> lock;
    Batch(chan_closure *m, long long n) : lock(m->ws_mu, std::try_to_lock)
    {
        const size_t xw = ((size_t)n * kIn + 63) / 64 * 64, yw = (size_t)n * kOut, bytes = (xw + yw + 1) * sizeof(float);
        if (n > kBatchKeep || !lock.owns_lock()) {
            e = cudaMalloc((void **)&own, bytes);
            X = own;
        } else {
            if (m->ws_bytes < bytes) {
                if (m->ws) cudaFree(m->ws);
                m->ws = nullptr;
                m->ws_bytes = 0;
                e = cudaMalloc((void **)&m->ws, bytes);
                if (e == cudaSuccess) m->ws_bytes = bytes;
            }
            X = m->ws;
        }
        Y = X ? X + xw : nullptr;
        err = X ? (int *)(Y + yw) : nullptr;
    }
    ~Batch() { if (own) cudaFree(own); }
    Batch(const Batch &) = delete;
    Batch &operator=(const Batch &) = delete;
};

int check_err(chan_closure *m, const int *err)
{
    int h = 0;
    CLK(m, cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, m->stream));
    CLK(m, cudaStreamSynchronize(m->stream));
    if (h) { m->msg = "tensor-core wait gave up"; return CHAN_ECUDA; }
    return CHAN_OK;
}

}  // namespace

int chan_internal_infer(chan_closure *m, const float *X, float *Y, long long n, bool soa, cudaStream_t stream,
                        int *flag, bool early, int *err)
{
    MlpParams P = base_params(m);
    P.X = X; P.Y = Y; P.n = n; P.rows = n; P.row0 = 0; P.flag = flag;
    if (err) P.err = err;
    if (soa) { P.xr = 1; P.xc = n; P.yr = 1; P.yc = n; }
    return launch_infer(m, P, stream, early);
}

int chan_internal_closure_device(chan_closure *m) { return m ? m->dev : -1; }

extern "C" {

int chan_selftest_umma(const uint16_t *A, const uint16_t *B, float *D, int32_t K, int32_t N, int32_t device)
{
    if (!A || !B || !D || K < 16 || K > 256 || K % 16 || N < 16 || N > 256 || N % 16) return CHAN_EINVAL;
    cudaError_t e = cudaSetDevice(device);
    __nv_bfloat16 *dA = nullptr, *dB = nullptr;
    float *dD = nullptr;
    int *derr = nullptr, herr = 0;
    const size_t smem = (size_t)(128 + N) * K * 2;
    if (e == cudaSuccess) e = cudaMalloc((void **)&dA, (size_t)128 * K * 2);
    if (e == cudaSuccess) e = cudaMalloc((void **)&dB, (size_t)N * K * 2);
    if (e == cudaSuccess) e = cudaMalloc((void **)&dD, (size_t)128 * N * 4);
    if (e == cudaSuccess) e = cudaMalloc((void **)&derr, sizeof(int));
    if (e == cudaSuccess) e = cudaMemcpy(dA, A, (size_t)128 * K * 2, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(dB, B, (size_t)N * K * 2, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(derr, 0, sizeof(int));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_umma_selftest, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) {
        k_umma_selftest<<<1, 128, smem>>>(dA, dB, dD, K, N, derr);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(D, dD, (size_t)128 * N * 4, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(&herr, derr, sizeof(int), cudaMemcpyDeviceToHost);
    if (dA) cudaFree(dA);
    if (dB) cudaFree(dB);
    if (dD) cudaFree(dD);
    if (derr) cudaFree(derr);
    if (e != cudaSuccess) {
        g_cl_error = cudaGetErrorString(e);
        return CHAN_ECUDA;
    }
    return herr ? CHAN_ECUDA : CHAN_OK;
}

int chan_closure_create(int32_t device, int64_t capacity, chan_closure **out)
{
    if (!out || capacity < 0) return CHAN_EINVAL;
    *out = nullptr;
    chan_closure *m = new chan_closure;
    m->dev = device;
    m->cap = capacity;
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking);
    // two allocations: the samples, X then T, and everything small.  A cudaMalloc of 2 MB and
    // more takes 0.3 to 1 ms, a smaller one shares a mapped block: the training kernel's sums
    // (3.3 MB) come with samples that are as large anyway, else from the first training call
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, device);
    const size_t xw = ((size_t)capacity * kIn + 63) / 64 * 64, tw = ((size_t)capacity * kOut + 63) / 64 * 64;
    const bool big = (xw + tw) * sizeof(float) >= (2u << 20);
    if (e == cudaSuccess && capacity > 0)
        e = cudaMalloc((void **)&m->X, (xw + tw + (big ? (size_t)m->sms * kPartStride : 0)) * sizeof(float));
    if (e == cudaSuccess && capacity > 0) {
        m->T = m->X + xw;
        m->part = big ? m->T + tw : nullptr;
        m->part_own = !big;
    }
    constexpr size_t accOff = 0, wOff = 44 * sizeof(double) + 32, imgOff = wOff + 4 * (size_t)kPStride * sizeof(float),
                     normOff = imgOff + WImages::bytes, lossOff = normOff + 48 * sizeof(float), errOff = lossOff + 16,
                     small = errOff + 16;
    static_assert(wOff % 128 == 0 && imgOff % 128 == 0 && normOff % 16 == 0, "alignment of a closure's arrays");
    if (e == cudaSuccess) e = cudaMalloc((void **)&m->block, small);
    if (e == cudaSuccess) e = cudaMemset(m->block, 0, small);
    if (e == cudaSuccess) {
        m->acc = (double *)(m->block + accOff);
        m->w = (float *)(m->block + wOff);
        m->img = m->block + imgOff;
        m->norm = (float *)(m->block + normOff);
        m->loss = (float *)(m->block + lossOff);
        m->err = (int *)(m->block + errOff);
    }
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, TrainSmem::bytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_mlp_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, InferSmem::bytes);
    if (e != cudaSuccess) {
        g_cl_error = std::string("chan_closure_create: ") + cudaGetErrorString(e);
        chan_closure_free(m);
        return CHAN_ECUDA;
    }
    m->m = m->w + kPStride;
    m->v = m->m + kPStride;
    m->g = m->v + kPStride;
    // identity normalisation until one is fitted or set
    float nrm[44];
    for (int i = 0; i < 44; i++) nrm[i] = (i >= 13 && i < 26) || i >= 35 ? 1.f : 0.f;
    cudaMemcpy(m->norm, nrm, sizeof(nrm), cudaMemcpyHostToDevice);
    *out = m;
    return CHAN_OK;
}

int chan_selftest_adam(float *w, float *mom1, float *mom2, const float *grad, float lr, int32_t failed, int32_t device)
{
    if (!w || !mom1 || !mom2 || !grad || !(lr > 0)) return CHAN_EINVAL;
    chan_closure *m = nullptr;
    int r = chan_closure_create(device, 0, &m);
    if (r) return r;
    std::vector<float> part(kPartStride, 0.f);
    for (int q = 0; q < kPartN; q++) part[q] = grad[part_param(q)];
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const int err = failed ? 1 : 0;
    constexpr size_t np = (size_t)kNParam * sizeof(float);
    cudaError_t e = ensure_part(m);
    if (e == cudaSuccess) e = cudaMemcpy(m->part, part.data(), kPartStride * sizeof(float), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(m->err, &err, sizeof(int), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(m->w, w, np, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(m->m, mom1, np, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(m->v, mom2, np, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaStreamSynchronize(cudaStreamLegacy);
    if (e == cudaSuccess)
        e = launch_kernel(false, k_adam, kSumBlocks, kSumThreads, 0, m->stream, m->w, m->m, m->v, m->part, 1, m->img,
                          m->err, lr, b1, b2, eps, 1.f - b1, 1.f - b2);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
    if (e == cudaSuccess) e = cudaMemcpy(w, m->w, np, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(mom1, m->m, np, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(mom2, m->v, np, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) g_cl_error = cudaGetErrorString(e);
    chan_closure_free(m);
    return e == cudaSuccess ? CHAN_OK : CHAN_ECUDA;
}

int chan_closure_sample(chan_closure *m, chan_ctx *dns, int32_t sx, int32_t sy, int32_t sz, int32_t fw,
                        int64_t *added)
{
    if (!m || !dns) return CHAN_EINVAL;
    long long a = 0;
    int r = chan_internal_sample(dns, m->X + m->count * kIn, m->T + m->count * kOut, m->cap - m->count, sx, sy, sz,
                                 fw, &a);
    if (r) { m->msg = "sampling failed (see chan_last_error of the context)"; return r; }
    m->count += a;
    if (added) *added = a;
    return CHAN_OK;
}

int chan_closure_add_data(chan_closure *m, const float *X, const float *T, int64_t n)
{
    if (!m || !X || !T || n < 0 || m->count + n > m->cap) return CHAN_EINVAL;
    CLK(m, cudaSetDevice(m->dev));
    CLK(m, host_copy(m, m->X + m->count * kIn, X, (size_t)n * kIn * sizeof(float), cudaMemcpyHostToDevice));
    CLK(m, host_copy(m, m->T + m->count * kOut, T, (size_t)n * kOut * sizeof(float), cudaMemcpyHostToDevice));
    m->count += n;
    return CHAN_OK;
}

int chan_closure_count(chan_closure *m, int64_t *count)
{
    if (!m || !count) return CHAN_EINVAL;
    *count = m->count;
    return CHAN_OK;
}

int chan_closure_get_data(chan_closure *m, int64_t first, int64_t n, float *X, float *T)
{
    if (!m || first < 0 || n < 0 || first + n > m->count) return CHAN_EINVAL;
    CLK(m, cudaSetDevice(m->dev));
    if (X) CLK(m, host_copy(m, X, m->X + first * kIn, (size_t)n * kIn * sizeof(float), cudaMemcpyDeviceToHost));
    if (T) CLK(m, host_copy(m, T, m->T + first * kOut, (size_t)n * kOut * sizeof(float), cudaMemcpyDeviceToHost));
    return CHAN_OK;
}

int chan_closure_fit_normalization(chan_closure *m, float *norm_out)
{
    if (!m || m->count < 2) return CHAN_EINVAL;
    CLK(m, cudaSetDevice(m->dev));
    std::lock_guard<std::mutex> lock(m->acc_mu);
    double *acc = m->acc;
    CLK(m, cudaMemsetAsync(acc, 0, 44 * sizeof(double), m->stream));
    k_colstats<kIn><<<2 * m->sms, 256, 0, m->stream>>>(m->X, m->count, acc, acc + 13);
    k_colstats<kOut><<<2 * m->sms, 256, 0, m->stream>>>(m->T, m->count, acc + 26, acc + 35);
    double h[44];
    cudaError_t e = cudaMemcpyAsync(h, acc, sizeof(h), cudaMemcpyDeviceToHost, m->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
    if (e != cudaSuccess) return cfail(m, "normalization", e);
    float nrm[44];
    const double n = (double)m->count;
    for (int c = 0; c < 13; c++) {
        const double mu = h[c] / n, var = h[13 + c] / n - mu * mu;
        nrm[c] = (float)mu;
        nrm[13 + c] = var > 1e-24 ? (float)std::sqrt(var) : 1.f;
    }
    for (int c = 0; c < 9; c++) {
        const double mu = h[26 + c] / n, var = h[35 + c] / n - mu * mu;
        nrm[26 + c] = (float)mu;
        nrm[35 + c] = var > 1e-24 ? (float)std::sqrt(var) : 1.f;
    }
    CLK(m, cudaMemcpy(m->norm, nrm, sizeof(nrm), cudaMemcpyHostToDevice));
    if (norm_out) std::memcpy(norm_out, nrm, sizeof(nrm));
    return CHAN_OK;
}

int chan_closure_set_normalization(chan_closure *m, const float *norm)
{
    if (!m || !norm) return CHAN_EINVAL;
    CLK(m, cudaSetDevice(m->dev));
    CLK(m, cudaMemcpy(m->norm, norm, 44 * sizeof(float), cudaMemcpyHostToDevice));
    return CHAN_OK;
}

int chan_closure_get_normalization(chan_closure *m, float *norm)
{
    if (!m || !norm) return CHAN_EINVAL;
    CLK(m, cudaSetDevice(m->dev));
    CLK(m, cudaMemcpy(norm, m->norm, 44 * sizeof(float), cudaMemcpyDeviceToHost));
    return CHAN_OK;
}

int chan_closure_nparams(void) { return kNParam; }

int chan_closure_init(chan_closure *m, uint64_t seed)
{
    if (!m) return CHAN_EINVAL;
    std::vector<float> w(kNParam, 0.f);
    uint64_t st = seed;
    auto uni = [&](double lim) { return (float)(((splitmix(st) >> 11) * (1.0 / 9007199254740992.0) * 2.0 - 1.0) * lim); };
    const double l1 = std::sqrt(6.0 / (kIn + kHid)), l2 = std::sqrt(6.0 / (kHid + kHid)), l3 = std::sqrt(6.0 / (kHid + kOut));
    for (int i = 0; i < kNW1; i++) w[i] = uni(l1);
    for (int i = 0; i < kNW2; i++) w[kOffW2 + i] = uni(l2);
    for (int i = 0; i < kNW3; i++) w[kOffW3 + i] = uni(l3);
    return chan_closure_set_params(m, w.data());
}

int chan_closure_set_params(chan_closure *m, const float *params)
{
    if (!m || !params) return CHAN_EINVAL;
    CLK(m, cudaSetDevice(m->dev));
    CLK(m, cudaMemcpy(m->w, params, (size_t)kNParam * sizeof(float), cudaMemcpyHostToDevice));
    CLK(m, cudaMemset(m->m, 0, 2 * (size_t)kPStride * sizeof(float)));
    m->adam_t = 0;
    int r = refresh_images(m);
    if (r) return r;
    CLK(m, cudaStreamSynchronize(m->stream));
    return CHAN_OK;
}

int chan_closure_get_params(chan_closure *m, float *params)
{
    if (!m || !params) return CHAN_EINVAL;
    CLK(m, cudaSetDevice(m->dev));
    CLK(m, cudaMemcpy(params, m->w, (size_t)kNParam * sizeof(float), cudaMemcpyDeviceToHost));
    return CHAN_OK;
}

int chan_closure_train(chan_closure *m, int32_t epochs, int32_t batch, double lr, uint64_t seed, double *losses)
{
    if (!m || epochs < 0 || batch < kTile || batch % kTile || !(lr > 0)) return CHAN_EINVAL;
    if (m->count < batch) { m->msg = "fewer samples than one batch"; return CHAN_EINVAL; }
    CLK(m, cudaSetDevice(m->dev));
    std::lock_guard<std::mutex> lock(m->sum_mu);
    CLK(m, ensure_part(m));
    CLK(m, cudaMemsetAsync(m->err, 0, sizeof(int), m->stream));
    const long long n = m->count, nb = n / batch;
    uint64_t st = seed;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    for (int ep = 0; ep < epochs; ep++) {
        // this epoch's order of the samples: row -> (a*row + b) mod n, a coprime to n
        long long a = (long long)(splitmix(st) % (uint64_t)n) | 1;
        while (gcd_ll(a, n) != 1) a = (a + 2) % n;
        const long long b = (long long)(splitmix(st) % (uint64_t)n);
        CLK(m, cudaMemsetAsync(m->loss, 0, sizeof(float), m->stream));
        for (long long bi = 0; bi < nb; bi++) {
            MlpParams P = base_params(m);
            P.X = m->X; P.T = m->T; P.n = n;
            P.perm_a = a; P.perm_b = b;
            P.row0 = bi * batch; P.rows = batch;
            P.inv_count = 2.f / (9.f * (float)batch);
            const int grid = train_grid(m, P.rows);
            CLK(m, launch_kernel(true, k_mlp_train, grid, kTrainThreads, TrainSmem::bytes, m->stream, P));
            m->adam_t++;
            const float c1 = 1.f - std::pow(b1, (float)m->adam_t), c2 = 1.f - std::pow(b2, (float)m->adam_t);
            CLK(m, launch_kernel(true, k_adam, kSumBlocks, kSumThreads, 0, m->stream, m->w, m->m, m->v, m->part, grid, m->img,
                                m->err, (float)lr, b1, b2, eps, c1, c2));
        }
        float l = 0.f;
        CLK(m, cudaMemcpyAsync(&l, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream));
        CLK(m, cudaStreamSynchronize(m->stream));
        if (losses) losses[ep] = (double)l / (9.0 * (double)batch * (double)nb);
        int r = check_err(m, m->err);
        if (r) return r;
    }
    return CHAN_OK;
}

int chan_closure_grad(chan_closure *m, const float *X, const float *T, int64_t n, float *grads, double *loss_sum)
{
    if (!m || !X || !T || n < 1) return CHAN_EINVAL;
    CLK(m, cudaSetDevice(m->dev));
    std::lock_guard<std::mutex> lock(m->sum_mu);
    CLK(m, ensure_part(m));
    Batch b(m, n);
    CLK(m, b.e);
    float *dX = b.X, *dT = b.Y;
    CLK(m, host_copy(m, dX, X, (size_t)n * kIn * sizeof(float), cudaMemcpyHostToDevice));
    CLK(m, host_copy(m, dT, T, (size_t)n * kOut * sizeof(float), cudaMemcpyHostToDevice));
    CLK(m, cudaMemsetAsync(m->loss, 0, sizeof(float), m->stream));
    CLK(m, cudaMemsetAsync(m->err, 0, sizeof(int), m->stream));
    MlpParams P = base_params(m);
    P.X = dX; P.T = dT; P.n = n; P.rows = n;
    P.inv_count = 2.f / (9.f * (float)n);
    const int grid = train_grid(m, n);
    k_mlp_train<<<grid, kTrainThreads, TrainSmem::bytes, m->stream>>>(P);
    CLK(m, cudaGetLastError());
    k_grad_sum<<<kSumBlocks, kSumThreads, 0, m->stream>>>(m->part, grid, m->g);
    CLK(m, cudaGetLastError());
    int r = CHAN_OK;
    float l = 0.f;
    if (!r) r = check_err(m, m->err);
    if (!r && grads) CLK(m, cudaMemcpy(grads, m->g, (size_t)kNParam * sizeof(float), cudaMemcpyDeviceToHost));
    if (!r) CLK(m, cudaMemcpy(&l, m->loss, sizeof(float), cudaMemcpyDeviceToHost));
    if (loss_sum) *loss_sum = l;
    return r;
}

int chan_closure_infer(chan_closure *m, const float *X, int64_t n, float *Y)
{
    if (!m || !X || !Y || n < 1) return CHAN_EINVAL;
    CLK(m, cudaSetDevice(m->dev));
    Batch b(m, n);
    CLK(m, b.e);
    float *dX = b.X, *dY = b.Y;
    CLK(m, host_copy(m, dX, X, (size_t)n * kIn * sizeof(float), cudaMemcpyHostToDevice));
    CLK(m, cudaMemsetAsync(b.err, 0, sizeof(int), m->stream));
    int r = chan_internal_infer(m, dX, dY, n, false, m->stream, nullptr, false, b.err);
    if (!r) r = check_err(m, b.err);
    if (!r) CLK(m, host_copy(m, Y, dY, (size_t)n * kOut * sizeof(float), cudaMemcpyDeviceToHost));
    return r;
}

const char *chan_closure_last_error(chan_closure *m) { return m ? m->msg.c_str() : g_cl_error.c_str(); }

void chan_closure_free(chan_closure *m)
{
    if (!m) return;
    cudaSetDevice(m->dev);
    if (m->stream) cudaStreamSynchronize(m->stream);
    if (m->X) cudaFree(m->X);
    if (m->block) cudaFree(m->block);
    if (m->part && m->part_own) cudaFree(m->part);
    if (m->ws) cudaFree(m->ws);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
}

}  // extern "C"
