// Learned initial guess: features, MLP inference and training kernels.
//
// Features (24 per free vertex, computed at the start of a step from the
// state, the adaptive guess, the inertial target and the step's OGC
// detection; `u` = |g| dt^2 is the displacement unit):
//   0-2   (y - x0) / u                      inertial displacement
//   3-5   (guess - x0) / u                  adaptive guess (prediction.rs)
//   6-8   mean over the 1-ring of the neighbours' guess displacement, minus own
//   9-11  (mean 1-ring position - x0) / mean 1-ring edge length
//   12-14 unit area-weighted normal of the incident triangles
//   15    100 * mean Green strain trace (E_ww + E_ff) of incident triangles
//   16    100 * mean |E_wf| shear of incident triangles
//   17    100 * max principal fibre strain max(E_ww, E_ff)
//   18    OGC nearest distance / query radius (radius / relaxation / rq)
//   19    contact terms incident to the vertex / 4 (capped at 16)
//   20-22 last step's correction (x_end - adaptive guess) / u, 0 without history
//   23    1 - ring size / 6
// The network maps them to a correction c; the learned guess is
// guess + u * c, clipped to the vertex's OGC ball.
#include <cuda_fp16.h>

#include <atomic>
#include <cmath>
#include <vector>

#include "learned.cuh"

namespace cc {

// GELU, tanh form (Hendrycks & Gimpel 2016): 0.5 z (1 + tanh(sqrt(2/pi) (z + 0.044715 z^3)))
__device__ __forceinline__ float gelu_f(float z) {
    const float c0 = 0.7978845608028654f, c1 = 0.044715f;
    float t = tanhf(c0 * (z + c1 * z * z * z));
    return 0.5f * z * (1.0f + t);
}
__device__ __forceinline__ void gelu_fg(float z, float& a, float& da) {
    const float c0 = 0.7978845608028654f, c1 = 0.044715f;
    float t = tanhf(c0 * (z + c1 * z * z * z));
    a = 0.5f * z * (1.0f + t);
    da = 0.5f * (1.0f + t) + 0.5f * z * (1.0f - t * t) * c0 * (1.0f + 3.0f * c1 * z * z);
}

// ------------------------------------------------------------- features
__global__ void k_features(FeatureView f, float* out) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < f.n; v += gridDim.x * blockDim.x) {
        if (f.pinned[v]) continue;
        float* o = out + (size_t)f.row[v] * kMlpIn;
        const double iu = 1.0 / f.unit;
        d3 x = ld3(f.x0, v), y = ld3(f.target, v), g = ld3(f.guess, v);
        d3 dy = (y - x) * iu, dg = (g - x) * iu;
        d3 nb_dg = mk(0, 0, 0), nb_x = mk(0, 0, 0);
        double elen = 0.0;
        uint32_t r0 = f.ring_off[v], r1 = f.ring_off[v + 1];
        for (uint32_t k = r0; k < r1; ++k) {
            uint32_t u = f.ring[k];
            d3 xu = ld3(f.x0, u);
            nb_x = nb_x + xu;
            elen += len(xu - x);
            nb_dg = nb_dg + (ld3(f.guess, u) - xu) * iu;
        }
        uint32_t cnt = r1 - r0;
        d3 rel = mk(0, 0, 0), lap = mk(0, 0, 0);
        if (cnt) {
            double ic = 1.0 / (double)cnt;
            rel = nb_dg * ic - dg;
            double el = elen * ic;
            lap = (nb_x * ic - x) * (1.0 / fmax(el, 1e-12));
        }
        d3 nrm = mk(0, 0, 0);
        double tr = 0.0, shs = 0.0, mx = -1e30;
        uint32_t nt = 0;
        for (uint32_t k = f.inc_off[v]; k < f.inc_off[v + 1]; ++k) {
            uint32_t ent = f.inc[k];
            if ((ent >> 30) != TERM_TRI) continue;
            uint32_t t = ent & 0x0fffffffu;
            int4 tv = f.tri_v[t];
            double4 cf = f.tri_coef[t];
            d3 a = ld3(f.x0, (uint32_t)tv.x), b = ld3(f.x0, (uint32_t)tv.y), c = ld3(f.x0, (uint32_t)tv.z);
            d3 ds0 = b - a, ds1 = c - a;
            nrm = nrm + cross(ds0, ds1);
            d3 w = ds0 * cf.x + ds1 * cf.y;
            d3 q = ds0 * cf.z + ds1 * cf.w;
            double ew = 0.5 * (dot(w, w) - 1.0), ef = 0.5 * (dot(q, q) - 1.0);
            tr += ew + ef;
            shs += fabs(dot(w, q));
            mx = fmax(mx, fmax(ew, ef));
            ++nt;
        }
        double nl = len(nrm);
        if (nl > 0.0) nrm = nrm * (1.0 / nl);
        if (nt) {
            tr /= (double)nt;
            shs /= (double)nt;
        } else {
            mx = 0.0;
        }
        double dmin = f.contacts.radii[v] / f.relaxation / f.query_radius;
        uint32_t nc = f.contacts.inc_off[v + 1] - f.contacts.inc_off[v];
        d3 pc = mk(0, 0, 0);
        if (f.history && *f.mismatch == 0) pc = ld3(f.prev_corr, v) * iu;
        double feat[kMlpIn] = {dy.x,
                               dy.y,
                               dy.z,
                               dg.x,
                               dg.y,
                               dg.z,
                               rel.x,
                               rel.y,
                               rel.z,
                               lap.x,
                               lap.y,
                               lap.z,
                               nrm.x,
                               nrm.y,
                               nrm.z,
                               100.0 * tr,
                               100.0 * shs,
                               100.0 * mx,
                               fmin(dmin, 1.0),
                               (double)min(nc, 16u) * 0.25,
                               pc.x,
                               pc.y,
                               pc.z,
                               1.0 - (double)cnt / 6.0};
#pragma unroll
        for (int k = 0; k < kMlpIn; ++k) o[k] = (float)feat[k];
    }
}

void launch_features(const FeatureView& f, float* out, cudaStream_t st) {
    if (f.n == 0) return;
    k_features<<<grid_for(f.n, 128), 128, 0, st>>>(f, out);
}

__global__ void k_learned_warm_start(FeatureView f, const float* corr, double alpha, double4* alt,
                                     unsigned int* clipped) {
    unsigned int cnt = 0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < f.n; v += gridDim.x * blockDim.x) {
        if (f.pinned[v]) {
            alt[v] = f.x0[v];
            continue;
        }
        const float* c = corr + (size_t)f.row[v] * kMlpOut;
        d3 p = ld3(f.guess, v) + mk((double)c[0], (double)c[1], (double)c[2]) * (f.unit * alpha);
        if (!isfin(p)) p = ld3(f.guess, v);  // a non-finite prediction falls back per vertex
        d3 ctr = ld3(f.contacts.centers, v);
        d3 d = p - ctr;
        double l = len(d);
        double b = f.contacts.radii[v];
        if (l > b) {  // ContactSet::truncate (src/ogc/world.rs:91-100)
            p = ctr + d * (b / l);
            ++cnt;
        }
        st3(alt, v, p);
    }
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(clipped, cnt);
}

void launch_learned_warm_start(const FeatureView& f, const float* corr, double alpha, double4* alt,
                               unsigned int* clipped, cudaStream_t st) {
    if (f.n == 0) return;
    k_learned_warm_start<<<grid_for(f.n, 256), 256, 0, st>>>(f, corr, alpha, alt, clipped);
}

__global__ void k_targets(FeatureView f, const double4* x, float* targets) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < f.n; v += gridDim.x * blockDim.x) {
        if (f.pinned[v]) continue;
        d3 c = (ld3(x, v) - ld3(f.guess, v)) * (1.0 / f.unit);
        float* o = targets + (size_t)f.row[v] * kMlpOut;
        o[0] = (float)c.x;
        o[1] = (float)c.y;
        o[2] = (float)c.z;
    }
}

void launch_targets(const FeatureView& f, const double4* x, float* targets, cudaStream_t st) {
    if (f.n == 0) return;
    k_targets<<<grid_for(f.n, 256), 256, 0, st>>>(f, x, targets);
}

// ------------------------------------------------------- FP32 inference
// One sample per thread. Weights and biases in shared memory (read as
// warp-wide broadcasts); each layer's input lives in registers and its output
// goes to a per-thread column of shared memory (conflict-free).
constexpr int kFwdBlock = 128;

template <int IN>
__device__ __forceinline__ void dense_gelu(const float* __restrict__ W, const float* __restrict__ b, const float* in,
                                           float* out_col) {
#pragma unroll 1
    for (int i = 0; i < kMlpHidden; i += 2) {
        float a0 = b[i], a1 = b[i + 1];
#pragma unroll
        for (int j = 0; j < IN; ++j) {
            a0 = fmaf(W[i * IN + j], in[j], a0);
            a1 = fmaf(W[(i + 1) * IN + j], in[j], a1);
        }
        out_col[i * kFwdBlock] = gelu_f(a0);
        out_col[(i + 1) * kFwdBlock] = gelu_f(a1);
    }
}

__global__ void __launch_bounds__(kFwdBlock) k_mlp_forward_f32(const float* __restrict__ P, const float* __restrict__ F,
                                                                 uint64_t n, float* __restrict__ out) {
    extern __shared__ float sm[];
    float* w = sm;                       // kMlpParams
    float* act = sm + kMlpParams + 1;    // [64][kFwdBlock]
    for (int i = threadIdx.x; i < kMlpParams; i += kFwdBlock) w[i] = P[i];
    __syncthreads();
    float* col = act + threadIdx.x;
    for (uint64_t s0 = (uint64_t)blockIdx.x * kFwdBlock; s0 < n; s0 += (uint64_t)gridDim.x * kFwdBlock) {
        uint64_t s = s0 + threadIdx.x;
        bool live = s < n;
        float x[kMlpIn];
#pragma unroll
        for (int j = 0; j < kMlpIn; ++j) x[j] = live ? F[s * kMlpIn + j] : 0.0f;
        dense_gelu<kMlpIn>(w + kOffW1, w + kOffB1, x, col);
        float h[kMlpHidden];
#pragma unroll
        for (int j = 0; j < kMlpHidden; ++j) h[j] = col[j * kFwdBlock];
        dense_gelu<kMlpHidden>(w + kOffW2, w + kOffB2, h, col);
#pragma unroll
        for (int j = 0; j < kMlpHidden; ++j) h[j] = col[j * kFwdBlock];
        dense_gelu<kMlpHidden>(w + kOffW3, w + kOffB3, h, col);
#pragma unroll
        for (int j = 0; j < kMlpHidden; ++j) h[j] = col[j * kFwdBlock];
        if (live) {
#pragma unroll
            for (int k = 0; k < kMlpOut; ++k) {
                float a = w[kOffB4 + k];
#pragma unroll
                for (int j = 0; j < kMlpHidden; ++j) a = fmaf(w[kOffW4 + k * kMlpHidden + j], h[j], a);
                out[s * kMlpOut + k] = a;
            }
        }
    }
}

// ------------------------------------------------------------- training
// One CTA of 256 threads per SM processes tiles of up to 64 samples: forward,
// loss gradient and back-propagation with every operand in shared memory, the
// weight gradients summed over the CTA's tiles in registers and written once
// into the CTA's row of `partial`; k_mlp_reduce sums the rows in a fixed order.
//
// All three products are FP32 FMA (no tensor-core format keeps FP32 operands),
// so the bound is 6 x 9,920 operations a sample: 16,384 samples are 13 us at
// ~75 TFLOP/s. A thread owns a 4 x 4 block of the result and reads two float4
// per 16 FMAs: weights transposed for the forward pass ([in][out]) and as they
// are for the backward one, activations unit-major (a row of kPitch samples), so
// that both sides of every product are contiguous float4. One thread per sample
// and unit range, weights from global memory and one weight gradient per thread
// at two shared-memory reads per FMA, took 315 us for the 16,384; this takes 58
// (clocks and caches as a launch-by-launch profile leaves them).
constexpr int kTile = 64;
constexpr int kPitch = kTile + 4;  // float4 rows; rows r and r + 1 lie 4 banks apart
constexpr int kTrainBlock = 256;
constexpr int kWPitch = kMlpHidden + 4;
// shared memory (floats): weights, then activations
constexpr int kSmW2 = 0;
constexpr int kSmW3 = kSmW2 + kMlpHidden * kMlpHidden;
constexpr int kSmW4 = kSmW3 + kMlpHidden * kMlpHidden;
constexpr int kSmT1 = kSmW4 + kMlpOut * kMlpHidden;
constexpr int kSmT2 = kSmT1 + kMlpIn * kWPitch;
constexpr int kSmT3 = kSmT2 + kMlpHidden * kWPitch;
constexpr int kSmB = kSmT3 + kMlpHidden * kWPitch;  // b1 b2 b3 b4 (+ 1)
constexpr int kSmX = kSmB + 3 * kMlpHidden + 4;
constexpr int kSmA1 = kSmX + kMlpIn * kPitch;  // activations A and GELU derivatives G, later the deltas in G's place
constexpr int kSmLayer = kMlpHidden * kPitch;
constexpr int kSmG1 = kSmA1 + kSmLayer, kSmA2 = kSmG1 + kSmLayer, kSmG2 = kSmA2 + kSmLayer;
constexpr int kSmA3 = kSmG2 + kSmLayer, kSmG3 = kSmA3 + kSmLayer, kSmD4 = kSmG3 + kSmLayer;
constexpr int kTrainFloats = kSmD4 + kMlpOut * kPitch;
static_assert(kSmX % 4 == 0 && kSmT1 % 4 == 0 && kTrainFloats * 4 <= 227 * 1024, "float4 rows, one block per SM");

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float a, float b, float c, float d) {
    *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
// acc[i][j] += w[i] * a[j]
__device__ __forceinline__ void outer4(float (&acc)[4][4], float4 w, float4 a) {
    const float wv[4] = {w.x, w.y, w.z, w.w}, av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(wv[i], av[j], acc[i][j]);
}

// hidden layer, units u0..u0+3 of samples s0..s0+3: A = gelu(W in + b), G = gelu'
template <int IN>
__device__ __forceinline__ void train_forward(const float* wt, const float* b, const float* in, int u0, int s0, float* A,
                                              float* G) {
    float z[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) z[i][j] = b[u0 + i];
#pragma unroll 8
    for (int k = 0; k < IN; ++k) outer4(z, ld4(wt + k * kWPitch + u0), ld4(in + k * kPitch + s0));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float a[4], d[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) gelu_fg(z[i][j], a[j], d[j]);
        st4(A + (u0 + i) * kPitch + s0, a[0], a[1], a[2], a[3]);
        st4(G + (u0 + i) * kPitch + s0, d[0], d[1], d[2], d[3]);
    }
}

// deltas of a hidden layer in the place of its GELU derivatives: G[i][s] *= sum_o W[o][i] D[o][s]
template <int OUTS>
__device__ __forceinline__ void train_backward(const float* w, const float* D, int u0, int s0, float* G) {
    float acc[4][4] = {};
#pragma unroll 8
    for (int o = 0; o < OUTS; ++o) outer4(acc, ld4(w + o * kMlpHidden + u0), ld4(D + o * kPitch + s0));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float* g = G + (u0 + i) * kPitch + s0;
        const float4 d = ld4(g);
        st4(g, d.x * acc[i][0], d.y * acc[i][1], d.z * acc[i][2], d.w * acc[i][3]);
    }
}

// acc[a][b] += sum_s D[4 og + a][s] A[ig + 16 b][s]: the weight gradients of outputs 4 og + a, inputs ig + 16 b
template <int NB>
__device__ __forceinline__ void train_weights(const float* D, const float* A, int og, int ig, int tile, int nb,
                                              float (&acc)[4][NB]) {
    for (int s = 0; s < tile; s += 4) {
        float4 d[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) d[a] = ld4(D + (4 * og + a) * kPitch + s);
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            if (b >= nb) break;
            const float4 x = ld4(A + (ig + 16 * b) * kPitch + s);
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                acc[a][b] = fmaf(d[a].x, x.x, acc[a][b]);
                acc[a][b] = fmaf(d[a].y, x.y, acc[a][b]);
                acc[a][b] = fmaf(d[a].z, x.z, acc[a][b]);
                acc[a][b] = fmaf(d[a].w, x.w, acc[a][b]);
            }
        }
    }
}

// `tile`: samples per tile, a multiple of 4 up to kTile
__global__ void __launch_bounds__(kTrainBlock) k_mlp_train_tile(const float* __restrict__ P, const float* __restrict__ F,
                                                                  const float* __restrict__ T,
                                                                  const uint32_t* __restrict__ index, uint64_t n,
                                                                  int tile, float inv_n, float* partial) {
    extern __shared__ __align__(16) float sm[];
    const int t = threadIdx.x;
    for (int e = t; e < kMlpHidden * kMlpHidden; e += kTrainBlock) {
        const int o = e / kMlpHidden, k = e % kMlpHidden;
        const float w2 = P[kOffW2 + e], w3 = P[kOffW3 + e];
        sm[kSmW2 + e] = w2;
        sm[kSmW3 + e] = w3;
        sm[kSmT2 + k * kWPitch + o] = w2;
        sm[kSmT3 + k * kWPitch + o] = w3;
    }
    for (int e = t; e < kMlpHidden * kMlpIn; e += kTrainBlock)
        sm[kSmT1 + (e % kMlpIn) * kWPitch + e / kMlpIn] = P[kOffW1 + e];
    if (t < kMlpOut * kMlpHidden) sm[kSmW4 + t] = P[kOffW4 + t];
    if (t < kMlpHidden) {
        sm[kSmB + t] = P[kOffB1 + t];
        sm[kSmB + kMlpHidden + t] = P[kOffB2 + t];
        sm[kSmB + 2 * kMlpHidden + t] = P[kOffB3 + t];
    }
    if (t < kMlpOut) sm[kSmB + 3 * kMlpHidden + t] = P[kOffB4 + t];
    const int u0 = 4 * (t >> 4), s0 = 4 * (t & 15), og = t >> 4, ig = t & 15;
    // gradients of this thread: its 4 x 4 blocks of W2 and W3, 4 x 2 of W1, one entry of W4 and one bias
    float g1[4][2] = {}, g2[4][4] = {}, g3[4][4] = {}, g4 = 0.0f, gb = 0.0f, loss = 0.0f;
    const int nb1 = ig < kMlpIn - 16 ? 2 : 1;
    const float* bias_rows = t < 64 ? sm + kSmG1 + t * kPitch
                                    : (t < 128 ? sm + kSmG2 + (t - 64) * kPitch
                                               : (t < 192 ? sm + kSmG3 + (t - 128) * kPitch
                                                          : sm + kSmD4 + (t < 195 ? t - 192 : 0) * kPitch));
    const uint64_t tiles = (n + tile - 1) / tile;
    for (uint64_t k = blockIdx.x; k < tiles; k += gridDim.x) {
        const uint64_t base = k * tile;
        const int valid = (int)(n - base < (uint64_t)tile ? n - base : (uint64_t)tile);
        __syncthreads();  // the weights are in place; the last tile is done with
        for (int e = t; e < kMlpIn * tile; e += kTrainBlock) {  // zero columns past the end
            const int ss = e / kMlpIn, j = e - ss * kMlpIn;
            float v = 0.0f;
            if (ss < valid) v = F[(index ? index[base + ss] : base + ss) * kMlpIn + j];
            sm[kSmX + j * kPitch + ss] = v;
        }
        __syncthreads();
        if (s0 < tile) train_forward<kMlpIn>(sm + kSmT1, sm + kSmB, sm + kSmX, u0, s0, sm + kSmA1, sm + kSmG1);
        __syncthreads();
        if (s0 < tile)
            train_forward<kMlpHidden>(sm + kSmT2, sm + kSmB + kMlpHidden, sm + kSmA1, u0, s0, sm + kSmA2, sm + kSmG2);
        __syncthreads();
        if (s0 < tile)
            train_forward<kMlpHidden>(sm + kSmT3, sm + kSmB + 2 * kMlpHidden, sm + kSmA2, u0, s0, sm + kSmA3,
                                      sm + kSmG3);
        __syncthreads();
        // output layer and dL/dout = 2 (out - t) / n (zero past the end)
        if (t < kMlpOut * kTile && (t & (kTile - 1)) < tile) {
            const int o = t / kTile, s = t & (kTile - 1);
            float v = sm[kSmB + 3 * kMlpHidden + o];
#pragma unroll 8
            for (int j = 0; j < kMlpHidden; ++j) v = fmaf(sm[kSmW4 + o * kMlpHidden + j], sm[kSmA3 + j * kPitch + s], v);
            float d = 0.0f;
            if (s < valid) {
                const uint64_t id = index ? index[base + s] : base + s;
                const float r = v - T[id * kMlpOut + o];
                loss += r * r;
                d = 2.0f * r * inv_n;
            }
            sm[kSmD4 + o * kPitch + s] = d;
        }
        __syncthreads();
        if (s0 < tile) train_backward<kMlpOut>(sm + kSmW4, sm + kSmD4, u0, s0, sm + kSmG3);
        if (t < kMlpOut * kMlpHidden) {
            const float *d = sm + kSmD4 + t / kMlpHidden * kPitch, *a = sm + kSmA3 + t % kMlpHidden * kPitch;
            for (int s = 0; s < tile; ++s) g4 = fmaf(d[s], a[s], g4);
        }
        __syncthreads();
        train_weights<4>(sm + kSmG3, sm + kSmA2, og, ig, tile, 4, g3);
        if (s0 < tile) train_backward<kMlpHidden>(sm + kSmW3, sm + kSmG3, u0, s0, sm + kSmG2);
        __syncthreads();
        train_weights<4>(sm + kSmG2, sm + kSmA1, og, ig, tile, 4, g2);
        if (s0 < tile) train_backward<kMlpHidden>(sm + kSmW2, sm + kSmG2, u0, s0, sm + kSmG1);
        __syncthreads();
        train_weights<2>(sm + kSmG1, sm + kSmX, og, ig, tile, nb1, g1);
        for (int s = 0; s < tile; ++s) gb += bias_rows[s];
    }
    float* row = partial + (size_t)blockIdx.x * (kMlpParams + 1);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            row[kOffW2 + (4 * og + a) * kMlpHidden + ig + 16 * b] = g2[a][b];
            row[kOffW3 + (4 * og + a) * kMlpHidden + ig + 16 * b] = g3[a][b];
        }
        for (int b = 0; b < nb1; ++b) row[kOffW1 + (4 * og + a) * kMlpIn + ig + 16 * b] = g1[a][b];
    }
    if (t < kMlpOut * kMlpHidden) row[kOffW4 + t] = g4;
    if (t < 64) row[kOffB1 + t] = gb;
    else if (t < 128) row[kOffB2 + t - 64] = gb;
    else if (t < 192) row[kOffB3 + t - 128] = gb;
    else if (t < 195) row[kOffB4 + t - 192] = gb;
    // loss: fixed-order block sum into the last slot of the row
    __shared__ float red[kTrainBlock];
    red[t] = loss;
    __syncthreads();
    for (int o = kTrainBlock / 2; o > 0; o >>= 1) {
        if (t < o) red[t] += red[t + o];
        __syncthreads();
    }
    if (t == 0) row[kMlpParams] = red[0] * inv_n;
}

// Column sums of the rows: 64 columns a block, four threads a column (rows r, r + 4, ...)
constexpr int kReduceCols = 64, kReduceParts = 4;
__global__ void __launch_bounds__(kReduceCols* kReduceParts) k_mlp_reduce(const float* partial, int rows, float* grads,
                                                                          float* loss) {
    __shared__ float part[kReduceParts][kReduceCols];
    const int c = threadIdx.x % kReduceCols, q = threadIdx.x / kReduceCols;
    const int p = blockIdx.x * kReduceCols + c;
    float a = 0.0f;
    if (p <= kMlpParams)
#pragma unroll 4
        for (int r = q; r < rows; r += kReduceParts) a += partial[(size_t)r * (kMlpParams + 1) + p];
    part[q][c] = a;
    __syncthreads();
    if (q == 0 && p <= kMlpParams) {
        a = (part[0][c] + part[1][c]) + (part[2][c] + part[3][c]);
        if (p < kMlpParams) grads[p] = a;
        else *loss = a;
    }
}

__global__ void k_adam(float* p, float* m, float* v, const float* g, float lr, float b1, float b2, float eps, float c1,
                       float c2) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kMlpParams; i += gridDim.x * blockDim.x) {
        float gi = g[i];
        float mi = b1 * m[i] + (1.0f - b1) * gi;
        float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

// ---------------------------------------------------------------- Mlp
namespace {
uint64_t splitmix64(uint64_t& s) {
    uint64_t z = (s += 0x9e3779b97f4a7c15ull);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
double uniform01(uint64_t& s) { return (double)(splitmix64(s) >> 11) * (1.0 / 9007199254740992.0); }
}  // namespace

Mlp::Mlp(uint64_t seed) {
    // Glorot-uniform weights (bound sqrt(6 / (fan_in + fan_out))), zero
    // biases; the output layer is scaled by 0.1 so the first corrections
    // are small.
    std::vector<float> h(kMlpParams, 0.0f);
    uint64_t st = seed;
    auto fill = [&](int off, int outs, int ins, double scale) {
        double b = std::sqrt(6.0 / (double)(ins + outs)) * scale;
        for (int k = 0; k < outs * ins; ++k) h[off + k] = (float)((2.0 * uniform01(st) - 1.0) * b);
    };
    fill(kOffW1, kMlpHidden, kMlpIn, 1.0);
    fill(kOffW2, kMlpHidden, kMlpHidden, 1.0);
    fill(kOffW3, kMlpHidden, kMlpHidden, 1.0);
    fill(kOffW4, kMlpOut, kMlpHidden, 0.1);
    p_.upload(h, nullptr);
    for (auto* b : {&m_, &v_}) {
        b->reserve(kMlpParams);
        b->zero(kMlpParams, nullptr);
    }
    g_.reserve(kMlpParams + 1);
    g_.zero(kMlpParams + 1, nullptr);
    CC_CUDA(cudaStreamSynchronize(nullptr));
}

void Mlp::set_params(const float* host, cudaStream_t st) {
    CC_CUDA(cudaMemcpyAsync(p_.ptr, host, kMlpParams * sizeof(float), cudaMemcpyHostToDevice, st));
    CC_CUDA(cudaMemsetAsync(m_.ptr, 0, kMlpParams * sizeof(float), st));
    CC_CUDA(cudaMemsetAsync(v_.ptr, 0, kMlpParams * sizeof(float), st));
    CC_CUDA(cudaStreamSynchronize(st));
    t_ = 0;
    w16_valid_ = false;
}

void Mlp::get_params(float* host, cudaStream_t st) const {
    CC_CUDA(cudaMemcpyAsync(host, p_.ptr, kMlpParams * sizeof(float), cudaMemcpyDeviceToHost, st));
    CC_CUDA(cudaStreamSynchronize(st));
}

void Mlp::forward(const float* features, uint64_t n, float* out, int precision, cudaStream_t st) {
    if (n == 0) return;
    if (precision == 1) {
        forward_tc(features, n, out, st);
        return;
    }
    size_t smem = (kMlpParams + 1 + kMlpHidden * kFwdBlock) * sizeof(float);
    allow_dynamic_smem(k_mlp_forward_f32, smem);
    uint64_t blocks = (n + kFwdBlock - 1) / kFwdBlock;
    unsigned grid = (unsigned)std::min<uint64_t>(blocks, 148ull * 4ull);
    k_mlp_forward_f32<<<grid, kFwdBlock, smem, st>>>(p_.ptr, features, n, out);
    CC_CUDA(cudaGetLastError());
}

void Mlp::gradients(const float* features, const float* targets, const uint32_t* index, uint64_t n, float* grads,
                    float* loss, cudaStream_t st) {
    if (n == 0) throw Failure{CC_ERR_INVALID_ARGUMENT, "MLP gradients need at least one sample"};
    constexpr size_t smem = (size_t)kTrainFloats * sizeof(float);
    static std::atomic<uint64_t> raised{0};  // devices on which the limit is raised
    allow_dynamic_smem_once(k_mlp_train_tile, smem, raised);
    // the smallest tile (a multiple of 4) with which every SM takes as many tiles
    // as 64-sample tiles would: 16,384 samples are 2 x 148 tiles of 56
    const uint64_t rounds = (n + 148ull * kTile - 1) / (148ull * kTile);
    const int tile = (int)(((n + 148ull * rounds - 1) / (148ull * rounds) + 3) & ~3ull);
    const uint64_t tiles = (n + tile - 1) / tile;
    int rows = (int)std::min<uint64_t>(tiles, 148ull);
    partial_.reserve((size_t)rows * (kMlpParams + 1));
    k_mlp_train_tile<<<rows, kTrainBlock, smem, st>>>(p_.ptr, features, targets, index, n, tile, 1.0f / (float)n,
                                                      partial_.ptr);
    k_mlp_reduce<<<(kMlpParams + kReduceCols) / kReduceCols, kReduceCols * kReduceParts, 0, st>>>(partial_.ptr, rows,
                                                                                                  grads, loss);
    CC_CUDA(cudaGetLastError());
}

void Mlp::adam(const float* grads, float lr, float beta1, float beta2, float eps, cudaStream_t st) {
    ++t_;
    float c1 = 1.0f - (float)std::pow((double)beta1, (double)t_);
    float c2 = 1.0f - (float)std::pow((double)beta2, (double)t_);
    k_adam<<<(kMlpParams + 255) / 256, 256, 0, st>>>(p_.ptr, m_.ptr, v_.ptr, grads, lr, beta1, beta2, eps, c1, c2);
    CC_CUDA(cudaGetLastError());
    w16_valid_ = false;
}

}  // namespace cc
