// The learned form selector's network: an MLP 12 -> 64 -> 64 -> 32 (ReLU, FP32) that predicts
// the log-time of each of the 32 engine forms from a matrix's structural features
// (k_features.cu), trained on the GPU by the kernels below (forward, backward, Adam).
//
// Parameters, one flat float array of 7,072 entries:
//   W1[64][12] @0   b1[64] @768   W2[64][64] @832   b2[64] @4928   W3[32][64] @4992   b3[32] @7040
// Loss: masked mean squared error over the outputs (a form that failed on a matrix has mask
// 0).  Every reduction runs in a fixed order, so a training run gives the same bits every time.

#include <math.h>
#include <string.h>

#include <vector>

#include "pava_internal.h"

namespace pava {

namespace {

constexpr int IN = PAVA_MLP_IN, HID = PAVA_MLP_HIDDEN, OUT = PAVA_MLP_OUT;
constexpr int OW1 = 0, OB1 = OW1 + HID * IN, OW2 = OB1 + HID, OB2 = OW2 + HID * HID,
              OW3 = OB2 + HID, OB3 = OW3 + OUT * HID, NP = OB3 + OUT;
static_assert(NP == PAVA_MLP_NPARAM, "parameter count");

// The network on tiles of TS samples, one 512-thread CTA per tile (grid-stride), the weights in
// shared memory for the whole launch.  GRAD = false: outputs O only.  GRAD = true: forward,
// backward and weight gradients of the CTA's tiles; the gradient sums stay in registers over
// the tiles (a 4 x 2 tile of W2 and 1 x 4 of W3 per thread, 2 of W1 for 384 threads, a bias
// each for 160) and go to part[blockIdx.x][NP], the CTA's loss sum to part_loss[blockIdx.x];
// reduce_kernel adds the CTAs.
//
// What bounds it: the latency of eight dependent phases between barriers, each a short chain of
// shared-memory reads and FMAs; an epoch moves well under 4 MB and 85 MFLOP at 2,000 samples.
// One CTA per sample read W2 with a stride of 256 bytes between lanes and left the weight
// gradients to 28 CTAs of 2,000-step serial sums: 183 us a training step at 2,000 samples (forward
// 51, backward 7, gradient 153, loss 42, Adam 4 us, each alone); this kernel and reduce_kernel
// take 17 us a step, 12.5 us at 500 samples.
// 16 samples per tile put 2,000 samples on 125 CTAs, one per SM (32 per tile would leave half
// of the SMs idle there), and 16 warps hide more of each phase than 8 (22 us a step).  Each thread
// has all of its weight loads in flight at once.
//
// Both kernels are launched as programmatic dependents of the one before: their launch and, here,
// the read of the inputs overlap its end.
//
// Rows of W2 and W3 are padded to 68 floats: a warp's 16-byte reads down the rows (forward) and
// its 4-byte reads along them (backward) are both free of bank conflicts.
constexpr int TS = 16, NT = 512, LDW = HID + 4;
constexpr int SH = TS * HID / NT, SO = TS * OUT / NT;  // samples per thread: hidden, output
static_assert(SH == 2 && SO == 1 && NP % 4 == 0, "thread mapping");
struct MlpSmem {
    float w1[HID * IN], b1[HID], w2[HID * LDW], b2[HID], w3[OUT * LDW], b3[OUT];
    float x[TS * IN], h1[TS * HID], h2[TS * HID], go[TS * OUT], g1[TS * HID], g2[TS * HID];
    float red[NT / 32];
};
static_assert(sizeof(MlpSmem) <= 48 * 1024, "default shared memory limit");

template <bool GRAD>
__global__ void __launch_bounds__(NT)
mlp_kernel(const float *P, const float *__restrict__ X, int B,
           const float *__restrict__ T, const float *__restrict__ Mk, float inv_count,
           float *O, float *part, float *part_loss) {
    __shared__ __align__(16) MlpSmem S;
    const int t = threadIdx.x;
    const int tiles = (B + TS - 1) / TS;
    auto load_x = [&](int tile) {
        const int b0 = tile * TS, nb = min(TS, B - b0);
        for (int q = t; q < TS * IN; q += NT) S.x[q] = q < nb * IN ? X[(long long)b0 * IN + q] : 0.f;
    };
    asm volatile("griddepcontrol.launch_dependents;");
    load_x(blockIdx.x);  // the grid has at most one CTA per tile
    // the step before has to be done: it wrote the weights, and read part
    asm volatile("griddepcontrol.wait;" ::: "memory");
    {
        constexpr int NV = (NP / 4 + NT - 1) / NT;
        float4 v[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int q = i * NT + t;
            if (q < NP / 4) v[i] = reinterpret_cast<const float4 *>(P)[q];
        }
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int q = 4 * (i * NT + t);  // the four entries lie in one row of one matrix
            if (q >= NP) continue;
            float *d = q < OB1   ? S.w1 + q
                       : q < OW2 ? S.b1 + (q - OB1)
                       : q < OB2 ? S.w2 + (q - OW2) / HID * LDW + (q - OW2) % HID
                       : q < OW3 ? S.b2 + (q - OB2)
                       : q < OB3 ? S.w3 + (q - OW3) / HID * LDW + (q - OW3) % HID
                                 : S.b3 + (q - OB3);
            *reinterpret_cast<float4 *>(d) = v[i];
        }
    }

    const int j = t & (HID - 1), s0 = (t / HID) * SH;  // hidden unit and SH samples
    const int o = t & (OUT - 1), s1 = (t / OUT) * SO;  // output and SO samples
    const int tj = (t >> 5) * 4, tk = (t & 31) * 2;    // W2 tile: rows tj.., columns tk, tk + 1
    const int to = t >> 4, tq = (t & 15) * 4;          // W3 tile: row to, columns tq..
    const int ti = (t >> 6) * 2;                       // W1: unit j, inputs ti, ti + 1 (t < 384)
    float a2[4][2] = {}, a3[4] = {}, a1[2] = {}, ab = 0.f, loss = 0.f;

    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int b0 = tile * TS, nb = min(TS, B - b0);
        if (tile != blockIdx.x) {
            __syncthreads();  // the previous tile's arrays are done with
            load_x(tile);
        }
        __syncthreads();
        // layer 1 (samples past the batch: zero activations, so they add nothing below)
        float z[SH];
#pragma unroll
        for (int u = 0; u < SH; ++u) z[u] = S.b1[j];
#pragma unroll
        for (int i = 0; i < IN; ++i) {
            const float w = S.w1[j * IN + i];
#pragma unroll
            for (int u = 0; u < SH; ++u) z[u] = fmaf(w, S.x[(s0 + u) * IN + i], z[u]);
        }
#pragma unroll
        for (int u = 0; u < SH; ++u) S.h1[(s0 + u) * HID + j] = s0 + u < nb && z[u] > 0.f ? z[u] : 0.f;
        __syncthreads();
        // layer 2
#pragma unroll
        for (int u = 0; u < SH; ++u) z[u] = S.b2[j];
#pragma unroll 8
        for (int k = 0; k < HID; k += 4) {
            const float4 w = *reinterpret_cast<const float4 *>(&S.w2[j * LDW + k]);
#pragma unroll
            for (int u = 0; u < SH; ++u) {
                const float4 h = *reinterpret_cast<const float4 *>(&S.h1[(s0 + u) * HID + k]);
                z[u] = fmaf(w.x, h.x, z[u]);
                z[u] = fmaf(w.y, h.y, z[u]);
                z[u] = fmaf(w.z, h.z, z[u]);
                z[u] = fmaf(w.w, h.w, z[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < SH; ++u) S.h2[(s0 + u) * HID + j] = s0 + u < nb && z[u] > 0.f ? z[u] : 0.f;
        __syncthreads();
        // output layer, its loss and gradient
        float y[SO];
#pragma unroll
        for (int u = 0; u < SO; ++u) y[u] = S.b3[o];
#pragma unroll 8
        for (int k = 0; k < HID; k += 4) {
            const float4 w = *reinterpret_cast<const float4 *>(&S.w3[o * LDW + k]);
#pragma unroll
            for (int u = 0; u < SO; ++u) {
                const float4 h = *reinterpret_cast<const float4 *>(&S.h2[(s1 + u) * HID + k]);
                y[u] = fmaf(w.x, h.x, y[u]);
                y[u] = fmaf(w.y, h.y, y[u]);
                y[u] = fmaf(w.z, h.z, y[u]);
                y[u] = fmaf(w.w, h.w, y[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < SO; ++u) {
            const bool in = s1 + u < nb;
            const long long q = (long long)(b0 + s1 + u) * OUT + o;
            if (!GRAD) {
                if (in) O[q] = y[u];
            } else {
                const float d = in ? y[u] - T[q] : 0.f, mk = in ? Mk[q] : 0.f;
                loss = fmaf(mk * d, d, loss);
                S.go[(s1 + u) * OUT + o] = in ? 2.f * mk * d * inv_count : 0.f;
            }
        }
        if (!GRAD) continue;
        __syncthreads();
        // dZ2 = (dO W3) through the ReLU
#pragma unroll
        for (int u = 0; u < SH; ++u) z[u] = 0.f;
#pragma unroll
        for (int k = 0; k < OUT; k += 4) {
            float w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) w[e] = S.w3[(k + e) * LDW + j];
#pragma unroll
            for (int u = 0; u < SH; ++u) {
                const float4 g = *reinterpret_cast<const float4 *>(&S.go[(s0 + u) * OUT + k]);
                z[u] = fmaf(g.x, w[0], z[u]);
                z[u] = fmaf(g.y, w[1], z[u]);
                z[u] = fmaf(g.z, w[2], z[u]);
                z[u] = fmaf(g.w, w[3], z[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < SH; ++u)
            S.g2[(s0 + u) * HID + j] = S.h2[(s0 + u) * HID + j] > 0.f ? z[u] : 0.f;
        __syncthreads();
        // dZ1 = (dZ2 W2) through the ReLU
#pragma unroll
        for (int u = 0; u < SH; ++u) z[u] = 0.f;
#pragma unroll 8
        for (int k = 0; k < HID; k += 4) {
            float w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) w[e] = S.w2[(k + e) * LDW + j];
#pragma unroll
            for (int u = 0; u < SH; ++u) {
                const float4 g = *reinterpret_cast<const float4 *>(&S.g2[(s0 + u) * HID + k]);
                z[u] = fmaf(g.x, w[0], z[u]);
                z[u] = fmaf(g.y, w[1], z[u]);
                z[u] = fmaf(g.z, w[2], z[u]);
                z[u] = fmaf(g.w, w[3], z[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < SH; ++u)
            S.g1[(s0 + u) * HID + j] = S.h1[(s0 + u) * HID + j] > 0.f ? z[u] : 0.f;
        __syncthreads();
        // weight gradients, summed over the samples in order
#pragma unroll 8
        for (int s = 0; s < TS; ++s) {
            const float4 g = *reinterpret_cast<const float4 *>(&S.g2[s * HID + tj]);
            const float2 h = *reinterpret_cast<const float2 *>(&S.h1[s * HID + tk]);
            const float4 h2 = *reinterpret_cast<const float4 *>(&S.h2[s * HID + tq]);
            const float go = S.go[s * OUT + to];
            const float gv[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                a2[r][0] = fmaf(gv[r], h.x, a2[r][0]);
                a2[r][1] = fmaf(gv[r], h.y, a2[r][1]);
            }
            a3[0] = fmaf(go, h2.x, a3[0]);
            a3[1] = fmaf(go, h2.y, a3[1]);
            a3[2] = fmaf(go, h2.z, a3[2]);
            a3[3] = fmaf(go, h2.w, a3[3]);
            if (t < 6 * HID) {
                const float g1 = S.g1[s * HID + j];
                a1[0] = fmaf(g1, S.x[s * IN + ti], a1[0]);
                a1[1] = fmaf(g1, S.x[s * IN + ti + 1], a1[1]);
                if (t < HID) ab += g1;
                else if (t < 2 * HID) ab += S.g2[s * HID + j];
                else if (t < 2 * HID + OUT) ab += S.go[s * OUT + o];
            }
        }
    }
    if (!GRAD) return;
    float *G = part + (long long)blockIdx.x * NP;
#pragma unroll
    for (int r = 0; r < 4; ++r)
        *reinterpret_cast<float2 *>(&G[OW2 + (tj + r) * HID + tk]) = make_float2(a2[r][0], a2[r][1]);
    *reinterpret_cast<float4 *>(&G[OW3 + to * HID + tq]) = make_float4(a3[0], a3[1], a3[2], a3[3]);
    if (t < 6 * HID)
        *reinterpret_cast<float2 *>(&G[OW1 + j * IN + ti]) = make_float2(a1[0], a1[1]);
    if (t < HID) G[OB1 + t] = ab;
    else if (t < 2 * HID) G[OB2 + j] = ab;
    else if (t < 2 * HID + OUT) G[OB3 + o] = ab;
    // the CTA's loss: fixed butterfly per warp, then the warps in order
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) loss += __shfl_xor_sync(FULL, loss, d);
    if ((t & 31) == 0) S.red[t >> 5] = loss;
    __syncthreads();
    if (t == 0) {
        float l = 0.f;
        for (int w = 0; w < NT / 32; ++w) l += S.red[w];
        part_loss[blockIdx.x] = l;
    }
}

// Sums the CTAs' gradients in a fixed order (warp w of RW takes the parts w, w + RW, ..., then the
// RW sums in order), 32 parameters per block, and either stores them (G) or applies an Adam
// step at once.  Block 0 also sums the loss.  Bound by latency: one round of L2 reads (3.5 MB at
// 125 parts, eight in flight per thread), the sum of the warps, the Adam step.
constexpr int RW = 16;
struct AdamStep {
    float *P, *Mm, *Vv;  // P = nullptr: store the gradient in G instead
    float lr, b1, b2, eps, c1, c2;
};
__global__ void __launch_bounds__(RW * 32)
reduce_kernel(const float *part, const float *part_loss, int parts,
              float inv_count, float *G, float *loss, AdamStep st) {
    __shared__ float red[RW][32];
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");  // mlp_kernel's parts
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int p = blockIdx.x * 32 + lane;
    static_assert(NP % 32 == 0 && NP % 4 == 0 && OW2 % 4 == 0 && OW3 % 4 == 0, "32 per block");
    float m0 = 0.f, v0 = 0.f, p0 = 0.f;
    if (w == 0 && st.P) {  // in flight beside the parts
        m0 = st.Mm[p];
        v0 = st.Vv[p];
        p0 = st.P[p];
    }
    float s = 0.f;
#pragma unroll 8
    for (int c = w; c < parts; c += RW) s += part[(long long)c * NP + p];
    red[w][lane] = s;
    __syncthreads();
    if (w == 0) {
        float g = red[0][lane];
#pragma unroll
        for (int q = 1; q < RW; ++q) g += red[q][lane];
        if (!st.P) {
            G[p] = g;
        } else {
            const float m = st.b1 * m0 + (1.f - st.b1) * g;
            const float v = st.b2 * v0 + (1.f - st.b2) * g * g;
            st.Mm[p] = m;
            st.Vv[p] = v;
            st.P[p] = p0 - st.lr * (m * st.c1) / (sqrtf(v * st.c2) + st.eps);
        }
    } else if (w == 1 && blockIdx.x == 0) {
        float l = 0.f;
        for (int c = lane; c < parts; c += 32) l += part_loss[c];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) l += __shfl_xor_sync(FULL, l, d);
        if (lane == 0) *loss = l * inv_count;
    }
}

// (x - mean) / std per feature.
__global__ void normalize_kernel(float *__restrict__ X, int B, const float *__restrict__ mu,
                                 const float *__restrict__ sd) {
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (long long)B * IN) return;
    const int i = (int)(q % IN);
    X[q] = (X[q] - mu[i]) / sd[i];
}

// splitmix64 -> uniform in [-1, 1)
uint64_t mix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

}  // namespace
}  // namespace pava

struct pava_mlp {
    float *P = nullptr, *G = nullptr, *Mm = nullptr, *Vv = nullptr;  // params, grad, Adam
    float *mu = nullptr, *sd = nullptr;                              // feature normalisation
    int B = 0, cap = 0;
    float *X = nullptr, *T = nullptr, *Mk = nullptr, *O = nullptr;   // current batch
    float *part = nullptr, *part_loss = nullptr;                     // per-CTA gradients, losses
    float *loss = nullptr;
    float *hist = nullptr;                                           // losses of a training run
    int hist_cap = 0;
    int max_ctas = 1;                                                // two per SM
    float inv_count = 0.f;
    int step = 0;
};

namespace {

using namespace pava;

pava_status mfail(cudaError_t e, const char *where) {
    set_last_error(std::string(where) + ": " + cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? PAVA_E_NOMEM : PAVA_E_CUDA;
}

void free_batch(pava_mlp *m) {
    float **bufs[] = {&m->X, &m->T, &m->Mk, &m->O, &m->part, &m->part_loss};
    for (float **b : bufs) { cudaFree(*b); *b = nullptr; }
    m->cap = 0;
}

int mlp_ctas(const pava_mlp *m, int B) {
    const int tiles = (B + TS - 1) / TS;
    return tiles < m->max_ctas ? tiles : m->max_ctas;
}

cudaError_t run_forward(pava_mlp *m) {
    mlp_kernel<false><<<mlp_ctas(m, m->B), NT>>>(m->P, m->X, m->B, nullptr, nullptr, 0.f, m->O,
                                                 nullptr, nullptr);
    return cudaGetLastError();
}

// The gradient of the current batch: into m->G (st.P null), or straight into an Adam step.
cudaError_t run_gradient(pava_mlp *m, float *loss, const AdamStep &st) {
    const int ctas = mlp_ctas(m, m->B);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(NT);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(
        &cfg, mlp_kernel<true>, (const float *)m->P, (const float *)m->X, m->B,
        (const float *)m->T, (const float *)m->Mk, m->inv_count, (float *)nullptr, m->part,
        m->part_loss);
    if (e != cudaSuccess) return e;
    cfg.gridDim = dim3(NP / 32);
    cfg.blockDim = dim3(RW * 32);
    return cudaLaunchKernelEx(&cfg, reduce_kernel, (const float *)m->part,
                              (const float *)m->part_loss, ctas, m->inv_count, m->G, loss, st);
}

}  // namespace

extern "C" {

pava_status pava_mlp_create(uint64_t seed, pava_mlp **out) {
    if (!out) { set_last_error("out is NULL"); return PAVA_E_INVALID_ARG; }
    *out = nullptr;
    pava_mlp *m = new (std::nothrow) pava_mlp();
    if (!m) return PAVA_E_NOMEM;
    int dev = 0, sms = 1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    m->max_ctas = 2 * sms;
    if (e == cudaSuccess) e = cudaMalloc(&m->P, sizeof(float) * NP);
    if (e == cudaSuccess) e = cudaMalloc(&m->G, sizeof(float) * NP);
    if (e == cudaSuccess) e = cudaMalloc(&m->Mm, sizeof(float) * NP);
    if (e == cudaSuccess) e = cudaMalloc(&m->Vv, sizeof(float) * NP);
    if (e == cudaSuccess) e = cudaMalloc(&m->mu, sizeof(float) * IN);
    if (e == cudaSuccess) e = cudaMalloc(&m->sd, sizeof(float) * IN);
    if (e == cudaSuccess) e = cudaMalloc(&m->loss, sizeof(float));
    // He-uniform weights (bound sqrt(6 / fan_in)), zero biases, identity normalisation
    std::vector<float> h(NP, 0.f);
    auto fill = [&](int off, int count, int fan_in, uint64_t tag) {
        const float bound = sqrtf(6.f / fan_in);
        for (int q = 0; q < count; ++q) {
            const uint64_t r = mix64(mix64(seed * 0xD6E8FEB86659FD93ull + tag) ^ (uint64_t)q);
            const float u = (float)((double)(r >> 11) * 0x1.0p-53) * 2.f - 1.f;
            h[off + q] = u * bound;
        }
    };
    fill(OW1, HID * IN, IN, 1);
    fill(OW2, HID * HID, HID, 2);
    fill(OW3, OUT * HID, HID, 3);
    std::vector<float> zero(IN, 0.f), one(IN, 1.f);
    if (e == cudaSuccess) e = cudaMemcpy(m->P, h.data(), sizeof(float) * NP, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(m->Mm, 0, sizeof(float) * NP);
    if (e == cudaSuccess) e = cudaMemset(m->Vv, 0, sizeof(float) * NP);
    if (e == cudaSuccess) e = cudaMemcpy(m->mu, zero.data(), sizeof(float) * IN, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(m->sd, one.data(), sizeof(float) * IN, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        pava_mlp_destroy(m);
        return mfail(e, "mlp create");
    }
    *out = m;
    return PAVA_SUCCESS;
}

pava_status pava_mlp_get_params(const pava_mlp *m, float *params, float *mean12, float *std12) {
    if (!m) { set_last_error("mlp is NULL"); return PAVA_E_INVALID_ARG; }
    cudaError_t e = cudaSuccess;
    if (params) e = cudaMemcpy(params, m->P, sizeof(float) * NP, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && mean12) e = cudaMemcpy(mean12, m->mu, sizeof(float) * IN, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && std12) e = cudaMemcpy(std12, m->sd, sizeof(float) * IN, cudaMemcpyDeviceToHost);
    return e == cudaSuccess ? PAVA_SUCCESS : mfail(e, "mlp get");
}

pava_status pava_mlp_set_params(pava_mlp *m, const float *params, const float *mean12,
                                const float *std12) {
    if (!m) { set_last_error("mlp is NULL"); return PAVA_E_INVALID_ARG; }
    if (std12)
        for (int i = 0; i < IN; ++i)
            if (!(std12[i] > 0.f)) { set_last_error("std must be > 0"); return PAVA_E_INVALID_ARG; }
    cudaError_t e = cudaSuccess;
    if (params) {
        e = cudaMemcpy(m->P, params, sizeof(float) * NP, cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemset(m->Mm, 0, sizeof(float) * NP);
        if (e == cudaSuccess) e = cudaMemset(m->Vv, 0, sizeof(float) * NP);
        m->step = 0;
    }
    if (e == cudaSuccess && mean12) e = cudaMemcpy(m->mu, mean12, sizeof(float) * IN, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && std12) e = cudaMemcpy(m->sd, std12, sizeof(float) * IN, cudaMemcpyHostToDevice);
    return e == cudaSuccess ? PAVA_SUCCESS : mfail(e, "mlp set");
}

pava_status pava_mlp_set_batch(pava_mlp *m, int B, const float *X, const float *T,
                               const float *mask) {
    if (!m || !X || B < 1) { set_last_error("mlp, X or B invalid"); return PAVA_E_INVALID_ARG; }
    cudaError_t e = cudaSuccess;
    if (B > m->cap) {
        free_batch(m);
        const size_t b = (size_t)B;
        const size_t ctas = (size_t)mlp_ctas(m, B);
        e = cudaMalloc(&m->X, sizeof(float) * b * IN);
        if (e == cudaSuccess) e = cudaMalloc(&m->T, sizeof(float) * b * OUT);
        if (e == cudaSuccess) e = cudaMalloc(&m->Mk, sizeof(float) * b * OUT);
        if (e == cudaSuccess) e = cudaMalloc(&m->O, sizeof(float) * b * OUT);
        if (e == cudaSuccess) e = cudaMalloc(&m->part, sizeof(float) * ctas * NP);
        if (e == cudaSuccess) e = cudaMalloc(&m->part_loss, sizeof(float) * ctas);
        if (e != cudaSuccess) { free_batch(m); return mfail(e, "mlp batch"); }
        m->cap = B;
    }
    m->B = B;
    e = cudaMemcpy(m->X, X, sizeof(float) * (size_t)B * IN, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        normalize_kernel<<<(unsigned)(((long long)B * IN + 255) / 256), 256>>>(m->X, B, m->mu, m->sd);
        e = cudaGetLastError();
    }
    std::vector<float> tt((size_t)B * OUT, 0.f), mk((size_t)B * OUT, 0.f);
    double count = 0;
    if (T) {
        for (size_t q = 0; q < tt.size(); ++q) {
            tt[q] = T[q];
            mk[q] = mask ? mask[q] : 1.f;
            count += mk[q];
        }
    }
    m->inv_count = count > 0 ? (float)(1.0 / count) : 0.f;
    if (e == cudaSuccess) e = cudaMemcpy(m->T, tt.data(), sizeof(float) * tt.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(m->Mk, mk.data(), sizeof(float) * mk.size(), cudaMemcpyHostToDevice);
    return e == cudaSuccess ? PAVA_SUCCESS : mfail(e, "mlp batch upload");
}

pava_status pava_mlp_forward(pava_mlp *m, float *Y) {
    if (!m || m->B < 1) { set_last_error("no batch set"); return PAVA_E_INVALID_ARG; }
    cudaError_t e = run_forward(m);
    if (e == cudaSuccess && Y)
        e = cudaMemcpy(Y, m->O, sizeof(float) * (size_t)m->B * OUT, cudaMemcpyDeviceToHost);
    return e == cudaSuccess ? PAVA_SUCCESS : mfail(e, "mlp forward");
}

pava_status pava_mlp_gradient(pava_mlp *m, float *grad, float *loss) {
    if (!m || m->B < 1) { set_last_error("no batch set"); return PAVA_E_INVALID_ARG; }
    cudaError_t e = run_gradient(m, m->loss, AdamStep{});
    if (e == cudaSuccess && grad) e = cudaMemcpy(grad, m->G, sizeof(float) * NP, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && loss) e = cudaMemcpy(loss, m->loss, sizeof(float), cudaMemcpyDeviceToHost);
    return e == cudaSuccess ? PAVA_SUCCESS : mfail(e, "mlp gradient");
}

pava_status pava_mlp_train(pava_mlp *m, int epochs, float lr, float *loss_hist) {
    if (!m || m->B < 1 || epochs < 0) { set_last_error("no batch set"); return PAVA_E_INVALID_ARG; }
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    cudaError_t e = cudaSuccess;
    if (epochs > m->hist_cap) {  // one loss per step, copied back once at the end
        cudaFree(m->hist);
        m->hist = nullptr;
        m->hist_cap = 0;
        e = cudaMalloc(&m->hist, sizeof(float) * (size_t)epochs);
        if (e != cudaSuccess) return mfail(e, "mlp train");
        m->hist_cap = epochs;
    }
    for (int ep = 0; ep < epochs && e == cudaSuccess; ++ep) {
        ++m->step;
        const float c1 = 1.f / (1.f - powf(b1, (float)m->step));
        const float c2 = 1.f / (1.f - powf(b2, (float)m->step));
        e = run_gradient(m, m->hist + ep, AdamStep{m->P, m->Mm, m->Vv, lr, b1, b2, eps, c1, c2});
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess && loss_hist && epochs > 0)
        e = cudaMemcpy(loss_hist, m->hist, sizeof(float) * (size_t)epochs, cudaMemcpyDeviceToHost);
    return e == cudaSuccess ? PAVA_SUCCESS : mfail(e, "mlp train");
}

pava_status pava_mlp_destroy(pava_mlp *m) {
    if (!m) return PAVA_SUCCESS;
    free_batch(m);
    cudaFree(m->P); cudaFree(m->G); cudaFree(m->Mm); cudaFree(m->Vv);
    cudaFree(m->mu); cudaFree(m->sd); cudaFree(m->loss); cudaFree(m->hist);
    delete m;
    return PAVA_SUCCESS;
}

}  // extern "C"
