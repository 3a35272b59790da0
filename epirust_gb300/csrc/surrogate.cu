// surrogate.cu -- the learned surrogate of include/epi_surrogate.h: a BF16 MLP trained and
// evaluated on the sm_103a tensor cores.
//
// Layers l = 0 .. L-1 map K_l inputs to N_l outputs (K_0 = in_dim padded to 64, N_{L-1} =
// out_dim padded to a multiple of 128, hidden widths in between).  Padding rows and columns
// are zero and stay zero: their inputs are zero, so are their gradients and Adam updates.
// Per layer the device holds the FP32 master weights W (N x K) and b, Adam moments, and two
// BF16 copies: W (the B operand of the forward product) and W^T (the B operand of the
// input-gradient product).  Training activations are kept in both orientations, written by the
// epilogues, so every product takes K-major operands:
//   forward  H_{l+1} = gelu(H_l W_l^T + b_l)          A = H_l      B = W_l
//   output   Y = H_{L-1} W^T + b, dY = 2 (Y - T) / (B * out_dim)   (fused, with the loss)
//   inputs   dZ_{l-1} = (dZ_l W_l) * gelu'(Z_{l-1})    A = dZ_l     B = W_l^T
//   weights  dW_l = dZ_l^T H_l                         A = dZ_l^T   B = H_l^T   (fused with Adam)
// A training step is 2 L launches (tc_train.cuh): L forward, then one launch per input
// gradient, each carrying the weight gradients that have become ready.  The minibatches of a
// chunk of steps are gathered by one launch; groups of kGroupSteps steps are one CUDA graph,
// kept by the handle.  Inference runs the products of tc_infer.cuh (tc_gemm.cuh where K > 512).
//
// A handle holds E = cfg.members networks of the same shape (an ensemble).  Every buffer
// carries a leading member axis and every kernel covers all members in one launch: the
// products through the third grid dimension and 3-D tensor maps {cols, rows, E}, the small
// kernels through blockIdx.y.  Member m is initialised from seed + m and, in training, draws
// its minibatches from shuffle_seed + m, so it equals a one-member network created and
// trained with those seeds.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/epi_surrogate.h"
#include "epi_internal.h"
#include "tc_gemm.cuh"
#include "tc_infer.cuh"
#include "tc_train.cuh"

using namespace epi::tc;

namespace {

constexpr uint32_t kInPad = 64;
constexpr uint32_t kMaxMembers = 64;
constexpr int kSmallThreads = 256;

// ---------------------------------------------------------------- small kernels
// Host arrays travel as the caller lays them out; padding, conversion and (un)packing are
// kernels (at 65,536 candidates the host loops they replace took a third of a score call).

// Rows of n x in_dim floats -> BF16 rows of kInPad, zero beyond in_dim and n (up to n_rows); xt,
// when given, also receives the transpose (kInPad x n_rows).  One thread per two columns.
__global__ void k_pad_inputs(const float* __restrict__ x, uint32_t n, uint32_t n_rows, uint32_t in_dim,
                             __nv_bfloat16* __restrict__ out, __nv_bfloat16* __restrict__ xt, uint32_t xt_pitch) {
    const size_t total = (size_t)n_rows * (kInPad / 2);
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (size_t)gridDim.x * blockDim.x) {
        const uint32_t r = (uint32_t)(q / (kInPad / 2)), c = 2u * (uint32_t)(q % (kInPad / 2));
        const float a = r < n && c < in_dim ? x[(size_t)r * in_dim + c] : 0.f;
        const float b = r < n && c + 1 < in_dim ? x[(size_t)r * in_dim + c + 1] : 0.f;
        const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
        reinterpret_cast<__nv_bfloat162*>(out)[q] = v;
        if (xt) {
            xt[(size_t)c * xt_pitch + r] = v.x;
            xt[(size_t)(c + 1) * xt_pitch + r] = v.y;
        }
    }
}

// Rows of n x cols floats <-> rows of `pitch` (padding zero when written).
__global__ void k_pad_rows(const float* __restrict__ in, uint32_t n, uint32_t cols, uint32_t pitch, float* __restrict__ out) {
    const size_t total = (size_t)n * pitch;
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (size_t)gridDim.x * blockDim.x) {
        const uint32_t c = (uint32_t)(q % pitch);
        out[q] = c < cols ? in[q / pitch * cols + c] : 0.f;
    }
}
__global__ void k_unpad_rows(const float* __restrict__ in, uint32_t n, uint32_t cols, uint32_t pitch, size_t member_in,
                             float* __restrict__ out) {
    const size_t total = (size_t)n * cols;
    in += blockIdx.y * member_in;
    out += blockIdx.y * total;
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (size_t)gridDim.x * blockDim.x)
        out[q] = in[q / cols * pitch + q % cols];
}

// One layer between the caller's flat layout (member blockIdx.y's block of `count` floats, W
// row by row and then b from `first`) and its padded arrays; the padding stays zero.
__global__ void k_params(float* __restrict__ flat, size_t count, size_t first, uint32_t n_real, uint32_t k_real,
                         float* __restrict__ w, float* __restrict__ b, uint32_t N, uint32_t K, int to_flat) {
    flat += blockIdx.y * count + first;
    w += (size_t)blockIdx.y * N * K;
    b += (size_t)blockIdx.y * N;
    const size_t nw = (size_t)n_real * k_real, total = nw + n_real;
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (size_t)gridDim.x * blockDim.x) {
        float* p = q < nw ? w + q / k_real * K + q % k_real : b + (q - nw);
        if (to_flat) flat[q] = *p;
        else *p = flat[q];
    }
}

// The minibatch inputs of a chunk of steps: row r of member e (grid rows / 32 x E) is sample
// idx[r / B][e][r % B], in both orientations (out rows x kInPad, out_t kInPad x rows per member).
__global__ void __launch_bounds__(256) k_gather(const __nv_bfloat16* __restrict__ xs, const uint32_t* __restrict__ idx,
                                                uint32_t B, uint32_t rows_cap, __nv_bfloat16* __restrict__ out,
                                                __nv_bfloat16* __restrict__ out_t) {
    __shared__ __nv_bfloat16 tile[32][kInPad + 2];
    const uint32_t e = blockIdx.y, r0 = blockIdx.x * 32u, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    out += (size_t)e * rows_cap * kInPad;
    out_t += (size_t)e * rows_cap * kInPad;
    for (uint32_t k = warp; k < 32u; k += 8u) {
        const uint32_t r = r0 + k, s = idx[((size_t)(r / B) * gridDim.y + e) * B + r % B];
        const __nv_bfloat162 v = reinterpret_cast<const __nv_bfloat162*>(xs + (size_t)s * kInPad)[lane];
        reinterpret_cast<__nv_bfloat162*>(out + (size_t)r * kInPad)[lane] = v;
        *reinterpret_cast<__nv_bfloat162*>(&tile[k][2u * lane]) = v;
    }
    __syncthreads();
    for (uint32_t c = warp; c < kInPad; c += 8u) out_t[(size_t)c * rows_cap + r0 + lane] = tile[lane][c];
}

// A chunk of n steps begins (t0 steps taken before it): what they read on the device.  One block.
__global__ void k_train_chunk(TrainDev* tr, const uint32_t* idx, const float* ys, float* loss, float4* corr, uint32_t n,
                              uint32_t t0, AdamHyper hp) {
    if (threadIdx.x == 0) {
        tr->local = 0u;
        tr->idx = idx;
        tr->ys = ys;
        tr->loss = loss;
        tr->corr = corr;
    }
    for (uint32_t s = threadIdx.x; s < n; s += blockDim.x) {
        const float t = (float)(t0 + s + 1u);
        const float c1 = 1.f - powf(hp.beta1, t), c2 = 1.f - powf(hp.beta2, t);
        corr[s] = make_float4(c1, c2, __frcp_rn(c1), __frcp_rn(c2));
    }
}
__global__ void k_step_end(TrainDev* tr, uint32_t steps) {
    tr->local += steps;
}

// BF16 copies of the master weights of member blockIdx.y (after initialisation or set_params).
__global__ void k_cast_weights(const float* __restrict__ w, __nv_bfloat16* __restrict__ wb, __nv_bfloat16* __restrict__ wtb,
                               uint32_t N, uint32_t K) {
    const size_t nw = (size_t)N * K, ow = (size_t)blockIdx.y * nw;
    w += ow; wb += ow; wtb += ow;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < nw; i += (size_t)gridDim.x * blockDim.x) {
        const __nv_bfloat16 q = __float2bfloat16_rn(w[i]);
        wb[i] = q;
        wtb[(i % K) * N + i / K] = q;
    }
}

// ---------------------------------------------------------------- host helpers
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

uint32_t round_up(uint32_t v, uint32_t a) { return (v + a - 1) / a * a; }

// splitmix64 (Steele, Lea & Flood 2014): the host stream for weight init and shuffles.
struct SplitMix {
    uint64_t s;
    uint64_t next() {
        uint64_t z = (s += 0x9E3779B97F4A7C15ull);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        return z ^ (z >> 31);
    }
    double uniform() { return (double)(next() >> 11) * (1.0 / 9007199254740992.0); }
};

}  // namespace

struct MlpLayer {
    uint32_t K = 0, N = 0;        // padded
    uint32_t k_real = 0, n_real = 0;
    // parameters, gradients and Adam moments, E members each
    float *w = nullptr, *b = nullptr, *mw = nullptr, *vw = nullptr, *mb = nullptr, *vb = nullptr;
    float *gw = nullptr, *gb = nullptr;
    __nv_bfloat16 *wb = nullptr, *wtb = nullptr;
    // training activations (batch rows, E members each; layer 0's are a chunk's minibatches)
    __nv_bfloat16 *h = nullptr, *ht = nullptr;     // input of this layer, B x K and K x B
    float* z = nullptr;                             // pre-activation output, B x N (hidden layers)
    __nv_bfloat16 *dz = nullptr, *dzt = nullptr;    // gradient at the pre-activation, B x N and N x B
    // training operands: A operands in boxes of 128 rows, B operands of 32 or 64
    CUtensorMap t_h, t_w32, t_w64, t_dzt, t_ht32, t_ht64, t_dz, t_wt32, t_wt64;
    CUtensorMap t_w;                                  // inference B operand (128 rows)
    // inference activations: the input layer's rows are shared by all members
    __nv_bfloat16* ph = nullptr;
    CUtensorMap t_ph;
};

struct epi_mlp {
    epi_mlp_config cfg{};
    uint32_t E = 1;  // members
    uint32_t L = 0, in_pad = kInPad, out_pad = 0, B = 0, sms = 0;
    std::vector<MlpLayer> layers;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    std::string err;
    int* d_err = nullptr;
    TrainDev* d_tr = nullptr;
    uint32_t adam_steps = 0;     // Adam's t of the last step
    float4* d_corr = nullptr;    // Adam's bias corrections of the chunk's steps
    float* d_t = nullptr;        // targets of a gradients call, B x out_pad (all members)
    float* d_loss = nullptr;     // per-step losses, steps x E
    size_t loss_cap = 0;
    __nv_bfloat16* d_chunk = nullptr;  // layer 0's input in both orientations
    uint32_t chunk = 0;          // steps whose minibatches layer 0's input has room for
    uint32_t chunk_most = 0;     // most steps whose minibatches are gathered at once
    uint32_t* d_idx = nullptr;   // minibatch indices of a train call, steps x E x B
    size_t idx_cap = 0;
    float* d_raw = nullptr;      // caller arrays on their way in or out
    size_t raw_cap = 0;
    __nv_bfloat16* d_xs = nullptr;  // dataset, n x 64 (bf16, padded)
    float* d_ys = nullptr;          // dataset, n x out_pad
    uint32_t n_data = 0;
    // inference
    uint32_t p_cap = 0;
    uint8_t* d_predict = nullptr; // the layers' ph, then
    float* d_py = nullptr;        // E x n x out_pad (the caller's rows before that)
    float* d_pscore = nullptr;    // E x n
    float* d_ptarget = nullptr;   // out_pad
    cudaGraphExec_t step_graph = nullptr, group_graph = nullptr;  // one step, kGroupSteps steps
    uint64_t launches = 0;
};

#define MCK(call)                                                                       \
    do {                                                                                \
        cudaError_t e_ = (call);                                                        \
        if (e_ != cudaSuccess) {                                                        \
            h->err = std::string(#call) + ": " + cudaGetErrorString(e_);                \
            return EPI_ERR_CUDA;                                                        \
        }                                                                               \
    } while (0)

namespace {

// 3-D map {cols, rows, depth} of depth stacked row-major BF16 matrices; a box is 64 columns
// x box_rows rows of one matrix.
int make_map(epi_mlp* h, CUtensorMap* map, const void* base, uint32_t rows, uint32_t cols, uint32_t box_rows,
             uint32_t depth) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) { h->err = "cuTensorMapEncodeTiled unavailable"; return EPI_ERR_CUDA; }
    const cuuint64_t dims[3] = {cols, rows, depth};
    const cuuint64_t strides[2] = {(cuuint64_t)cols * 2u, (cuuint64_t)cols * rows * 2u};
    const cuuint32_t box[3] = {(cuuint32_t)kBK, box_rows, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        h->err = "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")";
        return EPI_ERR_CUDA;
    }
    return EPI_OK;
}

// A launch that may be scheduled while the kernel before it runs (its CTAs wait on the device).
template <typename... KArgs, typename... Args>
int launch_overlapped(epi_mlp* h, void (*kern)(KArgs...), dim3 grid, int threads, uint32_t smem, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = h->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    MCK(cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...));
    h->launches++;
    return EPI_OK;
}

// One product per member (grid z = E); za = 0 when every member reads member 0's A.
template <int EP>
int gemm(epi_mlp* h, const CUtensorMap& ta, const CUtensorMap& tb, uint32_t M, uint32_t N, uint32_t K, const EpiArgs& a,
         uint32_t za = 1) {
    if (M % kBM || N % kGemmBN || K % kBK || K == 0) {
        h->err = "gemm shape " + std::to_string(M) + "x" + std::to_string(N) + "x" + std::to_string(K);
        return EPI_ERR_ARG;
    }
    return launch_overlapped(h, k_gemm<EP>, dim3(M / kBM, N / kGemmBN, h->E), kGemmThreads, kGemmSmem, ta, tb, M, N, K, a, za,
                             h->d_err);
}

// The same by k_infer, for K up to its resident panel (512); wider layers take k_gemm.  Whole
// rows per item, two blocks at a time, where the 128-row panels fill the SMs (65,536 rows x 5:
// 206 us a hidden layer, 235 a block at a time); below that one block per item (1,024 rows x 5:
// 14 us on 152 SMs; whole rows would leave 112 of them idle).  Just above the line some CTAs have
// two items and the others one: screens of 40 / 140 / 150 / 155 / 200 / 310 / 600 panels take 117 / 152 /
// 151 / 187 / 187 / 227 / 282 us, by k_gemm 146 / 206 / 214 / 223 / 243 / 313 / 504.
template <int EP>
int infer_product(epi_mlp* h, const CUtensorMap& ta, const CUtensorMap& tb, uint32_t M, uint32_t N, uint32_t K,
                  const EpiArgs& a, uint32_t za) {
    if (K / kBK > kInferMaxK) return gemm<EP>(h, ta, tb, M, N, K, a, za);
    const uint32_t panels = M / kBM * h->E, blocks = N / kInferBN;
    const uint32_t wide = panels < h->sms ? 1u : 2u, run = panels < h->sms ? 1u : blocks;
    const uint32_t items = panels * (blocks / run);
    return launch_overlapped(h, k_infer<EP>, dim3(std::min(items, h->sms)), kInferThreads, infer_smem(K / kBK), ta, tb, M, N,
                             K / kBK, wide, run, items, a, za, h->d_err);
}

#define MRC(x)                 \
    do {                       \
        int rc_ = (x);         \
        if (rc_) return rc_;   \
    } while (0)

int blocks_for(size_t n) { return (int)std::min<size_t>((n + kSmallThreads - 1) / kSmallThreads, 4096); }

int cast_all(epi_mlp* h) {
    for (auto& ly : h->layers) {
        k_cast_weights<<<dim3(blocks_for((size_t)ly.N * ly.K), h->E), kSmallThreads, 0, h->stream>>>(ly.w, ly.wb, ly.wtb,
                                                                                                     ly.N, ly.K);
        MCK(cudaGetLastError());
        h->launches++;
    }
    return EPI_OK;
}

// The forward and backward launches of one step: of the gathered chunk's step tr->local + off
// with its Adam updates, or (grads) of the one minibatch in row 0.. of the chunk buffers shared
// by all members, with targets d_t, the gradients stored in gw / gb and the losses in d_loss.
int enqueue_step(epi_mlp* h, uint32_t off, bool grads) {
    const uint32_t B = h->B, L = h->L, E = h->E;
    // Narrow tiles while a product's CTAs fit the SMs: one network's 256 x 512 product then
    // runs on 32 SMs (6.0 us a launch on one GB300).  Five networks' would take 160 CTAs, two
    // to an SM on some: 8.8 us, against 7.5 for 80 wide ones.
    auto wide = [&](uint32_t N) { return B / kBM * (N / kTrainBN) * E > h->sms; };
    // All K blocks in flight at once where a CTA has its SM to itself, else 4 (two CTAs an SM).
    auto stages_for = [&](uint32_t nk, uint32_t ctas) { return std::min(nk, ctas <= h->sms ? kTrainStages : 4u); };
    for (uint32_t l = 0; l < L; ++l) {
        MlpLayer& ly = h->layers[l];
        const bool out = l + 1 == L, w = wide(ly.N);
        const int bn = w ? kTrainWideBN : kTrainBN;
        const dim3 grid(B / kBM, ly.N / bn, E);
        ForwardArgs a{};
        a.M = B;
        a.N = ly.N;
        a.nk = ly.K / kBK;
        a.stages = stages_for(a.nk, grid.x * grid.y * grid.z);
        a.first = l == 0;
        a.shared_a = l == 0 && grads;
        a.off = off;
        a.bias = ly.b;
        a.z = ly.z;
        a.out = out ? ly.dz : h->layers[l + 1].h;
        a.out_t = out ? ly.dzt : h->layers[l + 1].ht;
        if (out) {
            a.target = grads ? h->d_t : nullptr;
            a.loss = grads ? h->d_loss : nullptr;
            a.n_valid = h->cfg.out_dim;
            a.grad_scale = 2.0f / ((float)B * (float)h->cfg.out_dim);
        }
        auto kern = out ? (w ? k_forward<true, kTrainWideBN> : k_forward<true, kTrainBN>)
                        : (w ? k_forward<false, kTrainWideBN> : k_forward<false, kTrainBN>);
        MRC(launch_overlapped(h, kern, grid, kTrainThreads, train_smem(bn, a.stages), ly.t_h, w ? ly.t_w64 : ly.t_w32, a,
                              (const TrainDev*)h->d_tr, h->d_err));
    }
    auto weight_job = [&](BackwardArgs& a, BackwardMaps& maps, int slot, uint32_t l, bool wide_w) {
        MlpLayer& ly = h->layers[l];
        WeightGrad& w = a.dw[slot];
        w.tiles = ly.N / kBM * (ly.K / (wide_w ? kTrainWideBN : kTrainBN));
        w.bias_blocks = (ly.N + kBiasRows - 1) / kBiasRows;
        w.N = ly.N;
        w.K = ly.K;
        w.nk = B / kBK;
        w.B = B;
        w.first = l == 0;
        w.shared_h = l == 0 && grads;
        w.w = ly.w; w.mw = ly.mw; w.vw = ly.vw;
        w.b = ly.b; w.mb = ly.mb; w.vb = ly.vb;
        w.wb = ly.wb; w.wtb = ly.wtb;
        w.dzt = ly.dzt;
        w.gw = grads ? ly.gw : nullptr;
        w.gb = grads ? ly.gb : nullptr;
        maps.dw_a[slot] = ly.t_dzt;
        maps.dw_b[slot] = wide_w ? ly.t_ht64 : ly.t_ht32;
    };
    // launch l computes dZ_{l-1} from dZ_l; W_{l+1}, whose last reader was the launch before,
    // takes its update beside it; the last launch has those of layers 1 and 0
    for (uint32_t l = L - 1; l + 1 > 0; --l) {
        BackwardArgs a{};
        BackwardMaps maps;
        std::memset(&maps, 0, sizeof maps);
        a.off = off;
        a.grads = grads;
        a.hp = AdamHyper{h->cfg.lr, h->cfg.beta1, h->cfg.beta2, h->cfg.eps};
        const bool w = l > 0 && wide(h->layers[l].K);
        // weight gradients: narrow while a hidden layer's fit two to an SM (200 steps on one
        // GB300, narrow / wide: 3 networks 12.4 / 12.4 ms, 8 networks 27.4 / 28.2, 16 networks
        // 46.8 / 44.9); in the last launch, which has nothing beside them, while they fit three
        // times (5 networks 19.3 / 20.5, 10 networks 32.3 / 33.1, 16 networks 45.2 / 44.9)
        const uint32_t narrow = h->cfg.hidden / kBM * (h->cfg.hidden / kTrainBN) * E;
        const bool ww = narrow > (l > 0 ? 2u : 6u) * h->sms;
        const int bn = w ? kTrainWideBN : kTrainBN;
        if (l > 0) {
            MlpLayer &ly = h->layers[l], &pv = h->layers[l - 1];
            a.dx.tiles = B / kBM * (ly.K / bn);
            a.dx.M = B;
            a.dx.N = ly.K;
            a.dx.nk = ly.N / kBK;
            a.dx.z = pv.z;
            a.dx.out = pv.dz;
            a.dx.out_t = pv.dzt;
            maps.dx_a = ly.t_dz;
            maps.dx_b = w ? ly.t_wt64 : ly.t_wt32;
            if (l + 1 < L) weight_job(a, maps, 0, l + 1, ww);
        } else {
            weight_job(a, maps, 0, 1, ww);
            weight_job(a, maps, 1, 0, ww);
        }
        const uint32_t blocks = a.dx.tiles + a.dw[0].tiles + a.dw[1].tiles + a.dw[0].bias_blocks + a.dw[1].bias_blocks;
        a.stages = stages_for(std::max(a.dx.nk, B / kBK), blocks * E);
        auto kern = w ? (ww ? k_backward<kTrainWideBN, kTrainWideBN> : k_backward<kTrainWideBN, kTrainBN>)
                      : (ww ? k_backward<kTrainBN, kTrainWideBN> : k_backward<kTrainBN, kTrainBN>);
        MRC(launch_overlapped(h, kern, dim3(blocks, E), kTrainThreads, train_smem(w || ww ? kTrainWideBN : kTrainBN, a.stages), maps, a,
                              (const TrainDev*)h->d_tr, h->d_err));
    }
    return EPI_OK;
}

// Adam steps of a captured group, so that the gap between graph launches is paid once in four.
constexpr uint32_t kGroupSteps = 4;

int step_graph(epi_mlp* h, uint32_t steps, cudaGraphExec_t* out) {
    if (*out) return EPI_OK;
    cudaGraph_t g;
    MCK(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    int rc = EPI_OK;
    for (uint32_t k = 0; k < steps && !rc; ++k) rc = enqueue_step(h, k, false);
    if (!rc) k_step_end<<<1, 1, 0, h->stream>>>(h->d_tr, steps);
    cudaError_t ce = cudaStreamEndCapture(h->stream, &g);
    if (rc) return rc;
    if (ce == cudaSuccess) {
        ce = cudaGraphInstantiate(out, g, 0);
        cudaGraphDestroy(g);
    }
    if (ce != cudaSuccess) { *out = nullptr; h->err = std::string("training graph: ") + cudaGetErrorString(ce); return EPI_ERR_CUDA; }
    return EPI_OK;
}

void drop_graphs(epi_mlp* h) {
    for (cudaGraphExec_t* g : {&h->step_graph, &h->group_graph}) {
        if (*g) cudaGraphExecDestroy(*g);
        *g = nullptr;
    }
}

// Device space for `floats` caller values.
int ensure_raw(epi_mlp* h, size_t floats) {
    if (floats <= h->raw_cap) return EPI_OK;
    MCK(cudaStreamSynchronize(h->stream));
    cudaFree(h->d_raw);
    h->d_raw = nullptr;
    h->raw_cap = 0;
    MCK(cudaMalloc(&h->d_raw, floats * sizeof(float)));
    h->raw_cap = floats;
    return EPI_OK;
}

int check_err(epi_mlp* h) {
    int e = 0;
    MCK(cudaMemcpyAsync(&e, h->d_err, sizeof e, cudaMemcpyDeviceToHost, h->stream));
    MCK(cudaStreamSynchronize(h->stream));
    if (e) {
        h->err = "tensor-core product: a bounded wait expired (flag " + std::to_string(e) + ")";
        MCK(cudaMemsetAsync(h->d_err, 0, sizeof(int), h->stream));
        return EPI_ERR_TIMEOUT;
    }
    return EPI_OK;
}

// n caller rows of in_dim floats into BF16 rows of kInPad on the device (n_rows of them).
int upload_inputs(epi_mlp* h, const float* x, uint32_t n, uint32_t n_rows, float* stage, __nv_bfloat16* out,
                  __nv_bfloat16* xt = nullptr, uint32_t xt_pitch = 0) {
    const size_t floats = (size_t)n * h->cfg.in_dim;
    if (!stage) {
        MRC(ensure_raw(h, floats));
        stage = h->d_raw;
    }
    MCK(cudaMemcpyAsync(stage, x, floats * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    k_pad_inputs<<<blocks_for((size_t)n_rows * (kInPad / 2)), kSmallThreads, 0, h->stream>>>(stage, n, n_rows,
                                                                                            h->cfg.in_dim, out, xt, xt_pitch);
    MCK(cudaGetLastError());
    h->launches++;
    return EPI_OK;
}

// n caller rows of out_dim floats into rows of out_pad on the device.
int upload_targets(epi_mlp* h, const float* y, uint32_t n, float* out) {
    const size_t floats = (size_t)n * h->cfg.out_dim;
    MRC(ensure_raw(h, floats));
    MCK(cudaMemcpyAsync(h->d_raw, y, floats * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    k_pad_rows<<<blocks_for((size_t)n * h->out_pad), kSmallThreads, 0, h->stream>>>(h->d_raw, n, h->cfg.out_dim, h->out_pad,
                                                                                   out);
    MCK(cudaGetLastError());
    h->launches++;
    return EPI_OK;
}

int ensure_predict(epi_mlp* h, uint32_t n_pad) {
    if (n_pad <= h->p_cap) return EPI_OK;
    cudaFree(h->d_predict);
    h->d_predict = nullptr;
    h->p_cap = 0;
    // one allocation for all of them (a first call of a few rows is mostly allocations)
    size_t bytes = 0;
    auto take = [&](size_t b) {
        const size_t at = bytes;
        bytes += (b + 255u) / 256u * 256u;
        return at;
    };
    std::vector<size_t> ph(h->L);
    for (uint32_t l = 0; l < h->L; ++l) ph[l] = take((size_t)(l == 0 ? 1u : h->E) * n_pad * h->layers[l].K * sizeof(__nv_bfloat16));
    const size_t py = take((size_t)h->E * n_pad * h->out_pad * sizeof(float)), ps = take((size_t)h->E * n_pad * sizeof(float));
    MCK(cudaMalloc(&h->d_predict, bytes));
    for (uint32_t l = 0; l < h->L; ++l) {
        MlpLayer& ly = h->layers[l];
        ly.ph = reinterpret_cast<__nv_bfloat16*>(h->d_predict + ph[l]);
        MRC(make_map(h, &ly.t_ph, ly.ph, n_pad, ly.K, kBM, l == 0 ? 1u : h->E));
    }
    h->d_py = reinterpret_cast<float*>(h->d_predict + py);
    h->d_pscore = reinterpret_cast<float*>(h->d_predict + ps);
    h->p_cap = n_pad;
    return EPI_OK;
}

// Whether the last product leaves the rows in d_py as the caller has them ([member][n][out_dim]):
// k_infer stores 32 bytes at a time, so out_dim is a multiple of 8.  Else they have out_pad columns
// and p_cap rows a member, and k_unpad_rows makes a copy for the caller.
bool outputs_as_asked(const epi_mlp* h) { return h->cfg.out_dim % 8u == 0u && h->layers[h->L - 1].K / kBK <= kInferMaxK; }

// Forward pass of n host samples through every member; outputs stay in d_py (and scores in
// d_pscore when target).  The buffers hold p_cap rows per member (the largest call so far):
// member m's rows start at m * p_cap in every buffer and tensor map, whatever n is.
int forward_n(epi_mlp* h, const float* x, uint32_t n, const float* target) {
    const uint32_t n_pad = std::max<uint32_t>(round_up(n, kBM), kBM);
    MRC(ensure_predict(h, n_pad));
    const uint64_t cap = h->p_cap;
    // (the outputs' buffer, unused until the last layer, holds the caller's rows: in_dim <= 64 < out_pad)
    MRC(upload_inputs(h, x, n, n_pad, h->d_py, h->layers[0].ph));
    if (target) {
        MCK(cudaMemcpyAsync(h->d_ptarget, target, h->cfg.out_dim * sizeof(float), cudaMemcpyHostToDevice, h->stream));
        MCK(cudaMemsetAsync(h->d_pscore, 0, (size_t)h->E * cap * sizeof(float), h->stream));
    }
    for (uint32_t l = 0; l < h->L; ++l) {
        MlpLayer& ly = h->layers[l];
        EpiArgs a;
        a.bias = ly.b;
        a.ms_bias = ly.N;
        const uint32_t za = l == 0 ? 0u : 1u;  // the input rows are shared
        if (l + 1 < h->L) {
            a.out = h->layers[l + 1].ph;
            a.ms_out = cap * ly.N;
            MRC(infer_product<kEpHidden>(h, ly.t_ph, ly.t_w, n_pad, ly.N, ly.K, a, za));
        } else {
            a.outf = target ? nullptr : h->d_py;
            a.score_target = target ? h->d_ptarget : nullptr;
            a.score = target ? h->d_pscore : nullptr;
            a.n_valid = h->cfg.out_dim;
            a.m_valid = n;
            a.ld_outf = outputs_as_asked(h) ? h->cfg.out_dim : ly.N;
            a.ms_outf = outputs_as_asked(h) ? (uint64_t)n * h->cfg.out_dim : cap * ly.N;
            a.ms_score = cap;
            MRC(infer_product<kEpOut>(h, ly.t_ph, ly.t_w, n_pad, ly.N, ly.K, a, za));
        }
    }
    return EPI_OK;
}

void free_all(epi_mlp* h) {
    drop_graphs(h);
    for (auto& ly : h->layers) {
        cudaFree(ly.w); cudaFree(ly.b); cudaFree(ly.mw); cudaFree(ly.vw); cudaFree(ly.mb); cudaFree(ly.vb);
        cudaFree(ly.gw); cudaFree(ly.gb); cudaFree(ly.wb); cudaFree(ly.wtb);
        if (&ly != &h->layers[0]) {  // (layer 0's lie in d_chunk)
            cudaFree(ly.h);
            cudaFree(ly.ht);
        }
        cudaFree(ly.z); cudaFree(ly.dz); cudaFree(ly.dzt);
    }
    cudaFree(h->d_chunk);
    cudaFree(h->d_err); cudaFree(h->d_tr); cudaFree(h->d_t); cudaFree(h->d_loss);
    cudaFree(h->d_idx); cudaFree(h->d_raw); cudaFree(h->d_corr);
    cudaFree(h->d_xs); cudaFree(h->d_ys); cudaFree(h->d_predict); cudaFree(h->d_ptarget);
    if (h->own_stream && h->stream) cudaStreamDestroy(h->stream);
}

// The operands that lie in a layer's input (rows of it a member).
int input_maps(epi_mlp* h, MlpLayer& ly, uint32_t rows) {
    MRC(make_map(h, &ly.t_h, ly.h, rows, ly.K, kBM, h->E));
    MRC(make_map(h, &ly.t_ht32, ly.ht, ly.K, rows, kTrainBN, h->E));
    MRC(make_map(h, &ly.t_ht64, ly.ht, ly.K, rows, kTrainWideBN, h->E));
    return EPI_OK;
}

// Room for the minibatches of so many steps in layer 0's input (nothing of the handle runs): one at
// first, for gradients, and as many as a training call gathers at once from that call on, so that
// handles that only predict do without (five members, batch 256: 42 MB).
int ensure_chunk(epi_mlp* h, uint32_t steps) {
    if (steps <= h->chunk) return EPI_OK;
    MlpLayer& ly = h->layers[0];
    drop_graphs(h);  // they bake the maps in
    cudaFree(h->d_chunk);
    h->d_chunk = nullptr;
    h->chunk = 0;
    const size_t elements = (size_t)h->E * steps * h->B * ly.K;  // (a multiple of 128 x 64)
    MCK(cudaMalloc(&h->d_chunk, 2 * elements * sizeof(__nv_bfloat16)));
    ly.h = h->d_chunk;
    ly.ht = h->d_chunk + elements;
    MRC(input_maps(h, ly, steps * h->B));
    h->chunk = steps;
    return EPI_OK;
}

int init(epi_mlp* h) {
    const epi_mlp_config& c = h->cfg;
    for (const void* k : {(const void*)k_gemm<kEpHidden>, (const void*)k_gemm<kEpOut>})
        MCK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmem));
    for (const void* k : {(const void*)k_infer<kEpHidden>, (const void*)k_infer<kEpOut>})
        MCK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)infer_smem(kInferMaxK)));
    for (const void* k : {(const void*)k_forward<false, kTrainBN>, (const void*)k_forward<false, kTrainWideBN>,
                          (const void*)k_forward<true, kTrainBN>, (const void*)k_forward<true, kTrainWideBN>,
                          (const void*)k_backward<kTrainBN, kTrainBN>, (const void*)k_backward<kTrainBN, kTrainWideBN>,
                          (const void*)k_backward<kTrainWideBN, kTrainBN>, (const void*)k_backward<kTrainWideBN, kTrainWideBN>})
        MCK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)train_smem(kTrainWideBN, kTrainStages)));
    int dev = 0, sms = 0;
    MCK(cudaGetDevice(&dev));
    MCK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    h->sms = (uint32_t)sms;
    const uint32_t E = h->E;
    h->L = c.hidden_layers + 1;
    h->B = c.batch;
    h->out_pad = round_up(c.out_dim, 128);
    MCK(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking));
    h->own_stream = true;
    MCK(cudaMalloc(&h->d_err, sizeof(int)));
    MCK(cudaMalloc(&h->d_tr, sizeof(TrainDev)));
    MCK(cudaMemset(h->d_err, 0, sizeof(int)));
    MCK(cudaMemset(h->d_tr, 0, sizeof(TrainDev)));
    MCK(cudaMalloc(&h->d_t, (size_t)h->B * h->out_pad * sizeof(float)));
    // steps gathered at once: up to 128, within 32 MB of inputs in each orientation
    h->chunk_most = (uint32_t)std::min<size_t>(128, std::max<size_t>(kGroupSteps, (32u << 20) / ((size_t)E * h->B * kInPad * 2)));
    h->chunk_most -= h->chunk_most % kGroupSteps;
    MCK(cudaMalloc(&h->d_corr, h->chunk_most * sizeof(float4)));
    MCK(cudaMalloc(&h->d_ptarget, (size_t)h->out_pad * sizeof(float)));
    h->layers.resize(h->L);
    for (uint32_t l = 0; l < h->L; ++l) {
        MlpLayer& ly = h->layers[l];
        ly.k_real = l == 0 ? c.in_dim : c.hidden;
        ly.n_real = l + 1 == h->L ? c.out_dim : c.hidden;
        ly.K = l == 0 ? kInPad : c.hidden;
        ly.N = l + 1 == h->L ? h->out_pad : c.hidden;
        const size_t nw = (size_t)E * ly.N * ly.K, nb = (size_t)E * ly.N, act_in = (size_t)E * h->B * ly.K,
                     act_out = (size_t)E * h->B * ly.N;
        for (float** p : {&ly.w, &ly.mw, &ly.vw, &ly.gw}) MCK(cudaMalloc(p, nw * sizeof(float)));
        for (float** p : {&ly.b, &ly.mb, &ly.vb, &ly.gb}) MCK(cudaMalloc(p, nb * sizeof(float)));
        MCK(cudaMalloc(&ly.wb, nw * sizeof(__nv_bfloat16)));
        MCK(cudaMalloc(&ly.wtb, nw * sizeof(__nv_bfloat16)));
        if (l == 0) {
            MRC(ensure_chunk(h, 1));
        } else {
            MCK(cudaMalloc(&ly.h, act_in * sizeof(__nv_bfloat16)));
            MCK(cudaMalloc(&ly.ht, act_in * sizeof(__nv_bfloat16)));
            MRC(input_maps(h, ly, h->B));
        }
        if (l + 1 < h->L) MCK(cudaMalloc(&ly.z, act_out * sizeof(float)));
        MCK(cudaMalloc(&ly.dz, act_out * sizeof(__nv_bfloat16)));
        MCK(cudaMalloc(&ly.dzt, act_out * sizeof(__nv_bfloat16)));
        for (float* p : {ly.mw, ly.vw, ly.gw}) MCK(cudaMemset(p, 0, nw * sizeof(float)));
        for (float* p : {ly.mb, ly.vb, ly.gb}) MCK(cudaMemset(p, 0, nb * sizeof(float)));
        // operands (and input_maps): forward A = h (B x K), B = W (N x K); weights A = dZ^T (N x B),
        // B = H^T (K x B); inputs A = dZ (B x N), B = W^T (K x N)
        MRC(make_map(h, &ly.t_w, ly.wb, ly.N, ly.K, 128, E));
        MRC(make_map(h, &ly.t_w32, ly.wb, ly.N, ly.K, kTrainBN, E));
        MRC(make_map(h, &ly.t_w64, ly.wb, ly.N, ly.K, kTrainWideBN, E));
        MRC(make_map(h, &ly.t_dzt, ly.dzt, ly.N, h->B, kBM, E));
        MRC(make_map(h, &ly.t_dz, ly.dz, h->B, ly.N, kBM, E));
        MRC(make_map(h, &ly.t_wt32, ly.wtb, ly.K, ly.N, kTrainBN, E));
        MRC(make_map(h, &ly.t_wt64, ly.wtb, ly.K, ly.N, kTrainWideBN, E));
    }
    // torch.nn.Linear's default: W and b uniform in +-1/sqrt(fan_in); member m draws from
    // seed + m, layer by layer (W row by row, then b)
    for (uint32_t m = 0; m < E; ++m) {
        SplitMix rng{c.seed + m};
        for (auto& ly : h->layers) {
            const size_t nw = (size_t)ly.N * ly.K;
            const double bound = 1.0 / std::sqrt((double)ly.k_real);
            std::vector<float> w(nw, 0.f), b(ly.N, 0.f);
            for (uint32_t n = 0; n < ly.n_real; ++n)
                for (uint32_t k = 0; k < ly.k_real; ++k) w[(size_t)n * ly.K + k] = (float)((2.0 * rng.uniform() - 1.0) * bound);
            for (uint32_t n = 0; n < ly.n_real; ++n) b[n] = (float)((2.0 * rng.uniform() - 1.0) * bound);
            MCK(cudaMemcpy(ly.w + m * nw, w.data(), nw * sizeof(float), cudaMemcpyHostToDevice));
            MCK(cudaMemcpy(ly.b + (size_t)m * ly.N, b.data(), ly.N * sizeof(float), cudaMemcpyHostToDevice));
        }
    }
    MRC(cast_all(h));
    MCK(cudaStreamSynchronize(h->stream));
    return EPI_OK;
}

uint64_t member_params(const epi_mlp* h) {
    uint64_t n = 0;
    for (auto& ly : h->layers) n += (uint64_t)ly.n_real * ly.k_real + ly.n_real;
    return n;
}

// Every layer's arrays (E padded members each) <-> the member-major unpadded layout in d_raw.
int move_params(epi_mlp* h, float* const MlpLayer::*wp, float* const MlpLayer::*bp, bool to_flat) {
    const uint64_t count = member_params(h);
    size_t o = 0;
    for (auto& ly : h->layers) {
        const size_t total = (size_t)ly.n_real * ly.k_real + ly.n_real;
        k_params<<<dim3(blocks_for(total), h->E), kSmallThreads, 0, h->stream>>>(h->d_raw, count, o, ly.n_real, ly.k_real,
                                                                                ly.*wp, ly.*bp, ly.N, ly.K, to_flat);
        MCK(cudaGetLastError());
        h->launches++;
        o += total;
    }
    return EPI_OK;
}
int download_params(epi_mlp* h, float* const MlpLayer::*wp, float* const MlpLayer::*bp, float* out) {
    const size_t floats = (size_t)member_params(h) * h->E;
    MRC(ensure_raw(h, floats));
    MRC(move_params(h, wp, bp, true));
    epi::touch_pages(out, floats * sizeof(float));
    MCK(cudaMemcpyAsync(out, h->d_raw, floats * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    MCK(cudaStreamSynchronize(h->stream));
    return EPI_OK;
}

}  // namespace

// ---------------------------------------------------------------- C ABI
extern "C" {

int epi_mlp_create(const epi_mlp_config* cfg, epi_mlp** out) {
    if (!cfg || !out) return EPI_ERR_ARG;
    *out = nullptr;
    if (cfg->in_dim == 0 || cfg->in_dim > kInPad || cfg->hidden == 0 || cfg->hidden % 128 || cfg->hidden_layers == 0 ||
        cfg->out_dim == 0 || cfg->batch == 0 || cfg->batch % 128 || !(cfg->lr > 0.f) || cfg->members > kMaxMembers)
        return EPI_ERR_CONFIG;
    epi_mlp* h = new epi_mlp();
    h->cfg = *cfg;
    h->E = cfg->members ? cfg->members : 1u;
    h->cfg.members = h->E;
    int rc = init(h);
    // on failure the handle is kept so that the caller can read the message, then destroy it
    *out = h;
    return rc;
}

int epi_mlp_destroy(epi_mlp* h) {
    if (!h) return EPI_OK;
    if (h->stream) cudaStreamSynchronize(h->stream);
    free_all(h);
    delete h;
    return EPI_OK;
}

const char* epi_mlp_last_error(const epi_mlp* h) { return h ? h->err.c_str() : "null handle"; }

int epi_mlp_set_stream(epi_mlp* h, void* cuda_stream) {
    if (!h) return EPI_ERR_ARG;
    MCK(cudaStreamSynchronize(h->stream));
    if (h->own_stream) cudaStreamDestroy(h->stream);
    h->stream = static_cast<cudaStream_t>(cuda_stream);
    h->own_stream = false;
    drop_graphs(h);
    return EPI_OK;
}

int epi_mlp_members(const epi_mlp* h, uint32_t* out) {
    if (!h || !out) return EPI_ERR_ARG;
    *out = h->E;
    return EPI_OK;
}

int epi_mlp_param_count(const epi_mlp* h, uint64_t* out) {
    if (!h || !out) return EPI_ERR_ARG;
    *out = member_params(h);
    return EPI_OK;
}

int epi_mlp_get_params(epi_mlp* h, float* out) {
    if (!h || !out) return EPI_ERR_ARG;
    MCK(cudaStreamSynchronize(h->stream));
    return download_params(h, &MlpLayer::w, &MlpLayer::b, out);
}

int epi_mlp_set_params(epi_mlp* h, const float* in) {
    if (!h || !in) return EPI_ERR_ARG;
    MCK(cudaStreamSynchronize(h->stream));
    const size_t floats = (size_t)member_params(h) * h->E;
    MRC(ensure_raw(h, floats));
    MCK(cudaMemcpyAsync(h->d_raw, in, floats * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    MRC(move_params(h, &MlpLayer::w, &MlpLayer::b, false));
    for (auto& ly : h->layers) {
        const size_t nw = (size_t)h->E * ly.N * ly.K * sizeof(float), nb = (size_t)h->E * ly.N * sizeof(float);
        for (float* p : {ly.mw, ly.vw}) MCK(cudaMemsetAsync(p, 0, nw, h->stream));
        for (float* p : {ly.mb, ly.vb}) MCK(cudaMemsetAsync(p, 0, nb, h->stream));
    }
    h->adam_steps = 0;
    MRC(cast_all(h));
    MCK(cudaStreamSynchronize(h->stream));
    return EPI_OK;
}

int epi_mlp_set_dataset(epi_mlp* h, const float* x, const float* y, uint32_t n) {
    if (!h || !x || !y || n == 0) return EPI_ERR_ARG;
    MCK(cudaStreamSynchronize(h->stream));
    cudaFree(h->d_xs);
    cudaFree(h->d_ys);
    h->d_xs = nullptr;
    h->d_ys = nullptr;
    h->n_data = 0;
    MCK(cudaMalloc(&h->d_xs, (size_t)n * kInPad * sizeof(__nv_bfloat16)));
    MCK(cudaMalloc(&h->d_ys, (size_t)n * h->out_pad * sizeof(float)));
    MRC(upload_inputs(h, x, n, n, nullptr, h->d_xs));
    MRC(upload_targets(h, y, n, h->d_ys));
    MCK(cudaStreamSynchronize(h->stream));
    h->n_data = n;
    return EPI_OK;
}

int epi_mlp_train(epi_mlp* h, uint32_t steps, uint64_t shuffle_seed, float* losses) {
    if (!h) return EPI_ERR_ARG;
    if (steps == 0) return EPI_OK;
    if (h->n_data < h->B) { h->err = "training set smaller than one minibatch"; return EPI_ERR_ARG; }
    const uint32_t E = h->E, B = h->B;
    // minibatch indices: member m shuffles from shuffle_seed + m, a fresh permutation every
    // epoch, whole batches only
    const uint32_t per_epoch = h->n_data / B;
    std::vector<uint32_t> idx((size_t)E * steps * B), perm(h->n_data);
    for (uint32_t m = 0; m < E; ++m) {
        SplitMix rng{shuffle_seed + m};
        for (uint32_t s = 0; s < steps; ++s) {
            if (s % per_epoch == 0) {
                for (uint32_t i = 0; i < h->n_data; ++i) perm[i] = i;
                for (uint32_t i = h->n_data - 1; i > 0; --i) std::swap(perm[i], perm[rng.next() % (i + 1)]);  // Fisher-Yates
            }
            std::memcpy(&idx[((size_t)s * E + m) * B], &perm[(size_t)(s % per_epoch) * B], B * sizeof(uint32_t));
        }
    }
    MCK(cudaStreamSynchronize(h->stream));
    if (idx.size() > h->idx_cap) {
        cudaFree(h->d_idx);
        h->d_idx = nullptr;
        h->idx_cap = 0;
        MCK(cudaMalloc(&h->d_idx, idx.size() * sizeof(uint32_t)));
        h->idx_cap = idx.size();
    }
    if ((size_t)steps * E > h->loss_cap) {
        cudaFree(h->d_loss);
        h->d_loss = nullptr;
        h->loss_cap = 0;
        MCK(cudaMalloc(&h->d_loss, (size_t)steps * E * sizeof(float)));
        h->loss_cap = (size_t)steps * E;
    }
    MRC(ensure_chunk(h, round_up(std::min(steps, h->chunk_most), kGroupSteps)));
    MCK(cudaMemcpyAsync(h->d_idx, idx.data(), idx.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, h->stream));
    MCK(cudaMemsetAsync(h->d_loss, 0, (size_t)steps * E * sizeof(float), h->stream));
    if (steps >= kGroupSteps) MRC(step_graph(h, kGroupSteps, &h->group_graph));
    if (steps % kGroupSteps) MRC(step_graph(h, 1, &h->step_graph));
    const AdamHyper hp{h->cfg.lr, h->cfg.beta1, h->cfg.beta2, h->cfg.eps};
    for (uint32_t s0 = 0; s0 < steps; s0 += h->chunk) {
        const uint32_t n = std::min(h->chunk, steps - s0);
        const uint32_t* idx0 = h->d_idx + (size_t)s0 * E * B;
        k_train_chunk<<<1, 128, 0, h->stream>>>(h->d_tr, idx0, h->d_ys, h->d_loss + (size_t)s0 * E, h->d_corr, n,
                                                h->adam_steps, hp);
        h->adam_steps += n;  // Adam's t keeps counting across calls
        k_gather<<<dim3(n * B / 32u, E), 256, 0, h->stream>>>(h->d_xs, idx0, B, h->chunk * B, h->layers[0].h,
                                                              h->layers[0].ht);
        MCK(cudaGetLastError());
        for (uint32_t k = 0; k < n;) {
            const uint32_t g = n - k >= kGroupSteps ? kGroupSteps : 1u;
            MCK(cudaGraphLaunch(g == kGroupSteps ? h->group_graph : h->step_graph, h->stream));
            h->launches += 2 * (uint64_t)h->L * g + 1;
            k += g;
        }
        h->launches += 2;
    }
    MRC(check_err(h));
    if (losses) {
        std::vector<float> l((size_t)steps * E);
        MCK(cudaMemcpy(l.data(), h->d_loss, l.size() * sizeof(float), cudaMemcpyDeviceToHost));
        const float inv = 1.0f / ((float)B * (float)h->cfg.out_dim);
        for (uint32_t m = 0; m < E; ++m)
            for (uint32_t s = 0; s < steps; ++s) losses[(size_t)m * steps + s] = l[(size_t)s * E + m] * inv;
    }
    return EPI_OK;
}

int epi_mlp_gradients(epi_mlp* h, const float* x, const float* y, uint32_t n, float* grads, float* loss) {
    if (!h || !x || !y || !grads) return EPI_ERR_ARG;
    if (n != h->B) { h->err = "gradients take exactly one minibatch"; return EPI_ERR_ARG; }
    MCK(cudaStreamSynchronize(h->stream));
    const uint32_t E = h->E;
    MRC(ensure_chunk(h, 1));
    MlpLayer& l0 = h->layers[0];
    // every member sees the same minibatch: row 0.. of the chunk buffers, member 0's
    MRC(upload_inputs(h, x, n, n, nullptr, l0.h, l0.ht, h->chunk * h->B));
    MRC(upload_targets(h, y, n, h->d_t));
    if (E > h->loss_cap) {
        cudaFree(h->d_loss);
        h->d_loss = nullptr;
        h->loss_cap = 0;
        MCK(cudaMalloc(&h->d_loss, E * sizeof(float)));
        h->loss_cap = E;
    }
    MCK(cudaMemsetAsync(h->d_loss, 0, E * sizeof(float), h->stream));
    MRC(enqueue_step(h, 0, true));
    std::vector<float> lsum(E, 0.f);
    MCK(cudaMemcpyAsync(lsum.data(), h->d_loss, E * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    MRC(check_err(h));
    if (loss)
        for (uint32_t m = 0; m < E; ++m) loss[m] = lsum[m] / ((float)n * (float)h->cfg.out_dim);
    return download_params(h, &MlpLayer::gw, &MlpLayer::gb, grads);
}

int epi_mlp_predict(epi_mlp* h, const float* x, uint32_t n, float* y) {
    if (!h || !x || !y) return EPI_ERR_ARG;
    if (n == 0) return EPI_OK;
    MRC(forward_n(h, x, n, nullptr));
    const size_t floats = (size_t)h->E * n * h->cfg.out_dim;
    const float* rows = h->d_py;
    if (!outputs_as_asked(h)) {
        MRC(ensure_raw(h, floats));
        k_unpad_rows<<<dim3(blocks_for((size_t)n * h->cfg.out_dim), h->E), kSmallThreads, 0, h->stream>>>(
            h->d_py, n, h->cfg.out_dim, h->out_pad, (size_t)h->p_cap * h->out_pad, h->d_raw);
        MCK(cudaGetLastError());
        h->launches++;
        rows = h->d_raw;
    }
    epi::touch_pages(y, floats * sizeof(float));
    MCK(cudaMemcpyAsync(y, rows, floats * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    MRC(check_err(h));
    return EPI_OK;
}

int epi_mlp_score(epi_mlp* h, const float* x, uint32_t n, const float* target, float* score) {
    if (!h || !x || !target || !score) return EPI_ERR_ARG;
    if (n == 0) return EPI_OK;
    MRC(forward_n(h, x, n, target));
    epi::touch_pages(score, (size_t)h->E * n * sizeof(float));
    MRC(check_err(h));
    for (uint32_t m = 0; m < h->E; ++m)
        MCK(cudaMemcpy(score + (size_t)m * n, h->d_pscore + (size_t)m * h->p_cap, (size_t)n * sizeof(float),
                       cudaMemcpyDeviceToHost));
    return EPI_OK;
}

int epi_mlp_kernels_launched(const epi_mlp* h, uint64_t* out) {
    if (!h || !out) return EPI_ERR_ARG;
    *out = h->launches;
    return EPI_OK;
}

}  // extern "C"
