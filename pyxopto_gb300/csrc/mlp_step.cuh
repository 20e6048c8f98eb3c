/*
 * mlp_step.cuh - one training step of the surrogate MLP as a chain of nine
 * launches for four layers.  Included by mlp.cu inside its anonymous
 * namespace, after mlp_tc.cuh and adamw_element.
 *
 * What bounds a step is latency: 3.4 GFLOP and 6 MB of weights and moments
 * are 2 us, but a launch that depends on the one before costs 3 to 5 us, and
 * the step was 26 of them, each called from Python.  So each pass over the
 * activations is fused into the GEMM that produces them, the weight gradients
 * of all layers are one launch, their slice sums, the bias and loss sums,
 * the tied columns and AdamW another, and every launch sets itself up
 * (barriers, TMEM) while the one before still runs (programmatic dependent
 * launch):
 *   step_forward   per layer: X W^T + b, pre-activation and GELU; the last
 *                  layer goes on to the loss, its gradient and their sums
 *   step_backward  per hidden layer: dPre W, times GELU', and column sums
 *   step_weights   every layer: dPre^T X over slices of the rows
 *   step_update    slice sums, tied columns, AdamW, bf16 and transposed copies
 * The products, roundings, formulas and sums are those of the separate
 * kernels, bit for bit; only the loss is summed in another order.
 * A step, the Python call included: batch 256 205 -> 53 us, 4096 208 -> 87 us,
 * 16384 296 -> 236 us.  A block and partial sum for each of the separate
 * kernel's slices (32 to 64 a layer, 18 MB of partial sums at 4096) cost 30 us
 * more; other sums (slices as long as fill the SMs once) 27 us less at 16384
 * and nothing at 4096, but biases that differ by an ulp flip bf16 roundings
 * of the next step.
 */
#pragma once

constexpr int STEP_MAX_LAYERS = MCGB_ADAMW_MAX_TENSORS / 2;

/* Column sums of a 128 x BN tile of dPre that the block has written to shared
   memory ([row][column], rows of BN + 1), as act_bwd_kernel takes them: for
   each 64 rows the sums over rows 8 apart, then those eight in order. */
template <int BN>
__device__ __forceinline__ void store_columns(float *tile, float *part, int r0, int c0, int ldc, int R) {
    float *red = tile + TBM * (BN + 1);   /* [chunk][row mod 8][column] */
    __syncthreads();
    for (int e = threadIdx.x; e < 16 * BN; e += TNT) {
        const int c = e % BN, row = e / BN / 8 * 64 + e / BN % 8;
        float s = 0.0f;
#pragma unroll
        for (int q = 0; q < 8; ++q) s += tile[(row + 8 * q) * (BN + 1) + c];
        red[e] = s;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 2 * BN; e += TNT) {
        const int c = e % BN, row = r0 + e / BN * 64;
        float t = 0.0f;
#pragma unroll
        for (int q = 0; q < 8; ++q) t += red[(e / BN * 8 + q) * BN + c];
        if (row < R && c0 + c < ldc) part[(size_t)(row / 64) * ldc + c0 + c] = t;
    }
}

/* The shared memory of the operand stages, free once the product is done. */
template <int BN>
__device__ __forceinline__ float *step_tile(uint8_t *tc_smem) {
    static_assert((TBM * (BN + 1) + 16 * BN) * 4 <= TcShape<BN>::BARS, "column sums fit the stages");
    return reinterpret_cast<float *>(tc_smem);
}

struct StepForward {
    const bf16 *x, *w;
    bf16 *copy;              /* x again, for a backward pass of its own; or NULL */
    const float *bias;
    bf16 *h;
    float *pre;
    int m, n, k, act;
    /* the last layer's loss (loss_grad_kernel) */
    const float *target, *wcol;
    bf16 *dpre;
    float *part, *loss_part;
    int nv, mode;
    float scale, clip;
};

template <int BN, bool LAST>
__global__ void __launch_bounds__(TNT) step_forward(const __grid_constant__ StepForward p) {
    extern __shared__ __align__(1024) uint8_t tc_smem[];
    const int r0 = blockIdx.y * TBM, c0 = blockIdx.x * BN;
    uint32_t tmem;
    const bool ok = tc_product<BN, false, false>(tc_smem, p.x, p.k, p.w, p.k, p.m, p.n, r0, c0, 0, p.k, tmem);
    const int r = r0 + tc_row();
    if (p.copy && blockIdx.x == 0 && threadIdx.x < TBM && r < p.m) {
        const uint4 *from = reinterpret_cast<const uint4 *>(p.x + (size_t)r * p.k);
        uint4 *to = reinterpret_cast<uint4 *>(p.copy + (size_t)r * p.k);
        for (int q = 0; q < p.k / 8; ++q) to[q] = from[q];
    }
    const float inv = 1.0f / ((float)p.m * (float)p.nv);
    float *tile = step_tile<BN>(tc_smem);
    float loss = 0.0f;
#pragma unroll 1
    for (int j = threadIdx.x >> 7; j < BN / 16; j += TNT / 128) {
        const int c = c0 + j * 16;
        float v[16];
        tc_row16(tmem, j, true, ok, v);
        if (c >= p.n) continue;
        const bool in = r < p.m;
        const size_t o = (size_t)r * p.n + c;
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] += p.bias[c + q];
        if (in) tc_store16(p.pre + o, v);
        if (LAST) {
            float t[16];
            if (in) tc_load16(p.target + o, t);
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                const float y = v[q];
                float g = 0.0f;
                if (in && c + q < p.nv) {
                    const float w = p.wcol ? p.wcol[c + q] : 1.0f;
                    if (p.mode == 0) {
                        const float d = y - t[q];
                        loss += w * d * d * inv;
                        g = 2.0f * w * d * inv;
                    } else {
                        const float ratio = t[q] * expf(-p.scale * y);
                        const float d = ratio - 1.0f;
                        loss += w * d * d * inv;
                        g = -2.0f * p.scale * w * (fminf(ratio, p.clip) - 1.0f) * inv;
                    }
                }
                t[q] = __bfloat162float(__float2bfloat16_rn(g));
            }
            if (in) {
                tc_store16(p.h + o, v);
                tc_store16(p.dpre + o, t);
            }
#pragma unroll
            for (int q = 0; q < 16; ++q) tile[tc_row() * (BN + 1) + j * 16 + q] = t[q];
        } else if (in) {
            if (p.act) {
#pragma unroll
                for (int q = 0; q < 16; ++q) v[q] = gelu(v[q]);
            }
            tc_store16(p.h + o, v);
        }
    }
    if (LAST) {
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, d);
        const int row = r0 + (int)(threadIdx.x & 96u);
        if ((threadIdx.x & 31) == 0 && row < p.m) p.loss_part[row / 32 * 2 + (threadIdx.x >> 7)] = loss;
        store_columns<BN>(tile, p.part, r0, c0, p.n, p.m);
    }
    tc_release<BN>(tmem);
}

struct StepBackward {
    const bf16 *dpre, *wt;   /* [m, n], [k, n] */
    const float *pre;        /* [m, k], of the layer below */
    bf16 *out;               /* its dPre [m, k] */
    float *part;
    int m, n, k, act;
};

template <int BN>
__global__ void __launch_bounds__(TNT) step_backward(const __grid_constant__ StepBackward p) {
    extern __shared__ __align__(1024) uint8_t tc_smem[];
    const int r0 = blockIdx.y * TBM, c0 = blockIdx.x * BN;
    uint32_t tmem;
    const bool ok = tc_product<BN, false, false>(tc_smem, p.dpre, p.n, p.wt, p.n, p.m, p.k, r0, c0, 0, p.n, tmem);
    const int r = r0 + tc_row();
    float *tile = step_tile<BN>(tc_smem);
#pragma unroll 1
    for (int j = threadIdx.x >> 7; j < BN / 16; j += TNT / 128) {
        const int c = c0 + j * 16;
        float v[16];
        tc_row16(tmem, j, true, ok, v);
        if (c >= p.k) continue;
        const size_t o = (size_t)r * p.k + c;
        if (r < p.m) {
            float pre[16];
            if (p.act) tc_load16(p.pre + o, pre);
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                /* dX leaves the product as bf16 */
                v[q] = __bfloat162float(__float2bfloat16_rn(v[q]));
                if (p.act) v[q] *= gelu_grad(pre[q]);
            }
            tc_store16(p.out + o, v);
        } else {
#pragma unroll
            for (int q = 0; q < 16; ++q) v[q] = 0.0f;
        }
#pragma unroll
        for (int q = 0; q < 16; ++q) tile[tc_row() * (BN + 1) + j * 16 + q] = v[q];
    }
    store_columns<BN>(tile, p.part, r0, c0, p.k, p.m);
    tc_release<BN>(tmem);
}

constexpr int STEP_COLS = 256;   /* accumulator columns of a weight-gradient CTA */

struct StepWeightLayer {
    const bf16 *dpre, *x;   /* [m, n], [m, k] */
    float *out;             /* [min(count, 8)][n][k] */
    int n, k, first;        /* first block */
    int rows, count;        /* the slices of mcgb_mlp_linear_bwd_weight */
};

struct StepWeights {
    StepWeightLayer layer[STEP_MAX_LAYERS];
    int layers, m;
};

/* Columns of a tile: an accumulator for every eighth slice fits STEP_COLS. */
__host__ __device__ __forceinline__ int step_width(int count) { return count > 32 ? 32 : 64; }

/* sum_slices adds slices w, w + 8, w + 16, ... of the separate kernel, then
   those eight sums in order.  Here one CTA takes the slices w, w + 8, ... of
   a tile, each in an accumulator of its own, and adds them: an eighth of the
   partial sums to write and read, and the same bits. */
template <int BN>
__device__ __forceinline__ void step_weights_tile(uint8_t *tc_smem, const StepWeightLayer &l, int m, int b) {
    const int tiles_k = (l.k + BN - 1) / BN, slices = min(l.count, 8);
    const int slice = b % slices;
    b /= slices;
    const int c0 = (b % tiles_k) * BN, r0 = (b / tiles_k) * TBM;
    const int sums = (l.count - slice + 7) / 8, part = l.rows / TBK;
    uint32_t tmem;
    const bool ok = tc_product<BN, true, true, STEP_COLS>(tc_smem, l.dpre, l.n, l.x, l.k, l.n, l.k, r0, c0,
                                                          slice * l.rows, m, tmem, sums * part, part, 8 * l.rows);
    const int r = r0 + tc_row();
#pragma unroll 1
    for (int j = threadIdx.x >> 7; j < BN / 16; j += TNT / 128) {
        const int c = c0 + j * 16;
        float v[16];
#pragma unroll
        for (int z = 0; z < 16; ++z) v[z] = 0.0f;
        for (int q = 0; q < sums; ++q) {
            float u[16];
            tc_row16(tmem + (uint32_t)(q * BN), j, true, ok, u);
#pragma unroll
            for (int z = 0; z < 16; ++z) v[z] += u[z];
        }
        if (r >= l.n || c >= l.k) continue;
        tc_store16(l.out + ((size_t)slice * l.n + r) * l.k + c, v);
    }
    tc_release<STEP_COLS>(tmem);
}

__global__ void __launch_bounds__(TNT) step_weights(const __grid_constant__ StepWeights p) {
    extern __shared__ __align__(1024) uint8_t tc_smem[];
    int i = p.layers - 1;
    while (i > 0 && (int)blockIdx.x < p.layer[i].first) --i;
    const StepWeightLayer &l = p.layer[i];
    if (step_width(l.count) == 64) step_weights_tile<64>(tc_smem, l, p.m, (int)blockIdx.x - l.first);
    else step_weights_tile<32>(tc_smem, l, p.m, (int)blockIdx.x - l.first);
}

struct StepUpdate {
    AdamwMulti a;                            /* weights and bias of layer i: tensors 2 i, 2 i + 1 */
    const float *dw[STEP_MAX_LAYERS];        /* [slices][n][k] */
    const float *db[STEP_MAX_LAYERS];        /* [row chunks][n] */
    uint64_t weights;                        /* elements of all weight tensors */
    uint64_t wstart[STEP_MAX_LAYERS + 1];
    int bstart[STEP_MAX_LAYERS + 1];         /* bias columns, in groups of 32 */
    int slices[STEP_MAX_LAYERS];
    int layers, chunks;                      /* row chunks of 64 */
    int tie_count, tie_shift;
    const float *loss_part;
    float *loss;
    int m, weight_blocks, bias_blocks;
};

/* The sum of at most eight values in order. */
__device__ __forceinline__ float sum_eight(const float *p, int count, size_t stride) {
    float s[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) s[q] = q < count ? p[(size_t)q * stride] : 0.0f;
    float t = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; ++q) t += s[q];
    return t;
}

/* Blocks: weight elements; groups of 32 bias columns; the loss sums. */
__global__ void __launch_bounds__(256) step_update(const __grid_constant__ StepUpdate p) {
    __shared__ float red[8][32];
    tc_after_previous();
    const AdamwMulti &a = p.a;
    int b = blockIdx.x;
    if (b < p.weight_blocks) {
        const uint64_t i = (uint64_t)b * 256 + threadIdx.x;
        if (i >= p.weights) return;
        int k = 0;
        while (k + 1 < p.layers && i >= p.wstart[k + 1]) ++k;
        const McgbAdamwTensor &T = a.t[2 * k];
        const size_t e = (size_t)(i - p.wstart[k]), size = (size_t)T.rows * T.cols;
        float g = sum_eight(p.dw[k] + e, p.slices[k], size);
        if (k == 0 && p.tie_count) {
            const int c = (int)(e % (size_t)T.cols);
            if (c < p.tie_count) g += sum_eight(p.dw[k] + e + p.tie_shift, p.slices[k], size);
            else if (c >= p.tie_shift && c < p.tie_shift + p.tie_count)
                g = sum_eight(p.dw[k] + e - p.tie_shift, p.slices[k], size) + g;
        }
        const_cast<float *>(T.grad)[e] = g;
        adamw_element(e, T.w, (bf16 *)T.w_bf16, (bf16 *)T.wt_bf16, T.grad, T.m, T.v, T.rows, T.cols, a.lr, a.b1,
                      a.b2, a.eps, T.weight_decay, a.c1, a.c2);
        return;
    }
    b -= p.weight_blocks;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (b < p.bias_blocks) {
        int k = 0;
        while (k + 1 < p.layers && b >= p.bstart[k + 1]) ++k;
        const McgbAdamwTensor &T = a.t[2 * k + 1];
        const int c = (b - p.bstart[k]) * 32 + lane;
        float s = 0.0f;
        if (c < T.cols)
            for (int z = w; z < p.chunks; z += 8) s += p.db[k][(size_t)z * T.cols + c];
        red[w][lane] = s;
        __syncthreads();
        if (w == 0 && c < T.cols) {
            float t = 0.0f;
#pragma unroll
            for (int q = 0; q < 8; ++q) t += red[q][lane];
            const_cast<float *>(T.grad)[c] = t;
            adamw_element(c, T.w, (bf16 *)T.w_bf16, nullptr, T.grad, T.m, T.v, 1, T.cols, a.lr, a.b1, a.b2, a.eps,
                          T.weight_decay, a.c1, a.c2);
        }
        return;
    }
    /* the loss of each 256 rows from its eight groups' two column halves */
    const int groups = (p.m + 31) / 32;
    for (int i = threadIdx.x; 8 * i < groups; i += 256) {
        const float *l = p.loss_part + 16 * i;
        const int n = min(8, groups - 8 * i);
        p.loss[i] = sum_eight(l, n, 2) + sum_eight(l + 1, n, 2);
    }
}

/* Launch behind the previous kernel of the stream, set-up overlapping it. */
template <class P>
cudaError_t step_launch(void (*kernel)(const P), dim3 grid, unsigned threads, size_t smem, cudaStream_t st,
                        const P &p) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, p);
}

template <class P>
cudaError_t step_launch_tc(void (*kernel)(const P), size_t smem, dim3 grid, cudaStream_t st, const P &p) {
    cudaError_t e = cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return e == cudaSuccess ? step_launch(kernel, grid, TNT, smem, st, p) : e;
}

/* The weight-gradient slices of mcgb_mlp_linear_bwd_weight. */
void step_slices(const McgbAdamwTensor &t, int m, int &rows, int &count) {
    const int fine = weight_slices(m, t.rows, t.cols, 0);
    rows = ((m + fine - 1) / fine + TBK - 1) / TBK * TBK;
    count = (m + rows - 1) / rows;
}
