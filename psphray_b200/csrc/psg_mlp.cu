// The chemistry surrogate's network, trained on the device: a 6 -> 64 -> 64
// -> 2 multilayer perceptron with SiLU activations, in FP32 (training) on
// the CUDA cores. Inference inside the ticks runs the same network in BF16
// on the tensor cores (psg_surrogate.cu).
//
// Parameters are one flat FP32 array (PSG_MLP_NPARAM floats):
//   W1[64][8] (inputs padded to 8), b1[64], W2[64][64], b2[64], W3[2][64], b3[2]
// Samples are rows of PSG_MLP_NIN (8) normalised inputs and 2 normalised
// targets. The loss is the mean over samples of the summed squared error.
//
// Gradients are deterministic: every block sums its samples' gradients in a
// fixed order into its own partial, and a second kernel adds the partials
// in block order.
#include <math.h>

#include "psg_internal.cuh"

namespace {

constexpr int NIN = PSG_MLP_NIN, H = 64, NOUT = 2;
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + H * NIN, OFF_W2 = OFF_B1 + H, OFF_B2 = OFF_W2 + H * H,
		OFF_W3 = OFF_B2 + H, OFF_B3 = OFF_W3 + NOUT * H, NPARAM = OFF_B3 + NOUT;
static_assert(NPARAM == PSG_MLP_NPARAM, "parameter layout");
constexpr int BS = 64;          // samples per block iteration
constexpr int TPB = 256;

__device__ __forceinline__ float sigm(float z) { return 1.0f / (1.0f + expf(-z)); }

// Rows of 64 are kept 68 floats apart, so that the 16-byte loads of eight
// lanes on eight rows fall on different banks.
constexpr int LD = H + 4;

struct __align__(16) MlpSmem {
	float W2[H][LD], h1[BS][LD], h2[BS][LD];
	float z1[BS][LD], z2[BS][LD];
	float x[BS][NIN];
	float p[NPARAM + 2];      // (W2 apart)
	float t[BS][NOUT];
	float y[BS][NOUT], dy[BS][NOUT];
	float g1[H * NIN + H], g2b[H], g3[NOUT * H + NOUT];
	float loss;
};

// A thread's part of a 64 x 64 x 64 product, both operands in rows along the
// summed index: acc[a][b] += sum over k of A[r0 + 16a][k] * B[c0 + 16b][k], k
// ascending. Two 16-byte loads per eight multiply-adds where a thread per
// output took sixteen 4-byte ones.
__device__ __forceinline__ void tile_dot(float acc[4][4], const float (*A)[LD], int r0, const float (*B)[LD], int c0) {
#pragma unroll 2
	for (int k = 0; k < H; k += 4) {
		float4 u[4], v[4];
#pragma unroll
		for (int i = 0; i < 4; i++) {
			u[i] = *(const float4 *)&A[r0 + 16 * i][k];
			v[i] = *(const float4 *)&B[c0 + 16 * i][k];
		}
#pragma unroll
		for (int a = 0; a < 4; a++)
#pragma unroll
			for (int b = 0; b < 4; b++) {
				acc[a][b] = fmaf(v[b].x, u[a].x, acc[a][b]);
				acc[a][b] = fmaf(v[b].y, u[a].y, acc[a][b]);
				acc[a][b] = fmaf(v[b].z, u[a].z, acc[a][b]);
				acc[a][b] = fmaf(v[b].w, u[a].w, acc[a][b]);
			}
	}
}

__device__ void load_params(MlpSmem &sm, const float *__restrict__ params) {
	for (int i = threadIdx.x; i < NPARAM; i += TPB) {
		const float v = params[i];
		const int w = i - OFF_W2;
		if (w >= 0 && w < H * H) sm.W2[w / H][w % H] = v;
		else sm.p[i] = v;
	}
}

// Forward pass of BS samples already in sm.x (rows >= nb are zero). A thread
// holds samples ts + 16a and units tj + 16b.
__device__ void forward(MlpSmem &sm) {
	const float *W1 = sm.p + OFF_W1, *b1 = sm.p + OFF_B1, *b2 = sm.p + OFF_B2;
	const float *W3 = sm.p + OFF_W3, *b3 = sm.p + OFF_B3;
	const int ts = threadIdx.x >> 4, tj = threadIdx.x & 15;
#pragma unroll
	for (int b = 0; b < 4; b++) {
		const int j = tj + 16 * b;
		float w[NIN];
#pragma unroll
		for (int k = 0; k < NIN; k++) w[k] = W1[j * NIN + k];
#pragma unroll
		for (int a = 0; a < 4; a++) {
			const int s = ts + 16 * a;
			float z = b1[j];
#pragma unroll
			for (int k = 0; k < NIN; k++) z = fmaf(w[k], sm.x[s][k], z);
			sm.z1[s][j] = z;
			sm.h1[s][j] = z * sigm(z);
		}
	}
	__syncthreads();
	{
		float z[4][4];
#pragma unroll
		for (int a = 0; a < 4; a++)
#pragma unroll
			for (int b = 0; b < 4; b++) z[a][b] = b2[tj + 16 * b];
		tile_dot(z, sm.h1, ts, sm.W2, tj);
#pragma unroll
		for (int a = 0; a < 4; a++)
#pragma unroll
			for (int b = 0; b < 4; b++) {
				sm.z2[ts + 16 * a][tj + 16 * b] = z[a][b];
				sm.h2[ts + 16 * a][tj + 16 * b] = z[a][b] * sigm(z[a][b]);
			}
	}
	__syncthreads();
	for (int i = threadIdx.x; i < BS * NOUT; i += TPB) {
		const int s = i / NOUT, o = i % NOUT;
		float y = b3[o];
#pragma unroll 4
		for (int k = 0; k < H; k += 4) {
			const float4 h = *(const float4 *)&sm.h2[s][k];
			y = fmaf(W3[o * H + k], h.x, y);
			y = fmaf(W3[o * H + k + 1], h.y, y);
			y = fmaf(W3[o * H + k + 2], h.z, y);
			y = fmaf(W3[o * H + k + 3], h.w, y);
		}
		sm.y[s][o] = y;
	}
	__syncthreads();
}

__device__ void load_rows(MlpSmem &sm, const float *X, const float *T, size_t s0, int nb) {
	for (int i = threadIdx.x; i < BS * NIN; i += TPB) {
		const int s = i / NIN, k = i % NIN;
		sm.x[s][k] = s < nb ? X[(s0 + s) * NIN + k] : 0.0f;
	}
	if (T)
		for (int i = threadIdx.x; i < BS * NOUT; i += TPB) {
			const int s = i / NOUT, o = i % NOUT;
			sm.t[s][o] = s < nb ? T[(s0 + s) * NOUT + o] : 0.0f;
		}
	__syncthreads();
}

__global__ void __launch_bounds__(TPB) k_mlp_forward(const float *__restrict__ params, const float *__restrict__ X,
		size_t n, float *__restrict__ Y) {
	extern __shared__ __align__(16) char smem_raw[];
	MlpSmem &sm = *reinterpret_cast<MlpSmem *>(smem_raw);
	load_params(sm, params);
	__syncthreads();
	for (size_t s0 = (size_t)blockIdx.x * BS; s0 < n; s0 += (size_t)gridDim.x * BS) {
		const int nb = (int)min((size_t)BS, n - s0);
		load_rows(sm, X, nullptr, s0, nb);
		forward(sm);
		for (int i = threadIdx.x; i < nb * NOUT; i += TPB) Y[s0 * NOUT + i] = sm.y[i / NOUT][i % NOUT];
		__syncthreads();
	}
}

// Loss and gradient partial of each block (partials[block][NPARAM + 1], the
// last entry the block's summed squared error). Every sum runs over its index
// in ascending order in one thread. Bound by shared-memory loads when each
// thread made one output at a time (two 4-byte loads per multiply-add); with
// 4 x 4 outputs per thread the kernel went from 43 to 28 us at 8192 samples,
// a training step of one context from 64 to 49 us (16384: 94 -> 66, 65536:
// 266 -> 157).
__global__ void __launch_bounds__(TPB) k_mlp_grad(const float *__restrict__ params, const float *__restrict__ X,
		const float *__restrict__ T, size_t n, float scale, float *__restrict__ partials) {
	extern __shared__ __align__(16) char smem_raw[];
	MlpSmem &sm = *reinterpret_cast<MlpSmem *>(smem_raw);
	load_params(sm, params);
	for (int i = threadIdx.x; i < H * NIN + H; i += TPB) sm.g1[i] = 0.0f;
	for (int i = threadIdx.x; i < NOUT * H + NOUT; i += TPB) sm.g3[i] = 0.0f;
	if (threadIdx.x < H) sm.g2b[threadIdx.x] = 0.0f;
	if (threadIdx.x == 0) sm.loss = 0.0f;
	__syncthreads();
	const float *W3 = sm.p + OFF_W3;
	const int tr = threadIdx.x >> 4, tc = threadIdx.x & 15;
	float gW2[4][4];      // rows 4 tr + a, columns 4 tc + b
#pragma unroll
	for (int a = 0; a < 4; a++)
#pragma unroll
		for (int b = 0; b < 4; b++) gW2[a][b] = 0.0f;
	for (size_t s0 = (size_t)blockIdx.x * BS; s0 < n; s0 += (size_t)gridDim.x * BS) {
		const int nb = (int)min((size_t)BS, n - s0);
		load_rows(sm, X, T, s0, nb);
		forward(sm);
		// dL/dy = 2 (y - t) * scale, zero for padding rows
		for (int i = threadIdx.x; i < BS * NOUT; i += TPB) {
			const int s = i / NOUT, o = i % NOUT;
			sm.dy[s][o] = s < nb ? 2.0f * (sm.y[s][o] - sm.t[s][o]) * scale : 0.0f;
		}
		__syncthreads();
		// layer 3, and on a warp of its own the summed squared error
		if (threadIdx.x < NOUT * H) {
			const int o = threadIdx.x / H, k = threadIdx.x % H;
			float a = 0.0f;
#pragma unroll 8
			for (int s = 0; s < nb; s++) a = fmaf(sm.dy[s][o], sm.h2[s][k], a);
			sm.g3[o * H + k] += a;
		} else if (threadIdx.x < NOUT * H + NOUT) {
			const int o = threadIdx.x - NOUT * H;
			float a = 0.0f;
			for (int s = 0; s < nb; s++) a += sm.dy[s][o];
			sm.g3[NOUT * H + o] += a;
		} else if (threadIdx.x == TPB - 1) {
			float l = 0.0f;
#pragma unroll 8
			for (int s = 0; s < nb; s++)
				for (int o = 0; o < NOUT; o++) {
					const float d = sm.y[s][o] - sm.t[s][o];
					l = fmaf(d, d, l);
				}
			sm.loss += l;
		}
		__syncthreads();
		// dZ2 into h2
		for (int i = threadIdx.x; i < BS * H; i += TPB) {
			const int s = i / H, k = i % H;
			float d = 0.0f;
			for (int o = 0; o < NOUT; o++) d = fmaf(sm.dy[s][o], W3[o * H + k], d);
			const float z = sm.z2[s][k], sg = sigm(z);
			sm.h2[s][k] = d * sg * (1.0f + z * (1.0f - sg));
		}
		__syncthreads();
		// layer 2
		{
			float g[4][4];
#pragma unroll
			for (int a = 0; a < 4; a++)
#pragma unroll
				for (int b = 0; b < 4; b++) g[a][b] = 0.0f;
#pragma unroll 4
			for (int s = 0; s < nb; s++) {
				const float4 u4 = *(const float4 *)&sm.h2[s][4 * tr], v4 = *(const float4 *)&sm.h1[s][4 * tc];
				const float u[4] = {u4.x, u4.y, u4.z, u4.w}, v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
				for (int a = 0; a < 4; a++)
#pragma unroll
					for (int b = 0; b < 4; b++) g[a][b] = fmaf(u[a], v[b], g[a][b]);
			}
#pragma unroll
			for (int a = 0; a < 4; a++)
#pragma unroll
				for (int b = 0; b < 4; b++) gW2[a][b] += g[a][b];
		}
		if (threadIdx.x < H) {
			float a = 0.0f;
#pragma unroll 8
			for (int s = 0; s < nb; s++) a += sm.h2[s][threadIdx.x];
			sm.g2b[threadIdx.x] += a;
		}
		__syncthreads();
		// dZ1 into h1: samples tr + 16a, inputs 4 tc + b
		{
			float d[4][4];
#pragma unroll
			for (int a = 0; a < 4; a++)
#pragma unroll
				for (int b = 0; b < 4; b++) d[a][b] = 0.0f;
#pragma unroll 2
			for (int j = 0; j < H; j += 4) {
				float4 u[4];
#pragma unroll
				for (int a = 0; a < 4; a++) u[a] = *(const float4 *)&sm.h2[tr + 16 * a][j];
#pragma unroll
				for (int q = 0; q < 4; q++) {
					const float4 w = *(const float4 *)&sm.W2[j + q][4 * tc];
#pragma unroll
					for (int a = 0; a < 4; a++) {
						const float x = q == 0 ? u[a].x : q == 1 ? u[a].y : q == 2 ? u[a].z : u[a].w;
						d[a][0] = fmaf(x, w.x, d[a][0]);
						d[a][1] = fmaf(x, w.y, d[a][1]);
						d[a][2] = fmaf(x, w.z, d[a][2]);
						d[a][3] = fmaf(x, w.w, d[a][3]);
					}
				}
			}
#pragma unroll
			for (int a = 0; a < 4; a++)
#pragma unroll
				for (int b = 0; b < 4; b++) {
					const float z = sm.z1[tr + 16 * a][4 * tc + b], sg = sigm(z);
					sm.h1[tr + 16 * a][4 * tc + b] = d[a][b] * sg * (1.0f + z * (1.0f - sg));
				}
		}
		__syncthreads();
		// layer 1
		for (int i = threadIdx.x; i < H * NIN; i += TPB) {
			const int j = i / NIN, k = i % NIN;
			float a = 0.0f;
#pragma unroll 8
			for (int s = 0; s < nb; s++) a = fmaf(sm.h1[s][j], sm.x[s][k], a);
			sm.g1[i] += a;
		}
		if (threadIdx.x < H) {
			float a = 0.0f;
#pragma unroll 8
			for (int s = 0; s < nb; s++) a += sm.h1[s][threadIdx.x];
			sm.g1[H * NIN + threadIdx.x] += a;
		}
		__syncthreads();
	}
	float *out = partials + (size_t)blockIdx.x * (NPARAM + 1);
	for (int i = threadIdx.x; i < H * NIN + H; i += TPB) out[OFF_W1 + i] = sm.g1[i];
#pragma unroll
	for (int a = 0; a < 4; a++)
#pragma unroll
		for (int b = 0; b < 4; b++) out[OFF_W2 + (4 * tr + a) * H + 4 * tc + b] = gW2[a][b];
	if (threadIdx.x < H) out[OFF_B2 + threadIdx.x] = sm.g2b[threadIdx.x];
	for (int i = threadIdx.x; i < NOUT * H + NOUT; i += TPB) out[OFF_W3 + i] = sm.g3[i];
	if (threadIdx.x == 0) out[NPARAM] = sm.loss;
}

// (sixteen blocks' entries in flight, added in block order)
__global__ void k_mlp_sum_partials(const float *__restrict__ partials, int nblocks, float *__restrict__ grad) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i > NPARAM) return;
	float a = 0.0f;
	for (int b = 0; b < nblocks; b += 16) {
		float v[16];
#pragma unroll
		for (int u = 0; u < 16; u++) v[u] = b + u < nblocks ? partials[(size_t)(b + u) * (NPARAM + 1) + i] : 0.0f;
#pragma unroll
		for (int u = 0; u < 16; u++)
			if (b + u < nblocks) a += v[u];
	}
	grad[i] = a;
}

__global__ void k_mlp_adam(float *__restrict__ params, const float *__restrict__ grad, float *__restrict__ m,
		float *__restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= NPARAM) return;
	const float g = grad[i];
	const float mi = b1 * m[i] + (1.0f - b1) * g;
	const float vi = b2 * v[i] + (1.0f - b2) * g * g;
	m[i] = mi;
	v[i] = vi;
	params[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

int mlp_smem(psg_context *ctx, const void *kern) {
	const int smem = (int)sizeof(MlpSmem);
	const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
	if (e != cudaSuccess) return psg_cuda_fail(ctx, e, "cudaFuncSetAttribute(mlp)", __FILE__, __LINE__);
	return PSG_OK;
}

}  // namespace

extern "C" int psg_mlp_forward(psg_context *ctx, const float *d_params, const float *d_x, size_t n, float *d_y) {
	if (!ctx) return PSG_E_INVAL;
	if (!d_params || !d_x || !d_y) return psg_fail(ctx, PSG_E_INVAL, "psg_mlp_forward: null pointer");
	if (n == 0) return PSG_OK;
	PSG_CUDA(cudaSetDevice(ctx->device));
	int rc = mlp_smem(ctx, (const void *)k_mlp_forward);
	if (rc) return rc;
	const unsigned grid = (unsigned)std::min<size_t>((n + BS - 1) / BS, 148 * 4);
	k_mlp_forward<<<grid, TPB, sizeof(MlpSmem), ctx->stream>>>(d_params, d_x, n, d_y);
	PSG_CHECK_LAUNCH();
	return PSG_OK;
}

extern "C" int psg_mlp_grad(psg_context *ctx, const float *d_params, const float *d_x, const float *d_t, size_t n,
		float *d_grad, float *d_loss) {
	if (!ctx) return PSG_E_INVAL;
	if (!d_params || !d_x || !d_t || !d_grad || n == 0) return psg_fail(ctx, PSG_E_INVAL, "psg_mlp_grad: bad argument");
	PSG_CUDA(cudaSetDevice(ctx->device));
	int rc = mlp_smem(ctx, (const void *)k_mlp_grad);
	if (rc) return rc;
	const int nblocks = (int)std::min<size_t>((n + BS - 1) / BS, 148 * 2);
	float *partials = (float *)psg_scratch(ctx, S_MLP, sizeof(float) * (size_t)nblocks * (NPARAM + 1));
	if (!partials) return PSG_E_NOMEM;
	k_mlp_grad<<<nblocks, TPB, sizeof(MlpSmem), ctx->stream>>>(d_params, d_x, d_t, n, 1.0f / (float)n, partials);
	PSG_CHECK_LAUNCH();
	// grad[NPARAM] receives the summed squared error
	float *gl = d_grad;
	k_mlp_sum_partials<<<(NPARAM + 64) / 64, 64, 0, ctx->stream>>>(partials, nblocks, gl);
	PSG_CHECK_LAUNCH();
	if (d_loss) PSG_CUDA(cudaMemcpyAsync(d_loss, gl + NPARAM, sizeof(float), cudaMemcpyDeviceToDevice, ctx->stream));
	return PSG_OK;
}

extern "C" int psg_mlp_adam(psg_context *ctx, float *d_params, const float *d_grad, float *d_m, float *d_v,
		float lr, float beta1, float beta2, float eps, int step) {
	if (!ctx) return PSG_E_INVAL;
	if (!d_params || !d_grad || !d_m || !d_v || step < 1) return psg_fail(ctx, PSG_E_INVAL, "psg_mlp_adam: bad argument");
	PSG_CUDA(cudaSetDevice(ctx->device));
	const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
	k_mlp_adam<<<(NPARAM + 255) / 256, 256, 0, ctx->stream>>>(d_params, d_grad, d_m, d_v, lr, beta1, beta2, eps, c1, c2);
	PSG_CHECK_LAUNCH();
	return PSG_OK;
}
