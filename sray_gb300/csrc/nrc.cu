/* nrc.cu -- the radiance cache: a small MLP that stands in for the photon-map
 * final gather of indirect light, trained online on the gather's own
 * estimates (no counterpart in the reference; the final gather it replaces is
 * shade_phong's diffuse rays + PhotonMap::radiance_est, src/shader.cc:154-187,
 * src/pmap.cc:143-178).
 *
 * Network: 9 inputs (position scaled to the scene box, normal, direction),
 * 12-band sin/cos encoding (216 features), 4 hidden layers of 64 ReLU units,
 * 3 linear outputs; relative L2 loss; Adam.  Weights are kept in FP32 (the
 * Adam master copy) and used as BF16 with FP32 accumulation: inference and
 * queries on the 5th-generation tensor cores (tcgen05.mma, a 128-sample tile
 * per MMA); the training step by warp-level MMAs (mma.sync m16n8k16: a warp
 * carries 16 samples through all five layers and back, the accumulator tile
 * of one layer becoming the operand tile of the next, and a share of the
 * block's weight gradients).
 *
 *   k_nrc_forward_tc<FWD_INFER>  inference: encode + 5 layers on the
 *                         5th-generation tensor cores (TMEM accumulators
 *                         and hidden operands, three tiles in flight per SM)
 *   k_nrc_forward_tc<FWD_QUERY>  the renderer's queries: the same, the output
 *                         weighted into the pixel's accumulator
 *   k_nrc_gradient        the training step's gradient: forward, loss, backward
 *                         and weight gradients of 128-sample tiles in one
 *                         kernel (warp-level MMA), activations in shared
 *                         memory, weight gradients in registers
 *   k_nrc_adam            Adam on the FP32 master, BF16 copies refreshed
 *
 * The CPU restatement (checker of these kernels) is oracle/nrc.py.
 */
#include <math.h>
#include <string.h>
#include <stdint.h>
#include <vector>
#include <mutex>
#include <string>
#include <cuda_bf16.h>
#include "sray_gpu.h"
#include "sray_rng.h"
#include "nrc.h"

namespace sray {

/* ---- parameter layout (packed FP32, the order of oracle/nrc.py) ---- */
enum {
	NRC_F = 216,            /* encoded features */
	NRC_FP = 224,           /* padded to 14 k-tiles of 16 */
	NRC_H = 64,
	NRC_O = 3,
	OFF_W1 = 0,
	OFF_B1 = OFF_W1 + NRC_H * NRC_F,
	OFF_W2 = OFF_B1 + NRC_H,
	OFF_B2 = OFF_W2 + NRC_H * NRC_H,
	OFF_W3 = OFF_B2 + NRC_H,
	OFF_B3 = OFF_W3 + NRC_H * NRC_H,
	OFF_W4 = OFF_B3 + NRC_H,
	OFF_B4 = OFF_W4 + NRC_H * NRC_H,
	OFF_W5 = OFF_B4 + NRC_H,
	OFF_B5 = OFF_W5 + NRC_O * NRC_H,
	NRC_NPARAM = OFF_B5 + NRC_O
};
static_assert(NRC_NPARAM == SRAY_NRC_PARAMS, "parameter count");

/* row strides (bf16 elements) of the weight images and of the training
 * step's shared memory, padded against bank conflicts */
enum { LD1 = 232, LDH = 72, LD5 = 24 };

/* BF16 weight images in global memory, in the training step's shared-memory
 * layout:
 *   w1  [64][LD1]      (in 0..215, zero up to 231)
 *   w2-4 [64][LDH]     (out rows, in columns)
 *   w5  [8][LDH]       (rows 3..7 zero)
 * plus the FP32 biases b1-b4 [64], b5 [8]. */
struct NrcDev {
	const __nv_bfloat16 *w1, *w2, *w3, *w4, *w5;
	const float *bias;            /* 4 x 64 + 8 */
};

enum {
	IMG_W1 = 0,
	IMG_W2 = IMG_W1 + 64 * LD1,
	IMG_W3 = IMG_W2 + 64 * LDH,
	IMG_W4 = IMG_W3 + 64 * LDH,
	IMG_W5 = IMG_W4 + 64 * LDH,
	IMG_END = IMG_W5 + 8 * LDH,
	NRC_NBIAS = 4 * 64 + 8
};

/* ---- warp-level MMA tiles ---- */
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
	asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
			: "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
			: "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
	__nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
	return *reinterpret_cast<uint32_t *>(&v);
}

__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

/* Four 8 x 8 BF16 blocks of a row-major shared matrix, one register each; the
 * lanes of eight give a block's row addresses.  T: each block transposed. */
template <bool T>
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t saddr)
{
	if(T)
		asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
				: "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(saddr) : "memory");
	else
		asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
				: "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(saddr) : "memory");
}

/* B operands of two k16 x n8 tiles (columns n0 and n0 + 8): r[0], r[1] and
 * r[2], r[3].  Element (k, n) is M[n0 + n][k0 + k]. */
__device__ __forceinline__ void load_b2(uint32_t (&r)[4], uint32_t M, int ld, int n0, int k0, int lane)
{
	int i = lane >> 3, row = n0 + (lane & 7) + (i >> 1) * 8, col = k0 + (i & 1) * 8;
	ldsm4<false>(r, M + (uint32_t)(row * ld + col) * 2);
}

/* the same where element (k, n) is M[k0 + k][n0 + n] */
__device__ __forceinline__ void load_bt2(uint32_t (&r)[4], uint32_t M, int ld, int n0, int k0, int lane)
{
	int i = lane >> 3, row = k0 + (lane & 7) + (i & 1) * 8, col = n0 + (i >> 1) * 8;
	ldsm4<true>(r, M + (uint32_t)(row * ld + col) * 2);
}

/* A operand of an m16 x k16 tile whose element (m, k) is M[k0 + k][m0 + m] */
__device__ __forceinline__ void load_at(uint32_t (&r)[4], uint32_t M, int ld, int m0, int k0, int lane)
{
	int i = lane >> 3, row = k0 + (lane & 7) + (i >> 1) * 8, col = m0 + (i & 1) * 8;
	ldsm4<true>(r, M + (uint32_t)(row * ld + col) * 2);
}

/* a 16 x 64 activation block as accumulators: 8 n-tiles x 4 floats */
struct Acc64 {
	float d[8][4];
};

/* accumulators of a layer -> A operand tiles of the next (BF16): k-tile kt
 * is made of n-tiles 2kt and 2kt+1 */
__device__ __forceinline__ void acc_to_a(const Acc64 &z, uint32_t (&a)[4][4], bool relu)
{
	#pragma unroll
	for(int kt = 0; kt < 4; kt++) {
		const float *lo = z.d[2 * kt], *hi = z.d[2 * kt + 1];
		float v[8] = {lo[0], lo[1], lo[2], lo[3], hi[0], hi[1], hi[2], hi[3]};
		if(relu) {
			#pragma unroll
			for(int i = 0; i < 8; i++) v[i] = fmaxf(v[i], 0.0f);
		}
		a[kt][0] = pack_bf16(v[0], v[1]);
		a[kt][1] = pack_bf16(v[2], v[3]);
		a[kt][2] = pack_bf16(v[4], v[5]);
		a[kt][3] = pack_bf16(v[6], v[7]);
	}
}

/* one encoded feature pair (sin, cos of pi 2^b x_v) for pair index p, 0 for padding */
__device__ __forceinline__ uint32_t feature_pair(const float *x, int p)
{
	if(p >= NRC_F / 2) return 0u;
	int v = p / 12, b = p - v * 12;
	float s, c;
	sincospif(x[v] * (float)(1 << b), &s, &c);
	return pack_bf16(s, c);
}

/* the A operand of k-tile kt of the encoded inputs, rows g and g + 8 */
__device__ __forceinline__ void encode_a(const float *xg, const float *xg8, int kt, int lane, uint32_t (&a)[4])
{
	int t = lane & 3;
	int p0 = kt * 8 + t, p1 = kt * 8 + 4 + t;
	a[0] = feature_pair(xg, p0);
	a[1] = feature_pair(xg8, p0);
	a[2] = feature_pair(xg, p1);
	a[3] = feature_pair(xg8, p1);
}

/* queries of the renderer: inputs x [n][9]; w[i] = weight rgb and the
 * accumulator slot; acc[slot] += w * max(y, 0); the count is read on the
 * device (n is the capacity) */
struct QueryOut {
	const int *count;
	const float4 *w;
	float4 *acc;
};

enum { FWD_INFER = 0, FWD_QUERY = 2 };

/* ---- The gradient of a batch ----
 * A block of eight warps takes tiles of 128 samples, 16 per warp.  Forward as
 * a chain of MMAs in registers, each layer's BF16 input also stored in shared
 * memory; loss and its gradient; backward through the same weights (read
 * transposed by ldmatrix).  After each layer's dZ the block's warps form its
 * weight gradient dW = dZ^T H over the tile's samples (both operands read
 * transposed), each warp a fixed part of it in registers -- 108 floats per
 * thread for all layers -- which go to the packed gradient once, after the
 * block's last tile, by vector atomics.  Weights and everything a sample needs
 * stay on the SM: the batch's inputs are read once, and nothing but the
 * gradient is written.
 *
 * Bound by the latency of its chain (weights, encoding, ten MMA layers with a
 * barrier each) up to a tile per SM, then by the warp-level tensor pipe.
 * As five kernels through global memory (forward, backward, a weight-gradient
 * kernel per layer whose operands were transposed element by element) a step
 * of 16,384 samples took 107 us on the device and 144 us per call; this way a
 * call takes 41 us (262,144 samples: 872 and 267 us, 155 TFLOP/s). */
#define GR_THREADS 256
#define GR_TILE 128
enum {
	GR_W = 0,                                   /* the images; w5 padded to 16 rows */
	GR_W5 = GR_W + IMG_W5 * 2,
	GR_BIAS = GR_W5 + 16 * LDH * 2,
	GR_DB = GR_BIAS + NRC_NBIAS * 4,            /* bias gradients: 4 x 64, then 3 */
	GR_H0 = GR_DB + NRC_NBIAS * 4,              /* encoded inputs [128][LD1] */
	GR_H1 = GR_H0 + GR_TILE * LD1 * 2,          /* hidden activations, four of [128][LDH] */
	GR_HSIZE = GR_TILE * LDH * 2,
	GR_DZ = GR_H1 + 4 * GR_HSIZE,               /* dZ of layers 4 and 2 (3 and 1: in place of h4) */
	GR_DZ5 = GR_DZ + GR_HSIZE,                  /* dZ of the outputs [128][LD5], 16 columns used */
	GR_SMEM = GR_DZ5 + GR_TILE * LD5 * 2
};
static_assert(GR_SMEM <= 232448, "shared memory of the gradient");
static_assert(GR_W5 % 16 == 0 && GR_BIAS % 16 == 0 && GR_H0 % 16 == 0 && GR_H1 % 16 == 0 && GR_DZ % 16 == 0 && GR_DZ5 % 16 == 0 &&
		LD1 * 2 % 16 == 0 && LDH * 2 % 16 == 0 && LD5 * 2 % 16 == 0 && IMG_END * 2 % 16 == 0, "16-byte rows for ldmatrix and cp.async");

__device__ __forceinline__ void red_add2(float *p, float a, float b)
{
	asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" :: "l"(p), "f"(a), "f"(b) : "memory");
}

/* 16 x 64 = A(16 x 64) W^T + bias: W [64][LDH] (out, in) at M */
__device__ __forceinline__ void layer64(const uint32_t (&a)[4][4], uint32_t M, const float *bias, int lane, Acc64 &z)
{
	int t = lane & 3;
	#pragma unroll
	for(int nt = 0; nt < 8; nt += 2) {
		#pragma unroll
		for(int h = 0; h < 2; h++) {
			float b0 = bias[(nt + h) * 8 + 2 * t], b1 = bias[(nt + h) * 8 + 2 * t + 1];
			z.d[nt + h][0] = b0; z.d[nt + h][1] = b1; z.d[nt + h][2] = b0; z.d[nt + h][3] = b1;
		}
		#pragma unroll
		for(int kt = 0; kt < 4; kt++) {
			uint32_t w[4];
			load_b2(w, M, LDH, nt * 8, kt * 16, lane);
			mma16816(z.d[nt], a[kt], w[0], w[1]);
			mma16816(z.d[nt + 1], a[kt], w[2], w[3]);
		}
	}
}

/* this warp's part of a 64 x 64 weight gradient over the tile: rows 16 mt ..,
 * columns 32 nh .. */
__device__ __forceinline__ void wgrad64(float (&g)[4][4], uint32_t dz, uint32_t h, int mt, int nh, int lane)
{
	#pragma unroll
	for(int k = 0; k < GR_TILE; k += 16) {
		uint32_t a[4], b[4];
		load_at(a, dz, LDH, mt * 16, k, lane);
		#pragma unroll
		for(int j = 0; j < 4; j += 2) {
			load_bt2(b, h, LDH, nh * 32 + j * 8, k, lane);
			mma16816(g[j], a, b[0], b[1]);
			mma16816(g[j + 1], a, b[2], b[3]);
		}
	}
}

__global__ void __launch_bounds__(GR_THREADS, 1) k_nrc_gradient(NrcDev net, int n, const float *x, const float *tgt, float *grad, float *loss_out)
{
	extern __shared__ __align__(16) unsigned char gsm[];
	const uint32_t sb = (uint32_t)__cvta_generic_to_shared(gsm);
	float *bias = reinterpret_cast<float *>(gsm + GR_BIAS), *sdb = reinterpret_cast<float *>(gsm + GR_DB);
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int g = lane >> 2, t = lane & 3;
	/* the weights arrive while the first tile is encoded */
	for(int i = threadIdx.x; i < IMG_END / 8; i += GR_THREADS)
		asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(sb + GR_W + i * 16), "l"(reinterpret_cast<const uint4 *>(net.w1) + i) : "memory");
	asm volatile("cp.async.commit_group;" ::: "memory");
	for(int i = threadIdx.x; i < 8 * LDH / 8; i += GR_THREADS)
		*reinterpret_cast<uint4 *>(gsm + GR_W5 + 8 * LDH * 2 + i * 16) = make_uint4(0u, 0u, 0u, 0u);
	for(int i = threadIdx.x; i < NRC_NBIAS; i += GR_THREADS) {
		bias[i] = net.bias[i];
		sdb[i] = 0.0f;
	}
	const uint32_t sW1 = sb + GR_W + IMG_W1 * 2, sW5 = sb + GR_W5, sH0 = sb + GR_H0, sDZ5 = sb + GR_DZ5;
	const int mt = warp & 3, nh = warp >> 2;       /* this warp's part of the weight gradients */
	float g1[14][4], gh[3][4][4], g5[4] = {0.0f, 0.0f, 0.0f, 0.0f};
	#pragma unroll
	for(int j = 0; j < 14; j++) g1[j][0] = g1[j][1] = g1[j][2] = g1[j][3] = 0.0f;
	#pragma unroll
	for(int l = 0; l < 3; l++)
		#pragma unroll
		for(int j = 0; j < 4; j++) gh[l][j][0] = gh[l][j][1] = gh[l][j][2] = gh[l][j][3] = 0.0f;
	float loss = 0.0f, db5[2] = {0.0f, 0.0f};
	const int ntiles = (n + GR_TILE - 1) / GR_TILE;
	const int lr = warp * 16 + g;                  /* this lane's rows in the tile: lr and lr + 8 */
	for(int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
		const int r0 = tile * GR_TILE + lr, r1 = r0 + 8;
		float xg[9], xg8[9];
		#pragma unroll
		for(int k = 0; k < 9; k++) {
			xg[k] = r0 < n ? x[(size_t)r0 * 9 + k] : 0.0f;
			xg8[k] = r1 < n ? x[(size_t)r1 * 9 + k] : 0.0f;
		}
		/* the encoded inputs, in the layout of the A operand */
		uint32_t *h0 = reinterpret_cast<uint32_t *>(gsm + GR_H0) + lr * (LD1 / 2) + t;
		#pragma unroll 2
		for(int kt = 0; kt < NRC_FP / 16; kt++) {
			uint32_t a[4];
			encode_a(xg, xg8, kt, lane, a);
			uint32_t *q = h0 + kt * 8;
			q[0] = a[0];
			q[8 * (LD1 / 2)] = a[1];
			q[4] = a[2];
			q[8 * (LD1 / 2) + 4] = a[3];
		}
		if(tile == (int)blockIdx.x) {
			asm volatile("cp.async.wait_group 0;" ::: "memory");
			__syncthreads();
		} else {
			__syncwarp();
		}
		/* layer 1 */
		Acc64 z;
		#pragma unroll
		for(int nt = 0; nt < 8; nt++) {
			float b0 = bias[nt * 8 + 2 * t], b1 = bias[nt * 8 + 2 * t + 1];
			z.d[nt][0] = b0; z.d[nt][1] = b1; z.d[nt][2] = b0; z.d[nt][3] = b1;
		}
		#pragma unroll 2
		for(int kt = 0; kt < NRC_FP / 16; kt++) {
			const uint32_t *q = h0 + kt * 8;
			const uint32_t a[4] = {q[0], q[8 * (LD1 / 2)], q[4], q[8 * (LD1 / 2) + 4]};
			#pragma unroll
			for(int nt = 0; nt < 8; nt += 2) {
				uint32_t w[4];
				load_b2(w, sW1, LD1, nt * 8, kt * 16, lane);
				mma16816(z.d[nt], a, w[0], w[1]);
				mma16816(z.d[nt + 1], a, w[2], w[3]);
			}
		}
		/* layers 2-4 and the inputs of the output layer; which activations
		 * are positive, a bit each */
		uint32_t a[4][4], on[4];
		#pragma unroll
		for(int l = 0; l < 4; l++) {
			acc_to_a(z, a, true);
			uint32_t *h = reinterpret_cast<uint32_t *>(gsm + GR_H1 + l * GR_HSIZE) + lr * (LDH / 2) + t;
			on[l] = 0;
			#pragma unroll
			for(int kt = 0; kt < 4; kt++) {
				h[kt * 8] = a[kt][0];
				h[kt * 8 + 8 * (LDH / 2)] = a[kt][1];
				h[kt * 8 + 4] = a[kt][2];
				h[kt * 8 + 4 + 8 * (LDH / 2)] = a[kt][3];
				#pragma unroll
				for(int i = 0; i < 4; i++)
					on[l] |= ((bf16_lo(a[kt][i]) > 0.0f ? 1u : 0u) | (bf16_hi(a[kt][i]) > 0.0f ? 2u : 0u)) << (kt * 8 + i * 2);
			}
			if(l < 3) layer64(a, sb + GR_W + (l == 0 ? IMG_W2 : (l == 1 ? IMG_W3 : IMG_W4)) * 2, bias + 64 * (l + 1), lane, z);
		}
		/* output layer: one n-tile (outputs 0..7, 3 used) */
		float o[4];
		o[0] = bias[256 + 2 * t]; o[1] = bias[256 + 2 * t + 1]; o[2] = o[0]; o[3] = o[1];
		#pragma unroll
		for(int kt = 0; kt < 4; kt++) {
			uint32_t w[4];
			load_b2(w, sW5, LDH, 0, kt * 16, lane);
			mma16816(o, a[kt], w[0], w[1]);
		}
		/* lane (g, t) holds outputs 2t, 2t+1 of rows g and g + 8: the loss and
		 * its gradient */
		uint32_t a5[4] = {0u, 0u, 0u, 0u};
		#pragma unroll
		for(int half = 0; half < 2; half++) {
			const int r = half ? r1 : r0;
			float dy[2];
			#pragma unroll
			for(int c = 0; c < 2; c++) {
				const int col = 2 * t + c;
				dy[c] = 0.0f;
				if(r < n && col < NRC_O) {
					float yv = o[2 * half + c], tv = tgt[(size_t)r * 3 + col];
					float den = yv * yv + 0.01f;
					float e = yv - tv;
					loss += e * e / den;
					dy[c] = 2.0f * e / den / (float)(3 * n);
				}
				db5[c] += dy[c];
			}
			a5[half] = pack_bf16(dy[0], dy[1]);
			uint32_t *q = reinterpret_cast<uint32_t *>(gsm + GR_DZ5) + (lr + 8 * half) * (LD5 / 2) + t;
			q[0] = a5[half];
			q[4] = 0u;
		}
		/* dZ of layer 4 from the outputs' */
		#pragma unroll
		for(int nt = 0; nt < 8; nt += 2) {
			uint32_t w[4];
			#pragma unroll
			for(int h = 0; h < 2; h++) z.d[nt + h][0] = z.d[nt + h][1] = z.d[nt + h][2] = z.d[nt + h][3] = 0.0f;
			load_bt2(w, sW5, LDH, nt * 8, 0, lane);
			mma16816(z.d[nt], a5, w[0], w[1]);
			mma16816(z.d[nt + 1], a5, w[2], w[3]);
		}
		__syncthreads();
		/* the output layer's weight gradient: columns 8 warp .. of h4 */
		#pragma unroll
		for(int k = 0; k < GR_TILE; k += 16) {
			uint32_t am[4], b[4];
			load_at(am, sDZ5, LD5, 0, k, lane);
			load_bt2(b, sb + GR_H1 + 3 * GR_HSIZE, LDH, (warp >> 1) * 16, k, lane);
			if(warp & 1) mma16816(g5, am, b[2], b[3]);
			else mma16816(g5, am, b[0], b[1]);
		}
		#pragma unroll
		for(int l = 4; l >= 1; l--) {
			/* dZ_l: masked by h_l > 0; bias sums, BF16 for the products.  The
			 * buffer it goes to was last read before the barrier of the layer
			 * after next (dZ_3 and dZ_1 in place of h4) */
			const uint32_t off = (l & 1) ? GR_H1 + 3 * GR_HSIZE : GR_DZ;
			uint32_t *dz = reinterpret_cast<uint32_t *>(gsm + off) + lr * (LDH / 2) + t;
			#pragma unroll
			for(int nt = 0; nt < 8; nt++) {
				const int kt = nt >> 1, i0 = (nt & 1) * 2;     /* this tile in the forward's A operand: registers i0 and i0 + 1 */
				const uint32_t m = on[l - 1] >> (kt * 8 + i0 * 2);
				if(!(m & 1u)) z.d[nt][0] = 0.0f;
				if(!(m & 2u)) z.d[nt][1] = 0.0f;
				if(!(m & 4u)) z.d[nt][2] = 0.0f;
				if(!(m & 8u)) z.d[nt][3] = 0.0f;
				float s0 = z.d[nt][0] + z.d[nt][2], s1 = z.d[nt][1] + z.d[nt][3];
				#pragma unroll
				for(int q = 4; q < 32; q <<= 1) {
					s0 += __shfl_xor_sync(0xffffffffu, s0, q);
					s1 += __shfl_xor_sync(0xffffffffu, s1, q);
				}
				if(g == 0) {
					atomicAdd(&sdb[(l - 1) * 64 + nt * 8 + 2 * t], s0);
					atomicAdd(&sdb[(l - 1) * 64 + nt * 8 + 2 * t + 1], s1);
				}
			}
			acc_to_a(z, a, false);
			#pragma unroll
			for(int kt = 0; kt < 4; kt++) {
				dz[kt * 8] = a[kt][0];
				dz[kt * 8 + 8 * (LDH / 2)] = a[kt][1];
				dz[kt * 8 + 4] = a[kt][2];
				dz[kt * 8 + 4 + 8 * (LDH / 2)] = a[kt][3];
			}
			if(l > 1) {
				/* dH_{l-1} = dZ_l W_l */
				const uint32_t W = sb + GR_W + (l == 4 ? IMG_W4 : (l == 3 ? IMG_W3 : IMG_W2)) * 2;
				#pragma unroll
				for(int nt = 0; nt < 8; nt += 2) {
					#pragma unroll
					for(int h = 0; h < 2; h++) z.d[nt + h][0] = z.d[nt + h][1] = z.d[nt + h][2] = z.d[nt + h][3] = 0.0f;
					#pragma unroll
					for(int kt = 0; kt < 4; kt++) {
						uint32_t w[4];
						load_bt2(w, W, LDH, nt * 8, kt * 16, lane);
						mma16816(z.d[nt], a[kt], w[0], w[1]);
						mma16816(z.d[nt + 1], a[kt], w[2], w[3]);
					}
				}
			}
			__syncthreads();
			if(l > 1) {
				wgrad64(gh[l - 2], sb + off, sb + GR_H1 + (l - 2) * GR_HSIZE, mt, nh, lane);
			} else {
				#pragma unroll 2
				for(int k = 0; k < GR_TILE; k += 16) {
					uint32_t am[4];
					load_at(am, sb + off, LDH, mt * 16, k, lane);
					#pragma unroll
					for(int j = 0; j < 14; j += 2) {
						uint32_t b[4];
						load_bt2(b, sH0, LD1, nh * 112 + j * 8, k, lane);
						mma16816(g1[j], am, b[0], b[1]);
						mma16816(g1[j + 1], am, b[2], b[3]);
					}
				}
			}
		}
		__syncthreads();      /* the next tile overwrites the activations */
	}
	/* the block's sums */
	for(int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
	if(lane == 0 && loss != 0.0f) atomicAdd(loss_out, loss / (float)(3 * n));
	for(int o = 4; o < 32; o <<= 1) {
		db5[0] += __shfl_xor_sync(0xffffffffu, db5[0], o);
		db5[1] += __shfl_xor_sync(0xffffffffu, db5[1], o);
	}
	if(g == 0) {
		if(2 * t < NRC_O) atomicAdd(&sdb[256 + 2 * t], db5[0]);
		if(2 * t + 1 < NRC_O) atomicAdd(&sdb[256 + 2 * t + 1], db5[1]);
	}
	#pragma unroll
	for(int half = 0; half < 2; half++) {
		const int row = mt * 16 + g + 8 * half;
		#pragma unroll
		for(int j = 0; j < 14; j++) {
			const int col = nh * 112 + j * 8 + 2 * t;
			if(col < NRC_F) red_add2(grad + OFF_W1 + row * NRC_F + col, g1[j][2 * half], g1[j][2 * half + 1]);
		}
		#pragma unroll
		for(int l = 0; l < 3; l++) {
			const int off = l == 0 ? OFF_W2 : (l == 1 ? OFF_W3 : OFF_W4);
			#pragma unroll
			for(int j = 0; j < 4; j++) red_add2(grad + off + row * 64 + nh * 32 + j * 8 + 2 * t, gh[l][j][2 * half], gh[l][j][2 * half + 1]);
		}
	}
	if(g < NRC_O) red_add2(grad + OFF_W5 + g * 64 + warp * 8 + 2 * t, g5[0], g5[1]);
	__syncthreads();
	const int boff[5] = {OFF_B1, OFF_B2, OFF_B3, OFF_B4, OFF_B5};
	for(int i = threadIdx.x; i < 256 + NRC_O; i += GR_THREADS) atomicAdd(&grad[boff[i >> 6] + (i & 63)], sdb[i]);
}
static_assert(OFF_W1 % 2 == 0 && OFF_W2 % 2 == 0 && OFF_W3 % 2 == 0 && OFF_W4 % 2 == 0 && OFF_W5 % 2 == 0 && NRC_F % 2 == 0,
		"pairs of the packed gradient for vector atomics");

/* ---- The inference and query forward on the 5th-generation tensor cores ----
 * tcgen05.mma with the accumulators in tensor memory (TMEM).  A CTA is
 * three groups of eight warps and a warp per group that issues its MMAs;
 * each group carries a tile of 128 samples through the five layers, two
 * threads per sample (row): its threads write the tile's encoded inputs (half
 * of a row's features each) into shared memory and arrive on the group's
 * "full" mbarrier, the issuing warp's elected thread issues the layer's MMAs
 * (M = 128, N = 64, K = 16 each; 14 for the 224-wide first layer, 5 for the
 * 80-wide others, N = 16 for the output layer) and commits them to the
 * group's other mbarrier, and the threads read their rows of the accumulator back from TMEM (tcgen05.ld,
 * 32x32b: warp w its lanes 32 (w mod 4) on; the two warps of a lane quarter
 * take 32 columns each) for the ReLU and BF16 rounding that make the next
 * layer's operand, which stays in TMEM (tcgen05.st; the MMA's A operand
 * there, two BF16 per column); the biases come with the products (a BF16 pair
 * per row of each weight tile against a constant pair in the operand).  The
 * features are read only by the first layer, so a group encodes its next
 * tile while the MMAs of the current one's layers 2-4 run (three, three and
 * one seventh of it after each of their issues), and that tile's first layer
 * is issued together with the current one's fifth: four waits per tile.  The
 * three groups interleave.
 *
 * The chain of round trips bounds a tile, then the encoding's instructions.
 * A call of 4,194,304 samples, host work (27 us) included: 362 us with five
 * waits per tile, 340 with four.  There a warp of each group issued the MMAs
 * from a branch that one lane took, every operand passing from vector to
 * uniform registers first: 299 us with elect.sync and operands that the
 * whole warp computes.  One issuing warp that polls all three groups 305,
 * one per group 260: no warp waits for the others of its group before it
 * encodes.  257 with the encoding split 3/3/1 over the windows (3/2/2 260,
 * 2/2/3 266, 4/2/1 278, 3/4 288).
 *
 * Shared memory, canonical K-major layouts without swizzle (8-row x 16-byte
 * core matrices; a descriptor's leading byte offset steps along K, its
 * stride byte offset along the rows):
 *   weights   W1 64 x 224, W2-W4 64 x 80, W5 its first 8 rows x 80 (rows 3-7
 *             zero; the MMA's rows 8-15 read the bytes that follow and land in
 *             output columns that are never read), row-group-major: the core
 *             matrices of a row group 128 bytes apart, row groups K/8 x 128
 *   per group the tile's 27 feature chunks, chunk-major: chunk c, row r at
 *             c x 2048 + r x 16 (leading byte offset 2048, stride 128)
 *   constant  2 KB of rows (1, 1, 0 ...), the features' bias pair (chunk 27),
 *             reached by the first layer's last K step through its leading
 *             byte offset
 * 228,672 bytes.  TMEM: 128 columns per group (the hidden accumulator, the
 * hidden operand, the output accumulator).  Every wait on an mbarrier is
 * bounded; one that runs out sets the error word and its warp stops, whereupon
 * the waits of the group's others run out (TMEM is released as usual). */
#define TC_NG 3                 /* groups (tiles in flight) per CTA */
#define TC_GROUP_THREADS 256
#define TC_THREADS (TC_NG * (TC_GROUP_THREADS + 32))   /* and a warp per group that issues its MMAs */
#define TC_WAIT_LIMIT (1 << 20)
#define TC_XH 5                 /* inputs a half of the encoding reads: 0-4 or 4-8 */

enum {
	TC_KH = 80,                         /* K of layers 2-5: 64 activations, the bias pair, zeros */
	TC_CHUNK = 128 * 16,                /* one 8-element K chunk of a 128-row operand */
	TC_W1 = 0,                          /* 64 x 224: 8 row groups x 28 K-chunks x 128 B */
	TC_W2 = TC_W1 + 64 * NRC_FP * 2,    /* 64 x 80 each */
	TC_W3 = TC_W2 + 64 * TC_KH * 2,
	TC_W4 = TC_W3 + 64 * TC_KH * 2,
	TC_W5 = TC_W4 + 64 * TC_KH * 2,     /* 8 x 80 */
	TC_GROUP0 = TC_W5 + 8 * TC_KH * 2,
	TC_GROUP_BYTES = (NRC_F / 8) * TC_CHUNK,        /* the 27 feature chunks */
	TC_CONST = TC_GROUP0 + TC_NG * TC_GROUP_BYTES,
	TC_MBAR = TC_CONST + TC_CHUNK,
	TC_FULL = TC_MBAR + 8 * TC_NG,      /* per group: its operands are written */
	TC_TMEM_SLOT = TC_FULL + 8 * TC_NG,
	TC_SMEM = TC_TMEM_SLOT + 16,
	TC_TMEM_COLS = 512,                 /* a power of two >= 128 per group */
	/* a group's TMEM columns, from 128 g: the hidden layers' accumulator,
	 * the hidden operand (80 BF16 = 40 columns), the output layer's
	 * accumulator */
	TC_TD = 0, TC_TA = 64, TC_TO = 112
};
static_assert(TC_SMEM <= 232448, "shared memory of the tensor-core forward");
static_assert(TC_GROUP0 % 128 == 0 && TC_CONST % 128 == 0 && TC_MBAR % 8 == 0, "operand alignment");

/* shared-memory matrix descriptor: start, leading and stride byte offsets, the
 * descriptor version of sm_100, no swizzle */
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
	uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
	d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
	d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
	d |= (uint64_t)1 << 46;
	return d;
}

/* instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both K-major, M x N */
__device__ __forceinline__ uint32_t tc_idesc(int m, int n)
{
	return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, int accumulate)
{
	asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
			"tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
			:: "r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

/* the same with the A operand in TMEM (M = 128 lanes, two BF16 per column) */
__device__ __forceinline__ void tc_mma_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, int accumulate)
{
	asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
			"tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
			:: "r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

__device__ __forceinline__ void tc_commit(uint32_t mbar)
{
	asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(mbar) : "memory");
}

__device__ __forceinline__ bool tc_wait(uint32_t mbar, uint32_t parity)
{
	for(int i = 0; i < TC_WAIT_LIMIT; i++) {
		uint32_t done;
		asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}\n"
				: "=r"(done) : "r"(mbar), "r"(parity) : "memory");
		if(done) return true;
	}
	return false;
}

/* one lane of a converged warp, the same one each time */
__device__ __forceinline__ bool tc_elect()
{
	uint32_t r;
	asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}\n" : "=r"(r) :: "memory");
	return r != 0;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

/* the same for a whole warp, which stays together */
__device__ __forceinline__ bool tc_wait_warp(uint32_t mbar, uint32_t parity)
{
	return __all_sync(0xffffffffu, tc_wait(mbar, parity));
}

/* the calling warp's part of its group's operands is written, and what it
 * reads of the accumulators has been read */
__device__ __forceinline__ void tc_arrive(uint32_t full, int lane)
{
	tc_fence_before();
	__syncwarp();
	if(lane == 0) asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}\n" :: "r"(full) : "memory");
}

/* 32 columns of the calling thread's accumulator row (its warp's 32 lanes) */
__device__ __forceinline__ void tc_ld32(uint32_t taddr, float (&v)[32])
{
	uint32_t r[32];
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
			"{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
			: "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
			  "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
			  "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
			  "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
			: "r"(taddr) : "memory");
	asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
	#pragma unroll
	for(int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tc_ld16(uint32_t taddr, float (&v)[16])
{
	uint32_t r[16];
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
			: "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
			  "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
			: "r"(taddr) : "memory");
	asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
	#pragma unroll
	for(int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

/* 16 columns of the calling thread's TMEM lane (its warp's 32 lanes), then
 * the wait for them */
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t (&r)[16])
{
	asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
			:: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
			   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
	asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

/* (sin, cos) of a + q quarter turns from (sin a, cos a); q mod 4 in the low bits of q */
__device__ __forceinline__ void quarter_turns(float &s, float &c, uint32_t q)
{
	float s1 = (q & 1u) ? c : s, c1 = (q & 1u) ? s : c;
	s = __uint_as_float(__float_as_uint(s1) ^ ((q << 30) & 0x80000000u));
	c = __uint_as_float(__float_as_uint(c1) ^ (((q + 1u) << 30) & 0x80000000u));
}

/* sin(pi t) and cos(pi t) of two arguments at once in packed FP32 (the
 * .f32x2 operations of sm_100 on), for |t| < 2^20.  Reduction: n = rint(2t)
 * by adding 1.5 x 2^23 (which rounds to an integer and leaves n in the low
 * bits of the sum), r = t - n/2 in [-1/4, 1/4] exactly (one FMA); then
 * sin(pi r) = r P(r^2) and cos(pi r) = 1 + r^2 Q(r^2) with P, Q of degree 3,
 * their coefficients fitted for this kernel by weighted least squares on 4000
 * Chebyshev nodes of [0, 1/4] (relative error of the sine, absolute of the
 * cosine), and n quarter turns.  Error within 8e-8 (against float64 sin and
 * cos of pi t over |t| <= 300, six million points). */
__device__ __forceinline__ void sincospi2(float2 t, float2 &sn, float2 &cs)
{
	const float MAGIC = 12582912.0f;
	const float2 u = __fadd2_rn(__fadd2_rn(t, t), make_float2(MAGIC, MAGIC));
	const float2 n = __fadd2_rn(u, make_float2(-MAGIC, -MAGIC));
	const float2 r = __ffma2_rn(n, make_float2(-0.5f, -0.5f), t);
	const float2 z = __fmul2_rn(r, r);
	float2 p = __ffma2_rn(z, make_float2(-0.5890136361122131f, -0.5890136361122131f),
			make_float2(2.5497612953186035f, 2.5497612953186035f));
	p = __ffma2_rn(p, z, make_float2(-5.167707920074463f, -5.167707920074463f));
	p = __ffma2_rn(p, z, make_float2(3.1415927410125732f, 3.1415927410125732f));
	float2 q = __ffma2_rn(z, make_float2(0.2314295470714569f, 0.2314295470714569f),
			make_float2(-1.3350584506988525f, -1.3350584506988525f));
	q = __ffma2_rn(q, z, make_float2(4.0587077140808105f, 4.0587077140808105f));
	q = __ffma2_rn(q, z, make_float2(-4.934802055358887f, -4.934802055358887f));
	sn = __fmul2_rn(p, r);
	cs = __ffma2_rn(q, z, make_float2(1.0f, 1.0f));
	quarter_turns(sn.x, cs.x, __float_as_uint(u.x));
	quarter_turns(sn.y, cs.y, __float_as_uint(u.y));
}

/* Pairs P0 .. P1 - 1 of this thread's half of a sample's encoded inputs:
 * the half is chunks C0 .. C0 + 13 of the 27 (chunk c = 3v + k holds the
 * (sin, cos) pairs of bands 4k .. 4k + 3 of input v; the bias pair, chunk
 * 27, is the constant block), from inputs C0/3 .. C0/3 + 4 (xv), two chunks
 * (a pair) at a time in packed FP32.  Band 4k from sincospi2 (exact
 * argument scaling), the next three by angle doubling, sin 2a = 2 sin a cos
 * a and cos 2a = 1 - 2 sin^2 a: 0.011 % of the features then round to
 * another BF16 value than the exact ones' (0.009 % from correctly rounded
 * bases). */
template <int C0, int P0, int P1>
__device__ __forceinline__ void tc_encode_pairs(unsigned char *A1, int row, const float (&xv)[TC_XH])
{
	const int v0 = C0 / 3;      /* the first input of this half: 0 or 4 */
	#pragma unroll
	for(int p = P0; p < P1; p++) {
		const int ca = C0 + 2 * p, cb = ca + 1 < NRC_F / 8 ? ca + 1 : ca;
		float2 sn, cs;
		sincospi2(__fmul2_rn(make_float2(xv[ca / 3 - v0], xv[cb / 3 - v0]),
				make_float2((float)(1 << (4 * (ca % 3))), (float)(1 << (4 * (cb % 3))))), sn, cs);
		uint32_t qa[4], qb[4];
		#pragma unroll
		for(int b = 0; b < 4; b++) {
			qa[b] = pack_bf16(sn.x, cs.x);
			qb[b] = pack_bf16(sn.y, cs.y);
			if(b < 3) {
				const float2 m = __fmul2_rn(sn, make_float2(-2.0f, -2.0f));
				const float2 s2 = __fmul2_rn(__fadd2_rn(sn, sn), cs);
				cs = __ffma2_rn(m, sn, make_float2(1.0f, 1.0f));
				sn = s2;
			}
		}
		*reinterpret_cast<uint4 *>(A1 + ca * TC_CHUNK + row * 16) = make_uint4(qa[0], qa[1], qa[2], qa[3]);
		if(cb != ca) *reinterpret_cast<uint4 *>(A1 + cb * TC_CHUNK + row * 16) = make_uint4(qb[0], qb[1], qb[2], qb[3]);
	}
}

template <int P0, int P1>
__device__ __forceinline__ void tc_encode_part(int hf, unsigned char *A1, int row, const float (&xv)[TC_XH])
{
	if(hf) tc_encode_pairs<NRC_FP / 16, P0, P1>(A1, row, xv);
	else tc_encode_pairs<0, P0, P1>(A1, row, xv);
}

/* the inputs of half hf of row `row` (zeros past n) */
__device__ __forceinline__ void tc_inputs(float (&xv)[TC_XH], const float *x, int n, int row, int hf)
{
	#pragma unroll
	for(int k = 0; k < TC_XH; k++) xv[k] = row < n ? x[(size_t)row * 9 + 4 * hf + k] : 0.0f;
}

/* byte offset of element row r, 8-element K-chunk c in the row-group-major layout of a tile with kc chunks */
__device__ __forceinline__ uint32_t tc_canon(int r, int c, int kc) { return (uint32_t)(((r >> 3) * kc + c) * 128 + (r & 7) * 16); }

/* a weight image [rows][ld] (BF16) into the row-group-major layout of kc
 * K-chunks: its first ks chunks, then in chunk ks the row's bias as a BF16
 * pair (hi, lo: b = hi + lo to 2^-17) that multiplies the operand's constant
 * pair (1, 1), the rest zero; rows beyond `rows` up to `rows_pad` zero */
__device__ __forceinline__ void tc_weights(unsigned char *dst, const __nv_bfloat16 *src, int rows, int rows_pad, int ld, int ks, int kc,
		const float *bias)
{
	for(int i = threadIdx.x; i < rows_pad * kc; i += blockDim.x) {
		int r = i / kc, c = i - r * kc;
		uint4 v = make_uint4(0u, 0u, 0u, 0u);
		if(r < rows && c < ks) v = *reinterpret_cast<const uint4 *>(src + (size_t)r * ld + c * 8);
		if(r < rows && c == ks) {
			float b = bias[r];
			__nv_bfloat16 hi = __float2bfloat16_rn(b);
			v.x = pack_bf16(__bfloat162float(hi), b - __bfloat162float(hi));
		}
		*reinterpret_cast<uint4 *>(dst + tc_canon(r, c, kc)) = v;
	}
}

/* two accumulator values as a BF16 pair after ReLU (lo in the low half) */
__device__ __forceinline__ uint32_t relu_bf16x2(float lo, float hi)
{
	uint32_t d;
	asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
	return d;
}

/* half `hf` (32 columns) of the hidden activations of the calling thread's
 * row (the bias came with the product): ReLU and BF16, into columns 16 hf ..
 * 16 hf + 15 of the next layer's operand in TMEM (ta: the operand's first
 * column in the thread's lane quarter) */
__device__ __forceinline__ void tc_hidden(uint32_t ta, int hf, const float (&v)[32])
{
	uint32_t q[16];
	#pragma unroll
	for(int i = 0; i < 16; i++) q[i] = relu_bf16x2(v[2 * i], v[2 * i + 1]);
	tc_st16(ta + (uint32_t)(hf * 16), q);
}

/* The issuing warp of group g: the MMAs of the group's next step once its
 * eight warps have arrived.  A group's steps are those of its warps: layer 5
 * of a tile with layer 1 of the next, then layers 2, 3 and 4 of that one. */
__device__ __forceinline__ void tc_issue(uint32_t sbase, uint32_t tmem, int g, int ntiles, int stride, unsigned *err)
{
	const uint32_t id64 = tc_idesc(128, 64), id16 = tc_idesc(128, 16);
	const uint32_t full = sbase + TC_FULL + 8 * g, mbar = sbase + TC_MBAR + 8 * g;
	const uint32_t tD = tmem + (uint32_t)(g * 128) + TC_TD, tA = tmem + (uint32_t)(g * 128) + TC_TA, tO = tmem + (uint32_t)(g * 128) + TC_TO;
	const uint32_t sA1 = sbase + TC_GROUP0 + g * TC_GROUP_BYTES, sA26 = sA1 + (NRC_F / 8 - 1) * TC_CHUNK;
	const uint64_t dA1 = tc_desc(sA1, TC_CHUNK, 128), dA26 = tc_desc(sA26, sbase + TC_CONST - sA26, 128);
	const uint64_t dW1 = tc_desc(sbase + TC_W1, 128, (NRC_FP / 8) * 128), dW2 = tc_desc(sbase + TC_W2, 128, TC_KH / 8 * 128);
	const uint64_t dW5 = tc_desc(sbase + TC_W5, 128, TC_KH / 8 * 128);
	uint32_t phase = 0;
	bool ok = true, have = false;
	int next = blockIdx.x * TC_NG + g;
	while(next < ntiles || have) {
		const bool more = next < ntiles;
		ok = tc_wait_warp(full, phase);
		if(!ok) break;
		phase ^= 1u;
		tc_fence_after();
		if(tc_elect()) {
			if(have) {
				#pragma unroll
				for(int j = 0; j < TC_KH / 16; j++) tc_mma_ta(tO, tA + (uint32_t)(8 * j), dW5 + j * 16, id16, j);
			}
			if(more) {
				#pragma unroll
				for(int j = 0; j < NRC_FP / 16 - 1; j++) tc_mma(tD, dA1 + j * (2 * TC_CHUNK >> 4), dW1 + j * 16, id64, j);
				/* the last K step: chunk 26, then the constant block's bias pairs */
				tc_mma(tD, dA26, dW1 + (NRC_FP / 16 - 1) * 16, id64, 1);
			}
			tc_commit(mbar);
		}
		__syncwarp();
		if(!more) break;
		have = true;
		next += stride;
		#pragma unroll
		for(int l = 1; l < 4; l++) {
			ok = tc_wait_warp(full, phase);
			if(!ok) break;
			phase ^= 1u;
			tc_fence_after();
			if(tc_elect()) {
				#pragma unroll
				for(int j = 0; j < TC_KH / 16; j++)
					tc_mma_ta(tD, tA + (uint32_t)(8 * j), dW2 + (l - 1) * ((TC_W3 - TC_W2) >> 4) + j * 16, id64, j);   /* W2, W3, W4 back to back */
				tc_commit(mbar);
			}
			__syncwarp();
		}
		if(!ok) break;
	}
	if(!ok && tc_elect()) atomicOr(err, 1u);
}

template <int MODE>
__global__ void __launch_bounds__(TC_THREADS, 1) k_nrc_forward_tc(NrcDev net, int n, const float *x, float *y, QueryOut qo,
		unsigned *err)
{
	if(MODE == FWD_QUERY) {
		int c = *qo.count;
		n = c < n ? c : n;
	}
	extern __shared__ __align__(1024) unsigned char tsm[];
	const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(tsm);
	tc_weights(tsm + TC_W1, net.w1, 64, 64, LD1, NRC_F / 8, NRC_FP / 8, net.bias);
	tc_weights(tsm + TC_W2, net.w2, 64, 64, LDH, 8, TC_KH / 8, net.bias + 64);
	tc_weights(tsm + TC_W3, net.w3, 64, 64, LDH, 8, TC_KH / 8, net.bias + 128);
	tc_weights(tsm + TC_W4, net.w4, 64, 64, LDH, 8, TC_KH / 8, net.bias + 192);
	tc_weights(tsm + TC_W5, net.w5, NRC_O, 8, LDH, 8, TC_KH / 8, net.bias + 256);
	for(int i = threadIdx.x; i < TC_CHUNK / 16; i += blockDim.x)
		*reinterpret_cast<uint4 *>(tsm + TC_CONST + i * 16) = make_uint4(pack_bf16(1.0f, 1.0f), 0u, 0u, 0u);
	/* group g: warps 8g .. 8g + 7; a warp's lane quarter (warp mod 4) gives
	 * its rows, its half (hf) the features and accumulator columns it takes */
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = warp >> 3, hf = (warp >> 2) & 1;
	const int tid = ((warp & 3) << 5) | lane;
	if(threadIdx.x == 0) {
		for(int k = 0; k < TC_NG; k++) {
			asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(sbase + TC_MBAR + 8 * k) : "memory");
			asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(sbase + TC_FULL + 8 * k), "n"(TC_GROUP_THREADS / 32) : "memory");
		}
	}
	if(warp == 0) {
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
				:: "r"(sbase + TC_TMEM_SLOT), "r"((uint32_t)TC_TMEM_COLS) : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
	}
	/* the weights and constants are read by the tensor cores (async proxy) */
	proxy_fence();
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem = *reinterpret_cast<const uint32_t *>(tsm + TC_TMEM_SLOT);
	const int ntiles = (n + 127) >> 7, stride = gridDim.x * TC_NG;
	if(g >= TC_NG) {
		tc_issue(sbase, __shfl_sync(0xffffffffu, tmem, 0), __shfl_sync(0xffffffffu, warp, 0) - TC_NG * TC_GROUP_THREADS / 32, ntiles, stride, err);
	} else {
		unsigned char *A1 = tsm + TC_GROUP0 + g * TC_GROUP_BYTES;
		const uint32_t mbar = sbase + TC_MBAR + 8 * g, full = sbase + TC_FULL + 8 * g;
		const uint32_t mine = tmem + (uint32_t)(g * 128) + ((uint32_t)((warp & 3) * 32) << 16);   /* the warp's lanes of the group's columns */
		if(hf == 0) {
			/* the hidden operand's last K step: the bias pair (1, 1), then zeros */
			uint32_t q[16] = {pack_bf16(1.0f, 1.0f)};
			tc_st16(mine + TC_TA + 32, q);
		}
		uint32_t phase = 0;
		/* A round of a group: layer 5 of its tile and layer 1 of its next one,
		 * then layers 2, 3 and 4 of that one, under whose MMAs (which read the
		 * hidden operand, not the features) the features of the one after it
		 * are encoded.  xv holds the inputs of the tile to encode next. */
		int next = blockIdx.x * TC_NG + g;
		int row = -1;          /* this thread's sample in the tile before next, -1 none */
		bool ok = true;        /* the warp's waits so far */
		float xv[TC_XH];
		tc_inputs(xv, x, n, next * 128 + tid, hf);
		if(next < ntiles) tc_encode_part<0, 7>(hf, A1, tid, xv);
		while(next < ntiles || row >= 0) {
			const bool more = next < ntiles;
			proxy_fence();     /* the features are read by the tensor cores (async proxy) */
			tc_arrive(full, lane);
			const int after = next + stride;
			if(after < ntiles) tc_inputs(xv, x, n, after * 128 + tid, hf);
			ok = tc_wait_warp(mbar, phase);
			if(!ok) break;
			phase ^= 1u;
			tc_fence_after();
			if(more) {
				float v[32];
				tc_ld32(mine + TC_TD + (uint32_t)(hf * 32), v);
				tc_hidden(mine + TC_TA, hf, v);
			}
			if(row >= 0 && hf == 0) {
				float v[16];
				tc_ld16(mine + TC_TO, v);
				if(row < n) {
					const float *o = v;   /* the bias came with the product */
					if(MODE == FWD_QUERY) {
						float4 wv = qo.w[row];
						float *a = reinterpret_cast<float *>(qo.acc + __float_as_int(wv.w));
						atomicAdd(a, wv.x * fmaxf(o[0], 0.0f));
						atomicAdd(a + 1, wv.y * fmaxf(o[1], 0.0f));
						atomicAdd(a + 2, wv.z * fmaxf(o[2], 0.0f));
					} else {
						y[(size_t)row * 3] = o[0];
						y[(size_t)row * 3 + 1] = o[1];
						y[(size_t)row * 3 + 2] = o[2];
					}
				}
			}
			if(!more) break;
			row = next * 128 + tid;
			next = after;
			#pragma unroll
			for(int l = 1; l < 4; l++) {
				tc_arrive(full, lane);
				if(next < ntiles) {
					if(l == 1) tc_encode_part<0, 3>(hf, A1, tid, xv);
					else if(l == 2) tc_encode_part<3, 6>(hf, A1, tid, xv);
					else tc_encode_part<6, 7>(hf, A1, tid, xv);
				}
				ok = tc_wait_warp(mbar, phase);
				if(!ok) break;
				phase ^= 1u;
				tc_fence_after();
				float v[32];
				tc_ld32(mine + TC_TD + (uint32_t)(hf * 32), v);
				tc_hidden(mine + TC_TA, hf, v);
			}
			if(!ok) break;
		}
		if(!ok) {
			/* what was committed may still be running: a last bounded wait */
			if(lane == 0) atomicOr(err, 1u);
			tc_wait(mbar, phase);
		}
	}
	__syncwarp();
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	if(warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"((uint32_t)TC_TMEM_COLS) : "memory");
}

/* Adam on the FP32 master; the BF16 images are rewritten from it */
__global__ void k_nrc_adam(float *p, float *m, float *v, float *grad, const int *step_dev, float lr)
{
	const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
	int step = *step_dev + 1;   /* the step counter lives on the device, so that a captured graph replays */
	float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < NRC_NPARAM; i += gridDim.x * blockDim.x) {
		float gi = grad[i];
		grad[i] = 0.0f;
		float mi = b1 * m[i] + (1.0f - b1) * gi;
		float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
		m[i] = mi;
		v[i] = vi;
		float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
		p[i] = pi;
	}
}

/* the BF16 images and FP32 biases of the current master weights; after an
 * Adam step (count_step) also the step counter */
__global__ void k_nrc_images(const float *p, __nv_bfloat16 *img, float *bias, int *step_dev, int count_step)
{
	if(count_step && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(step_dev, 1);
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < IMG_END; i += gridDim.x * blockDim.x) {
		float v = 0.0f;
		if(i < IMG_W2) {
			int o = i / LD1, c = i - o * LD1;
			if(c < NRC_F) v = p[OFF_W1 + o * NRC_F + c];
		} else if(i < IMG_W5) {
			int l = (i - IMG_W2) / (64 * LDH), r = i - IMG_W2 - l * 64 * LDH;
			int o = r / LDH, c = r - o * LDH;
			const int offs[3] = {OFF_W2, OFF_W3, OFF_W4};
			if(c < 64) v = p[offs[l] + o * 64 + c];
		} else {
			int r = i - IMG_W5, o = r / LDH, c = r - o * LDH;
			if(o < NRC_O && c < 64) v = p[OFF_W5 + o * 64 + c];
		}
		img[i] = __float2bfloat16_rn(v);
	}
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < NRC_NBIAS; i += gridDim.x * blockDim.x) {
		float v = 0.0f;
		if(i < 256) {
			const int offs[4] = {OFF_B1, OFF_B2, OFF_B3, OFF_B4};
			v = p[offs[i >> 6] + (i & 63)];
		} else if(i - 256 < NRC_O) {
			v = p[OFF_B5 + i - 256];
		}
		bias[i] = v;
	}
}

/* ---------------- host side ---------------- */

struct NrcState {
	int device = -1;
	float *p = nullptr, *m = nullptr, *v = nullptr, *grad = nullptr, *loss = nullptr, *bias = nullptr;
	int *step_dev = nullptr;         /* Adam steps taken (device copy of `step`) */
	unsigned *tc_err = nullptr;      /* set when a tensor-core forward's bounded wait ran out */
	int nsm = 0;
	/* the per-frame training steps as a CUDA graph, replayed while the
	 * batch shape and buffers stay the same */
	cudaGraphExec_t graph = nullptr;
	cudaStream_t cap = nullptr;      /* stream the graph is captured on (the caller's may be the legacy stream) */
	int g_steps = 0, g_per = 0;
	const float *g_x = nullptr, *g_t = nullptr;
	float g_lr = 0.0f;
	__nv_bfloat16 *img = nullptr;
	int step = 0;
	bool ready = false;
	std::string err;
};

static NrcState g_nrc;
static std::mutex g_nrc_mu;

static int nrc_fail(cudaError_t e, const char *where)
{
	g_nrc.err = std::string(where) + ": " + cudaGetErrorString(e);
	return SRAY_ECUDA;
}

#define NCK(call, where) do { cudaError_t e_ = (call); if(e_ != cudaSuccess) return nrc_fail(e_, where); } while(0)

static NrcDev nrc_dev()
{
	NrcDev d;
	const __nv_bfloat16 *b = g_nrc.img;
	d.w1 = b + IMG_W1; d.w2 = b + IMG_W2; d.w3 = b + IMG_W3; d.w4 = b + IMG_W4; d.w5 = b + IMG_W5;
	d.bias = g_nrc.bias;
	return d;
}

static int nrc_alloc()
{
	int dev = 0;
	NCK(cudaGetDevice(&dev), "device");
	if(g_nrc.ready && g_nrc.device == dev) return 0;
	NCK(cudaMalloc(&g_nrc.p, NRC_NPARAM * sizeof(float)), "radiance cache weights");
	NCK(cudaMalloc(&g_nrc.m, NRC_NPARAM * sizeof(float)), "radiance cache moments");
	NCK(cudaMalloc(&g_nrc.v, NRC_NPARAM * sizeof(float)), "radiance cache moments");
	NCK(cudaMalloc(&g_nrc.grad, NRC_NPARAM * sizeof(float)), "radiance cache gradient");
	NCK(cudaMalloc(&g_nrc.loss, sizeof(float)), "radiance cache loss");
	NCK(cudaMalloc(&g_nrc.bias, NRC_NBIAS * sizeof(float)), "radiance cache biases");
	NCK(cudaMalloc(&g_nrc.img, IMG_END * sizeof(__nv_bfloat16)), "radiance cache images");
	NCK(cudaMalloc(&g_nrc.step_dev, sizeof(int)), "radiance cache step");
	NCK(cudaMalloc(&g_nrc.tc_err, sizeof(unsigned)), "radiance cache error word");
	NCK(cudaMemset(g_nrc.tc_err, 0, sizeof(unsigned)), "radiance cache error word");
	NCK(cudaDeviceGetAttribute(&g_nrc.nsm, cudaDevAttrMultiProcessorCount, dev), "multiprocessors");
	NCK(cudaFuncSetAttribute(k_nrc_forward_tc<FWD_INFER>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM), "smem");
	NCK(cudaFuncSetAttribute(k_nrc_forward_tc<FWD_QUERY>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM), "smem");
	NCK(cudaFuncSetAttribute(k_nrc_gradient, cudaFuncAttributeMaxDynamicSharedMemorySize, GR_SMEM), "smem");
	g_nrc.device = dev;
	g_nrc.ready = true;
	return 0;
}

static int nrc_set(const float *host_p, cudaStream_t s)
{
	NCK(cudaMemcpyAsync(g_nrc.p, host_p, NRC_NPARAM * sizeof(float), cudaMemcpyHostToDevice, s), "upload weights");
	NCK(cudaMemsetAsync(g_nrc.m, 0, NRC_NPARAM * sizeof(float), s), "reset moments");
	NCK(cudaMemsetAsync(g_nrc.v, 0, NRC_NPARAM * sizeof(float), s), "reset moments");
	NCK(cudaMemsetAsync(g_nrc.grad, 0, NRC_NPARAM * sizeof(float), s), "reset gradient");
	NCK(cudaMemsetAsync(g_nrc.step_dev, 0, sizeof(int), s), "reset step");
	k_nrc_images<<<64, 256, 0, s>>>(g_nrc.p, g_nrc.img, g_nrc.bias, g_nrc.step_dev, 0);
	NCK(cudaGetLastError(), "radiance cache images");
	g_nrc.step = 0;
	return 0;
}

/* He-uniform weights from a Philox stream, zero biases */
static void nrc_init_host(uint64_t seed, std::vector<float> &p)
{
	p.assign(NRC_NPARAM, 0.0f);
	struct L { int off, out, in; } ls[5] = {{OFF_W1, 64, NRC_F}, {OFF_W2, 64, 64}, {OFF_W3, 64, 64}, {OFF_W4, 64, 64}, {OFF_W5, 3, 64}};
	sray_rng r;
	sray_rng_init(&r, seed, SRAY_DOM_USER, 0x4e5243u, 0);
	for(const L &l : ls) {
		float lim = sqrtf(6.0f / (float)l.in);
		for(int i = 0; i < l.out * l.in; i++) p[l.off + i] = (2.0f * sray_rng_uniform_f(&r) - 1.0f) * lim;
	}
}

/* gradient of the loss over a batch, added into grad (8-byte aligned); the
 * loss into *loss */
static int nrc_gradient(int n, const float *x, const float *t, float *grad, float *loss, cudaStream_t s)
{
	NCK(cudaMemsetAsync(loss, 0, sizeof(float), s), "reset loss");
	int tiles = (n + GR_TILE - 1) / GR_TILE, cap = g_nrc.nsm > 0 ? g_nrc.nsm : 152;
	k_nrc_gradient<<<tiles < cap ? tiles : cap, GR_THREADS, GR_SMEM, s>>>(nrc_dev(), n, x, t, grad, loss);
	NCK(cudaGetLastError(), "radiance cache gradient");
	return 0;
}

int nrc_ensure_ready(uint64_t seed, cudaStream_t s)
{
	bool fresh = !g_nrc.ready;
	int r = nrc_alloc();
	if(r) return r;
	if(fresh) {
		std::vector<float> p;
		nrc_init_host(seed, p);
		if((r = nrc_set(p.data(), s))) return r;
		NCK(cudaStreamSynchronize(s), "radiance cache init");
	}
	return 0;
}

/* CTAs of the tensor-core forward for up to n samples: one per SM at
 * most, TC_NG 128-sample tiles in flight each */
static int tc_grid(int n)
{
	int tiles = (n + 127) / 128;
	int blocks = (tiles + TC_NG - 1) / TC_NG;
	int cap = g_nrc.nsm > 0 ? g_nrc.nsm : 152;
	if(blocks > cap) blocks = cap;
	return blocks < 1 ? 1 : blocks;
}

int nrc_infer(int n, const float *x, float *y, cudaStream_t s)
{
	if(n <= 0) return 0;
	k_nrc_forward_tc<FWD_INFER><<<tc_grid(n), TC_THREADS, TC_SMEM, s>>>(nrc_dev(), n, x, y, QueryOut(), g_nrc.tc_err);
	NCK(cudaGetLastError(), "radiance cache inference");
	return 0;
}

int nrc_device_error(cudaStream_t s)
{
	if(!g_nrc.ready) return 0;
	unsigned h = 0;
	NCK(cudaMemcpyAsync(&h, g_nrc.tc_err, sizeof h, cudaMemcpyDeviceToHost, s), "radiance cache error word");
	NCK(cudaStreamSynchronize(s), "radiance cache error word");
	if(h) {
		g_nrc.err = "radiance cache: a tensor-core wait ran out";
		NCK(cudaMemsetAsync(g_nrc.tc_err, 0, sizeof(unsigned), s), "radiance cache error word");
		return SRAY_EDEVICE;
	}
	return 0;
}

int nrc_query(const int *count, int cap, const float *x, const float4 *w, float4 *acc, cudaStream_t s)
{
	if(cap <= 0) return 0;
	QueryOut qo;
	qo.count = count;
	qo.w = w;
	qo.acc = acc;
	k_nrc_forward_tc<FWD_QUERY><<<tc_grid(cap), TC_THREADS, TC_SMEM, s>>>(nrc_dev(), cap, x, nullptr, qo, g_nrc.tc_err);
	NCK(cudaGetLastError(), "radiance cache queries");
	return 0;
}

int nrc_train(int n, const float *x, const float *t, float lr, cudaStream_t s)
{
	if(n <= 0) return 0;
	int r = nrc_gradient(n, x, t, g_nrc.grad, g_nrc.loss, s);
	if(r) return r;
	g_nrc.step++;
	k_nrc_adam<<<64, 256, 0, s>>>(g_nrc.p, g_nrc.m, g_nrc.v, g_nrc.grad, g_nrc.step_dev, lr);
	k_nrc_images<<<64, 256, 0, s>>>(g_nrc.p, g_nrc.img, g_nrc.bias, g_nrc.step_dev, 1);
	NCK(cudaGetLastError(), "radiance cache training");
	return 0;
}

/* `steps` Adam steps over consecutive batches of `per` samples: captured
 * once as a CUDA graph (gradient, Adam and weight images of every step: steps *
 * NRC_TRAIN_KERNELS kernels) and replayed
 * while the shape, buffers and rate stay the same */
int nrc_train_steps(int steps, int per, const float *x, const float *t, float lr, cudaStream_t s)
{
	if(steps <= 0 || per <= 0) return 0;
	NrcState &G = g_nrc;
	if(!(G.graph && G.g_steps == steps && G.g_per == per && G.g_x == x && G.g_t == t && G.g_lr == lr)) {
		if(G.graph) {
			cudaGraphExecDestroy(G.graph);
			G.graph = nullptr;
		}
		int r = 0;
		if(!G.cap) NCK(cudaStreamCreateWithFlags(&G.cap, cudaStreamNonBlocking), "capture stream");
		cudaGraph_t g = nullptr;
		NCK(cudaStreamBeginCapture(G.cap, cudaStreamCaptureModeThreadLocal), "capture training steps");
		int step0 = G.step;
		for(int i = 0; i < steps && !r; i++) r = nrc_train(per, x + (size_t)i * per * 9, t + (size_t)i * per * 3, lr, G.cap);
		G.step = step0;
		cudaError_t e = cudaStreamEndCapture(G.cap, &g);
		if(r) {
			if(g) cudaGraphDestroy(g);
			return r;
		}
		if(e != cudaSuccess) return nrc_fail(e, "capture training steps");
		e = cudaGraphInstantiate(&G.graph, g, 0);
		cudaGraphDestroy(g);
		if(e != cudaSuccess) {
			G.graph = nullptr;
			return nrc_fail(e, "instantiate training graph");
		}
		G.g_steps = steps;
		G.g_per = per;
		G.g_x = x;
		G.g_t = t;
		G.g_lr = lr;
	}
	NCK(cudaGraphLaunch(G.graph, s), "training graph");
	G.step += steps;
	return 0;
}

const char *nrc_error() { return g_nrc.err.c_str(); }

float *nrc_loss_ptr() { return g_nrc.loss; }

}  // namespace sray

using namespace sray;

extern "C" {

static thread_local std::string t_nrc_err;

static int nrc_err_ret(int r)
{
	if(r) t_nrc_err = g_nrc.err;
	return r;
}

int sray_nrc_reset(uint64_t seed)
{
	std::lock_guard<std::mutex> lk(g_nrc_mu);
	int r = nrc_alloc();
	if(r) return nrc_err_ret(r);
	std::vector<float> p;
	nrc_init_host(seed, p);
	r = nrc_set(p.data(), 0);
	if(!r) { cudaError_t e = cudaStreamSynchronize(0); if(e != cudaSuccess) r = nrc_fail(e, "reset"); }
	return nrc_err_ret(r);
}

int sray_nrc_set_params(const float *p, int n)
{
	std::lock_guard<std::mutex> lk(g_nrc_mu);
	if(!p || n != NRC_NPARAM) { g_nrc.err = "expected SRAY_NRC_PARAMS parameters"; return nrc_err_ret(SRAY_EINVAL); }
	int r = nrc_alloc();
	if(!r) r = nrc_set(p, 0);
	if(!r) { cudaError_t e = cudaStreamSynchronize(0); if(e != cudaSuccess) r = nrc_fail(e, "set parameters"); }
	return nrc_err_ret(r);
}

int sray_nrc_get_params(float *p, int n)
{
	std::lock_guard<std::mutex> lk(g_nrc_mu);
	if(!p || n != NRC_NPARAM) { g_nrc.err = "expected SRAY_NRC_PARAMS parameters"; return nrc_err_ret(SRAY_EINVAL); }
	if(!g_nrc.ready) { g_nrc.err = "radiance cache not initialised"; return nrc_err_ret(SRAY_ESTATE); }
	cudaError_t e = cudaMemcpy(p, g_nrc.p, NRC_NPARAM * sizeof(float), cudaMemcpyDeviceToHost);
	return nrc_err_ret(e == cudaSuccess ? 0 : nrc_fail(e, "get parameters"));
}

int sray_nrc_infer(int n, const float *x, float *y, void *stream)
{
	std::lock_guard<std::mutex> lk(g_nrc_mu);
	if(n < 0 || (n > 0 && (!x || !y))) { g_nrc.err = "bad arguments"; return nrc_err_ret(SRAY_EINVAL); }
	if(!g_nrc.ready) { g_nrc.err = "radiance cache not initialised"; return nrc_err_ret(SRAY_ESTATE); }
	cudaStream_t s = (cudaStream_t)stream;
	int r = nrc_infer(n, x, y, s);
	if(!r) { cudaError_t e = cudaStreamSynchronize(s); if(e != cudaSuccess) r = nrc_fail(e, "inference"); }
	if(!r) r = nrc_device_error(s);
	return nrc_err_ret(r);
}

int sray_nrc_infer_async(int n, const float *x, float *y, void *stream)
{
	std::lock_guard<std::mutex> lk(g_nrc_mu);
	if(n < 0 || (n > 0 && (!x || !y))) { g_nrc.err = "bad arguments"; return nrc_err_ret(SRAY_EINVAL); }
	if(!g_nrc.ready) { g_nrc.err = "radiance cache not initialised"; return nrc_err_ret(SRAY_ESTATE); }
	return nrc_err_ret(nrc_infer(n, x, y, (cudaStream_t)stream));
}

int sray_nrc_check(void *stream)
{
	std::lock_guard<std::mutex> lk(g_nrc_mu);
	if(!g_nrc.ready) return 0;
	cudaStream_t s = (cudaStream_t)stream;
	int r = 0;
	cudaError_t e = cudaStreamSynchronize(s);
	if(e != cudaSuccess) r = nrc_fail(e, "inference");
	if(!r) r = nrc_device_error(s);
	return nrc_err_ret(r);
}

int sray_nrc_gradients(int n, const float *x, const float *t, float *grad, float *loss, void *stream)
{
	std::lock_guard<std::mutex> lk(g_nrc_mu);
	if(n <= 0 || !x || !t || !grad || !loss) { g_nrc.err = "bad arguments"; return nrc_err_ret(SRAY_EINVAL); }
	if(!g_nrc.ready) { g_nrc.err = "radiance cache not initialised"; return nrc_err_ret(SRAY_ESTATE); }
	cudaStream_t s = (cudaStream_t)stream;
	/* straight into the caller's buffers (the gradient by way of the cache's
	 * own where its pairs are not aligned) */
	float *gr = (uintptr_t)grad % 8 ? g_nrc.grad : grad;
	int r = 0;
	cudaError_t e = cudaMemsetAsync(gr, 0, NRC_NPARAM * sizeof(float), s);
	if(e != cudaSuccess) r = nrc_fail(e, "reset gradient");
	if(!r) r = nrc_gradient(n, x, t, gr, loss, s);
	if(!r && gr != grad) {
		e = cudaMemcpyAsync(grad, gr, NRC_NPARAM * sizeof(float), cudaMemcpyDeviceToDevice, s);
		if(e == cudaSuccess) e = cudaMemsetAsync(gr, 0, NRC_NPARAM * sizeof(float), s);
		if(e != cudaSuccess) r = nrc_fail(e, "copy gradient");
	}
	if(!r) { e = cudaStreamSynchronize(s); if(e != cudaSuccess) r = nrc_fail(e, "gradients"); }
	return nrc_err_ret(r);
}

int sray_nrc_train(int n, const float *x, const float *t, float *loss, void *stream)
{
	std::lock_guard<std::mutex> lk(g_nrc_mu);
	if(n <= 0 || !x || !t) { g_nrc.err = "bad arguments"; return nrc_err_ret(SRAY_EINVAL); }
	if(!g_nrc.ready) { g_nrc.err = "radiance cache not initialised"; return nrc_err_ret(SRAY_ESTATE); }
	cudaStream_t s = (cudaStream_t)stream;
	int r = nrc_train(n, x, t, 1e-3f, s);
	if(!r && loss) { cudaError_t e = cudaMemcpyAsync(loss, g_nrc.loss, sizeof(float), cudaMemcpyDeviceToDevice, s); if(e != cudaSuccess) r = nrc_fail(e, "copy loss"); }
	if(!r) { cudaError_t e = cudaStreamSynchronize(s); if(e != cudaSuccess) r = nrc_fail(e, "training"); }
	return nrc_err_ret(r);
}

int sray_nrc_last_error(char *buf, size_t len)
{
	if(!buf || len == 0) return SRAY_EINVAL;
	size_t n = t_nrc_err.size() < len - 1 ? t_nrc_err.size() : len - 1;
	memcpy(buf, t_nrc_err.data(), n);
	buf[n] = 0;
	return 0;
}

}  /* extern "C" */
