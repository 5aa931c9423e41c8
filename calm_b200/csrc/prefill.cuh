// prefill.cuh -- batched prompt pass (reference behaviour replaced: run.c:206-209 feeds the prompt one
// token at a time through forward(), README.md:80).  T prompt tokens go through every layer together, so each weight
// matrix is read once per 128-token tile instead of once per token and the projections become real GEMMs on the
// 5th-generation tensor cores:
//
//   k_pf_gemm   D[128 weight rows][128 tokens] (+)= W_tile . X_tile^T with tcgen05.mma (kind::f16, cta_group::1), fp32
//               accumulators in TMEM.  A = the weight tile, dequantised ON THE FLY by four warps from the model's own
//               format (fp16 / e5m2 / gf4: all exact in f16) into the 128-byte-swizzled K-major shared-memory layout
//               the MMA reads; B = the activations as TWO f16 matrices hi + lo (x = hi + lo to 22 bits, so the result
//               carries fp32-grade inputs: two MMAs per k-step into the same accumulator), brought in by 2-D TMA
//               (cp.async.bulk.tensor, SWIZZLE_128B).  One warp issues TMA, one thread issues MMAs, completion flows
//               through mbarriers (tcgen05.commit), the epilogue reads TMEM with tcgen05.ld and applies what the
//               decode kernels apply: bias / clip / RoPE / KV-cache append (QKV), residual add (wo, w2),
//               act(w1 x) * (w3 x) with both accumulators side by side in TMEM (FFN up).
//   k_pf_attn   causal attention of the block against the cache (online softmax in fp32; reference infer.c:238-267), scores and
//               values on warp-level tensor cores with hi + lo queries and weights against the cached fp16 / e5m2 entries.
//   k_pf_norm   RMSNorm / LayerNorm per token (reference infer.c:183-207) -> hi / lo f16 rows.
//
// Parity contract (tests/test_prefill_gpu.py): after forward_prefill_cuda(tokens, n, pos0) the KV cache and the logits of
// the following token equal those of n serial forward(FF_UPDATE_KV_ONLY) calls within the stated tolerances.
#pragma once

#include <cuda.h>

#include "stages.cuh"
#include "tc05.cuh"

#define PF_BM 128 // weight rows per tile  (TMEM lanes)
#define PF_BN 128 // tokens per tile       (TMEM columns per accumulator)
#define PF_BK 64  // k per stage: 64 f16 = 128 bytes = one swizzle atom
#define PF_THREADS 192
enum { PF_QKV = 0, PF_WO = 1, PF_UP = 2, PF_DOWN = 3 };

// instruction descriptor, kind::f16: D = f32, A = B = f16, both K-major, M = 128, N = 128
#define PF_IDESC ((1u << 4) | ((uint32_t)(PF_BN >> 3) << 17) | ((uint32_t)(PF_BM >> 4) << 24))

// ---------------------------------------------------------------- small kernels

// f32 -> (hi, lo) f16 pair with x = hi + lo up to 2^-22 |x|
__device__ __forceinline__ void split_hl(float x, __half& hi, __half& lo) {
	hi = __float2half_rn(x);
	lo = __float2half_rn(x - __half2float(hi));
}

// X[t][:] = decode(E[tokens[t]])  (reference infer.c:335-347)
template <int DBITS>
__global__ void k_pf_embed(float* X, const void* table, const int* tokens, int n, int dim) {
	pdl_enter();
	const int t = blockIdx.x;
	if (t >= n) return;
	const size_t base = (size_t)tokens[t] * dim;
	for (int i = threadIdx.x; i < dim; i += blockDim.x) X[(size_t)t * dim + i] = weight_at<DBITS>(table, base + i);
}

// rope[t][j] = (cos, sin)((pos0 + t) * freq[j])
__global__ void k_pf_rope(float2* rope, const float* freq, int n, int half_hd, int pos0) {
	pdl_enter();
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n * half_hd) return;
	float s, c;
	sincosf((float)(pos0 + i / half_hd) * freq[i % half_hd], &s, &c);
	rope[i] = make_float2(c, s);
}

// one CTA per token: norm (infer.c:183-207) then hi / lo split; rows beyond n (tile padding) are zeroed once at allocation
__global__ void __launch_bounds__(256) k_pf_norm(const float* X, const float* normw, __half* hi, __half* lo, int n, int dim, float eps, int ln) {
	pdl_enter();
	__shared__ float red[32];
	const int t = blockIdx.x;
	if (t >= n) return;
	const float* x = X + (size_t)t * dim;
	float mean = 0.f;
	if (ln) {
		float s = 0.f;
		for (int i = threadIdx.x; i < dim; i += blockDim.x) s += x[i];
		mean = block_sum(s, red) / dim;
	}
	float ss = 0.f;
	for (int i = threadIdx.x; i < dim; i += blockDim.x) {
		const float d = x[i] - mean;
		ss = fmaf(d, d, ss);
	}
	ss = block_sum(ss, red);
	const float scale = 1.0f / sqrtf(ss / dim + eps);
	for (int i = threadIdx.x; i < dim; i += blockDim.x) {
		const float v = (x[i] - mean) * scale * normw[i];
		__half h, l;
		split_hl(v, h, l);
		hi[(size_t)t * dim + i] = h, lo[(size_t)t * dim + i] = l;
	}
}

// ---------------------------------------------------------------- the GEMM

struct PfGemmArgs {
	const void* w[3]; // QKV: wq, wk, wv   UP: w1, w3   WO / DOWN: w
	int K, n_tokens;
	// QKV epilogue
	float* Q;         // [T][q_dim]
	int q_dim, kv_dim, head_dim, seq_len, pos0;
	const float* bias;
	float clip;
	const float2* rope; // [T][head_dim / 2]
	void* kc;           // this layer: [n_kv_heads][seq_len][head_dim]
	void* vc;
	// WO / DOWN epilogue
	float* X; // [T][dim] residual stream
	int dim;
	// UP epilogue
	__half* Hhi;
	__half* Hlo;
	int hidden, gelu;
};

// 64 weights of one row (one k-stage) -> 8 swizzled 16-byte chunks of f16 in the A tile
template <int DBITS>
__device__ __forceinline__ void pf_load_raw(const unsigned char* row, int kb, uint4 (&raw)[DBITS / 2]) {
	const uint4* p = reinterpret_cast<const uint4*>(row + (size_t)kb * (PF_BK * DBITS / 8));
#pragma unroll
	for (int i = 0; i < DBITS / 2; ++i) raw[i] = ldg_stream(p + i);
}
template <int DBITS>
__device__ __forceinline__ void pf_store_a(unsigned char* tile, int r, const uint4 (&raw)[DBITS / 2]) {
	unsigned char* rowp = tile + r * 128;
	auto put = [&](int c, uint4 v) { *reinterpret_cast<uint4*>(rowp + ((c ^ (r & 7)) << 4)) = v; };
	if constexpr (DBITS == 16) {
#pragma unroll
		for (int c = 0; c < 8; ++c) put(c, raw[c]);
	} else if constexpr (DBITS == 8) { // an e5m2 byte is the high byte of the f16 (reference infer.c:28-35)
#pragma unroll
		for (int i = 0; i < 4; ++i) {
			const uint32_t w[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
			put(2 * i, make_uint4(__byte_perm(w[0], 0, 0x1404), __byte_perm(w[0], 0, 0x3424), __byte_perm(w[1], 0, 0x1404), __byte_perm(w[1], 0, 0x3424)));
			put(2 * i + 1, make_uint4(__byte_perm(w[2], 0, 0x1404), __byte_perm(w[2], 0, 0x3424), __byte_perm(w[3], 0, 0x1404), __byte_perm(w[3], 0, 0x3424)));
		}
	} else { // gf4: (q - 4) * s / -4 (reference infer.c:37-40); at most 6 significant bits: exact in f16
#pragma unroll
		for (int i = 0; i < 2; ++i) {
			const uint32_t w[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
#pragma unroll
			for (int j = 0; j < 4; ++j) {
				const float sf = e5m2_to_float((uint8_t)(w[j] & 0xff)) * -0.25f;
				uint32_t h[4];
#pragma unroll
				for (int k = 0; k < 4; ++k) {
					const float a0 = (float)((int)((w[j] >> (8 + 6 * k)) & 7) - 4) * sf, a1 = (float)((int)((w[j] >> (11 + 6 * k)) & 7) - 4) * sf;
					h[k] = pack_h2(__float2half_rn(a0), __float2half_rn(a1));
				}
				put(4 * i + j, make_uint4(h[0], h[1], h[2], h[3]));
			}
		}
	}
}

template <int MODE>
__host__ __device__ constexpr int pf_stages() {
	return MODE == PF_UP ? 3 : 4;
}
template <int MODE>
__host__ __device__ constexpr size_t pf_stage_bytes() {
	return (size_t)(MODE == PF_UP ? 2 : 1) * PF_BM * 128 + 2 * PF_BN * 128; // A tile(s) + B hi + B lo
}
template <int MODE>
__host__ __device__ constexpr size_t pf_smem_bytes() {
	return pf_stages<MODE>() * pf_stage_bytes<MODE>() + 1024; // + alignment slack
}

template <int MODE, int DBITS, typename KVT>
__global__ void __launch_bounds__(PF_THREADS, 1) k_pf_gemm(const __grid_constant__ CUtensorMap tm_hi, const __grid_constant__ CUtensorMap tm_lo, const PfGemmArgs a) {
	constexpr int STAGES = pf_stages<MODE>(), NA = MODE == PF_UP ? 2 : 1;
	constexpr uint32_t TMEM_COLS = NA * PF_BN;
	extern __shared__ unsigned char smem_dyn[];
	__shared__ __align__(8) uint64_t full[STAGES], empty[STAGES], accum;
	__shared__ uint32_t tmem_base_s;
	unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int row0 = blockIdx.x * PF_BM, tok0 = blockIdx.y * PF_BN;
	const int nkb = a.K / PF_BK;
	auto a_tile = [&](int s, int i) { return smem + (size_t)s * pf_stage_bytes<MODE>() + (size_t)i * PF_BM * 128; };
	auto b_tile = [&](int s, int i) { return smem + (size_t)s * pf_stage_bytes<MODE>() + (size_t)NA * PF_BM * 128 + (size_t)i * PF_BN * 128; };

	pdl_launch_next();
	if (tid == 0) {
		for (int s = 0; s < STAGES; ++s) mbar_init(&full[s], 1 + 4), mbar_init(&empty[s], 1);
		mbar_init(&accum, 1);
		mbar_init_fence();
	}
	if (warp == 1) tmem_alloc(&tmem_base_s, TMEM_COLS);
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem_base = tmem_base_s;
	pdl_wait_prev(); // activations (and, for the KV rows, the cache) come from the previous kernels of the layer

	if (warp == 0) {
		// ===== TMA producer: the two activation tiles of every k-stage
		if (lane == 0) {
			for (int kb = 0; kb < nkb; ++kb) {
				const int s = kb % STAGES;
				mbar_wait_guard(&empty[s], ((kb / STAGES) & 1) ^ 1);
				mbar_expect_tx(&full[s], 2 * PF_BN * 128);
				tma_load_2d(b_tile(s, 0), &tm_hi, kb * PF_BK, tok0, &full[s]);
				tma_load_2d(b_tile(s, 1), &tm_lo, kb * PF_BK, tok0, &full[s]);
			}
		}
	} else if (warp == 1) {
		// ===== MMA issuer
		if (lane == 0) {
			for (int kb = 0; kb < nkb; ++kb) {
				const int s = kb % STAGES;
				mbar_wait_guard(&full[s], (kb / STAGES) & 1);
				tc_fence_after();
#pragma unroll
				for (int k = 0; k < PF_BK / 16; ++k) { // 16 f16 = 32 bytes along K inside the swizzle atom: +2 in the 16-byte address field
					const uint64_t db_hi = umma_desc_sw128(b_tile(s, 0)) + 2 * k, db_lo = umma_desc_sw128(b_tile(s, 1)) + 2 * k;
#pragma unroll
					for (int i = 0; i < NA; ++i) {
						const uint64_t da = umma_desc_sw128(a_tile(s, i)) + 2 * k;
						umma_f16(tmem_base + i * PF_BN, da, db_hi, PF_IDESC, (kb | k) ? 1u : 0u);
						umma_f16(tmem_base + i * PF_BN, da, db_lo, PF_IDESC, 1u);
					}
				}
				umma_commit(&empty[s]); // frees the stage when these MMAs have read it
			}
			umma_commit(&accum);
		}
	} else {
		// ===== dequantising producers (one tile row per thread), then the epilogue (one accumulator row per thread)
		const int r = tid - 64; // 0..127
		const unsigned char* rowp[NA];
		{
			const size_t rowbytes = (size_t)a.K * DBITS / 8;
			const int gr = row0 + r;
			if constexpr (MODE == PF_QKV) {
				const void* w = gr < a.q_dim ? a.w[0] : (gr < a.q_dim + a.kv_dim ? a.w[1] : a.w[2]);
				const int k = gr < a.q_dim ? gr : (gr < a.q_dim + a.kv_dim ? gr - a.q_dim : gr - a.q_dim - a.kv_dim);
				rowp[0] = reinterpret_cast<const unsigned char*>(w) + (size_t)k * rowbytes;
			} else if constexpr (MODE == PF_UP) {
				rowp[0] = reinterpret_cast<const unsigned char*>(a.w[0]) + (size_t)gr * rowbytes;
				rowp[1] = reinterpret_cast<const unsigned char*>(a.w[1]) + (size_t)gr * rowbytes;
			} else {
				rowp[0] = reinterpret_cast<const unsigned char*>(a.w[0]) + (size_t)gr * rowbytes;
			}
		}
		uint4 raw[NA][DBITS / 2];
#pragma unroll
		for (int i = 0; i < NA; ++i) pf_load_raw<DBITS>(rowp[i], 0, raw[i]);
		for (int kb = 0; kb < nkb; ++kb) {
			const int s = kb % STAGES;
			mbar_wait_guard(&empty[s], ((kb / STAGES) & 1) ^ 1);
#pragma unroll
			for (int i = 0; i < NA; ++i) pf_store_a<DBITS>(a_tile(s, i), r, raw[i]);
			if (kb + 1 < nkb) { // the next stage's bytes travel while this one is being multiplied
#pragma unroll
				for (int i = 0; i < NA; ++i) pf_load_raw<DBITS>(rowp[i], kb + 1, raw[i]);
			}
			fence_async_smem();
			__syncwarp();
			if (lane == 0) mbar_arrive(&full[s]);
		}

		mbar_wait_guard(&accum, 0);
		tc_fence_after();
		const int q4 = warp & 3; // the TMEM lane quarter this warp may read
		const int lr = q4 * 32 + lane, gr = row0 + lr;
		for (int c0 = 0; c0 < PF_BN; c0 += 32) {
			float v[32];
			tmem_ld32(tmem_base + ((uint32_t)(q4 * 32) << 16) + c0, v);
			if constexpr (MODE == PF_QKV) {
				const bool is_q = gr < a.q_dim, is_k = !is_q && gr < a.q_dim + a.kv_dim;
				const int k = is_q ? gr : (is_k ? gr - a.q_dim : gr - a.q_dim - a.kv_dim);
				const int d = k % a.head_dim, h = k / a.head_dim;
				const float b = a.bias ? a.bias[gr] : 0.f;
#pragma unroll
				for (int j = 0; j < 32; ++j) {
					const int t = tok0 + c0 + j;
					float x = fminf(fmaxf(v[j] + b, -a.clip), a.clip);
					const float other = __shfl_xor_sync(0xffffffffu, x, 1); // the row pair a rotation mixes sits in adjacent lanes
					if (t < a.n_tokens) {
						if (is_q || is_k) {
							const float2 cs = a.rope[(size_t)t * (a.head_dim / 2) + (d >> 1)];
							x = (lane & 1) ? fmaf(other, cs.y, x * cs.x) : fmaf(-other, cs.y, x * cs.x);
						}
						if (is_q) {
							a.Q[(size_t)t * a.q_dim + k] = x;
						} else {
							KVT* dst = reinterpret_cast<KVT*>(is_k ? a.kc : a.vc) + ((size_t)h * a.seq_len + a.pos0 + t) * a.head_dim + d;
							kv_store(dst, x);
						}
					}
				}
			} else if constexpr (MODE == PF_UP) {
				float v3[32];
				tmem_ld32(tmem_base + ((uint32_t)(q4 * 32) << 16) + PF_BN + c0, v3);
#pragma unroll
				for (int j = 0; j < 32; ++j) {
					const int t = tok0 + c0 + j;
					if (t < a.n_tokens) {
						const float hv = (a.gelu ? act_gelu(v[j]) : act_silu(v[j])) * v3[j];
						__half hh, hl;
						split_hl(hv, hh, hl);
						a.Hhi[(size_t)t * a.hidden + gr] = hh, a.Hlo[(size_t)t * a.hidden + gr] = hl;
					}
				}
			} else {
#pragma unroll
				for (int j = 0; j < 32; ++j) {
					const int t = tok0 + c0 + j;
					if (t < a.n_tokens) a.X[(size_t)t * a.dim + gr] += v[j];
				}
			}
		}
		tc_fence_before();
	}
	__syncthreads();
	if (warp == 1) {
		tc_fence_after();
		tmem_dealloc(tmem_base, TMEM_COLS);
	}
}

// ---------------------------------------------------------------- causal attention of the block against the cache
// Flash attention on warp-level tensor cores (mma.m16n8k16, fp32 accumulators).  A CTA serves KM of the query heads that share a kv
// head: warp = (head, 16 consecutive tokens), so one 64-key tile of K and V in shared memory feeds up to 128 rows.  The cache
// entries (fp16, or e5m2 widened on the way in) are exact f16 operands; queries and softmax weights travel as an f16 hi + lo
// pair, two MMAs into the same fp32 accumulator, so they keep 22 bits.  A query row is first scaled by the power of two that
// brings its largest entry into [1, 2) (exact; the score is scaled back), so no query leaves the f16 range.  Running maximum,
// exponentials and the denominator are fp32.
// Bound: the MMA rate (4 x 64 MMAs per warp and tile against 32 KB of ldmatrix traffic).  Tokens are taken 16 per warp and not 32 because
// 64 accumulator and 64 query registers per 16 rows already fill the file at 8 warps; the last blocks of the prompt, which see
// the most keys, are started first.  2047 tokens, 32 / 8 heads of 128: 1550 us a layer as fp32 FMAs, one token per warp; about 360 us here.
#define PFA_TILE 64 // keys per tile

struct PfAttnArgs {
	const float* Q; // [T][q_dim]
	const void* kc; // this layer
	const void* vc;
	__half* Ohi;    // [T][q_dim]
	__half* Olo;
	int n_tokens, pos0, seq_len, q_dim, kv_mul;
	int km, tb; // query heads and 16-token blocks per CTA: km * tb warps, km divides kv_mul
	float inv_sqrt_hd;
};

template <int HD>
__host__ __device__ constexpr size_t pfa_smem_bytes() { // two buffers of K and V
	return (size_t)2 * 2 * PFA_TILE * HD * sizeof(__half);
}

__device__ __forceinline__ void ldsm_x4(const void* p, uint32_t (&r)[4]) {
	asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)));
}
__device__ __forceinline__ void ldsm_x4_t(const void* p, uint32_t (&r)[4]) {
	asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)));
}
__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
	asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
	             : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
	             : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool in) { // 16 bytes, zeros when !in
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
// two floats -> (hi, lo) f16 pairs
__device__ __forceinline__ void split_hl2(float x, float y, uint32_t& hi, uint32_t& lo) {
	const __half2 h = __floats2half2_rn(x, y);
	const float2 f = __half22float2(h);
	const __half2 l = __floats2half2_rn(x - f.x, y - f.y);
	hi = *reinterpret_cast<const uint32_t*>(&h), lo = *reinterpret_cast<const uint32_t*>(&l);
}

template <typename KVT, int HD>
__global__ void __launch_bounds__(256, 1) k_pf_attn(const PfAttnArgs a) {
	pdl_enter();
	constexpr int CH = HD / 8;   // 16-byte chunks of a tile row
	constexpr int NT = PFA_TILE / 8, KS = HD / 16, TILE = PFA_TILE * HD;
	extern __shared__ __align__(128) __half sm[];
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
	const int per_kv = a.kv_mul / a.km; // CTAs per kv head and token block
	const int kvh = blockIdx.y / per_kv, head = kvh * a.kv_mul + (blockIdx.y % per_kv) * a.km + warp % a.km;
	const int c0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * 16 * a.tb; // first token of the CTA (the longest rows first)
	const int t0 = c0 + (warp / a.km) * 16;                            // first token of the warp
	const int last = a.pos0 + min(a.n_tokens, c0 + 16 * a.tb) - 1;     // last key position any row of the CTA sees
	const int wlast = a.pos0 + min(a.n_tokens, t0 + 16) - 1;           // ... of this warp (below pos0 + t0: no live row)
	const KVT* kbase = reinterpret_cast<const KVT*>(a.kc) + (size_t)kvh * a.seq_len * HD;
	const KVT* vbase = reinterpret_cast<const KVT*>(a.vc) + (size_t)kvh * a.seq_len * HD;
	// row r, chunk c of a tile lies at chunk c ^ (r & 7): ldmatrix reads 8 rows of one chunk without bank conflicts
	auto at = [&](int buf, int which, int r, int c) { return sm + (size_t)(buf * 2 + which) * TILE + r * HD + ((c ^ (r & 7)) << 3); };
	auto fetch = [&](int buf, int k0) {
		for (int i = tid; i < 2 * PFA_TILE * CH; i += blockDim.x) {
			const int which = i / (PFA_TILE * CH), r = (i / CH) % PFA_TILE, c = i % CH;
			const bool in = k0 + r <= last;
			const KVT* src = (which ? vbase : kbase) + (size_t)(in ? k0 + r : 0) * HD + c * 8;
			if constexpr (sizeof(KVT) == 2) {
				cp_async16(at(buf, which, r, c), src, in);
			} else { // an e5m2 byte is the high byte of the f16
				const uint2 w = in ? __ldcg(reinterpret_cast<const uint2*>(src)) : make_uint2(0, 0);
				*reinterpret_cast<uint4*>(at(buf, which, r, c)) = make_uint4(__byte_perm(w.x, 0, 0x1404), __byte_perm(w.x, 0, 0x3424), __byte_perm(w.y, 0, 0x1404), __byte_perm(w.y, 0, 0x3424));
			}
		}
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
	fetch(0, 0);

	// queries of rows t0 + g and t0 + g + 8 as MMA fragments
	uint32_t qh[KS][4], ql[KS][4];
	float smul[2]; // score factor of the two rows
	{
		float2 q[2][KS][2];
#pragma unroll
		for (int r = 0; r < 2; ++r) {
			const int t = t0 + g + 8 * r;
			const float* qp = a.Q + (size_t)t * a.q_dim + (size_t)head * HD + 2 * t4;
			float mx = 0.f;
#pragma unroll
			for (int k = 0; k < KS; ++k)
#pragma unroll
				for (int j = 0; j < 2; ++j) {
					q[r][k][j] = t < a.n_tokens ? __ldcg(reinterpret_cast<const float2*>(qp + 16 * k + 8 * j)) : make_float2(0.f, 0.f);
					mx = fmaxf(mx, fmaxf(fabsf(q[r][k][j].x), fabsf(q[r][k][j].y)));
				}
			mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1)), mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
			const uint32_t e = __float_as_uint(mx) >> 23; // biased exponent of the largest entry
			const bool normal = e > 0 && e < 254;
			const float down = normal ? __uint_as_float((254 - e) << 23) : 1.f; // 2^(127 - e)
			smul[r] = (normal ? __uint_as_float(e << 23) : 1.f) * a.inv_sqrt_hd;
#pragma unroll
			for (int k = 0; k < KS; ++k)
#pragma unroll
				for (int j = 0; j < 2; ++j) split_hl2(q[r][k][j].x * down, q[r][k][j].y * down, qh[k][2 * j + r], ql[k][2 * j + r]);
		}
	}
	float o[HD / 8][4], m[2] = {-FLT_MAX, -FLT_MAX}, l[2] = {0.f, 0.f};
#pragma unroll
	for (int n = 0; n < HD / 8; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;

	for (int k0 = 0, buf = 0; k0 <= last; k0 += PFA_TILE, buf ^= 1) {
		asm volatile("cp.async.wait_group 0;" ::: "memory");
		__syncthreads(); // the tile has arrived, and the other buffer is no longer being read
		if (k0 + PFA_TILE <= last) fetch(buf ^ 1, k0 + PFA_TILE);
		if (k0 > wlast) continue; // (warp-uniform) nothing of this tile is visible to this warp's rows
		float s[NT][4];
#pragma unroll
		for (int n = 0; n < NT; ++n) {
			s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll
			for (int k = 0; k < KS; k += 2) {
				uint32_t b[4]; // key block n, dims 16k .. 16k + 31
				ldsm_x4(at(buf, 0, n * 8 + (lane & 7), 2 * k + (lane >> 3)), b);
				mma_f16(s[n], qh[k], b[0], b[1]), mma_f16(s[n], ql[k], b[0], b[1]);
				mma_f16(s[n], qh[k + 1], b[2], b[3]), mma_f16(s[n], ql[k + 1], b[2], b[3]);
			}
		}
		float mx[2] = {-FLT_MAX, -FLT_MAX};
		const int p0 = a.pos0 + t0 + g; // position of row 0
		const bool whole = k0 + PFA_TILE - 1 <= a.pos0 + t0; // every row of the warp sees every key of the tile
#pragma unroll
		for (int n = 0; n < NT; ++n)
#pragma unroll
			for (int e = 0; e < 4; ++e) {
				const int r = e >> 1, key = k0 + n * 8 + 2 * t4 + (e & 1);
				s[n][e] = whole || key <= p0 + 8 * r ? s[n][e] * smul[r] : -FLT_MAX;
				mx[r] = fmaxf(mx[r], s[n][e]);
			}
		float corr[2];
#pragma unroll
		for (int r = 0; r < 2; ++r) {
			mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1)), mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
			const float mn = fmaxf(m[r], mx[r]);
			corr[r] = expf(m[r] - mn);
			m[r] = mn, l[r] *= corr[r];
		}
#pragma unroll
		for (int n = 0; n < HD / 8; ++n) o[n][0] *= corr[0], o[n][1] *= corr[0], o[n][2] *= corr[1], o[n][3] *= corr[1];
#pragma unroll
		for (int kk = 0; kk < PFA_TILE / 16; ++kk) { // 16 keys: their weights, then their values
			uint32_t ph[4], pl[4];
#pragma unroll
			for (int j = 0; j < 2; ++j)
#pragma unroll
				for (int r = 0; r < 2; ++r) {
					const float x = s[2 * kk + j][2 * r], y = s[2 * kk + j][2 * r + 1];
					const float px = x == -FLT_MAX ? 0.f : expf(x - m[r]), py = y == -FLT_MAX ? 0.f : expf(y - m[r]);
					l[r] += px + py;
					split_hl2(px, py, ph[2 * j + r], pl[2 * j + r]);
				}
#pragma unroll
			for (int n = 0; n < HD / 8; n += 2) {
				uint32_t b[4]; // (keys 0-7, dims n), (keys 8-15, dims n), (keys 0-7, dims n + 1), (keys 8-15, dims n + 1)
				ldsm_x4_t(at(buf, 1, kk * 16 + (lane & 15), n + (lane >> 4)), b);
				mma_f16(o[n], ph, b[0], b[1]), mma_f16(o[n], pl, b[0], b[1]);
				mma_f16(o[n + 1], ph, b[2], b[3]), mma_f16(o[n + 1], pl, b[2], b[3]);
			}
		}
	}
#pragma unroll
	for (int r = 0; r < 2; ++r) {
		l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1), l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
		const int t = t0 + g + 8 * r;
		if (t >= a.n_tokens) continue;
		const float inv = 1.0f / l[r];
		const size_t at0 = (size_t)t * a.q_dim + (size_t)head * HD + 2 * t4;
#pragma unroll
		for (int n = 0; n < HD / 8; ++n) {
			uint32_t hi, lo;
			split_hl2(o[n][2 * r] * inv, o[n][2 * r + 1] * inv, hi, lo);
			*reinterpret_cast<uint32_t*>(a.Ohi + at0 + 8 * n) = hi, *reinterpret_cast<uint32_t*>(a.Olo + at0 + 8 * n) = lo;
		}
	}
}
