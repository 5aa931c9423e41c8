// prefill.cuh -- batched prompt pass (reference behaviour replaced: run.c:206-209 feeds the prompt one
// token at a time through forward()).  T prompt tokens go through every layer together, so each weight
// matrix is read once per tile of 64 to 256 tokens instead of once per token and the projections become real GEMMs on the
// 5th-generation tensor cores:
//
//   k_pf_gemm   D[128 weight rows][<= 256 tokens] = W_tile . X_tile^T with tcgen05.mma (kind::f16, cta_group::1), fp32
//               accumulators in TMEM.  A = the weight tile, widened ON THE FLY from the model's own format (fp16 / e5m2 /
//               gf4: all exact in f16); B = the activations as TWO f16 matrices hi + lo (x = hi + lo to 22 bits, so the
//               result carries fp32-grade inputs), multiplied as one operand of both or one after the other (pf_side).  The epilogue applies
//               what the decode kernels apply: bias / clip / RoPE / KV-cache append (QKV), residual add (wo, w2),
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

#define PF_BM 128  // weight rows per tile  (TMEM lanes)
#define PF_BK 64   // k per stage: 64 f16 = 128 bytes = one swizzle atom
#define PF_PAD 128 // activation rows are allocated in multiples of this
enum { PF_QKV = 0, PF_RES = 1 /* wo, w2 */, PF_UP = 2 };

// ---------------------------------------------------------------- small kernels

// f32 -> (hi, lo) f16 pair with x = hi + lo up to 2^-22 |x|
__device__ __forceinline__ void split_hl(float x, __half& hi, __half& lo) {
	hi = __float2half_rn(x);
	lo = __float2half_rn(x - __half2float(hi));
}

// two floats -> (hi, lo) f16 pairs
__device__ __forceinline__ void split_hl2(float x, float y, uint32_t& hi, uint32_t& lo) {
	const __half2 h = __floats2half2_rn(x, y);
	const float2 f = __half22float2(h);
	const __half2 l = __floats2half2_rn(x - f.x, y - f.y);
	hi = *reinterpret_cast<const uint32_t*>(&h), lo = *reinterpret_cast<const uint32_t*>(&l);
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

// one CTA per token: norm (infer.c:183-207) then hi / lo split; rows beyond n (tile padding) are zeroed once at allocation.  dim is a multiple of 4;
// a row of up to 8192 is read once, 16 bytes at a time, and stays in registers (the 64 norms of a 333-token Mistral-7B prompt: 0.9 of its 18.7 ms saved)
#define PFN_REGS 8
__global__ void __launch_bounds__(256) k_pf_norm(const float* X, const float* normw, __half* hi, __half* lo, int n, int dim, float eps, int ln) {
	pdl_enter();
	__shared__ float red[32];
	const int t = blockIdx.x, n4 = dim >> 2;
	if (t >= n) return;
	const float4* x = reinterpret_cast<const float4*>(X + (size_t)t * dim);
	float4 v[PFN_REGS];
#pragma unroll
	for (int k = 0; k < PFN_REGS; ++k) {
		const int i = threadIdx.x + k * 256;
		if (i < n4) v[k] = __ldcg(x + i);
	}
	auto each = [&](auto&& f) { // f(group, value of the group)
#pragma unroll
		for (int k = 0; k < PFN_REGS; ++k)
			if ((int)threadIdx.x + k * 256 < n4) f(threadIdx.x + k * 256, v[k]);
		for (int i = threadIdx.x + PFN_REGS * 256; i < n4; i += 256) f(i, __ldcg(x + i));
	};
	float mean = 0.f;
	if (ln) {
		float s = 0.f;
		each([&](int, float4 a) { s += (a.x + a.y) + (a.z + a.w); });
		mean = block_sum(s, red) / dim;
	}
	float ss = 0.f;
	each([&](int, float4 a) {
		a.x -= mean, a.y -= mean, a.z -= mean, a.w -= mean;
		ss += (a.x * a.x + a.y * a.y) + (a.z * a.z + a.w * a.w);
	});
	ss = block_sum(ss, red);
	const float scale = 1.0f / sqrtf(ss / dim + eps);
	each([&](int i, float4 a) {
		const float4 w = __ldg(reinterpret_cast<const float4*>(normw) + i);
		uint2 h, l;
		split_hl2((a.x - mean) * scale * w.x, (a.y - mean) * scale * w.y, h.x, l.x);
		split_hl2((a.z - mean) * scale * w.z, (a.w - mean) * scale * w.w, h.y, l.y);
		reinterpret_cast<uint2*>(hi + (size_t)t * dim)[i] = h, reinterpret_cast<uint2*>(lo + (size_t)t * dim)[i] = l;
	});
}

// ---------------------------------------------------------------- the GEMM
//
// Persistent: a CTA walks work items = (one or two tiles of 128 weight rows, K-slice, bn tokens), token tiles fastest, so that
// the CTAs running at one time share a weight tile's bytes in L2.  Roles, each with its own ring so that none waits for another's
// latency: two warps stream the hi and the lo activation tiles and one the weight bytes in the model's format (TMA; a warp gets one copy on its
// way every 300 cycles or so), four or eight widen them to f16 in the swizzled layout of the MMA (fp16 weights arrive in it), warp 1
// issues the MMAs, warps 2-5 drain one of two TMEM accumulators while the other is being filled.
// Bound: the MMA warp's hand-overs (tensor pipe 42 to 61 % active).  Everything a stage needs arrives on one barrier (with a wait and a commit for the weights,
// for hi and for lo, FFN up took a fifth longer) and an item is as large as TMEM allows.  14336 x 2 rows, K 4096, 2047 tokens: fp8 733 us,
// fp16 717 us (1310 and 1340 TFLOP/s, hi and lo counted; 1324 us (fp8) when every thread loaded its weight row one stage ahead); 4096 rows:
// 135 and 118 us (387 us).
//
// Slices of a tile that fit a thread-block cluster (up to eight, and all clusters at a time) are folded through distributed shared memory: each CTA leaves its sums
// where its stages were, and adds up, with all its threads, a share of the tile's tokens.  Through memory the last slice to arrive waited for 32 tokens of
// two slices at a time, with four warps, behind a fence and a counter: 5000 cycles and 15 more per slice, row tile and token, where this costs 2500 and 30 in all.  With it slices pay
// for products that were whole.  Qwen2-0.5B fp16, us a layer without the classifier's token: 20 / 61 / 130 / 400 tokens 73.9 -> 53.8, 86.9 -> 62.9, 88.7 -> 73.7, 114.6 -> 109.2;
// Llama-3-8B fp8 61 / 130 / 300: 184 -> 176, 304 -> 295, 435 -> 418; Mistral-7B gf4 61 / 333: 198 -> 180, 447 -> 429.
struct PfMaps {
	CUtensorMap x[2]; // activations, hi and lo: f16 [tokens][K], box = bn rows x 64 columns, 128-byte swizzle
	CUtensorMap w[3]; // weights: QKV: wq, wk, wv   UP: w1, w3   WO / DOWN: w
};

struct PfGemmArgs {
	int K, n_tokens;
	// work items
	int rows, na, bn; // weight rows; row tiles per item (UP: 2, w1 and w3); tokens per tile (64, 128 or 256, na * bn <= 256)
	int tail, splits; // the last `tail` tiles are cut into K-slices, an item each (tail * splits of them, at most one per SM); the others are one item
	int stages;               // in flight
	float* ws;            // [slice of a tail tile][na][bn][128] partial sums
	unsigned* counter;    // [tail tile] slices that have arrived, zero between launches
	int* err;             // mapped host word: code of a wait that gave up
	unsigned wait_limit;  // tries of a wait before it gives up
	// QKV epilogue
	float* Q;         // [T][q_dim]
	int q_dim, kv_dim, head_dim, seq_len, pos0, kvbits;
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

#define PF_TILE_BYTES (PF_BM * 128)
#define PF_MAX_STAGES 6
template <int DBITS>
__host__ __device__ constexpr int pf_raw_bytes() {
	return PF_BM * PF_BK * DBITS / 8;
}
// shared memory: weight tiles as stored (fp16: none), then stages = widened weight tiles, hi tile, lo tile
template <int DBITS>
__host__ __device__ constexpr int pf_raw_tiles() {
	return DBITS == 16 ? 0 : 32768 / pf_raw_bytes<DBITS>();
}
template <int DBITS>
__host__ __device__ constexpr size_t pf_fixed_bytes() { // everything but the stages
	return (size_t)pf_raw_tiles<DBITS>() * pf_raw_bytes<DBITS>() + 1024; // + alignment slack
}
__host__ __device__ inline size_t pf_stage_bytes(int na, int bn) {
	return (size_t)na * PF_TILE_BYTES + 2 * bn * 128;
}
// Tiles whose accumulators leave room multiply hi and lo as one operand, so that the weight tile is read from shared memory once for both: those reads, the
// activations', the copies and the widening share its 128 bytes a cycle, which is what bounds a stage (FFN up 14336 x 4096 fp8: 135 tokens 188 -> 150 us, 20 tokens 70 -> 57).
__host__ __device__ constexpr bool pf_side(int na, int bn) { return na * bn <= 128; }
template <int DBITS>
__host__ __device__ constexpr int pf_widen_warps() { // FFN up as above, side by side: fp8 696 us with four warps and 802 with eight (more arrivals per stage), gf4 871 and 825 (19 instructions per 8 weights)
	return DBITS == 16 ? 0 : DBITS == 8 ? 4 : 8;
}
template <int DBITS>
__host__ __device__ constexpr int pf_threads() {
	return (8 + pf_widen_warps<DBITS>()) * 32;
}

// 16 bytes i of row r (one k-stage of it) out of the copied bytes.  The copy swizzles them (64-byte pattern for fp8, 32-byte for gf4), so that a
// row per lane reads without bank conflicts.
template <int DBITS>
__device__ __forceinline__ uint4 pf_load_raw(const unsigned char* raw, int r, int i) {
	const int c = DBITS == 8 ? i ^ ((r >> 1) & 3) : i ^ ((r >> 2) & 1);
	uint4 w;
	// volatile: these reads stay ahead of the arrival that lets the copy engine overwrite the slot
	asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w) : "r"(smem_u32(raw + r * (PF_BK * DBITS / 8) + (c << 4))) : "memory");
	return w;
}
// ... widened: 16 / 32 weights are 2 / 4 16-byte chunks of f16
template <int DBITS>
__device__ __forceinline__ void pf_widen(const uint4& raw, uint4* out) {
	const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
	if constexpr (DBITS == 8) { // an e5m2 byte is the high byte of the f16 (reference infer.c:28-35)
		out[0] = make_uint4(__byte_perm(w[0], 0, 0x1404), __byte_perm(w[0], 0, 0x3424), __byte_perm(w[1], 0, 0x1404), __byte_perm(w[1], 0, 0x3424));
		out[1] = make_uint4(__byte_perm(w[2], 0, 0x1404), __byte_perm(w[2], 0, 0x3424), __byte_perm(w[3], 0, 0x1404), __byte_perm(w[3], 0, 0x3424));
	} else { // gf4 (reference infer.c:37-40)
#pragma unroll
		for (int j = 0; j < 4; ++j) {
			uint32_t h[4];
			gf4_to_h2(w[j], h);
			out[j] = make_uint4(h[0], h[1], h[2], h[3]);
		}
	}
}

// What the decode kernels apply, on N tokens of one weight row: gr = row (lanes = consecutive rows), t0 = first token, v (v3: FFN up's second matrix) the sums.
// Values are formed without asking whether their token is there, several at a time, and only the stores ask: a condition around each value kept the
// values apart (q/k/v of 20 / 135 tokens, 6144 x 4096 fp8: 31 -> 26, 65 -> 50 us).
template <int MODE, int N>
__device__ __forceinline__ void pf_epilogue(const PfGemmArgs& a, int gr, int lane, int t0, int left, const float (&v)[N], const float (&v3)[N]) {
	if constexpr (MODE == PF_QKV) { // bias / clip / RoPE / KV-cache append
		const bool is_q = gr < a.q_dim, is_k = !is_q && gr < a.q_dim + a.kv_dim; // uniform over a tile: the dims are multiples of 128
		const int k = is_q ? gr : (is_k ? gr - a.q_dim : gr - a.q_dim - a.kv_dim);
		const int d = k % a.head_dim, h = k / a.head_dim;
		const float b = a.bias ? a.bias[gr] : 0.f;
		const size_t kv0 = ((size_t)h * a.seq_len + a.pos0 + t0) * a.head_dim + d;
		void* const cache = is_k ? a.kc : a.vc;
		constexpr int G = N < 16 ? N : 16;
#pragma unroll
		for (int j0 = 0; j0 < N; j0 += G) { // the angles of up to 16 tokens at a time, all loads before the first store (one by one they cost a round trip each)
			float x[G];
#pragma unroll
			for (int j = 0; j < G; ++j) x[j] = fminf(fmaxf(v[j0 + j] + b, -a.clip), a.clip);
			if (is_q || is_k) {
				float2 cs[G];
#pragma unroll
				for (int j = 0; j < G; ++j) cs[j] = j0 + j < left ? __ldcg(a.rope + (size_t)(t0 + j0 + j) * (a.head_dim / 2) + (d >> 1)) : make_float2(1.f, 0.f);
#pragma unroll
				for (int j = 0; j < G; ++j) {
					const float other = __shfl_xor_sync(0xffffffffu, x[j], 1); // the row pair a rotation mixes sits in adjacent lanes
					x[j] = (lane & 1) ? fmaf(other, cs[j].y, x[j] * cs[j].x) : fmaf(-other, cs[j].y, x[j] * cs[j].x);
				}
			}
			auto store = [&](auto* p, size_t step, auto&& put) {
#pragma unroll
				for (int j = 0; j < G; ++j)
					if (j0 + j < left) put(p + j * step, x[j]);
			};
			const size_t hd = a.head_dim, o = kv0 + (size_t)j0 * hd;
			if (is_q) store(a.Q + (size_t)(t0 + j0) * a.q_dim + k, a.q_dim, [](float* q, float y) { *q = y; });
			else if (a.kvbits == 16) store(reinterpret_cast<__half*>(cache) + o, hd, [](__half* q, float y) { kv_store(q, y); });
			else store(reinterpret_cast<uint8_t*>(cache) + o, hd, [](uint8_t* q, float y) { kv_store(q, y); });
		}
	} else if constexpr (MODE == PF_UP) { // act(w1 x) * (w3 x)
		__half* const ph = a.Hhi + (size_t)t0 * a.hidden + gr;
		__half* const pl = a.Hlo + (size_t)t0 * a.hidden + gr;
		constexpr int G = N < 8 ? N : 8;
#pragma unroll
		for (int j0 = 0; j0 < N; j0 += G) {
			__half hh[G], hl[G];
			if (a.gelu) {
#pragma unroll
				for (int j = 0; j < G; ++j) split_hl(act_gelu(v[j0 + j]) * v3[j0 + j], hh[j], hl[j]);
			} else {
#pragma unroll
				for (int j = 0; j < G; ++j) split_hl(act_silu(v[j0 + j]) * v3[j0 + j], hh[j], hl[j]);
			}
#pragma unroll
			for (int j = 0; j < G; ++j)
				if (j0 + j < left) ph[(size_t)(j0 + j) * a.hidden] = hh[j], pl[(size_t)(j0 + j) * a.hidden] = hl[j];
		}
	} else { // residual add: all loads before the first store
		float x[N];
		float* p = a.X + (size_t)t0 * a.dim + gr;
#pragma unroll
		for (int j = 0; j < N; ++j) x[j] = j < left ? __ldcg(p + (size_t)j * a.dim) : 0.f;
#pragma unroll
		for (int j = 0; j < N; ++j)
			if (j < left) p[(size_t)j * a.dim] = x[j] + v[j];
	}
}

// named barrier of `threads` threads that also tells whether `p` held for all of them
__device__ __forceinline__ bool bar_and(int id, int threads, bool p) {
	int all;
	asm volatile(
	    "{\n\t.reg .pred p, q;\n\t"
	    "setp.ne.s32 p, %3, 0;\n\t"
	    "barrier.cta.red.and.pred q, %1, %2, p;\n\t"
	    "selp.s32 %0, 1, 0, q;\n\t}"
	    : "=r"(all)
	    : "r"(id), "r"(threads), "r"((int)p)
	    : "memory");
	return all != 0;
}

// CLUSTER: every tile is cut, the slices of a tile are one thread-block cluster, and each of its CTAs has one item
template <int MODE, int DBITS, bool CLUSTER>
__global__ void __launch_bounds__(pf_threads<DBITS>(), 1) k_pf_gemm(const __grid_constant__ PfMaps m, const PfGemmArgs a) {
	constexpr int WIDEN = pf_widen_warps<DBITS>(), W_WARP = 6 + WIDEN, LO_WARP = W_WARP + 1;
	constexpr int ROLES = 2 + (DBITS == 16 ? 1 : WIDEN); // arrivals that make a stage full: hi, lo, then the weight copy or the widening warps
	constexpr int RT = pf_raw_tiles<DBITS>(), RAW = pf_raw_bytes<DBITS>();
	extern __shared__ unsigned char smem_dyn[];
	__shared__ __align__(8) uint64_t full[PF_MAX_STAGES], empty[PF_MAX_STAGES], r_full[RT ? RT : 1], r_empty[RT ? RT : 1], acc_full[2], acc_empty[2];
	__shared__ uint32_t tmem_base_s;
	__shared__ int last_s;
	__shared__ int handed[ROLES], raw_handed, multiplied, accumulated; // stages and items that each role got to (read when a wait has given up)
	unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int nkb = a.K / PF_BK, ns = a.stages, bn = a.bn, splits = a.splits, tail = a.tail, na = MODE == PF_UP ? 2 : a.na;
	const int rs = RT / na; // slots of na weight tiles
	const int row_tiles = a.rows / PF_BM, tok_tiles = (a.n_tokens + bn - 1) / bn;
	const int whole = (MODE == PF_UP ? row_tiles : (row_tiles + na - 1) / na) * tok_tiles - tail, items = whole + tail * splits;
	const int b_bytes = bn * 128;
	const bool side = pf_side(na, bn);
	const int ac = side ? 2 * bn : bn; // accumulator columns of a weight tile: its sums with hi and with lo side by side, or both in one
	const size_t stage_bytes = pf_stage_bytes(na, bn);
	auto r_tile = [&](int s, int i) { return smem + (size_t)(s * na + i) * RAW; };
	auto a_tile = [&](int s, int i) { return smem + (size_t)RT * RAW + s * stage_bytes + (size_t)i * PF_TILE_BYTES; };
	auto b_tile = [&](int s) { return smem + (size_t)RT * RAW + s * stage_bytes + (size_t)na * PF_TILE_BYTES; };
	float* const partial = reinterpret_cast<float*>(smem + (size_t)RT * RAW); // a cluster's slice: [na][bn][128] sums where the stages were
	// item -> first weight row, tiles, first token, k-stages [k0, k1), which slice of the tail it is (slices of one k next to each other; -1: none)
	struct Item {
		int row0, cnt, tok0, k0, k1, part;
	};
	auto item_of = [&](int it) {
		Item r;
		r.part = it < whole ? -1 : it - whole;
		const int tile = it < whole ? it : CLUSTER ? r.part / splits : whole + r.part % tail, sp = it < whole ? 0 : CLUSTER ? r.part % splits : r.part / tail, of = it < whole ? 1 : splits, rt = tile / tok_tiles * (MODE == PF_UP ? 1 : na);
		r.tok0 = (tile % tok_tiles) * bn, r.row0 = rt * PF_BM, r.cnt = MODE == PF_UP ? 2 : min(na, row_tiles - rt);
		r.k0 = (int)((long)nkb * sp / of), r.k1 = (int)((long)nkb * (sp + 1) / of);
		return r;
	};
	// every wait is bounded: a role whose wait gives up (whole warps at a time) records a code and leaves its loop, the others follow, what is on its
	// way into shared memory or TMEM is waited for, and the host reads the code
	auto gave_up = [&](int code) {
		if (a.err) *reinterpret_cast<volatile int*>(a.err) = code;
		return false;
	};

	pdl_launch_next();
	if (tid == 0) {
		for (int s = 0; s < RT; ++s) mbar_init(&r_full[s], 1), mbar_init(&r_empty[s], WIDEN);
		for (int s = 0; s < ns; ++s) mbar_init(&full[s], ROLES), mbar_init(&empty[s], 1);
		for (int s = 0; s < 2; ++s) mbar_init(&acc_full[s], 1), mbar_init(&acc_empty[s], 4);
		mbar_init_fence();
	}
	if (warp == 1) tmem_alloc(&tmem_base_s, 512);
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem_base = tmem_base_s; // accumulator i of buffer b: columns 256 b + ac i

	// The one-thread roles keep their warp together and elect a lane for the issuing: addresses and descriptors then live in uniform registers
	// (one lane in a branch of its own spent 60 cycles per MMA on moving them).
	bool ok = true;
	if (warp == 0 || warp == LO_WARP) { // ===== activations: one warp the hi, one the lo tile of a stage
		pdl_wait_prev();
		const bool el = elect_one();
		const int lo = warp != 0;
		int s = 0, n = 0;
		unsigned ph = 1;
		for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
			const Item t = item_of(it);
			for (int kb = t.k0; kb < t.k1; ++kb) {
				if (!mbar_wait_warp(&empty[s], ph, a.wait_limit)) {
					ok = gave_up(9301);
					break;
				}
				if (el) {
					mbar_expect_tx(&full[s], b_bytes);
					tma_load_2d(b_tile(s) + lo * b_bytes, &m.x[lo], kb * PF_BK, t.tok0, &full[s]);
				}
				++n;
				if (++s == ns) s = 0, ph ^= 1;
			}
		}
		if (lane == 0) handed[lo] = n;
	} else if (warp == 1) { // ===== MMAs
		// kind::f16: D = f32, A = B = f16, both K-major, M = 128, N = ac (the lo tile lies right behind the hi tile: as one operand they are 2 bn rows)
		const uint32_t idesc = (1u << 4) | ((uint32_t)(ac >> 3) << 17) | ((uint32_t)(PF_BM >> 4) << 24);
		const bool el = elect_one();
		int s = 0, n = 0;
		unsigned ph = 0, q = 0;
		for (int it = blockIdx.x; it < items; it += gridDim.x, ++q) {
			const Item t = item_of(it);
			const uint32_t acc = tmem_base + (q & 1) * 256;
			if (!mbar_wait_warp(&acc_empty[q & 1], ((q >> 1) & 1) ^ 1, a.wait_limit)) ok = gave_up(9302);
			tc_fence_after();
			for (int kb = t.k0; kb < t.k1 && ok; ++kb) {
				if (!mbar_wait_warp(&full[s], ph, a.wait_limit)) {
					ok = gave_up(9303);
					break;
				}
				if (el) {
					const uint64_t db = umma_desc_sw128(b_tile(s)), da = umma_desc_sw128(a_tile(s, 0));
#pragma unroll
					for (int k = 0; k < PF_BK / 16; ++k) // 16 f16 = 32 bytes along K inside the swizzle atom: +2 in the 16-byte address field
#pragma unroll
						for (int i = 0; i < 2; ++i)
							if (i < t.cnt) {
								const uint64_t dw = da + i * (PF_TILE_BYTES >> 4) + 2 * k;
								umma_f16(acc + i * ac, dw, db + 2 * k, idesc, (kb > t.k0 || k) ? 1u : 0u);
								if (!side) umma_f16(acc + i * ac, dw, db + (b_bytes >> 4) + 2 * k, idesc, 1u);
							}
					umma_commit(&empty[s]); // frees the stage when these MMAs have read it
				}
				__syncwarp();
				++n;
				if (++s == ns) s = 0, ph ^= 1;
			}
			if (!ok) break;
			if (el) umma_commit(&acc_full[q & 1]);
			__syncwarp();
		}
		if (lane == 0) multiplied = n, accumulated = q;
	} else if (warp < 6) { // ===== epilogue: one accumulator row per thread
		pdl_wait_prev();
		const int q4 = warp & 3, lr = q4 * 32 + lane; // the TMEM lane quarter this warp may read
		unsigned q = 0;
		for (int it = blockIdx.x; it < items; it += gridDim.x, ++q) {
			const Item t = item_of(it);
			const uint32_t acc = tmem_base + (q & 1) * 256 + ((uint32_t)(q4 * 32) << 16);
			// the four warps go on together or leave together: none is left alone at a named barrier
			if (!bar_and(1, 128, mbar_wait_bounded(&acc_full[q & 1], (q >> 1) & 1, a.wait_limit))) {
				ok = gave_up(9305);
				break;
			}
			tc_fence_after();
			const int cols = min(bn, a.n_tokens - t.tok0);
			float v[32], v3[32];
			auto sums = [&](int i, int c0, float(&to)[32]) { // of tile i, 32 tokens from c0
				tmem_ld32(acc + i * ac + c0, to);
				if (side) {
					float lo[32];
					tmem_ld32(acc + i * ac + bn + c0, lo);
#pragma unroll
					for (int j = 0; j < 32; ++j) to[j] += lo[j];
				}
			};
			if (t.part < 0) {
				for (int i = 0; i < (MODE == PF_UP ? 1 : t.cnt); ++i)
					for (int c0 = 0; c0 < cols; c0 += 32) {
						sums(i, c0, v);
						if (MODE == PF_UP) sums(1, c0, v3);
						pf_epilogue<MODE, 32>(a, t.row0 + i * PF_BM + lr, lane, t.tok0 + c0, a.n_tokens - t.tok0 - c0, v, v3);
					}
			} else if constexpr (CLUSTER) { // the ring is free: every stage has been multiplied
				for (int i = 0; i < t.cnt; ++i)
					for (int c0 = 0; c0 < cols; c0 += 32) {
						sums(i, c0, v);
						float* p = partial + (size_t)(i * bn + c0) * PF_BM + lr;
#pragma unroll
						for (int j = 0; j < 32; ++j) p[j * PF_BM] = v[j];
					}
			} else {
				for (int i = 0; i < t.cnt; ++i)
					for (int c0 = 0; c0 < cols; c0 += 32) {
						sums(i, c0, v);
						float* p = a.ws + ((size_t)(t.part * na + i) * bn + c0) * PF_BM + lr;
#pragma unroll
						for (int j = 0; j < 32; ++j) __stcg(p + j * PF_BM, v[j]);
					}
			}
			tc_fence_before();
			__syncwarp();
			if (lane == 0) mbar_arrive(&acc_empty[q & 1]);
			if (!CLUSTER && t.part >= 0) { // the last slice of a tile to arrive adds all of them up in slice order
				const int tile = t.part % tail;
				__threadfence();
				asm volatile("bar.sync 1, 128;" ::: "memory");
				if (tid == 64) {
					const bool last = atomicAdd(a.counter + tile, 1u) == (unsigned)splits - 1;
					if (last) a.counter[tile] = 0;
					last_s = last;
				}
				asm volatile("bar.sync 1, 128;" ::: "memory");
				const bool last = last_s;
				asm volatile("bar.sync 1, 128;" ::: "memory");
				if (!last) continue;
				__threadfence();
				auto fold = [&](int i, int c0, float(&sum)[32]) {
#pragma unroll
					for (int j = 0; j < 32; ++j) sum[j] = 0.f;
					constexpr int AHEAD = DBITS == 4 ? 1 : 2; // slices whose loads are out at a time
#pragma unroll AHEAD
					for (int sp = 0; sp < splits; ++sp) {
						const float* p = a.ws + ((size_t)((tile + sp * tail) * na + i) * bn + c0) * PF_BM + lr;
#pragma unroll
						for (int j = 0; j < 32; ++j) sum[j] += __ldcg(p + j * PF_BM);
					}
				};
				for (int i = 0; i < (MODE == PF_UP ? 1 : t.cnt); ++i)
					for (int c0 = 0; c0 < cols; c0 += 32) {
						fold(i, c0, v);
						if (MODE == PF_UP) fold(1, c0, v3);
						pf_epilogue<MODE, 32>(a, t.row0 + i * PF_BM + lr, lane, t.tok0 + c0, a.n_tokens - t.tok0 - c0, v, v3);
					}
			}
		}
	} else if (warp == W_WARP) { // ===== weights: immutable, so the first tiles are requested before the previous kernel has finished
		uint64_t* wfull = DBITS == 16 ? full : r_full;
		uint64_t* wempty = DBITS == 16 ? empty : r_empty;
		const int ws = DBITS == 16 ? ns : rs;
		const bool el = elect_one();
		int s = 0, n = 0;
		unsigned ph = 1;
		for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
			const Item t = item_of(it);
			for (int kb = t.k0; kb < t.k1; ++kb) {
				if (!mbar_wait_warp(&wempty[s], ph, a.wait_limit)) {
					ok = gave_up(9306);
					break;
				}
				if (el) {
					mbar_expect_tx(&wfull[s], t.cnt * RAW);
					for (int i = 0; i < t.cnt; ++i) {
						int row = t.row0 + (MODE == PF_UP ? 0 : i * PF_BM), which = MODE == PF_UP ? i : 0;
						if (MODE == PF_QKV && row >= a.q_dim) {
							row -= a.q_dim, which = 1;
							if (row >= a.kv_dim) row -= a.kv_dim, which = 2;
						}
						tma_load_2d(DBITS == 16 ? a_tile(s, i) : r_tile(s, i), &m.w[which], kb * (DBITS == 16 ? PF_BK : PF_BK * DBITS / 8), row, &wfull[s]);
					}
				}
				++n;
				if (++s == ws) s = 0, ph ^= 1;
			}
		}
		if (lane == 0) (DBITS == 16 ? handed[2] : raw_handed) = n;
	} else if constexpr (DBITS != 16) { // ===== widening: a row per thread; with eight warps a tile each of two, or half the row each of one
		constexpr int NV = DBITS / 2, PER = 8 / NV, NT = WIDEN == 4 ? 2 : 1; // 16-byte vectors of a row's k-stage, chunks of f16 from each, tiles per thread
		const int r = (tid - 192) & 127, part = (tid - 192) >> 7;
		const bool whole = WIDEN == 4 || na == 2;
		const int tile0 = WIDEN == 8 && na == 2 ? part : 0, i0 = whole ? 0 : part * (NV / 2);
		int sr = 0, sa = 0, n = 0;
		unsigned pr = 0, pe = 1;
		for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
			const Item t = item_of(it);
			const int nt = min(NT, t.cnt - tile0);
			for (int kb = t.k0; kb < t.k1; ++kb) {
				uint4 raw[NT][NV];
				if (!mbar_wait_warp(&r_full[sr], pr, a.wait_limit)) {
					ok = gave_up(9307);
					break;
				}
#pragma unroll
				for (int j = 0; j < NT; ++j)
					if (j < nt) {
#pragma unroll
						for (int i = 0; i < NV; ++i)
							if (whole || i < NV / 2) raw[j][i] = pf_load_raw<DBITS>(r_tile(sr, tile0 + j), r, i0 + i);
					}
				fence_async_smem(); // the copy engine writes next what was read here
				__syncwarp();
				if (lane == 0) mbar_arrive(&r_empty[sr]);
				if (!mbar_wait_warp(&empty[sa], pe, a.wait_limit)) {
					ok = gave_up(9308);
					break;
				}
#pragma unroll
				for (int j = 0; j < NT; ++j)
					if (j < nt) {
						unsigned char* const dst = a_tile(sa, tile0 + j) + r * 128;
#pragma unroll
						for (int i = 0; i < NV; ++i)
							if (whole || i < NV / 2) {
								uint4 out[PER];
								pf_widen<DBITS>(raw[j][i], out);
#pragma unroll
								for (int c = 0; c < PER; ++c) *reinterpret_cast<uint4*>(dst + ((((i0 + i) * PER + c) ^ (r & 7)) << 4)) = out[c];
							}
					}
				fence_async_smem();
				__syncwarp();
				if (lane == 0) mbar_arrive(&full[sa]);
				++n;
				if (++sr == rs) sr = 0, pr ^= 1;
				if (++sa == ns) sa = 0, pe ^= 1;
			}
		}
		if (lane == 0) handed[warp - 4] = n;
	}
	tc_fence_before();
	if (__syncthreads_or(!ok)) { // a wait gave up: the copies and MMAs already issued end before the CTA does
		if (tid == 0) {
			int most = 0;
			for (int r = 0; r < ROLES; ++r) most = max(most, handed[r]);
			// no role is ns stages ahead of another, so each barrier is in the phase of one of the last ns stages; it gets the arrivals of the roles that
			// did not come that far and then completes with its copies
			for (int i = max(0, most - ns); i < most; ++i) {
				for (int r = 0; r < ROLES; ++r)
					if (handed[r] <= i) mbar_arrive(&full[i % ns]);
				mbar_wait_bounded(&full[i % ns], (i / ns) & 1);
			}
			if constexpr (RT > 0)
				for (int i = max(0, raw_handed - rs); i < raw_handed; ++i) mbar_wait_bounded(&r_full[i % rs], (i / rs) & 1);
			if (multiplied) mbar_wait_bounded(&empty[(multiplied - 1) % ns], ((multiplied - 1) / ns) & 1);
			if (accumulated) mbar_wait_bounded(&acc_full[(accumulated - 1) & 1], ((accumulated - 1) >> 1) & 1);
		}
		__syncthreads();
	}
	if constexpr (CLUSTER) { // each CTA of a tile adds up, in slice order, and finishes its share of the tile's tokens
		pdl_wait_prev(); // (roles that touch nothing of the previous kernel have not waited for it)
		cluster_sync();
		const Item t = item_of(blockIdx.x);
		const int cols = min(bn, a.n_tokens - t.tok0), rank = blockIdx.x % splits;
		const int lo = cols * rank / splits, hi = cols * (rank + 1) / splits, groups = pf_threads<DBITS>() / PF_BM, lr = tid % PF_BM;
		for (int i = 0; i < (MODE == PF_UP ? 1 : t.cnt); ++i)
			for (int c = lo + tid / PF_BM * 4; c < hi; c += 4 * groups) { // four tokens of a row a thread
				float v[4] = {0.f, 0.f, 0.f, 0.f}, v3[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
				for (int sp = 0; sp < splits; ++sp) {
					const uint32_t peer = cluster_addr(partial + (size_t)(i * bn + c) * PF_BM + lr, sp);
#pragma unroll
					for (int j = 0; j < 4; ++j)
						if (c + j < hi) {
							v[j] += cluster_load_f32(peer + j * PF_BM * 4);
							if (MODE == PF_UP) v3[j] += cluster_load_f32(peer + (bn + j) * PF_BM * 4);
						}
				}
				pf_epilogue<MODE, 4>(a, t.row0 + i * PF_BM + lr, lane, t.tok0 + c, hi - c, v, v3);
			}
		cluster_sync(); // no CTA leaves while another reads its sums
	}
	if (warp == 1) {
		tc_fence_after();
		tmem_dealloc(tmem_base, 512);
	}
}

// ---------------------------------------------------------------- causal attention of the block against the cache
// Flash attention on warp-level tensor cores (mma.m16n8k16, fp32 accumulators).  A CTA serves KM of the query heads that share a kv
// head: warp = (head, 16 consecutive tokens), so one 64-key tile of K and V in shared memory feeds up to 128 rows.  The cache
// entries (fp16, or e5m2 widened on the way in) are exact f16 operands; queries and softmax weights travel as an f16 hi + lo
// pair, two MMAs into the same fp32 accumulator, so they keep 22 bits.  A query row is first scaled by the power of two that
// brings its largest entry into [1, 2) (exact; the score is scaled back), so no query leaves the f16 range.  The weights (at most 1) carry a factor
// of 2^15, which the denominator shares: 22 bits down to 2^-18 of the largest, steps of 2^-39 of it below (without the factor 2^-24: a
// thousand keys of 2^-26 were lost).  Running maximum, exponentials and the denominator are fp32.
// Bound: the MMA rate (4 x 64 MMAs per warp and tile against 32 KB of ldmatrix traffic).  Tokens are taken 16 per warp and not 32 because
// 64 accumulator and 64 query registers per 16 rows already fill the file at 8 warps; the last blocks of the prompt, which see
// the most keys, are started first.  2047 tokens, 32 / 8 heads of 128: 1550 us a layer as fp32 FMAs, one token per warp; 365 us here (tensor pipe 35 % active).
#define PFA_TILE 64 // keys per tile
#define PFA_ONE 32768.f // weight of the largest score

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

__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
	asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
	             : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
	             : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool in) { // 16 bytes, zeros when !in
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
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
			const int kb = k0 + kk * 16;
			if (kb > wlast) continue; // (warp-uniform) seen by no row of the warp
			uint32_t ph[4], pl[4];
#pragma unroll
			for (int j = 0; j < 2; ++j)
#pragma unroll
				for (int r = 0; r < 2; ++r) {
					const float x = s[2 * kk + j][2 * r], y = s[2 * kk + j][2 * r + 1];
					const float px = x == -FLT_MAX ? 0.f : expf(x - m[r]) * PFA_ONE, py = y == -FLT_MAX ? 0.f : expf(y - m[r]) * PFA_ONE;
					l[r] += px + py;
					split_hl2(px, py, ph[2 * j + r], pl[2 * j + r]);
				}
			if (sizeof(KVT) == 2 && kb + 15 > a.pos0 + t0) { // some rows do not see some of the keys: a weight of zero must not meet an infinity (e5m2 entries are finite)
				bool finite = true;
#pragma unroll
				for (int n = 0; n < HD / 8; n += 2) {
					uint32_t b[4];
					ldsm_x4_t(at(buf, 1, kk * 16 + (lane & 15), n + (lane >> 4)), b);
#pragma unroll
					for (int i = 0; i < 4; ++i) finite &= __vcmpeq2(b[i] & 0x7c007c00u, 0x7c007c00u) == 0;
				}
				if (!__all_sync(0xffffffffu, finite)) { // key by key, for the rows that see it
#pragma unroll 1
					for (int i = 0; i < 16; ++i) {
						float p[2];
						const int key = kb + i, half = i >> 3, src = (lane & ~3) | ((i & 7) >> 1); // the lane of the quad that has the key's weights
#pragma unroll
						for (int r = 0; r < 2; ++r) {
							const uint32_t hw = __shfl_sync(0xffffffffu, half ? ph[2 + r] : ph[r], src), lw = __shfl_sync(0xffffffffu, half ? pl[2 + r] : pl[r], src);
							const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&hw)), l2 = __half22float2(*reinterpret_cast<const __half2*>(&lw));
							p[r] = i & 1 ? h.y + l2.y : h.x + l2.x;
						}
#pragma unroll
						for (int n = 0; n < HD / 8; ++n) {
							const float2 v = __half22float2(*reinterpret_cast<const __half2*>(at(buf, 1, kk * 16 + i, n) + 2 * t4));
							if (key <= p0) o[n][0] = fmaf(p[0], v.x, o[n][0]), o[n][1] = fmaf(p[0], v.y, o[n][1]);
							if (key <= p0 + 8) o[n][2] = fmaf(p[1], v.x, o[n][2]), o[n][3] = fmaf(p[1], v.y, o[n][3]);
						}
					}
					continue;
				}
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
