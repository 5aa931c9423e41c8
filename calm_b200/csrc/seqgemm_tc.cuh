// seqgemm_tc.cuh -- the layer-list products on the 5th-generation tensor cores (bf16 mode, many tokens):
//   D[128 weight rows][128 tokens] += W_tile . X_tile^T with tcgen05.mma (kind::f16 on bf16 operands, cta_group::1; large products: 256 x 256 on
//   pairs of CTAs, cta_group::2),
//   fp32 accumulators in TMEM.  Both operands are K-major bf16 matrices in global memory (weights as stored,
//   activations as the producing kernels wrote them) and come in by TMA (cp.async.bulk.tensor, SWIZZLE_128B; edges of M,
//   N and K are zero-filled by the copy).  One lane issues the copies, one lane the MMAs, completion flows through
//   mbarriers (tcgen05.commit); four warps read the accumulators back (tcgen05.ld) and apply the epilogue of the product, in an instance of
//   the kernel for each common one (tg_epilogue; the same arithmetic as gemm_store, which serves the rest and the other kernels).  blockIdx.z walks a batch of per-head products
//   (3-D tensor maps; an operand shared by the batch keeps a 2-D map).
// Every wait is bounded: a stalled pipeline records a code in `err`, every role falls through to the common exit, TMEM
// is released and the host reports the code after the step.
#pragma once

#include <algorithm>
#include <map>
#include <tuple>
#include <type_traits>

#include "seqkernels.cuh"
#include "tc05.cuh"

#define TG_BM 128
#define TG_BN 128
#define TG_BK 64
#define TG_STAGES 3
#define TG_THREADS 192
#define TG_STAGE_BYTES ((TG_BM + TG_BN) * TG_BK * 2)
#define TG_SMEM (TG_STAGES * TG_STAGE_BYTES + 1024)
// kind::f16 instruction descriptor: D = f32 (bit 4), A = B = bf16 (bits 7, 10), both K-major, N at bit 17 (>> 3), M at bit 24 (>> 4)
#define TG_IDESC ((1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TG_BN >> 3) << 17) | ((uint32_t)(TG_BM >> 4) << 24))

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
	asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)), "l"(map),
	             "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
	             : "memory");
}
// The epilogue of one warp: its 32 weight rows (lane = row m) against the tile's tokens, 32 at a time.  E: what the epilogue does when it is one
// of the plain ones -- a bias and a factor at most, and for EPI_F32 columns past `split` in the activation type -- with everything that does not
// depend on the token worked out before the loop.  The additions to the residual stream load 16 tokens' rows ahead of the stores: one after the
// other, each store bars the next load (164 us for 2048 x 2048 x 5632).  TG_ANY: gemm_store decides per element, in a loop that is not
// unrolled: 32 copies of every epilogue do not fit the instruction cache, which costs more than the accumulators' way through local memory.  What is left to it,
// as a loop and unrolled: factors per row, all products of a Sopepel step of 2048 / 700 tokens 1194 / 763 and 1286 / 823 us; capped logits, of
// a Tabisun step with 512 tokens' logits 838 and 852 us.
// All products of a 2048-token step with attention and two linear attentions: 1735 us with residual additions, decays and squared rectifiers in the
// unrolled TG_ANY, 743 in instances of their own, 652 without conditions per element, 545 with the large ones on pairs of CTAs (below).
#define TG_ANY (-1)
#define TG_ACT_GATE 100 // EPI_ACT times sigmoid(gate)
#define TG_EPILOGUES 8  // EPI_*
// Tokens [c0, c1) of the tile.  A run of 32 tokens that are all there, for 32 rows that are all there, takes a path without a condition per element: with
// them a warp stored one token in a hundred cycles, and a 256 x 256 tile's epilogue took as long as its products (K = 2048).
template <int E>
__device__ __forceinline__ void tg_epilogue(const GemmArgs& a, int z, const GemmRows& gr, int n0, int c0, int c1, int m, int lane, uint32_t tmem) {
	const int rows = min(c1, gr.count - n0);
	const bool live = m < a.M;
	const float bias = E != TG_ANY && a.bias && live ? ldf(a.bias + (size_t)z * a.M + m) : 0.f;
	const float scale = a.out_scale != 0.f ? a.out_scale : 1.f;
	const bool aside = E == EPI_F32 && a.split > 0 && m >= a.split; // this weight row's results go to Y2
	const bool f32 = (E == EPI_F32 && !aside) || E == EPI_DECAY;    // fp32 results
	const bool alike = __all_sync(0xffffffffu, live) && (E != EPI_F32 || __all_sync(0xffffffffu, aside) || !__any_sync(0xffffffffu, aside));
	const long ld = aside ? a.ldy2 : a.ldy;
	const size_t o = aside ? (size_t)(gr.base + n0) * a.ldy2 + (m - a.split) : (size_t)z * a.ybs + (size_t)(gr.base + n0) * a.ldy + (E == EPI_GLU ? m >> 1 : m);
	float* const yf = (float*)a.Y + o;
	bf16* const yb = (bf16*)(aside ? a.Y2 : a.Y) + o;
	const float* const gate = E == TG_ACT_GATE ? a.gate + (size_t)z * a.gbs + (size_t)(gr.base + n0) * a.ldgate + m : nullptr;
	for (; c0 < rows; c0 += 32) {
		float v[32];
		tmem_ld32(tmem + c0, v);
		if constexpr (E == TG_ANY) {
#pragma unroll 1
			for (int j = 0; j < 32; ++j) gemm_store<bf16>(a, z, gr, n0 + c0 + j, m, v[j]); // lanes = consecutive weight rows: coalesced
			continue;
		}
		auto run = [&](auto whole) { // whole: all 32 tokens and rows are there
			constexpr bool W = decltype(whole)::value;
			const int left = W ? 32 : live ? rows - c0 : 0; // of this row's tokens
			if constexpr (E == EPI_RES || E == EPI_DYT_RES) {
				float* p = yf + (size_t)c0 * ld;
				const float* rp = E == EPI_RES && a.res ? a.res + o + (size_t)c0 * ld : nullptr;
				const float na = E == EPI_DYT_RES ? ldf(a.na) : 0.f, nw = E == EPI_DYT_RES && live ? ldf(a.nw + m) : 0.f, nb = E == EPI_DYT_RES && live ? ldf(a.nb + m) : 0.f;
				const bool next = E == EPI_DYT_RES && a.xw;
				const float xa = next ? ldf(a.xa) : 0.f, xw = next && live ? ldf(a.xw + m) : 0.f, xb = next && live ? ldf(a.xb + m) : 0.f;
				bf16* px = next ? (bf16*)a.Y2 + (size_t)(gr.base + n0 + c0) * a.ldy2 + m : nullptr;
				constexpr int B = W ? 32 : 16; // loads ahead of the stores
#pragma unroll
				for (int j0 = 0; j0 < 32; j0 += B) {
					float y[B], r[B];
					float* py = p;
#pragma unroll
					for (int i = 0; i < B; ++i, py += ld) y[i] = j0 + i < left ? *py : 0.f;
					if (rp) {
#pragma unroll
						for (int i = 0; i < B; ++i, rp += ld) r[i] = j0 + i < left ? *rp : 0.f;
					}
#pragma unroll
					for (int i = 0; i < B; ++i, p += ld) {
						const float x = (v[j0 + i] + bias) * scale;
						if (j0 + i < left) *p = y[i] += E == EPI_DYT_RES ? tanhf(na * x) * nw + nb : rp ? r[i] + x : x;
					}
					if (next) {
#pragma unroll
						for (int i = 0; i < B; ++i, px += a.ldy2)
							if (j0 + i < left) *px = __float2bfloat16_rn(tanhf(xa * y[i]) * xw + xb);
					}
				}
			} else if constexpr (E == EPI_GLU) { // lanes 2c (gate) and 2c + 1 (up) share the unit's tokens: the even lane forms token j, the odd one token j + 1
				const int odd = lane & 1;
				bf16* q = yb + (size_t)(c0 + odd) * ld;
#pragma unroll
				for (int j = 0; j < 32; j += 2, q += 2 * ld) {
					const float x0 = v[j] + bias, x1 = v[j + 1] + bias;
					const float other = __shfl_xor_sync(0xffffffffu, odd ? x0 : x1, 1);
					if (j + odd < left) *q = __float2bfloat16_rn(glu_unit(odd ? other : x0, odd ? x1 : other, a.glu_limit, a.glu_mode));
				}
			} else {
				// the row pointers advance by one addition per token: 32 separate row offsets would cost k_seq_gemm_tc its second CTA per SM
				auto each = [&](auto* q, long step, auto&& store) { // store(where, value, token)
#pragma unroll
					for (int j = 0; j < 32; ++j, q += step)
						if (j < left) store(q, (v[j] + bias) * scale, j);
				};
				float* const qf = yf + (size_t)c0 * ld;
				bf16* const qb = yb + (size_t)c0 * ld;
				auto square = [](float x) { // of the positive part
					const float pos = fmaxf(x, 0.f);
					return pos * pos;
				};
				if constexpr (E == EPI_F32) {
					if (!aside) each(qf, ld, [&](float* q, float x, int) { *q = x; });
					else if (a.split_act) each(qb, ld, [&](bf16* q, float x, int) { *q = __float2bfloat16_rn(x); });
					else each(qb, ld, [&](bf16* q, float x, int) { *q = __float2bfloat16_rn(square(x)); });
				} else if constexpr (E == EPI_DECAY) each(qf, ld, [&](float* q, float x, int) { *q = expf(-softplusf_(-x) * a.epi_f); });
				else if constexpr (E == EPI_ACT_RELU2) each(qb, ld, [&](bf16* q, float x, int) { *q = __float2bfloat16_rn(square(x)); });
				else if constexpr (E == EPI_ACT) each(qb, ld, [&](bf16* q, float x, int) { *q = __float2bfloat16_rn(x); });
				else if constexpr (E == TG_ACT_GATE) {
					const float* g = gate + (size_t)c0 * a.ldgate;
					float gv[32];
#pragma unroll
					for (int j = 0; j < 32; ++j, g += a.ldgate) gv[j] = j < left ? *g : 0.f;
					each(qb, ld, [&](bf16* q, float x, int j) { *q = __float2bfloat16_rn(x * sigmoidf_(gv[j])); });
				} else
					each(qb, ld, [&](bf16* q, float x, int) {
						const bf16 h = __float2bfloat16_rn(x);
						q[0] = h, q[a.split3] = h, q[2 * a.split3] = __float2bfloat16_rn(x - __bfloat162float(h));
					});
			}
		};
		if (alike && rows - c0 >= 32) run(std::true_type{});
		else run(std::false_type{});
	}
}
// which instance serves a product
static inline int tg_kind(const GemmArgs& a) {
	const bool plain = a.out_cap == 0.f && !a.rs && (a.split == 0 || a.epi == EPI_F32) && (a.out_scale == 0.f || a.epi != EPI_GLU);
	if (a.gate) return plain && a.epi == EPI_ACT ? TG_ACT_GATE : TG_ANY;
	return plain ? a.epi : TG_ANY;
}

template <int E>
__global__ void __launch_bounds__(TG_THREADS, 2) k_seq_gemm_tc(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, const GemmArgs a, int w3d, int x3d,
                                                             int* err) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	extern __shared__ unsigned char smem_dyn[];
	__shared__ __align__(8) uint64_t full[TG_STAGES], empty[TG_STAGES], accum;
	__shared__ uint32_t tmem_base_s;
	unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int m0 = blockIdx.x * TG_BM, n0 = blockIdx.y * TG_BN, z = blockIdx.z;
	const int nkb = (a.K + TG_BK - 1) / TG_BK;
	const GemmRows gr = gemm_rows(a, z);
	if (a.band_mode == 1 && !a.band.meets(n0, min(n0 + TG_BN, gr.count) - 1, m0, m0 + TG_BM - 1)) return; // scores that no row of the tile sees
	if (n0 >= gr.count) return; // a grouped product's tile past the end of its group (uniform over the CTA, before any barrier or TMEM allocation)
	// 64-deep step kb of the sum: left out when none of the tile's rows meets its columns
	auto skips = [&](int kb) {
		if (a.band_mode != 2) return false;
		const int c = kb * TG_BK - (a.band_cp > 0 && kb * TG_BK >= a.band_cp ? a.band_cp : 0);
		return !a.band.meets(n0, min(n0 + TG_BN, gr.count) - 1, c, c + TG_BK - 1);
	};
	auto a_tile = [&](int s) { return smem + (size_t)s * TG_STAGE_BYTES; };
	auto b_tile = [&](int s) { return smem + (size_t)s * TG_STAGE_BYTES + TG_BM * TG_BK * 2; };
	if (tid == 0) {
		for (int s = 0; s < TG_STAGES; ++s) mbar_init(&full[s], 1), mbar_init(&empty[s], 1);
		mbar_init(&accum, 1);
		mbar_init_fence();
	}
	if (warp == 1) tmem_alloc(&tmem_base_s, TG_BN);
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem_base = tmem_base_s;
	bool ok = true;
	int copied = 0; // thread 0: stages requested

	if (warp == 0) {
		if (lane == 0) {
			for (int kb = 0; kb < nkb; ++kb) {
				if (skips(kb)) continue;
				const int s = copied % TG_STAGES;
				if (!mbar_wait_bounded(&empty[s], ((copied / TG_STAGES) & 1) ^ 1)) {
					atomicExch(err, 1);
					ok = false;
					break;
				}
				++copied;
				mbar_expect_tx(&full[s], TG_STAGE_BYTES);
				if (w3d) tma_load_3d(a_tile(s), &tm_w, kb * TG_BK, m0, z, &full[s]);
				else tma_load_2d(a_tile(s), &tm_w, kb * TG_BK, m0, &full[s]);
				if (x3d) tma_load_3d(b_tile(s), &tm_x, kb * TG_BK, n0, z, &full[s]);
				else tma_load_2d(b_tile(s), &tm_x, kb * TG_BK, gr.base + n0, &full[s]); // rows past the group are other groups' (or zero fill): never stored
			}
		}
	} else if (warp == 1) {
		if (lane == 0) {
			for (int kb = 0, it = 0; kb < nkb; ++kb) {
				if (skips(kb)) continue;
				const int s = it % TG_STAGES;
				if (!mbar_wait_bounded(&full[s], (it / TG_STAGES) & 1)) {
					atomicExch(err, 2);
					ok = false;
					break;
				}
				tc_fence_after();
#pragma unroll
				for (int k = 0; k < TG_BK / 16; ++k) // 16 bf16 = 32 bytes along K inside the swizzle atom: +2 in the 16-byte address field
					umma_f16(tmem_base, umma_desc_sw128(a_tile(s)) + 2 * k, umma_desc_sw128(b_tile(s)) + 2 * k, TG_IDESC, (it | k) ? 1u : 0u);
				umma_commit(&empty[s]);
				++it;
			}
			umma_commit(&accum); // arrives when everything issued so far has completed, also after a stall
		}
	} else {
		ok = mbar_wait_warp(&accum, 0);
		if (!ok && lane == 0) atomicExch(err, 3);
		tc_fence_after();
		if (ok) {
			const int q4 = warp & 3; // the TMEM lane quarter this warp may read
			tg_epilogue<E>(a, z, gr, n0, 0, TG_BN, m0 + q4 * 32 + lane, lane, tmem_base + ((uint32_t)(q4 * 32) << 16));
		}
		tc_fence_before();
	}
	if (__syncthreads_or(!ok)) { // a wait gave up: the copies and MMAs already issued end before the CTA does
		if (tid == 0) {
			for (int i = max(0, copied - TG_STAGES); i < copied; ++i) mbar_wait_bounded(&full[i % TG_STAGES], (i / TG_STAGES) & 1);
			mbar_wait_bounded(&accum, 0);
		}
		__syncthreads();
	}
	if (warp == 1) {
		tc_fence_after();
		tmem_dealloc(tmem_base, TG_BN);
	}
}

// The same product with tiles of 256 weight rows x 256 tokens on pairs of CTAs (cta_group::2), persistent.  A 128 x 128 tile asks L2 for 32 KB per 64-deep
// step, 256 cycles of the tensor core; here a CTA asks for its 128 weight rows and half of the tokens, the same 32 KB, in 512.  Roles as above, and
// two accumulators of 256 columns, so that a tile's epilogue runs under the next tile's products.  A step takes 580 cycles where the tensor core
// needs 512; a tile's epilogue 4300 (fp32 results) to 20000 (two addends from memory), read by eight warps.  13888 x 2048 rows and K, 2048 tokens: 83 us (1400 TFLOP/s;
// under a profiler the tensor pipe is active 74 %), 118 with tiles of 128.
#define TP_BM 256
#define TP_BN 256
#define TP_STAGES 6
#define TP_STAGE_BYTES (2 * 128 * TG_BK * 2) // per CTA
#define TP_THREADS 320 // a copying and a multiplying warp, eight that read results
#define TP_SMEM (TP_STAGES * TP_STAGE_BYTES + 1024)
template <int E>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TP_THREADS, 1) k_seq_gemm_pair(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, const GemmArgs a, int* err, unsigned tries) {
	extern __shared__ unsigned char smem_dyn[];
	__shared__ __align__(8) uint64_t full[TP_STAGES], empty[TP_STAGES], acc_full[2], acc_empty[2]; // full, acc_empty: rank 0's are used
	__shared__ uint32_t tmem_base_s;
	__shared__ int gave_up_s[2]; // whether a wait gave up in each of the CTAs
	__shared__ int asked[2], multiplied_s, handed_s; // rank 0's, read when one did: stages that each CTA's copies got to, stages multiplied, accumulators handed over
	unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rank = (int)cluster_rank(), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
	const int nkb = (a.K + TG_BK - 1) / TG_BK, tok_tiles = (a.N + TP_BN - 1) / TP_BN, tiles = (a.M + TP_BM - 1) / TP_BM * tok_tiles;
	auto a_tile = [&](int s) { return smem + (size_t)s * TP_STAGE_BYTES; };
	auto b_tile = [&](int s) { return smem + (size_t)s * TP_STAGE_BYTES + TP_STAGE_BYTES / 2; };
	// tokens of a tile that the MMAs run over: whole tiles, or what is left in steps of 32
	auto width = [&](int n0) { return min(TP_BN, (a.N - n0 + 31) & ~31); };
	pdl_launch_next();
	if (tid == 0) {
		for (int s = 0; s < TP_STAGES; ++s) mbar_init(&full[s], 1), mbar_init(&empty[s], 1);
		for (int s = 0; s < 2; ++s) mbar_init(&acc_full[s], 1), mbar_init(&acc_empty[s], 16);
		asked[0] = asked[1] = multiplied_s = handed_s = 0;
		mbar_init_fence();
	}
	if (warp == 1) pair_tmem_alloc(&tmem_base_s, 512);
	tc_fence_before();
	cluster_sync(); // the other CTA's barriers are there too
	tc_fence_after();
	const uint32_t tmem_base = tmem_base_s;
	bool ok = true;
	pdl_wait_prev();
	if (warp == 0) {
		int it = 0;
		for (int t = pair; t < tiles && ok; t += pairs) {
			const int m0 = t / tok_tiles * TP_BM + rank * 128, n0 = t % tok_tiles * TP_BN, n1 = n0 + rank * (width(n0) / 2);
			for (int kb = 0; kb < nkb; ++kb, ++it) {
				const int s = it % TP_STAGES;
				ok = mbar_wait_warp(&empty[s], ((it / TP_STAGES) & 1) ^ 1, tries);
				if (!ok) break;
				if (elect_one()) {
					const uint32_t bar = cluster_addr(&full[s], 0);
					if (rank == 0) mbar_expect_tx(&full[s], 2 * TP_STAGE_BYTES);
					pair_tma_load_2d(a_tile(s), &tm_w, kb * TG_BK, m0, bar);
					pair_tma_load_2d(b_tile(s), &tm_x, kb * TG_BK, n1, bar);
				}
				__syncwarp();
			}
		}
		if (lane == 0) cluster_store(cluster_addr(&asked[rank], 0), it);
		// the stages' last releases arrive in this CTA: they do before it ends
		const bool copied = ok;
		for (int i = max(0, it - TP_STAGES); i < it && ok; ++i) ok = mbar_wait_warp(&empty[i % TP_STAGES], (i / TP_STAGES) & 1, tries);
		if (!ok && lane == 0) atomicExch(err, copied ? 4 : 1);
	} else if (warp == 1) {
		if (rank == 0) {
			int it = 0, n = 0, handed = 0;
			for (int t = pair; t < tiles && ok; t += pairs, ++n) {
				const int buf = n & 1;
				const uint32_t d = tmem_base + buf * 256, idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(width(t % tok_tiles * TP_BN) >> 3) << 17) | ((uint32_t)(TP_BM >> 4) << 24);
				ok = mbar_wait_warp(&acc_empty[buf], ((n >> 1) & 1) ^ 1, tries);
				tc_fence_after();
				for (int kb = 0; kb < nkb && ok; ++kb, ++it) {
					const int s = it % TP_STAGES;
					ok = mbar_wait_warp(&full[s], (it / TP_STAGES) & 1, tries);
					if (!ok) break;
					if (elect_one()) {
						const uint64_t da = umma_desc_sw128(a_tile(s)), db = umma_desc_sw128(b_tile(s));
#pragma unroll
						for (int k = 0; k < TG_BK / 16; ++k) pair_umma_f16(d, da + 2 * k, db + 2 * k, idesc, (kb | k) ? 1u : 0u);
						pair_umma_commit(&empty[s]);
						if (kb + 1 == nkb) pair_umma_commit(&acc_full[buf]);
					}
					__syncwarp();
				}
				handed += ok;
			}
			if (!ok && lane == 0) atomicExch(err, 2);
			if (lane == 0) multiplied_s = it, handed_s = handed;
		}
	} else {
		const int q4 = warp & 3, half = (warp - 2) / 4 * (TP_BN / 2); // the TMEM lane quarter this warp may read, and its half of the tokens
		const GemmRows gr = gemm_rows(a, 0);
		int n = 0;
		for (int t = pair; t < tiles; t += pairs, ++n) {
			const int buf = n & 1, m0 = t / tok_tiles * TP_BM + rank * 128, n0 = t % tok_tiles * TP_BN;
			if constexpr (E == EPI_RES || E == EPI_DYT_RES) // what the tile's results are added to travels to L2 while they are formed (the 11 products of a 2048-token step 550 -> 545 us)
				for (int i = n0 + half + lane; i < min(n0 + half + TP_BN / 2, a.N) && m0 + q4 * 32 < a.M; i += 32) {
					asm volatile("prefetch.global.L2 [%0];" ::"l"((const float*)a.Y + (size_t)i * a.ldy + m0 + q4 * 32));
					if (E == EPI_RES && a.res) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.res + (size_t)i * a.ldy + m0 + q4 * 32));
				}
			ok = mbar_wait_warp(&acc_full[buf], (n >> 1) & 1, tries);
			if (!ok) break;
			tc_fence_after();
			tg_epilogue<E>(a, 0, gr, n0, half, half + TP_BN / 2, m0 + q4 * 32 + lane, lane, tmem_base + buf * 256 + ((uint32_t)(q4 * 32) << 16));
			tc_fence_before();
			__syncwarp();
			if (lane == 0) mbar_arrive_cluster(cluster_addr(&acc_empty[buf], 0));
		}
		if (!ok && lane == 0) atomicExch(err, 3);
	}
	const int gave_up = __syncthreads_or(!ok);
	if (tid < 2) cluster_store(cluster_addr(&gave_up_s[rank], tid), gave_up);
	cluster_sync();
	// a wait gave up, in either CTA: what is on its way ends before the CTAs do.  Copies are counted in rank 0 (a stage that one CTA alone asked for never
	// fills: that wait runs out); what the MMAs release and hand over arrives in both, and each CTA waits for its own arrivals
	if (tid == 0 && (gave_up_s[0] | gave_up_s[1])) {
		const int multiplied = cluster_load(cluster_addr(&multiplied_s, 0)), handed = cluster_load(cluster_addr(&handed_s, 0)), most = rank == 0 ? max(asked[0], asked[1]) : 0;
		for (int i = max(0, most - TP_STAGES); i < most; ++i) mbar_wait_bounded(&full[i % TP_STAGES], (i / TP_STAGES) & 1, MBAR_SPINS / 16);
		for (int i = max(0, multiplied - TP_STAGES); i < multiplied; ++i) mbar_wait_bounded(&empty[i % TP_STAGES], (i / TP_STAGES) & 1, MBAR_SPINS / 16);
		for (int i = max(0, handed - 2); i < handed; ++i) mbar_wait_bounded(&acc_full[i & 1], (i >> 1) & 1, MBAR_SPINS / 16);
	}
	cluster_sync();
	if (warp == 1) {
		tc_fence_after();
		pair_tmem_dealloc(tmem_base, 512);
	}
}

// ---------------------------------------------------------------- host side
typedef CUresult (*TgEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                               CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
struct TgState {
	TgEncodeFn encode = nullptr;
	int* err_host = nullptr; // pinned + mapped
	int* err_dev = nullptr;
	int pairs = 0; // clusters of two CTAs that the device holds at a time
	uint64_t pair_launches[TG_EPILOGUES] = {}; // by EPI_*
	unsigned tries = MBAR_SPINS; // of a wait in the pairs' kernel
	std::map<std::tuple<const void*, long, long, long, long, int>, CUtensorMap> maps;
};
static TgState g_tg;
// the pairs' kernel has no instances for the epilogues of products per head, of a decay's low rank and of rows that are all squared rectifiers (a shared unit
// without gate and router rows): none of the families has large ones of them
static constexpr bool tg_pair_instance(int kind) { return kind != EPI_SPLIT3 && kind != TG_ACT_GATE && kind != EPI_DECAY && kind != EPI_ACT_RELU2; }
// f(instance) for every instance of the kernels
template <typename F>
static inline void tg_each(F&& f) {
	f(std::integral_constant<int, TG_ANY>{}), f(std::integral_constant<int, EPI_F32>{}), f(std::integral_constant<int, EPI_ACT>{}), f(std::integral_constant<int, EPI_SPLIT3>{});
	f(std::integral_constant<int, EPI_GLU>{}), f(std::integral_constant<int, TG_ACT_GATE>{}), f(std::integral_constant<int, EPI_RES>{}), f(std::integral_constant<int, EPI_DYT_RES>{});
	f(std::integral_constant<int, EPI_ACT_RELU2>{}), f(std::integral_constant<int, EPI_DECAY>{});
}

static inline void gemm_tc_setup() {
	if (g_tg.encode) return;
	cudaDriverEntryPointQueryResult qres;
	void* fn = nullptr;
	CUDA_CHECK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres));
	if (!fn || qres != cudaDriverEntryPointSuccess) CALM_FATAL("cuTensorMapEncodeTiled is not available from this driver");
	g_tg.encode = (TgEncodeFn)fn;
	CUDA_CHECK(cudaHostAlloc((void**)&g_tg.err_host, sizeof(int), cudaHostAllocMapped));
	*g_tg.err_host = 0;
	CUDA_CHECK(cudaHostGetDevicePointer((void**)&g_tg.err_dev, g_tg.err_host, 0));
	tg_each([&](auto e) {
		constexpr int E = decltype(e)::value;
		CUDA_CHECK(cudaFuncSetAttribute(k_seq_gemm_tc<E>, cudaFuncAttributeMaxDynamicSharedMemorySize, TG_SMEM));
		if constexpr (tg_pair_instance(E)) CUDA_CHECK(cudaFuncSetAttribute(k_seq_gemm_pair<E>, cudaFuncAttributeMaxDynamicSharedMemorySize, TP_SMEM));
	});
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3(2 * 74), cfg.blockDim = dim3(TP_THREADS), cfg.dynamicSmemBytes = TP_SMEM;
	if (const char* e = getenv("CALM_B200_SEQ_WAIT")) g_tg.tries = (unsigned)atol(e); // tests make the waits run out
	CUDA_CHECK(cudaOccupancyMaxActiveClusters(&g_tg.pairs, k_seq_gemm_pair<EPI_F32>, &cfg));
}
// a stalled pipeline leaves its code here; read after the stream has been synchronised
static inline int gemm_tc_error() { return g_tg.err_host ? *g_tg.err_host : 0; }

// bf16 [batch][rows][cols] with row stride ld and batch stride bs (elements); box = 64 columns x `box_rows` rows
static inline const CUtensorMap* tg_map(const void* base, long rows, long cols, long ld, long bs, int batch, int box_rows) {
	const auto key = std::make_tuple(base, rows, cols, ld, bs, batch * 1024 + box_rows);
	auto it = g_tg.maps.find(key);
	if (it != g_tg.maps.end()) return &it->second;
	CUtensorMap m;
	const bool three = bs != 0 && batch > 1;
	const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)batch};
	const cuuint64_t strides[2] = {(cuuint64_t)ld * 2, (cuuint64_t)bs * 2};
	const cuuint32_t box[3] = {TG_BK, (cuuint32_t)box_rows, 1}, estr[3] = {1, 1, 1};
	CUresult r = g_tg.encode(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, three ? 3 : 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
	                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
	if (r != CUDA_SUCCESS) return nullptr; // a layout the copy engine does not describe: the caller keeps the mma.sync kernel
	return &(g_tg.maps[key] = m);
}

// shapes the kernel takes: enough tokens to fill its tiles (a matrix of few rows, a router's, fills the rest of its tile with the copy's zeros), 16-byte aligned rows and bases
static inline bool gemm_tc_fits(const GemmArgs& a, int batch) {
	auto al8 = [](long v) { return v % 8 == 0; };
	return a.N >= 64 && a.M >= 8 && a.K >= 32 && al8(a.ldx) && al8(a.ldw) && al8(a.xbs) && al8(a.wbs) && ((uintptr_t)a.X & 15) == 0 && ((uintptr_t)a.W & 15) == 0 &&
	       batch < 65536;
}
// the tensor maps of both operands; false: no map for one of them
static inline bool gemm_tc_maps(const GemmArgs& a, int batch, const CUtensorMap*& mw, const CUtensorMap*& mx) {
	if (g_tg.maps.size() > 8192) g_tg.maps.clear(); // before the look-ups: their results point into the map
	mw = tg_map(a.W, a.M, a.K, a.ldw, a.wbs, batch, TG_BM);
	mx = tg_map(a.X, a.seg ? a.x_rows : a.N, a.K, a.ldx, a.xbs, batch, TG_BN);
	return mw && mx;
}
// Products that run on pairs of CTAs, by estimated cycles: a 64-deep step takes a 256 x 256 tile 590 and a 128 x 128 tile 900 (two CTAs to an SM, or one), and
// larger tiles bring 9000 more of launch, first loads and epilogue, more where the epilogue reads what it adds to: nothing runs over the epilogues of a single wave,
// and the smaller tiles' are half as long and, two to an SM, run over each other's products.  us alone with tiles of 128 / on pairs, K = 2048 unless given:
//   plain, 13888 rows, 2048 tokens 118 / 83; 700 tokens 58 / 43; 8192 rows, 64 tokens 16.9 / 13.7, 128 17.6 / 14.9, 512 21.3 / 20.6; K = 1024 10.1 / 9.8, 11.0 / 10.7,
//   13.6 / 14.3; 3072 rows, K = 1024, 256 tokens 10.7 / 13.2; gated units, 11264 rows, 64 tokens 23.5 / 20.1, 256 29.5 / 26.9, 2048 130.5 / 84.3;
//   Dynamic Tanh added to the stream, 2048 rows, 256 tokens 24.2 / 26.3, 1024 28.0 / 28.1, 2048 32.2 / 30.3; K = 5632 43.7 / 38.3, 46.5 / 41.1, 51.6 / 45.2;
//   added to the stream, 2048 rows, 64 tokens 17.4 / 17.5, 128 21.1 / 23.0, 256 22.3 / 26.8, 2048 26.2 / 30.4; K = 5632 38.5 / 29.5, 41.9 / 34.9, 42.6 / 43.8, 54.6 / 54.2;
//   8192 rows, 512 tokens 30.2 / 34.2, 1024 (two waves) 60.4 / 53.4; 4096 rows, K = 1024, 2048 tokens (two waves) 41.9 / 43.8.
// Between other launches a pair's start is hidden.  us more on pairs a product in whole steps, added to the stream, 64 / 128 / 200 / 256 / 512 / 1024 / 2048 tokens:
//   2048 rows, K = 2048 -2.3, -1.3, 3.5, 2.4, 4.0, 4.1, 1.8; K = 5632 -11.4, -9.1, -4.4, 0.0, 1.9, -4.0, -2.3; 1024 rows, K = 2816 -8.3, -3.5, -2.0, 5.4, 3.9, 1.8, 0.3;
//   4096 rows, K = 4096 -6.1, -2.6, -2.5, 0.7, -0.5, -0.3, -20.5 (two waves); K = 2048 -2.1, 2.5, -0.8, 3.5, 1.4, 2.4, -5.8.
static inline bool tg_pairs_pay(long M, long N, long K, int epi, long pairs) {
	const long steps = (K + TG_BK - 1) / TG_BK, slots = 4 * pairs; // CTAs of the smaller tiles at a time
	const long small = ((M + TG_BM - 1) / TG_BM) * ((N + TG_BN - 1) / TG_BN), large = ((M + TP_BM - 1) / TP_BM) * ((N + TP_BN - 1) / TP_BN);
	const bool alone = small <= 5 * pairs / 2; // the smaller tiles are about one to an SM
	long more = 9000;
	if (epi == EPI_RES) more = large > pairs ? 14000 : N <= 128 ? 9000 : N <= 224 ? 13000 : alone ? 24000 : 20000;
	else if (epi == EPI_DYT_RES && N > 224 && alone) more = 15500;
	return (large + pairs - 1) / pairs * steps * 590 + more < (small + slots - 1) / slots * steps * 900;
}
static inline bool tg_pairs(const GemmArgs& a, int batch) {
	if (batch > 1 || a.seg || a.band_mode || g_tg.pairs < 1 || !tg_pair_instance(tg_kind(a))) return false;
	return tg_pairs_pay(a.M, a.N, a.K, a.epi, g_tg.pairs);
}
// false: nothing was launched
static inline bool gemm_tc_launch(const GemmArgs& a, int batch, cudaStream_t stream, bool pdl) {
	const CUtensorMap *mw, *mx;
	if (!gemm_tc_maps(a, batch, mw, mx)) return false;
	const bool pair = tg_pairs(a, batch);
	const long tiles = (long)((a.M + TP_BM - 1) / TP_BM) * ((a.N + TP_BN - 1) / TP_BN);
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = pair ? dim3(2 * (int)std::min<long>(tiles, g_tg.pairs)) : dim3((a.M + TG_BM - 1) / TG_BM, (a.N + TG_BN - 1) / TG_BN, batch);
	cfg.blockDim = dim3(pair ? TP_THREADS : TG_THREADS), cfg.dynamicSmemBytes = pair ? TP_SMEM : TG_SMEM, cfg.stream = stream;
	cudaLaunchAttribute at[1];
	at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	at[0].val.programmaticStreamSerializationAllowed = 1;
	cfg.attrs = at, cfg.numAttrs = pdl ? 1 : 0;
	const int kind = tg_kind(a);
	if (pair) ++g_tg.pair_launches[a.epi];
	tg_each([&](auto e) {
		constexpr int E = decltype(e)::value;
		if (E != kind) return;
		if constexpr (tg_pair_instance(E))
			if (pair) {
				CUDA_CHECK(cudaLaunchKernelEx(&cfg, k_seq_gemm_pair<E>, *mw, *mx, a, g_tg.err_dev, g_tg.tries));
				return;
			}
		CUDA_CHECK(cudaLaunchKernelEx(&cfg, k_seq_gemm_tc<E>, *mw, *mx, a, (int)(a.wbs != 0 && batch > 1), (int)(a.xbs != 0 && batch > 1), g_tg.err_dev));
	});
	return true;
}
