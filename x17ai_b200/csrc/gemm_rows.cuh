// GEMM for few rows of A (a decode step's tokens): a pass over the weights, bound by HBM.
//
// The persistent forms of gemm.cuh put at most one CTA on each 256-column tile: an 8192-column output keeps 32 of 148
// SMs busy, and 128 accumulator rows are multiplied whatever the number of tokens. Here the operands change places:
// the weights are the MMA's 128-row side, the tokens its N (16 .. 48 columns), so a K block of 128 weight rows costs
// 16 KB of weights, the tokens' few KB and a few dozen MMA cycles, and the accumulator is a few TMEM columns. A cluster of
// up to four CTAs splits K; the parts are exchanged through the cluster's shared memory (no workspace, no second
// launch) and added up in K order. Small CTAs (shared memory for two per SM) keep enough bytes in flight
// on every SM although the tile counts do not divide evenly.
//
// Epilogue: thread = output column (weight row), registers = tokens. Gate and value of a pair sit in neighbouring
// lanes: each lane of a pair takes half of the tokens. Output bytes are collected in shared memory and leave in 16-byte
// stores along the rows.
//
// Measured at 16 rows, weights cold, back to back (before: one CTA per 128 x 256 tile): [12288, 4096] int8 20.7 -> 15.5 us,
// [8192, 4096] 21 -> 11.4, [28672, 4096] 29.6 -> 22 (5.4 TB/s), [8192, 2 x 14336] e4m3 100 -> 41 (5.8 TB/s).
#pragma once

#include "gemm.cuh"

namespace x17 {

struct RowsParams {
	u32 split;    // CTAs per tile = cluster size: 1, 2 or 4
	u32 n_tok;    // MMA N: the rows of A rounded up to 16
	u32 a_box;    // rows of A's box: rounded up to 8
	u32 stages;
};

namespace rows_cfg {
constexpr u32 WM = 128;        // weight rows per tile
constexpr u32 BK = 128;
constexpr u32 MAX_TOK = 48;
constexpr u32 MAX_STAGES = 8;
constexpr u32 THREADS = 192;
constexpr u32 ACC_PITCH = WM + 1;   // f32 / i32 words per token of the L2-norm epilogue's copy of the tile
__host__ __device__ constexpr u32 stage_bytes(u32 a_box) { return a_box * BK + WM * BK; }
// What the epilogue lays over the ring: the other CTAs' parts, then the output bytes, then (per-head L2 norm) the tile
// and its scales.
__host__ __device__ constexpr u32 parts_bytes(u32 split, u32 n_tok) { return (split - 1) * WM * n_tok * 4; }
constexpr u32 tail_bytes(u32 split, u32 n_tok, bool heads) {
	return parts_bytes(split, n_tok) + WM * n_tok + (heads ? n_tok * ACC_PITCH * 4 + 2 * n_tok * 4 : 0u);
}
constexpr u32 smem_bytes(u32 a_box, u32 stages) { return stages * stage_bytes(a_box) + 1024 /*alignment slack*/ + 256 /*barriers*/; }
}  // namespace rows_cfg

template <int EPI, bool F8>
__global__ void __launch_bounds__(rows_cfg::THREADS)
gemm_rows_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_w, const GemmParams p,
				 const RowsParams rp) {
	using namespace rows_cfg;
	constexpr bool HEADS = EPI == EPI_QKVG || EPI == EPI_L2NORM_KV;
	constexpr bool PAIRS = EPI == EPI_GEGLU_E4M3 || EPI == EPI_RESID_E4M3 || EPI == EPI_RESID_I8;
	extern __shared__ u8 smem_raw[];
	u32 const smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
	u8 *const smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
	u32 const st_bytes = stage_bytes(rp.a_box);
	u32 const bar_base = smem_base + rp.stages * st_bytes;
	auto full_bar = [&](u32 s) { return bar_base + 8 * s; };
	auto empty_bar = [&](u32 s) { return bar_base + 8 * (MAX_STAGES + s); };
	u32 const acc_full_bar = bar_base + 8 * (2 * MAX_STAGES);
	u32 const tmem_slot = acc_full_bar + 8;
	volatile u32 *const tmem_slot_gen = reinterpret_cast<volatile u32 *>(smem_gen + (tmem_slot - smem_base));
	volatile u32 *const abort_flag = tmem_slot_gen + 1;
	WaitCtx const ctx{abort_flag, p.status};

	u32 const warp = threadIdx.x >> 5;
	u32 const lane = threadIdx.x & 31;
	u32 const rank = cluster_cta_rank();
	u32 const w0 = (blockIdx.x / rp.split) * WM;   // first weight row = output column of the tile
	u32 const k_blocks = p.k / BK;
	u32 const kb_begin = rank * k_blocks / rp.split, kb_end = (rank + 1) * k_blocks / rp.split;
	u32 const tmem_cols = rp.n_tok <= 32 ? 32u : 64u;

	if (threadIdx.x == 0) {
		for (u32 s = 0; s < rp.stages; ++s) {
			mbar_init(full_bar(s), 1);
			mbar_init(empty_bar(s), 1);
		}
		mbar_init(acc_full_bar, 1);
		*abort_flag = 0;
		mbar_fence_init();
	}
	if (warp == 1) {
		tmem_alloc(tmem_slot, tmem_cols);
		tmem_relinquish();
	}
	if (threadIdx.x == 0) {
		// the first weights start on their way to L2 while the kernel in front of this one finishes
		tma_prefetch_desc(&tm_a);
		tma_prefetch_desc(&tm_w);
		for (u32 i = 0; i < 2 * rp.stages && kb_begin + i < kb_end; ++i) tma_prefetch_2d(&tm_w, i32((kb_begin + i) * BK), i32(w0));
	}
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	u32 const tmem_base = *tmem_slot_gen;
	pdl_launch_dependents();
	pdl_wait();

	bool ok = true;
	if (warp == 0) {
		if (elect_one()) {
			for (u32 kb = kb_begin, s = 0, ph = 0; kb < kb_end; ++kb) {
				if (!mbar_wait(empty_bar(s), ph ^ 1, ctx, ST_WAIT_STAGE_EMPTY, s)) break;
				u32 const dst = smem_base + s * st_bytes;
				mbar_expect_tx(full_bar(s), st_bytes);
				tma_load_2d(dst + rp.a_box * BK, &tm_w, full_bar(s), i32(kb * BK), i32(w0));
				tma_load_2d(dst, &tm_a, full_bar(s), i32((kb * BK) % p.k_a), 0);
				if (++s == rp.stages) {
					s = 0;
					ph ^= 1;
				}
			}
		}
	} else if (warp == 1) {
		if (elect_one()) {
			u32 const idesc = F8 ? make_idesc(DFMT_F32, FMT_E4M3, FMT_E4M3, 0, 0, WM, rp.n_tok)
								 : make_idesc(DFMT_S32, FMT_S8, FMT_S8, 0, 0, WM, rp.n_tok);
			bool done = true;
			for (u32 kb = kb_begin, s = 0, ph = 0; kb < kb_end; ++kb) {
				if (!mbar_wait(full_bar(s), ph, ctx, ST_WAIT_TMA_FULL, s)) {
					done = false;
					break;
				}
				tc_fence_after();
				// the token rows behind A's box are whatever follows it in shared memory: they only reach accumulator
				// columns that are never stored
				u64 const tdesc = make_smem_desc(smem_base + s * st_bytes, 128);
				u64 const wdesc = make_smem_desc(smem_base + s * st_bytes + rp.a_box * BK, 128);
#pragma unroll
				for (u32 ks = 0; ks < BK / 32; ++ks) {
					u32 const accumulate = kb != kb_begin || ks != 0 ? 1u : 0u;
					if constexpr (F8) mma_f8_ss(tmem_base, wdesc + 2 * ks, tdesc + 2 * ks, idesc, accumulate);
					else mma_i8_ss(tmem_base, wdesc + 2 * ks, tdesc + 2 * ks, idesc, accumulate);
				}
				tc_commit(empty_bar(s));
				if (++s == rp.stages) {
					s = 0;
					ph ^= 1;
				}
			}
			if (done) tc_commit(acc_full_bar);
		}
	} else {
		ok = mbar_wait_warp(acc_full_bar, 0, ctx, ST_WAIT_ACC_FULL, 0);
		tc_fence_after();
	}
	__syncwarp();

	u32 const quarter = warp & 3;           // of the tile's weight rows
	u32 const wrow = quarter * 32 + lane;
	u32 const t_base = tmem_base + ((quarter * 32u) << 16);
	u32 const groups = rp.n_tok / 16;
	// Tiles with per-head L2 norm are finished by the cluster's first CTA, the quarters of other tiles are dealt out.
	SegOut seg{};
	if constexpr (HEADS) seg = segment_of<EPI>(p, w0);
	auto owner_of = [&](u32 q) { return HEADS && seg.heads ? 0u : q % rp.split; };
	u32 const slot_bytes = WM * rp.n_tok * 4;   // [quarter][n_tok / 4][lane][16 bytes]
	auto part_at = [&](u32 slot, u32 t4) { return smem_base + slot * slot_bytes + ((quarter * (rp.n_tok / 4) + t4) * 32 + lane) * 16; };
	if (rp.split > 1) {
		cluster_sync_all();   // every CTA's MMAs have finished: its ring takes the others' parts
		u32 const owner = owner_of(quarter);
		if (warp >= 2 && ok && owner != rank) {
			for (u32 g = 0; g < groups; ++g) {
				u32 r[16];
				tmem_ld_32x32b_x16(t_base + 16 * g, r);
				tmem_wait_ld();
				u32 const dst = map_to_cta(part_at(rank < owner ? rank : rank - 1, 4 * g), owner);
#pragma unroll
				for (u32 i = 0; i < 4; ++i) st_cluster_v4(dst + i * 512, r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
			}
		}
		cluster_sync_all();   // the parts have arrived
	}
	bool const works = warp >= 2 && ok && owner_of(quarter) == rank;
	// tokens [16 g, 16 g + 16) of this thread's output column, added up over the cluster in K order
	auto whole_group = [&](u32 g, u32 (&acc)[16]) {
		tmem_ld_32x32b_x16(t_base + 16 * g, acc);
		tmem_wait_ld();
		if (rp.split > 1) {
			u32 own[16];
#pragma unroll
			for (u32 i = 0; i < 16; ++i) own[i] = acc[i];
#pragma unroll 1
			for (u32 src = 0; src < rp.split; ++src) {
#pragma unroll
				for (u32 i = 0; i < 4; ++i) {
					uint4 v = make_uint4(own[4 * i], own[4 * i + 1], own[4 * i + 2], own[4 * i + 3]);
					if (src != rank) v = ld_shared_v4(part_at(src < rank ? src : src - 1, 4 * g + i));
					u32 const w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
					for (u32 j = 0; j < 4; ++j) {
						u32 &a = acc[4 * i + j];
						if (src == 0) a = w[j];
						else if constexpr (F8) a = __float_as_uint(__fadd_rn(__uint_as_float(a), __uint_as_float(w[j])));
						else a += w[j];
					}
				}
			}
		}
	};
	// output bytes [token][WM or WM / 2 columns]
	constexpr u32 OUT_COLS = PAIRS ? WM / 2 : WM;
	u32 const out_off = parts_bytes(rp.split, rp.n_tok);
	u8 *const out_s = smem_gen + out_off;
	if constexpr (EPI == EPI_RAW_I32) {
		if (works) {
			for (u32 g = 0; g < groups; ++g) {
				u32 r[16];
				whole_group(g, r);
#pragma unroll
				for (u32 i = 0; i < 16; ++i) {
					if (16 * g + i < p.m) static_cast<u32 *>(p.c)[u64(16 * g + i) * p.c_stride + w0 + wrow] = r[i];
				}
			}
		}
	} else {
		if constexpr (HEADS) {
			if (seg.heads && rank == 0) {   // uniform over the CTA
				// thread t sums the squares of a head's K columns of token t in column order, as the other forms do
				u32 *const tile_s = reinterpret_cast<u32 *>(out_s + WM * rp.n_tok);
				f32 *const scale_s = reinterpret_cast<f32 *>(tile_s + rp.n_tok * ACC_PITCH);
				if (works) {
					for (u32 g = 0; g < groups; ++g) {
						u32 r[16];
						whole_group(g, r);
#pragma unroll
						for (u32 i = 0; i < 16; ++i) tile_s[(16 * g + i) * ACC_PITCH + wrow] = r[i];
					}
				}
				u32 const d = p.head_dim;
				u32 const heads = d == 128 ? (seg.col0 % 256 == 0 ? 1u : 0u) : WM / (2 * d);   // K heads in the tile
				if (warp >= 2) {
					named_barrier_sync(1, 128);
					for (u32 i = threadIdx.x - 64; i < heads * rp.n_tok; i += 128) {
						u32 const h = i / rp.n_tok, t = i % rp.n_tok;
						u32 const *src = tile_s + t * ACC_PITCH + h * 2 * d;
						f32 ssum = 0.0f;
#pragma unroll 16
						for (u32 c = 0; c < d; ++c) {
							f32 const f = acc_to_f32<F8>(src[c]);
							ssum = __fmaf_rn(f, f, ssum);
						}
						f32 const ks = __fmul_rn(rsqrt_approx(__fadd_rn(ssum, p.k0)), p.k1);
						scale_s[i] = ks;
						if (t < p.m) p.rrms[u64(t) * p.rrms_cols + seg.col0 / (2 * d) + h] = ks;
					}
					named_barrier_sync(1, 128);
				}
				if (works) {
					u32 const col = seg.col0 + wrow;
					bool const is_k = col % (2 * d) < d;
					f32 const *const ks = scale_s + (d == 128 ? 0u : wrow / (2 * d)) * rp.n_tok;
#pragma unroll 4
					for (u32 t = 0; t < rp.n_tok; ++t) {
						f32 const f = acc_to_f32<F8>(tile_s[t * ACC_PITCH + wrow]);
						out_s[t * OUT_COLS + wrow] = u8(f32_to_fixedi8(__fmul_rn(f, is_k ? ks[t] : seg.scale)));
					}
				}
			}
		}
		bool const plain = !(HEADS && seg.heads);
		if (works && plain) {
			for (u32 g = 0; g < groups; ++g) {
				u32 r[16];
				whole_group(g, r);
				if constexpr (PAIRS) {
					// the even lane holds the gates, the odd lane the values; the even lane takes tokens 0-7 of the
					// group, the odd lane 8-15
					bool const odd = (lane & 1) != 0;
					u32 const t0 = 16 * g + (odd ? 8u : 0u);
					u32 const col = (w0 + wrow) / 2;
#pragma unroll
					for (u32 i = 0; i < 8; ++i) {
						u32 const other = __shfl_xor_sync(0xffffffffu, odd ? r[i] : r[8 + i], 1);
						f32 const gate = acc_to_f32<F8>(odd ? other : r[i]), val = acc_to_f32<F8>(odd ? r[8 + i] : other);
						u32 b;
						if constexpr (EPI == EPI_GEGLU_E4M3) {
							b = f32_to_e4m3(geglu_val(gate, val, p));
						} else {
							i8 const code = t0 + i < p.m ? p.residual[u64(t0 + i) * p.resid_stride + col] : i8(0);
							f32 const v = resid_val(gate, val, f32(i32(code)), p);
							b = EPI == EPI_RESID_E4M3 ? f32_to_e4m3(v) : u32(f32_to_fixedi8(v));
						}
						out_s[(t0 + i) * OUT_COLS + wrow / 2] = u8(b);
					}
				} else {
					f32 const sc = HEADS ? seg.scale : p.k0;
#pragma unroll
					for (u32 i = 0; i < 16; ++i) {
						out_s[(16 * g + i) * OUT_COLS + wrow] = u8(f32_to_fixedi8(__fmul_rn(acc_to_f32<F8>(r[i]), sc)));
					}
				}
			}
		}
		if (warp >= 2) {
			named_barrier_sync(1, 128);   // the bytes are in place
			// 16-byte chunks along the rows; a quarter's columns are stored by the CTA that finished them
			constexpr u32 CH = OUT_COLS / 16, CH_QUARTER = CH / 4;
			u32 const col0 = HEADS ? seg.col0 : PAIRS ? w0 / 2 : w0;
			u8 *const dst = HEADS ? reinterpret_cast<u8 *>(seg.base) : static_cast<u8 *>(p.c);
			u64 const stride = HEADS ? seg.stride : p.c_stride;
			for (u32 i = threadIdx.x - 64; ok && i < p.m * CH; i += 128) {
				u32 const t = i / CH, ch = i % CH;
				if (owner_of(ch / CH_QUARTER) != rank) continue;
				*reinterpret_cast<uint4 *>(dst + u64(t) * stride + col0 + ch * 16) = *reinterpret_cast<uint4 const *>(out_s + t * OUT_COLS + ch * 16);
			}
		}
	}

	tc_fence_before();
	__syncthreads();
	if (warp == 1) {
		__syncwarp();
		tc_fence_after();
		tmem_dealloc(tmem_base, tmem_cols);
	}
}

}  // namespace x17
