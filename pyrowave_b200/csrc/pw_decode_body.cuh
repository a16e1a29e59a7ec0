// Device bodies of the decoder stages, shared by the per-stage kernels
// (pw_decode.cu) and the batched form's persistent kernel (pw_encode.cu):
// the dequantiser of one 32x32 block and the inverse transform of one tile.
//
// Reference behaviour followed (file:line in the reference tree):
//   dequantiser   shaders/wavelet_dequant.comp:100-391 (STORAGE_MODE 0), pyrowave_decoder.cpp:280-381
//   inverse level shaders/idwt.comp:25-214, pyrowave_decoder.cpp:699-778
//
// Every payload read is bounds-checked against the payload size: the payload
// comes from the network and a malformed packet must decode to garbage, never
// to an out-of-bounds access. Reads past the end return zero.
#pragma once

#include "pw_device.cuh"

namespace pw
{
namespace
{
struct PayloadReader
{
	const uint32_t *words;
	uint32_t nwords;
	__device__ __forceinline__ uint32_t w32(uint32_t i) const { return i < nwords ? __ldcg(words + i) : 0u; }
	__device__ __forceinline__ uint32_t u8(uint32_t i) const { return (w32(i >> 2) >> (8u * (i & 3u))) & 0xffu; }
	__device__ __forceinline__ uint32_t u16(uint32_t i) const { return (w32(i >> 1) >> (16u * (i & 1u))) & 0xffffu; }
};

// A block's words staged in shared memory: words [base, base + count) of the
// payload come from `s`, anything else from the bounds-checked global reader,
// so reads of a malformed block behave exactly as with PayloadReader alone.
struct StagedReader
{
	const uint32_t *s;
	uint32_t base, count;
	PayloadReader g;
	__device__ __forceinline__ uint32_t w32(uint32_t i) const
	{
		const uint32_t r = i - base;
		return r < count ? s[r] : g.w32(i);
	}
	__device__ __forceinline__ uint32_t u8(uint32_t i) const { return (w32(i >> 2) >> (8u * (i & 3u))) & 0xffu; }
	__device__ __forceinline__ uint32_t u16(uint32_t i) const { return (w32(i >> 1) >> (16u * (i & 1u))) & 0xffffu; }
};

constexpr uint32_t kSpeculativeWords = 128; // staged with the header when the block size is not yet known

// s[i] = payload word off + i for i in [begin, end), by kThreads threads with
// up to eight loads per thread in flight together.
template <int kThreads = 128>
__device__ __forceinline__ void stage_words(uint32_t *s, const PayloadReader &g, uint32_t off, uint32_t begin,
                                            uint32_t end, int t)
{
	for (uint32_t base = begin + uint32_t(t); base < end; base += kThreads * 8)
	{
		uint32_t v[8];
#pragma unroll
		for (int u = 0; u < 8; u++)
		{
			const uint32_t i = base + uint32_t(kThreads) * u;
			v[u] = i < end ? g.w32(off + i) : 0u;
		}
#pragma unroll
		for (int u = 0; u < 8; u++)
		{
			const uint32_t i = base + uint32_t(kThreads) * u;
			if (i < end)
				s[i] = v[u];
		}
	}
}

// The barrier of a block's thread group: hardware barrier `bar` of 128
// threads, or the whole CTA when a CTA holds one smaller group.
template <int kSubs> __device__ __forceinline__ void block_sync(int bar)
{
	if constexpr (kSubs == 1)
		group_sync(bar);
	else
		__syncthreads();
}

__device__ __forceinline__ void store_coef(float *c32, __half *c16, bool fp16, int64_t idx, float v)
{
	if (fp16)
		c16[idx] = __float2half_rn(v);
	else
		c32[idx] = v;
}

// One 32x32 block per thread group; thread = one 4x2 sub-block (the
// reference's mapping, wavelet_dequant.comp:222-238), or kSubs sub-blocks two
// 8x8 rows apart. The group with `clear_error` set clears the decode's error
// word: every inverse level runs after the dequantiser has completed, so the
// clear precedes any error report.
struct DequantShared
{
	uint32_t s_words[kMaxBlockWords];
	uint32_t s_plane_off[16];
	uint32_t s_sign_base;
	uint32_t s_sig[4];
};

// One 32x32 block on a group of 128 / kSubs threads: with kSubs = 1 the group
// is threadIdx.x & 127, synchronised with hardware barrier `bar`; with kSubs =
// 2 the whole 64-thread CTA, each thread decoding the sub-blocks of 8x8 rows
// ly and ly + 2.
template <int kSubs = 1>
__device__ __forceinline__ void dequant_body(DequantShared &sh, const BlockParams &p, const DecodeInput &in,
                                             const int blk, const bool clear_error, const int bar)
{
	static_assert(kSubs == 1 || kSubs == 2, "one or two sub-blocks per thread");
	constexpr int kGroup = 128 / kSubs;
	constexpr int kRowStep = 4 / kSubs;
	uint32_t *const s_words = sh.s_words;
	uint32_t *const s_plane_off = sh.s_plane_off;
	uint32_t &s_sign_base = sh.s_sign_base;
	uint32_t *const s_sig = sh.s_sig;
	pdl_trigger();
	const int k = find_band(p, blk);
	const BandEntry &B = p.band[k];
	const LevelDesc &L = p.level[B.level];
	const int rel = blk - B.block32_offset;
	const int by32 = rel / B.block32_stride, bx32 = rel - by32 * B.block32_stride;
	const bool f16 = L.fp16 != 0;
	const int t = threadIdx.x & (kGroup - 1), lane = t & 31;
	const int sub = t & 7, lx = (t >> 3) & 3, ly0 = t >> 5;
	const int ox = bx32 * 32 + lx * 8 + sub_x(sub);
	pdl_wait();
	if (clear_error && t == 0 && in.error)
		*in.error = 0u;
	if (clear_error && in.state && t < int(sizeof(DecodeState) / 4))
		reinterpret_cast<uint32_t *>(in.state)[t] = 0u;

	uint32_t off, words = 0;
	const bool sized_by_header = in.offsets || in.keys;
	if (in.keys)
	{
		const unsigned long long key = __ldcg(in.keys + blk);
		off = key == ~0ull ? 0xffffffffu : uint32_t(key & 0x3fffffffull);
	}
	else if (in.offsets)
		off = __ldcg(in.offsets + blk);
	else
	{
		const uint2 m = __ldcg(reinterpret_cast<const uint2 *>(in.block_meta) + blk);
		off = m.y ? m.x : 0xffffffffu;
		words = m.y;
	}

	if (off == 0xffffffffu)
	{
		// Missing block: all coefficients are zero (wavelet_dequant.comp:242-248).
		const float zero[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
		for (int h = 0; h < kSubs; h++)
		{
			const int oy = by32 * 32 + (ly0 + h * kRowStep) * 8 + sub_y(sub);
			store_subblock(in.coef32, in.coef16, f16, B.offset + int64_t(oy) * L.pitch + ox, L.pitch, zero);
		}
		return;
	}

	// Stage the block's words in shared memory with all loads in flight at
	// once; every read below is then a shared-memory read. With only an offset
	// table the size comes from the block header, so the first
	// kSpeculativeWords are fetched together with it.
	const PayloadReader grd{in.payload, in.payload_words};
	uint32_t staged;
	if (sized_by_header)
	{
		stage_words<kGroup>(s_words, grd, off, 0, kSpeculativeWords, t);
		block_sync<kSubs>(bar);
		words = (s_words[0] >> 16) & 0xfffu;
		staged = min(max(words, kSpeculativeWords), uint32_t(kMaxBlockWords));
		stage_words<kGroup>(s_words, grd, off, kSpeculativeWords, staged, t);
	}
	else
	{
		staged = min(words, uint32_t(kMaxBlockWords));
		stage_words<kGroup>(s_words, grd, off, 0, staged, t);
	}
	block_sync<kSubs>(bar);
	const StagedReader rd{s_words, off, staged, grd};
	const uint32_t ballot = rd.w32(off) & 0xffffu;
	const uint32_t q_code = rd.w32(off + 1) & 0xffu;
	const uint32_t n = uint32_t(__popc(ballot));

	if (t < 16)
	{
		uint32_t cw = 0, qb = 0;
		if ((ballot >> t) & 1u)
		{
			const uint32_t local = uint32_t(__popc(ballot & ((1u << t) - 1u)));
			cw = rd.u16(off * 2 + 4 + local);
			qb = rd.u8(off * 4 + 8 + n * 2 + local) & 0xfu;
		}
		const uint32_t lsbs = cw & 0x5555u;
		uint32_t msbs = cw & 0xaaaau;
		msbs |= msbs >> 1;
		const uint32_t cost = uint32_t(__popc(lsbs) + __popc(msbs)) + qb * 8u;
		uint32_t inc = cost;
#pragma unroll
		for (int o = 1; o < 16; o *= 2)
		{
			const uint32_t y = __shfl_up_sync(0x0000ffffu, inc, o);
			if (t >= o)
				inc += y;
		}
		const uint32_t base = off * 4 + 8 + 3 * n;
		s_plane_off[t] = base + inc - cost;
		if (t == 15)
			s_sign_base = 8u * (base + inc);
	}
	block_sync<kSubs>(bar);

	float v[kSubs][8];
#pragma unroll
	for (int h = 0; h < kSubs; h++)
	{
		const int grp = (ly0 + h * kRowStep) * 4 + lx;
#pragma unroll
		for (int i = 0; i < 8; i++)
			v[h][i] = 0.0f;
		if ((ballot >> grp) & 1u)
		{
			const uint32_t local = uint32_t(__popc(ballot & ((1u << grp) - 1u)));
			const uint32_t cw = rd.u16(off * 2 + 4 + local);
			const uint32_t cw2 = rd.u8(off * 4 + 8 + n * 2 + local);
			const uint32_t qb = cw2 & 0xfu;
			if (cw != 0)
			{
				const uint32_t mask = (1u << (2 * sub)) - 1u;
				const uint32_t lsbs = cw & 0x5555u;
				uint32_t msbs = cw & 0xaaaau;
				msbs |= msbs >> 1;
				uint32_t byte_offset =
				    uint32_t(__popc(lsbs & mask) + __popc(msbs & mask)) + qb * uint32_t(sub) + s_plane_off[grp];
				const int planes = int(qb + ((cw >> (2 * sub)) & 3u));
				uint32_t dec[8] = {0, 0, 0, 0, 0, 0, 0, 0};
				if (planes <= 16)
				{
					// Plane bytes (most significant first) as the rows of two 8x8 bit
					// matrices; transposed, byte i holds coefficient i's magnitude bits.
					unsigned long long lo = 0, hi = 0;
					for (int pl = planes - 1; pl >= 0; pl--)
					{
						const unsigned long long bits = rd.u8(byte_offset++);
						if (pl < 8)
							lo |= bits << (8 * pl);
						else
							hi |= bits << (8 * (pl - 8));
					}
					lo = transpose8x8(lo);
					hi = transpose8x8(hi);
#pragma unroll
					for (int i = 0; i < 8; i++)
						dec[i] = uint32_t((lo >> (8 * i)) & 0xffu) | (uint32_t((hi >> (8 * i)) & 0xffu) << 8);
				}
				else
				{
					// Only a malformed header gives more than 16 planes.
					for (int pl = planes - 1; pl >= 0; pl--)
					{
						const uint32_t bits = rd.u8(byte_offset++);
#pragma unroll
						for (int i = 0; i < 8; i++)
							dec[i] |= ((bits >> i) & 1u) << pl;
					}
				}
#pragma unroll
				for (int i = 0; i < 8; i++)
				{
					float f = float(dec[i]);
					if (f != 0.0f)
						f = __fadd_rn(f, 0.5f);
					v[h][i] = f;
				}
			}
			const float inv_scale = __fmul_rn(decode_quant(q_code), decode_quant_scale((cw2 >> 4) & 0xfu));
#pragma unroll
			for (int i = 0; i < 8; i++)
				v[h][i] = __fmul_rn(v[h][i], inv_scale);
		}
	}

	// Sign bits: position = number of significant coefficients before this one
	// (in sub-block order: 8x8 rows, then the 32 sub-blocks of a row).
	uint32_t nsig[kSubs], inc[kSubs];
#pragma unroll
	for (int h = 0; h < kSubs; h++)
	{
		nsig[h] = 0;
#pragma unroll
		for (int i = 0; i < 8; i++)
			nsig[h] += v[h][i] != 0.0f ? 1u : 0u;
		inc[h] = nsig[h];
#pragma unroll
		for (int o = 1; o < 32; o *= 2)
		{
			const uint32_t y = __shfl_up_sync(0xffffffffu, inc[h], o);
			if (lane >= o)
				inc[h] += y;
		}
		if (lane == 31)
			s_sig[ly0 + h * kRowStep] = inc[h];
	}
	block_sync<kSubs>(bar);
#pragma unroll
	for (int h = 0; h < kSubs; h++)
	{
		const int ly = ly0 + h * kRowStep;
		uint32_t bitpos = s_sign_base + inc[h] - nsig[h];
		for (int w = 0; w < ly; w++)
			bitpos += s_sig[w];
		// This thread's (at most 8) sign bits are consecutive: one 64-bit window.
		const uint32_t sw = bitpos >> 5, shift = bitpos & 31u;
		const uint64_t window = (uint64_t(rd.w32(sw + 1)) << 32 | rd.w32(sw)) >> shift;
		int nth = 0;
#pragma unroll
		for (int i = 0; i < 8; i++)
		{
			if (v[h][i] != 0.0f)
			{
				if ((window >> nth) & 1u)
					v[h][i] = -v[h][i];
				nth++;
			}
		}
		const int oy = by32 * 32 + ly * 8 + sub_y(sub);
		store_subblock(in.coef32, in.coef16, f16, B.offset + int64_t(oy) * L.pitch + ox, L.pitch, v[h]);
	}
}

constexpr int kBandTile = 36; // 32 band samples + 2 on each side
// Band tiles are stored as rows of 40 samples from 4 before the tile (16-byte
// aligned in the band, so an interior tile is one TMA box per band): band
// sample j of the tile (0 = 2 before it) is at column j + kBandCol0.
constexpr int kBandRow = 40;
constexpr int kBandCol0 = 2;
constexpr uint32_t kBandBoxBytes = kBandTile * kBandRow * 4;
constexpr uint32_t kTmaMaxPolls = 1u << 20; // bounded wait for a tile load

// Work split of an inverse level: outputs per lifting item. Whole tiles favour
// few instructions (24 samples lifted for 16 kept), stripes and 1024-thread
// CTAs a short chain.
template <int kThreads, int kStripes> struct IdwtSplit
{
	static constexpr int kOutRows = 64 / kStripes;       // output rows of the CTA
	static constexpr int kBandRows = kOutRows / 2 + 4;   // band rows it reads
	static constexpr int kOut = kStripes > 1 ? 4 : (kThreads >= 1024 ? 8 : 16);
};

template <int kOutRows> struct IdwtSharedT
{
	int xl[kBandRow], xh[kBandRow], yl[kBandTile], yh[kBandTile]; // mirrored band indices (edge tiles)
	alignas(128) float band[4][kOutRows / 2 + 4][kBandRow];
	alignas(16) float v[2][kOutRows][kBandTile]; // after vertical lifting: [horizontal low/high][output row][band column]
	uint64_t tile_bar;                           // completion of the TMA tile loads
};
using IdwtShared = IdwtSharedT<64>;

// Store of kOut consecutive 8-bit samples (four to a word) of a row, the first
// `left` of them inside the plane, with the widest stores the address allows.
template <int kOut> __device__ __forceinline__ void store_samples8(uint8_t *dst, const uint32_t (&w)[kOut / 4], int left)
{
	const uintptr_t a = reinterpret_cast<uintptr_t>(dst);
	if (left >= kOut && kOut >= 8 && (a & (kOut - 1)) == 0)
	{
		if constexpr (kOut == 16)
			*reinterpret_cast<uint4 *>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
		else if constexpr (kOut == 8)
			*reinterpret_cast<uint2 *>(dst) = make_uint2(w[0], w[1]);
	}
	else if (left >= kOut && (a & 3u) == 0)
	{
#pragma unroll
		for (int k = 0; k < kOut / 4; k++)
			reinterpret_cast<uint32_t *>(dst)[k] = w[k];
	}
	else if (left >= kOut && (a & 1u) == 0)
	{
#pragma unroll
		for (int k = 0; k < kOut / 2; k++)
			reinterpret_cast<uint16_t *>(dst)[k] = uint16_t(w[k >> 1] >> (16 * (k & 1)));
	}
	else
	{
#pragma unroll
		for (int k = 0; k < kOut; k++)
			if (k < left)
				dst[k] = uint8_t(w[k >> 2] >> (8 * (k & 3)));
	}
}

// The same for 16-bit samples (two to a word, 2-byte aligned rows).
template <int kOut> __device__ __forceinline__ void store_samples16(uint16_t *dst, const uint32_t (&w)[kOut / 2], int left)
{
	const uintptr_t a = reinterpret_cast<uintptr_t>(dst);
	if (left >= kOut && kOut >= 8 && (a & 15u) == 0)
	{
		if constexpr (kOut >= 8)
		{
#pragma unroll
			for (int k = 0; k < kOut / 8; k++)
				reinterpret_cast<uint4 *>(dst)[k] = make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
		}
	}
	else if (left >= kOut && (a & 3u) == 0)
	{
#pragma unroll
		for (int k = 0; k < kOut / 2; k++)
			reinterpret_cast<uint32_t *>(dst)[k] = w[k];
	}
	else if (left >= kOut)
	{
		// An odd sample position: words shifted by one sample between the ends.
		dst[0] = uint16_t(w[0]);
#pragma unroll
		for (int k = 0; k + 1 < kOut / 2; k++)
			*reinterpret_cast<uint32_t *>(dst + 1 + 2 * k) = __byte_perm(w[k], w[k + 1], 0x5432);
		dst[kOut - 1] = uint16_t(w[kOut / 2 - 1] >> 16);
	}
	else
	{
#pragma unroll
		for (int k = 0; k < kOut; k++)
			if (k < left)
				dst[k] = uint16_t(w[k >> 1] >> (16 * (k & 1)));
	}
}

// Two decoded samples (one of each row of a pair) as integers in the low bits:
// clamp(e + 0.5) * scale + 0.5 truncated (R8_UNORM / R16_UNORM store). The sum
// is in [0.5, 65535.5], so adding 2^23 rounded toward zero leaves its integer
// part in the low mantissa bits.
__device__ __forceinline__ void quantise_samples2(f32x2 e, float scale, uint32_t &u0, uint32_t &u1)
{
	float a, b;
	f2_unpack(e, a, b);
	a = __fmul_rn(__saturatef(__fadd_rn(a, 0.5f)), scale);
	b = __fmul_rn(__saturatef(__fadd_rn(b, 0.5f)), scale);
	const f32x2 t = f2_add_rz(f2_add_rn(f2_pack(a, b), f2_pack(0.5f, 0.5f)), f2_pack(8388608.0f, 8388608.0f));
	f2_unpack(t, a, b);
	u0 = __float_as_uint(a);
	u1 = __float_as_uint(b);
}

// One inverse level for a 64x64 output tile (32x32 band tile) of one component.
// Large levels run 256-thread CTAs, several per SM; the batched form's small
// levels run 1024-thread CTAs whose lifting items cover half as many outputs.
// With kStripes = 4 a CTA computes one stripe of 16 output rows of the tile
// (small levels: four times the CTAs, each with a quarter of the lifting and
// a third of the loads), with the same arithmetic per output.
//
// Bound by instruction issue on the large levels, by latency on the small ones.
// Both passes lift packed pairs (two FP32 operations per instruction): adjacent
// columns in the vertical pass, rows (r, r + rows / 2) in the horizontal one.
// The scaling by K and 1/K, one multiplication per sample, puts each pair into
// adjacent registers, so the packing costs nothing. It stays scalar: a packed
// product that feeds a packed sum was seen rounded once, as a fused operation,
// which is off by an ulp from the two roundings wanted. Measured against scalar
// lifting: decode of a 1080p 4:2:0 frame 41.7 -> 32.8 us, 4K 4:4:4 133 -> 118 us;
// 16-bit 4:4:4 at 1365x767 (rows of no common alignment) encode + decode 124 ->
// 96 us.
template <int kThreads, int kStripes = 1>
__device__ __forceinline__ void idwt_body(IdwtSharedT<IdwtSplit<kThreads, kStripes>::kOutRows> &sh, const LevelParams &p,
                                          const DecodeInput &in, const PlaneOutput &out, const LevelTileMap *maps,
                                          const int tile, const int comp_index, const int stripe = 0)
{
	using Split = IdwtSplit<kThreads, kStripes>;
	constexpr int kOut = Split::kOut, kWin = kOut + 8;
	constexpr int kRows = Split::kBandRows;
	pdl_trigger();
	const int level = p.level;
	const int comp = (level == 0 && !p.chroma444) ? 0 : comp_index;
	const LevelDesc &L = p.L;
	const int tx = tile % L.tiles_x, ty = tile / L.tiles_x;
	const int nx = L.width, ny = L.height;
	const bool final_level = level == 0 || (level == 1 && comp != 0 && !p.chroma444);
	const bool f16 = L.fp16 != 0;

	// Interior tiles read every band sample at its own position. Interior FP32
	// tiles of a decoder with tensor maps take one TMA box per band (barrier and
	// maps made ready before the dependency wait); the others load vectors of
	// four samples, gathered through the mirrored index tables where they cross
	// an edge.
	const int x0 = tx * 32 - 4, y0 = ty * 32 - 2 + stripe * (Split::kOutRows / 2); // column 0, row 0 of the band tiles
	const bool y_inside = y0 >= 0 && y0 + kRows <= ny;
	const bool interior = x0 >= 0 && x0 + kBandRow <= nx && y_inside;
	const bool use_tma = kThreads == 256 && kStripes == 1 && interior && maps && ((maps->valid >> comp) & 1u) && !f16 &&
	                     !L.stage16;
	if (!interior)
	{
		for (int k = threadIdx.x; k < 2 * kBandRow + 2 * kRows; k += kThreads)
		{
			if (k < kBandRow)
				sh.xl[k] = inv_index_low(x0 + k, nx);
			else if (k < 2 * kBandRow)
				sh.xh[k - kBandRow] = inv_index_high(x0 + k - kBandRow, nx);
			else if (k < 2 * kBandRow + kRows)
				sh.yl[k - 2 * kBandRow] = inv_index_low(y0 + k - 2 * kBandRow, ny);
			else
				sh.yh[k - 2 * kBandRow - kRows] = inv_index_high(y0 + k - 2 * kBandRow - kRows, ny);
		}
		__syncthreads();
	}
	else if (use_tma)
	{
		if (threadIdx.x == 0)
		{
			mbarrier_init(&sh.tile_bar, 1);
			prefetch_tensor_map(&maps->map);
		}
		__syncthreads();
	}
	pdl_wait();

	if (use_tma)
	{
		if (threadIdx.x == 0)
		{
			mbarrier_expect_tx(&sh.tile_bar, 4 * kBandBoxBytes);
#pragma unroll
			for (int b = 0; b < 4; b++)
				tma_load_2d(&sh.band[b][0][0], &maps->map, x0, maps->row[comp][b] + y0, &sh.tile_bar);
		}
		const bool done = mbarrier_wait(&sh.tile_bar, 0, kTmaMaxPolls) && !maps->test_fail_wait;
		if (__syncthreads_or(!done))
		{
			// Give up on this tile: record it, and keep the CTA alive (its shared
			// memory is the copy's destination) for one more bounded wait.
			if (threadIdx.x == 0 && in.error)
				atomicOr(in.error, kDecodeErrorTileWait);
			(void)mbarrier_wait(&sh.tile_bar, 0, kTmaMaxPolls);
			return;
		}
	}
	else
	{
		// A thread keeps one group of four columns: its mirrored indices are read
		// once, and every load of its rows is in flight at once.
		constexpr int kVecPerRow = kBandRow / 4;
		constexpr int kLoadRows = kThreads / kVecPerRow;
		constexpr int kIters = (4 * kRows + kLoadRows - 1) / kLoadRows;
		const int j = threadIdx.x % kVecPerRow, br0 = threadIdx.x / kVecPerRow;
		const bool loader = threadIdx.x < kLoadRows * kVecPerRow;
		const int x = x0 + 4 * j;
		const bool inside = x >= 0 && x + 4 <= nx;
		int4 lo = make_int4(x, x + 1, x + 2, x + 3), hi = lo;
		if (!inside)
		{
			lo = *reinterpret_cast<const int4 *>(&sh.xl[4 * j]);
			hi = *reinterpret_cast<const int4 *>(&sh.xh[4 * j]);
		}
		float4 v[kIters];
#pragma unroll
		for (int u = 0; u < kIters; u++)
		{
			const int br = br0 + u * kLoadRows;
			v[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
			if (!loader || br >= 4 * kRows)
				continue;
			const int b = br / kRows, i = br - b * kRows;
			const int yy = y_inside ? y0 + i : ((b >> 1) ? sh.yh[i] : sh.yl[i]);
			const int64_t row = p.band[comp][b].offset + int64_t(yy) * L.pitch;
			if (!inside)
			{
				const int4 xi = (b & 1) ? hi : lo;
				v[u] = make_float4(load_coef(in.coef32, in.coef16, f16, row + xi.x),
				                   load_coef(in.coef32, in.coef16, f16, row + xi.y),
				                   load_coef(in.coef32, in.coef16, f16, row + xi.z),
				                   load_coef(in.coef32, in.coef16, f16, row + xi.w));
			}
			else if (f16)
			{
				const uint2 hv = __ldcg(reinterpret_cast<const uint2 *>(in.coef16 + row + x));
				const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&hv.x));
				const float2 c = __half22float2(*reinterpret_cast<const __half2 *>(&hv.y));
				v[u] = make_float4(a.x, a.y, c.x, c.y);
			}
			else
				v[u] = __ldcg(reinterpret_cast<const float4 *>(in.coef32 + row + x));
		}
#pragma unroll
		for (int u = 0; u < kIters; u++)
		{
			const int br = br0 + u * kLoadRows;
			if (!loader || br >= 4 * kRows)
				continue;
			const int b = br / kRows, i = br - b * kRows;
			float4 f = v[u];
			if (L.stage16)
			{
				f.x = round_to_half(f.x);
				f.y = round_to_half(f.y);
				f.z = round_to_half(f.z);
				f.w = round_to_half(f.w);
			}
			*reinterpret_cast<float4 *>(&sh.band[b][i][4 * j]) = f;
		}
	}
	__syncthreads();

	// Vertical lifting: 18 pairs of band columns x {horizontal low: LL/LH,
	// horizontal high: HL/HH} x segments of kOut rows. Items start at another
	// warp from tile to tile: they fill half the warps, and warps of one index
	// share an issue port.
	{
		constexpr int kPairs = kBandTile / 2, kSegs = Split::kOutRows / kOut;
		const int t0 = kStripes == 1 ? (threadIdx.x + 32 * (tile & 3)) & (kThreads - 1) : threadIdx.x;
		for (int item = t0; item < kPairs * 2 * kSegs; item += kThreads)
		{
			const int pair = item % kPairs;
			const int which = (item / kPairs) & 1;
			const int seg = item / (2 * kPairs);
			f32x2 e[kWin];
#pragma unroll
			for (int jj = 0; jj < kWin; jj += 2)
			{
				const int i = (seg * kOut + jj) >> 1;
				const float2 a = *reinterpret_cast<const float2 *>(&sh.band[which][i][2 * pair + kBandCol0]);
				const float2 b = *reinterpret_cast<const float2 *>(&sh.band[which + 2][i][2 * pair + kBandCol0]);
				e[jj] = f2_pack(__fmul_rn(a.x, kK), __fmul_rn(a.y, kK));
				e[jj + 1] = f2_pack(__fmul_rn(b.x, kInvK), __fmul_rn(b.y, kInvK));
			}
			lift_inverse2(e);
#pragma unroll
			for (int jj = 4; jj < 4 + kOut; jj++)
			{
				if (L.stage16)
				{
					float a, b;
					f2_unpack(e[jj], a, b);
					e[jj] = f2_pack(round_to_half(a), round_to_half(b));
				}
				*reinterpret_cast<f32x2 *>(&sh.v[which][seg * kOut + jj - 4][2 * pair]) = e[jj];
			}
		}
	}
	__syncthreads();

	// Horizontal lifting of row pairs, segments of kOut outputs.
	constexpr int kPairRows = Split::kOutRows / 2;
	for (int item = threadIdx.x; item < kPairRows * (64 / kOut); item += kThreads)
	{
		const int pr = item % kPairRows, seg = item / kPairRows;
		f32x2 e[kWin];
		// Band columns seg * kOut / 2 + jj / 2 of the two rows, kV at a time.
		constexpr int kV = kOut >= 8 ? 4 : 2;
#pragma unroll
		for (int jj = 0; jj < kWin; jj += 2 * kV)
		{
#pragma unroll
			for (int which = 0; which < 2; which++)
			{
				float a[kV], b[kV];
				const float *ra = &sh.v[which][pr][(seg * kOut + jj) >> 1];
				const float *rb = &sh.v[which][pr + kPairRows][(seg * kOut + jj) >> 1];
				if constexpr (kV == 4)
				{
					const float4 qa = *reinterpret_cast<const float4 *>(ra), qb = *reinterpret_cast<const float4 *>(rb);
					a[0] = qa.x, a[1] = qa.y, a[2] = qa.z, a[3] = qa.w;
					b[0] = qb.x, b[1] = qb.y, b[2] = qb.z, b[3] = qb.w;
				}
				else
				{
					const float2 qa = *reinterpret_cast<const float2 *>(ra), qb = *reinterpret_cast<const float2 *>(rb);
					a[0] = qa.x, a[1] = qa.y;
					b[0] = qb.x, b[1] = qb.y;
				}
				const float k = which ? kInvK : kK;
#pragma unroll
				for (int m = 0; m < kV; m++)
					e[jj + 2 * m + which] = f2_pack(__fmul_rn(a[m], k), __fmul_rn(b[m], k));
			}
		}
		lift_inverse2(e);
		if (L.stage16)
		{
#pragma unroll
			for (int jj = 4; jj < 4 + kOut; jj++)
			{
				float a, b;
				f2_unpack(e[jj], a, b);
				e[jj] = f2_pack(round_to_half(a), round_to_half(b));
			}
		}
		const int gy = ty * 64 + stripe * Split::kOutRows + pr; // and gy + kPairRows
		const int gx0 = tx * 64 + seg * kOut;
		if (final_level)
		{
			const int pw = p.plane_width[comp], ph = p.plane_height[comp];
			uint8_t *const plane = comp == 0 ? out.data[0] : (comp == 1 ? out.data[1] : out.data[2]);
			const int opitch = comp == 0 ? out.pitch[0] : (comp == 1 ? out.pitch[1] : out.pitch[2]);
			if (out.sample16)
			{
				uint32_t w0[kOut / 2], w1[kOut / 2];
#pragma unroll
				for (int k = 0; k < kOut / 2; k++)
				{
					uint32_t a0, a1, b0, b1;
					quantise_samples2(e[4 + 2 * k], 65535.0f, a0, a1);
					quantise_samples2(e[5 + 2 * k], 65535.0f, b0, b1);
					w0[k] = __byte_perm(a0, b0, 0x5410);
					w1[k] = __byte_perm(a1, b1, 0x5410);
				}
				if (gy < ph)
					store_samples16<kOut>(reinterpret_cast<uint16_t *>(plane + size_t(gy) * opitch) + gx0, w0, pw - gx0);
				if (gy + kPairRows < ph)
					store_samples16<kOut>(reinterpret_cast<uint16_t *>(plane + size_t(gy + kPairRows) * opitch) + gx0, w1,
					                      pw - gx0);
			}
			else
			{
				uint32_t w0[kOut / 4], w1[kOut / 4];
#pragma unroll
				for (int k = 0; k < kOut / 4; k++)
				{
					uint32_t a[4], b[4];
#pragma unroll
					for (int m = 0; m < 4; m++)
						quantise_samples2(e[4 + 4 * k + m], 255.0f, a[m], b[m]);
					w0[k] = __byte_perm(__byte_perm(a[0], a[1], 0x0040), __byte_perm(a[2], a[3], 0x0040), 0x5410);
					w1[k] = __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
				}
				if (gy < ph)
					store_samples8<kOut>(plane + size_t(gy) * opitch + gx0, w0, pw - gx0);
				if (gy + kPairRows < ph)
					store_samples8<kOut>(plane + size_t(gy + kPairRows) * opitch + gx0, w1, pw - gx0);
			}
		}
		else
		{
			const LevelDesc &P = p.P;
			const int64_t ll = comp == 0 ? p.prev_ll[0] : (comp == 1 ? p.prev_ll[1] : p.prev_ll[2]);
			const bool pf16 = P.fp16 != 0;
			float r[2][kOut];
#pragma unroll
			for (int k = 0; k < kOut; k++)
				f2_unpack(e[4 + k], r[0][k], r[1][k]);
#pragma unroll
			for (int h = 0; h < 2; h++)
			{
				const int y = gy + h * kPairRows;
				if (y >= P.height)
					continue;
				const int64_t base = ll + int64_t(y) * P.pitch + gx0;
				if (gx0 + kOut > P.width)
				{
#pragma unroll
					for (int k = 0; k < kOut; k++)
						if (gx0 + k < P.width)
							store_coef(in.coef32, in.coef16, pf16, base + k, r[h][k]);
				}
				else if (pf16)
				{
#pragma unroll
					for (int k = 0; k < kOut; k += 4)
					{
						const __half2 a = __floats2half2_rn(r[h][k], r[h][k + 1]),
						              b = __floats2half2_rn(r[h][k + 2], r[h][k + 3]);
						*reinterpret_cast<uint2 *>(in.coef16 + base + k) =
						    make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
					}
				}
				else
				{
#pragma unroll
					for (int k = 0; k < kOut; k += 4)
						*reinterpret_cast<float4 *>(in.coef32 + base + k) =
						    make_float4(r[h][k], r[h][k + 1], r[h][k + 2], r[h][k + 3]);
				}
			}
		}
	}
}

} // namespace
} // namespace pw
