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
};

// A block's words staged in shared memory, addressed from the block's first
// word. With kChecked, words beyond `count` come from the bounds-checked global
// reader (a malformed block reads on into what follows it, never out of
// bounds); without, the caller has made sure that every word read is staged.
template <bool kChecked> struct BlockReader
{
	const uint32_t *s;
	uint32_t off, count;
	PayloadReader g;
	__device__ __forceinline__ uint32_t w32(uint32_t r) const
	{
		if constexpr (kChecked)
			return r < count ? s[r] : g.w32(off + r);
		else
			return s[r];
	}
	__device__ __forceinline__ uint32_t u8(uint32_t r) const
	{
		if constexpr (kChecked)
			return (w32(r >> 2) >> (8u * (r & 3u))) & 0xffu;
		else
			return reinterpret_cast<const uint8_t *>(s)[r];
	}
	__device__ __forceinline__ uint32_t u16(uint32_t r) const
	{
		if constexpr (kChecked)
			return (w32(r >> 1) >> (16u * (r & 1u))) & 0xffffu;
		else
			return reinterpret_cast<const uint16_t *>(s)[r];
	}
};

constexpr uint32_t kSpeculativeWords = 128; // staged with the header when the block size is not yet known

// s[i] = payload word off + i for i in [begin, end), by one warp with up to
// eight loads per lane in flight together.
__device__ __forceinline__ void stage_words(uint32_t *s, const PayloadReader &g, uint32_t off, uint32_t begin,
                                            uint32_t end)
{
	for (uint32_t base = begin + (threadIdx.x & 31); base < end; base += 32 * 8)
	{
		uint32_t v[8];
#pragma unroll
		for (int u = 0; u < 8; u++)
			v[u] = base + 32u * u < end ? g.w32(off + base + 32u * u) : 0u;
#pragma unroll
		for (int u = 0; u < 8; u++)
			if (base + 32u * u < end)
				s[base + 32u * u] = v[u];
	}
}

__device__ __forceinline__ void store_coef(float *c32, __half *c16, bool fp16, int64_t idx, float v)
{
	if (fp16)
		c16[idx] = __float2half_rn(v);
	else
		c32[idx] = v;
}

// A warp's staging area: the block's words and room for the reads of whole
// words just past them.
struct DequantShared
{
	uint32_t words[kMaxBlockWords + 4];
};

// Magnitudes and signs of one staged block (see dequant_body), its four rows'
// sub-blocks stored as coefficients.
template <bool kChecked>
__device__ __forceinline__ void dequant_block(const BlockReader<kChecked> &rd, const uint32_t ballot,
                                              const uint32_t header, const uint32_t first_byte, uint32_t sign_bit,
                                              const float quant, const DecodeInput &in, const bool f16, const int64_t at,
                                              const int pitch)
{
	const unsigned full = 0xffffffffu;
	const int lane = threadIdx.x & 31, sub = lane & 7, lx = lane >> 3;
	float v[4][8];
	uint32_t sig4 = 0;
#pragma unroll
	for (int h = 0; h < 4; h++)
	{
#pragma unroll
		for (int i = 0; i < 8; i++)
			v[h][i] = 0.0f;
		if (((ballot >> (4 * h)) & 0xfu) == 0)
			continue; // no coded 8x8 in the row
		// Lane grp of the header pass holds 8x8 grp: code word, Q bits, scale.
		const int grp = 4 * h + lx;
		const uint32_t cw = __shfl_sync(full, header, grp);
		uint32_t byte = __shfl_sync(full, first_byte, grp);
		const uint32_t qb = (cw >> 16) & 0xfu;
		const uint32_t before = (1u << (2 * sub)) - 1u;
		byte += uint32_t(plane_code_sum(cw & before, 0)) + qb * uint32_t(sub);
		const uint32_t planes = (cw & 0xffffu) != 0 ? qb + ((cw >> (2 * sub)) & 3u) : 0u;
		const float scale = __fmul_rn(quant, decode_quant_scale((cw >> 20) & 0xfu));
		uint32_t sig = 0;
		if (__reduce_max_sync(full, planes) <= 8)
		{
			// The sub-block's plane bytes (most significant first) as one 64-bit
			// window, turned round and moved down so that byte k is plane k: the
			// rows of an 8x8 bit matrix; transposed, byte i is coefficient i.
			unsigned long long m = 0;
			if (planes != 0)
			{
				const uint32_t w = byte >> 2, sh = 8u * (byte & 3u);
				const uint32_t a = rd.w32(w), b = rd.w32(w + 1), c = rd.w32(w + 2);
				const uint32_t lo = __funnelshift_r(a, b, sh), hi = __funnelshift_r(b, c, sh);
				m = ((unsigned long long)(__byte_perm(lo, 0, 0x0123)) << 32 | __byte_perm(hi, 0, 0x0123)) >>
				    (8u * (8u - planes));
			}
			sig = uint32_t(m) | uint32_t(m >> 32);
			sig |= sig >> 16;
			sig = (sig | (sig >> 8)) & 0xffu;
			m = transpose8x8(m);
#pragma unroll
			for (int i = 0; i < 8; i += 2)
			{
				// Magnitude + 0.5: the byte over the exponent of 2^23, minus 2^23 - 0.5.
				const uint32_t w = i < 4 ? uint32_t(m) : uint32_t(m >> 32);
				const f32x2 f = f2_add_rn(f2_pack(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440 + (i & 3))),
				                                  __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7441 + (i & 3)))),
				                          f2_pack(-8388607.5f, -8388607.5f));
				f2_unpack(f, v[h][i], v[h][i + 1]);
			}
		}
		else
		{
			// More than eight planes somewhere in the row, as rows of every frame's LL
			// blocks have (9 to 12; more than sixteen only a malformed one): plane by plane.
			uint32_t dec[8] = {0, 0, 0, 0, 0, 0, 0, 0};
			for (int pl = int(planes) - 1; pl >= 0; pl--)
			{
				const uint32_t bits = rd.u8(byte++);
#pragma unroll
				for (int i = 0; i < 8; i++)
					dec[i] |= ((bits >> i) & 1u) << pl;
			}
#pragma unroll
			for (int i = 0; i < 8; i++)
			{
				sig |= dec[i] != 0 ? 1u << i : 0u;
				v[h][i] = __fadd_rn(float(dec[i]), 0.5f);
			}
		}
		sig4 |= sig << (8 * h);
#pragma unroll
		for (int i = 0; i < 8; i++)
			v[h][i] = __fmul_rn(v[h][i], scale);
	}

	// Sign bits: position = number of significant coefficients before this one
	// (in sub-block order: 8x8 rows, then the 32 sub-blocks of a row); two rows'
	// counts to a word.
	uint32_t s01 = uint32_t(__popc(sig4 & 0xffu)) | (uint32_t(__popc(sig4 & 0xff00u)) << 16),
	         s23 = uint32_t(__popc(sig4 & 0xff0000u)) | (uint32_t(__popc(sig4 & 0xff000000u)) << 16);
	const uint32_t n01 = s01, n23 = s23;
#pragma unroll
	for (int o = 1; o < 32; o *= 2)
	{
		const uint32_t a = __shfl_up_sync(full, s01, o), b = __shfl_up_sync(full, s23, o);
		if (lane >= o)
		{
			s01 += a;
			s23 += b;
		}
	}
	const uint32_t t01 = __shfl_sync(full, s01, 31), t23 = __shfl_sync(full, s23, 31);
	s01 -= n01;
	s23 -= n23;
	const uint32_t total = (t01 & 0xffffu) + (t01 >> 16) + (t23 & 0xffffu) + (t23 >> 16);
	const bool signs_staged = sign_bit + total <= 32 * rd.count;
	const BlockReader<true> checked{rd.s, rd.off, rd.count, rd.g};
#pragma unroll
	for (int h = 0; h < 4; h++)
	{
		const uint32_t sig = (sig4 >> (8 * h)) & 0xffu;
		if (((ballot >> (4 * h)) & 0xfu) != 0)
		{
			const uint32_t bit = sign_bit + (((h < 2 ? s01 : s23) >> (16 * (h & 1))) & 0xffffu);
			uint32_t signs = 0;
			if (sig != 0)
				signs = signs_staged ? __funnelshift_r(rd.s[bit >> 5], rd.s[(bit >> 5) + 1], bit & 31u)
				                     : __funnelshift_r(checked.w32(bit >> 5), checked.w32((bit >> 5) + 1), bit & 31u);
#pragma unroll
			for (int i = 0; i < 8; i++)
			{
				const bool on = (sig >> i) & 1u;
				v[h][i] = on ? __uint_as_float(__float_as_uint(v[h][i]) ^ (signs << 31)) : 0.0f;
				signs >>= on ? 1 : 0;
			}
			sign_bit += ((h < 2 ? t01 : t23) >> (16 * (h & 1))) & 0xffffu;
		}
		store_subblock(in.coef32, in.coef16, f16, at + int64_t(8 * h) * pitch, pitch, v[h]);
	}
}

// One 32x32 block per warp, four 4x2 sub-blocks per lane (8x8 rows 0..3 of
// column lane >> 3, sub-block lane & 7: the reference's mapping,
// wavelet_dequant.comp:222-238). No CTA barrier: the block's words are staged in
// the warp's shared memory, the header's prefixes are warp scans. Planes and
// signs that lie inside the staged words (every valid block's) are read without
// per-word checks; the area has room for the words just past them that a
// window may touch. Bound by instruction issue at 4K, by latency at 1080p.
// Measured against two sub-blocks per thread of a 64-thread CTA: decode of a 4K
// 4:4:4 frame (1.2 MB) 118 -> 105 us, 1080p 32.8 -> 31.9 us.
//
// The warp with `clear_error` set clears the decode's error word: every
// inverse level runs after the dequantiser has completed, so the clear precedes
// any error report.
__device__ __forceinline__ void dequant_body(DequantShared &sh, const BlockParams &p, const DecodeInput &in,
                                             const int blk, const bool clear_error)
{
	const unsigned full = 0xffffffffu;
	pdl_trigger();
	const BandEntry &B = p.band[find_band(p, blk)];
	const LevelDesc &L = p.level[B.level];
	const int rel = blk - B.block32_offset;
	const int by32 = rel / B.block32_stride, bx32 = rel - by32 * B.block32_stride;
	const bool f16 = L.fp16 != 0;
	const int lane = threadIdx.x & 31, sub = lane & 7, lx = lane >> 3;
	const int pitch = L.pitch;
	const int64_t at = B.offset + int64_t(by32 * 32 + sub_y(sub)) * pitch + bx32 * 32 + lx * 8 + sub_x(sub);
	pdl_wait();
	if (clear_error && lane == 0 && in.error)
		*in.error = 0u;
	if (clear_error && in.state && lane < int(sizeof(DecodeState) / 4))
		reinterpret_cast<uint32_t *>(in.state)[lane] = 0u;

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
		for (int h = 0; h < 4; h++)
			store_subblock(in.coef32, in.coef16, f16, at + int64_t(8 * h) * pitch, pitch, zero);
		return;
	}

	// Stage the block's words in shared memory with all loads in flight at
	// once; every read below is then a shared-memory read. With only an offset
	// table the size comes from the block header, so the first
	// kSpeculativeWords are fetched together with it.
	const PayloadReader grd{in.payload, in.payload_words};
	uint32_t *const s = sh.words;
	uint32_t staged;
	if (sized_by_header)
	{
		stage_words(s, grd, off, 0, kSpeculativeWords);
		__syncwarp();
		words = (s[0] >> 16) & 0xfffu;
		staged = min(max(words, kSpeculativeWords), uint32_t(kMaxBlockWords));
		stage_words(s, grd, off, kSpeculativeWords, staged);
	}
	else
	{
		staged = min(words, uint32_t(kMaxBlockWords));
		stage_words(s, grd, off, 0, staged);
	}
	__syncwarp();

	// Header: lane t < 16 reads 8x8 t and finds where its planes start.
	const BlockReader<true> checked{s, off, staged, grd};
	const uint32_t ballot = checked.w32(0) & 0xffffu;
	const float quant = decode_quant(checked.w32(1) & 0xffu);
	const uint32_t n = uint32_t(__popc(ballot));
	uint32_t header = 0; // code word, Q bits << 16, scale << 20
	if (lane < 16 && ((ballot >> lane) & 1u))
	{
		const uint32_t local = uint32_t(__popc(ballot & ((1u << lane) - 1u)));
		header = checked.u16(4 + local) | (checked.u8(8 + n * 2 + local) << 16);
	}
	const uint32_t cost = uint32_t(plane_code_sum(header, 0)) + ((header >> 16) & 0xfu) * 8u;
	uint32_t inc = cost;
#pragma unroll
	for (int o = 1; o < 16; o *= 2)
	{
		const uint32_t y = __shfl_up_sync(full, inc, o);
		if (lane >= o)
			inc += y;
	}
	const uint32_t base = 8 + 3 * n;
	const uint32_t plane_end = base + __shfl_sync(full, inc, 15);
	const uint32_t first_byte = base + inc - cost;
	if (plane_end <= 4 * staged)
		dequant_block(BlockReader<false>{s, off, staged, grd}, ballot, header, first_byte, 8u * plane_end, quant, in, f16, at,
		              pitch);
	else
		dequant_block(checked, ballot, header, first_byte, 8u * plane_end, quant, in, f16, at, pitch);
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

// Mirrored band indices of a window that crosses an edge: columns and rows of
// the low-pass and the high-pass bands.
template <int kRows, int kCols> struct BandTables
{
	alignas(16) int xl[kCols], xh[kCols];
	int yl[kRows], yh[kRows];
};

template <int kThreads, int kRows, int kCols>
__device__ __forceinline__ void fill_band_tables(BandTables<kRows, kCols> &t, const LevelDesc &L, const int x0, const int y0)
{
	for (int k = threadIdx.x; k < 2 * (kCols + kRows); k += kThreads)
	{
		if (k < kCols)
			t.xl[k] = inv_index_low(x0 + k, L.width);
		else if (k < 2 * kCols)
			t.xh[k - kCols] = inv_index_high(x0 + k - kCols, L.width);
		else if (k < 2 * kCols + kRows)
			t.yl[k - 2 * kCols] = inv_index_low(y0 + k - 2 * kCols, L.height);
		else
			t.yh[k - 2 * kCols - kRows] = inv_index_high(y0 + k - 2 * kCols - kRows, L.height);
	}
}

// Rows [y0, y0 + kRows) and columns [x0, x0 + kCols) (x0 a multiple of 4) of
// bands kFirst..3 of a level into dst[band][row][column], rows of kCols samples.
// A thread keeps one group of four columns: its mirrored indices are read once,
// and every load of its rows is in flight at once.
template <int kThreads, int kFirst, int kRows, int kCols, bool kHalf>
__device__ __forceinline__ void load_bands(float *dst, const BandTables<kRows, kCols> &t, const LevelDesc &L,
                                           const BandParam (&band)[4], const DecodeInput &in, const int x0, const int y0)
{
	constexpr int kVecPerRow = kCols / 4, kBands = 4 - kFirst;
	constexpr int kLoadRows = kThreads / kVecPerRow;
	constexpr int kIters = (kBands * kRows + kLoadRows - 1) / kLoadRows;
	const bool f16 = kHalf && L.fp16 != 0, stage16 = kHalf && L.stage16 != 0;
	const bool y_inside = y0 >= 0 && y0 + kRows <= L.height;
	const int j = threadIdx.x % kVecPerRow, br0 = threadIdx.x / kVecPerRow;
	const bool loader = threadIdx.x < kLoadRows * kVecPerRow;
	const int x = x0 + 4 * j;
	const bool inside = x >= 0 && x + 4 <= L.width;
	int4 lo = make_int4(x, x + 1, x + 2, x + 3), hi = lo;
	if (!inside)
	{
		lo = *reinterpret_cast<const int4 *>(&t.xl[4 * j]);
		hi = *reinterpret_cast<const int4 *>(&t.xh[4 * j]);
	}
	float4 v[kIters];
#pragma unroll
	for (int u = 0; u < kIters; u++)
	{
		const int br = br0 + u * kLoadRows;
		v[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
		if (!loader || br >= kBands * kRows)
			continue;
		const int b = kFirst + br / kRows, i = br % kRows;
		const int yy = y_inside ? y0 + i : ((b >> 1) ? t.yh[i] : t.yl[i]);
		const int64_t row = band[b].offset + int64_t(yy) * L.pitch;
		if (!inside)
		{
			const int4 xi = (b & 1) ? hi : lo;
			v[u] = make_float4(load_coef(in.coef32, in.coef16, f16, row + xi.x), load_coef(in.coef32, in.coef16, f16, row + xi.y),
			                   load_coef(in.coef32, in.coef16, f16, row + xi.z), load_coef(in.coef32, in.coef16, f16, row + xi.w));
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
		if (!loader || br >= kBands * kRows)
			continue;
		float4 f = v[u];
		if (stage16)
		{
			f.x = round_to_half(f.x);
			f.y = round_to_half(f.y);
			f.z = round_to_half(f.z);
			f.w = round_to_half(f.w);
		}
		*reinterpret_cast<float4 *>(dst + ((kFirst + br / kRows) * kRows + br % kRows) * kCols + 4 * j) = f;
	}
}

template <int kOutRows> struct IdwtSharedT
{
	BandTables<kOutRows / 2 + 4, kBandRow> tables; // edge tiles
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

// Both lifting passes of a loaded tile or stripe, and the store of planes or of
// the finer level's LL.
template <int kThreads, int kStripes, bool kHalf>
__device__ __forceinline__ void idwt_lift_store(IdwtSharedT<IdwtSplit<kThreads, kStripes>::kOutRows> &sh,
                                                const LevelParams &p, const DecodeInput &in, const PlaneOutput &out,
                                                const int comp, const int tx, const int ty, const int tile,
                                                const int stripe)
{
	using Split = IdwtSplit<kThreads, kStripes>;
	constexpr int kOut = Split::kOut, kWin = kOut + 8;
	const bool stage16 = kHalf && p.L.stage16 != 0;
	const bool final_level = p.level == 0 || (p.level == 1 && comp != 0 && !p.chroma444);

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
				if (stage16)
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
		// Neighbouring lanes take neighbouring segments of a row: their stores fill
		// whole sectors (with a row to each lane, every store touched half of one:
		// 4K 4:4:4 decode 105 -> 97 us, 1080p 32.6 -> 29.1), and their loads still meet no bank conflict.
		const int seg = item % (64 / kOut), pr = item / (64 / kOut);
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
		if (stage16)
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
			const bool pf16 = kHalf && P.fp16 != 0;
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
				else if constexpr (kOut >= 8)
				{
#pragma unroll
					for (int k = 0; k < kOut; k += 8)
						store_f32x8(in.coef32 + base + k, r[h][k], r[h][k + 1], r[h][k + 2], r[h][k + 3], r[h][k + 4],
						            r[h][k + 5], r[h][k + 6], r[h][k + 7]);
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
//
// kHalf: the level, or the finer one it writes, is stored in FP16, or lifting is
// staged through it; the all-FP32 form carries none of that code.
template <int kThreads, int kStripes, bool kHalf>
__device__ __forceinline__ void idwt_body(IdwtSharedT<IdwtSplit<kThreads, kStripes>::kOutRows> &sh, const LevelParams &p,
                                          const DecodeInput &in, const PlaneOutput &out, const LevelTileMap *maps,
                                          const int tile, const int comp_index, const int stripe = 0)
{
	using Split = IdwtSplit<kThreads, kStripes>;
	constexpr int kRows = Split::kBandRows;
	pdl_trigger();
	const int level = p.level;
	const int comp = (level == 0 && !p.chroma444) ? 0 : comp_index;
	const LevelDesc &L = p.L;
	const int tx = tile % L.tiles_x, ty = tile / L.tiles_x;
	const int nx = L.width, ny = L.height;
	const bool f16 = kHalf && L.fp16 != 0, stage16 = kHalf && L.stage16 != 0;

	// Interior tiles read every band sample at its own position. Interior FP32
	// tiles of a decoder with tensor maps take one TMA box per band (barrier and
	// maps made ready before the dependency wait); the others load vectors of
	// four samples, gathered through the mirrored index tables where they cross
	// an edge.
	const int x0 = tx * 32 - 4, y0 = ty * 32 - 2 + stripe * (Split::kOutRows / 2); // column 0, row 0 of the band tiles
	const bool y_inside = y0 >= 0 && y0 + kRows <= ny;
	const bool interior = x0 >= 0 && x0 + kBandRow <= nx && y_inside;
	const bool use_tma = kThreads == 256 && kStripes == 1 && interior && maps && ((maps->valid >> comp) & 1u) && !f16 &&
	                     !stage16;
	if (!interior)
	{
		fill_band_tables<kThreads>(sh.tables, L, x0, y0);
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
		load_bands<kThreads, 0, kRows, kBandRow, kHalf>(&sh.band[0][0][0], sh.tables, L, p.band[comp], in, x0, y0);
	}
	__syncthreads();
	idwt_lift_store<kThreads, kStripes, kHalf>(sh, p, in, out, comp, tx, ty, tile, stripe);
}

// Two small inverse levels in one launch: a stripe of 16 output rows of a tile
// of level `p`, whose LL input (12 rows x 40 columns) the CTA computes itself
// from level `c`, the next coarser one, instead of reading what a launch of that
// level stored: 10 x 24 samples of its four bands, lifted as that level lifts
// them, so with the same results. Neighbouring stripes repeat some of that work,
// a third of what a stripe does anyway; a launch costs about 3 us of launch,
// dependency and memory latency whatever it computes. Measured against
// a launch per level: encode + decode of 256x144 43.4 -> 40.6 us, decode of a 1080p
// 4:2:0 frame 29.6 -> 28.0 us, 4K 4:4:4 96.6 -> 93.8 us.
constexpr int kPairRows = 12, kPairBandRows = kPairRows / 2 + 4, kPairBandCols = kBandRow / 2 + 4;
struct IdwtPairShared
{
	IdwtSharedT<16> fine;
	BandTables<kPairBandRows, kPairBandCols> tables;
	alignas(16) float band[4][kPairBandRows][kPairBandCols];
	alignas(16) float v[2][kPairRows][kPairBandCols];
	alignas(16) float ll[kPairRows][kBandRow]; // the LL window, where the fine level mirrors it
};

template <bool kHalf>
__device__ __forceinline__ void idwt_pair_body(IdwtPairShared &sh, const LevelParams &p, const LevelParams &c,
                                               const DecodeInput &in, const PlaneOutput &out, const int tile,
                                               const int comp, const int stripe)
{
	constexpr int kThreads = 256, kStripes = 4, kOut = 4, kWin = kOut + 8;
	static_assert(IdwtSplit<kThreads, kStripes>::kBandRows == kPairRows, "the LL window of a stripe");
	pdl_trigger();
	const LevelDesc &L = p.L;
	const int ty = tile / L.tiles_x, tx = tile - ty * L.tiles_x;
	const int x0 = tx * 32 - 4, y0 = ty * 32 - 2 + stripe * 8; // the LL window, both even
	const int cx0 = x0 / 2 - 2, cy0 = (y0 - 4) >> 1;           // and the window of the coarser bands under it
	const bool interior = x0 >= 0 && x0 + kBandRow <= L.width && y0 >= 0 && y0 + kPairRows <= L.height;
	const bool stage16 = kHalf && L.stage16 != 0;
	if (!interior)
		fill_band_tables<kThreads>(sh.fine.tables, L, x0, y0);
	fill_band_tables<kThreads>(sh.tables, c.L, cx0, cy0);
	__syncthreads();
	pdl_wait();
	load_bands<kThreads, 0, kPairBandRows, kPairBandCols, kHalf>(&sh.band[0][0][0], sh.tables, c.L, c.band[comp], in, cx0, cy0);
	load_bands<kThreads, 1, kPairRows, kBandRow, kHalf>(&sh.fine.band[0][0][0], sh.fine.tables, L, p.band[comp], in, x0, y0);
	__syncthreads();

	// The coarser level: vertical, then horizontal lifting, four outputs per item.
	for (int item = threadIdx.x; item < (kPairBandCols / 2) * 2 * (kPairRows / kOut); item += kThreads)
	{
		const int pair = item % (kPairBandCols / 2), which = (item / (kPairBandCols / 2)) & 1, seg = item / kPairBandCols;
		f32x2 e[kWin];
#pragma unroll
		for (int jj = 0; jj < kWin; jj += 2)
		{
			const int i = (seg * kOut + jj) >> 1;
			const float2 a = *reinterpret_cast<const float2 *>(&sh.band[which][i][2 * pair]);
			const float2 b = *reinterpret_cast<const float2 *>(&sh.band[which + 2][i][2 * pair]);
			e[jj] = f2_pack(__fmul_rn(a.x, kK), __fmul_rn(a.y, kK));
			e[jj + 1] = f2_pack(__fmul_rn(b.x, kInvK), __fmul_rn(b.y, kInvK));
		}
		lift_inverse2(e);
#pragma unroll
		for (int jj = 4; jj < 4 + kOut; jj++)
		{
			float a, b;
			f2_unpack(e[jj], a, b);
			if (stage16)
			{
				a = round_to_half(a);
				b = round_to_half(b);
			}
			*reinterpret_cast<float2 *>(&sh.v[which][seg * kOut + jj - 4][2 * pair]) = make_float2(a, b);
		}
	}
	__syncthreads();
	float(*const ll)[kBandRow] = interior ? sh.fine.band[0] : sh.ll;
	for (int item = threadIdx.x; item < (kPairRows / 2) * (kBandRow / kOut); item += kThreads)
	{
		const int seg = item % (kBandRow / kOut), pr = item / (kBandRow / kOut); // rows pr and pr + 6
		f32x2 e[kWin];
#pragma unroll
		for (int jj = 0; jj < kWin; jj += 2)
		{
			const int i = (seg * kOut + jj) >> 1;
			e[jj] = f2_pack(__fmul_rn(sh.v[0][pr][i], kK), __fmul_rn(sh.v[0][pr + kPairRows / 2][i], kK));
			e[jj + 1] = f2_pack(__fmul_rn(sh.v[1][pr][i], kInvK), __fmul_rn(sh.v[1][pr + kPairRows / 2][i], kInvK));
		}
		lift_inverse2(e);
#pragma unroll
		for (int k = 0; k < kOut; k++)
		{
			float a, b;
			f2_unpack(e[4 + k], a, b);
			if (stage16 || (kHalf && L.fp16))
			{
				a = round_to_half(a); // as stored in the fine level's LL, or staged from it
				b = round_to_half(b);
			}
			ll[pr][seg * kOut + k] = a;
			ll[pr + kPairRows / 2][seg * kOut + k] = b;
		}
	}
	__syncthreads();
	if (!interior)
	{
		// Mirrored samples; those beyond what any stored output reads are clamped to the window.
		for (int k = threadIdx.x; k < kPairRows * kBandRow; k += kThreads)
		{
			const int i = k / kBandRow, j = k - i * kBandRow;
			const int r = min(max(sh.fine.tables.yl[i] - y0, 0), kPairRows - 1);
			sh.fine.band[0][i][j] = sh.ll[r][min(max(sh.fine.tables.xl[j] - x0, 0), kBandRow - 1)];
		}
		__syncthreads();
	}
	idwt_lift_store<kThreads, kStripes, kHalf>(sh.fine, p, in, out, comp, tx, ty, tile, stripe);
}

} // namespace
} // namespace pw
