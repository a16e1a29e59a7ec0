// Device-side packet assembly for the decoder: the packets of a frame, as
// received into device memory, are parsed and turned into the per-block
// table the dequantiser reads, with the sequence and first-copy rules of the
// reference's host parser (pyrowave_decoder.cpp:154-262, as restated by the
// host parser in pw_host.cpp), so nothing of the frame passes through the host.
//
// The parser's state is the sequence of the frame being assembled (none or
// 0..7). Pushing one packet maps a state to a state, so the state before every
// packet follows from a scan of the packets' state maps:
//   1. packet_tables_kernel  one CTA per packet: the packet's items are found
//      (below) and the packet is evaluated from each of the 9 possible states:
//      the state after it, the last restart (the reference's clear()) inside
//      it, the block total of the last accepted sequence header, and whether
//      the parser rejects it. The last CTA to finish scans the state maps of
//      all packets: the state before each packet, the last restart of the
//      whole list, the frame's sequence and block total. Meanwhile every CTA
//      clears its share of the first-copy table.
//   2. packet_blocks_kernel  one CTA per packet from the last restart on:
//      every block the parser keeps proposes (packet, item, word offset) and
//      the smallest, the first copy pushed, wins by a 64-bit atomicMin; the
//      winners are counted. The dequantiser reads the winning keys directly.
#include "pw_device.cuh"

namespace pw
{
namespace
{
constexpr uint32_t kNoneState = 0;          // states: 0 = no sequence yet, 1 + s = sequence s
constexpr uint32_t kNoPos = 0xffffu;        // no restart inside the packet
constexpr uint32_t kNoTotal = 0xffffffffu;  // no sequence header accepted
constexpr uint32_t kMaxItems = 1u << 14;    // items (headers + blocks) per packet
constexpr unsigned long long kNoKey = ~0ull;
constexpr uint32_t kNoBlock = 0xffffffffu;  // listed item is a sequence header

struct WalkResult
{
	uint32_t state;
	uint32_t restart; // item index of the last restart, kNoPos if none
	uint32_t total;   // blocks announced by the last header after the last restart
	bool error;       // the host parser returns false for this packet
};

// One pass of the host parser over one packet (push_packet). `word(i)` reads
// word i of the packet; `size` is the packet's size in bytes. on_block(block,
// word position, item index) is called for every block the parser keeps.
template <typename R, typename F>
__device__ WalkResult walk_packet(R word, uint32_t size, uint32_t state, const PacketParams &pp, F on_block)
{
	WalkResult res{state, kNoPos, kNoTotal, false};
	uint32_t pos = 0; // in words
	for (uint32_t item = 0; size >= 8; item++)
	{
		if (item >= kMaxItems)
		{
			res.error = true;
			return res;
		}
		const uint32_t w0 = word(pos), w1 = word(pos + 1);
		const uint32_t seq = (w0 >> 28) & 7u;
		const bool fresh = res.state == kNoneState;
		const uint32_t diff = fresh ? 0u : ((seq - (res.state - 1)) & 7u);
		if ((w0 >> 31) & 1u)
		{
			// Start-of-frame sequence header (bitstream.md:250-265).
			if (((w1 >> 26) & 1u) != uint32_t(pp.chroma444))
			{
				res.error = true;
				return res;
			}
			if (!fresh && diff > 3)
				return res; // an older sequence: the rest of the packet is ignored
			if (fresh || diff != 0)
			{
				res.state = 1 + seq;
				res.restart = item;
				res.total = kNoTotal;
			}
			if (((w1 >> 24) & 3u) != 0 || int(w0 & 0x3fffu) + 1 != pp.width ||
			    int((w0 >> 14) & 0x3fffu) + 1 != pp.height)
			{
				res.error = true;
				return res;
			}
			res.total = w1 & 0xffffffu;
			pos += 2;
			size -= 8;
			continue;
		}
		const uint32_t words = (w0 >> 16) & 0xfffu;
		if (words * 4u > size)
		{
			res.error = true;
			return res;
		}
		if (!fresh && diff > 3)
			return res;
		if (fresh || diff != 0)
		{
			res.state = 1 + seq;
			res.restart = item;
			res.total = kNoTotal;
		}
		const uint32_t block = (w1 >> 8) & 0xffffffu;
		// A block shorter than its own header makes the packet invalid; it is
		// left missing.
		if (block >= uint32_t(pp.block_count) || words < 2)
		{
			res.error = true;
			return res;
		}
		on_block(block, pos, item);
		pos += words;
		size -= words * 4u;
	}
	res.error = res.error || size != 0;
	return res;
}

// The packet's bytes, or why it cannot be read as words.
__device__ __forceinline__ bool packet_span(const PacketParams &pp, int p, uint32_t &first_word, uint32_t &size)
{
	const unsigned long long off = pp.packets[2 * p], sz = pp.packets[2 * p + 1];
	if ((off & 3u) != 0 || off > pp.data_bytes || sz > pp.data_bytes - off || sz > 0xffffffffull)
		return false;
	first_word = uint32_t(off >> 2);
	size = uint32_t(sz);
	return true;
}

// ---------------------------------------------------------------------------
// Item discovery. A packet is a chain of items (sequence headers of 2 words,
// blocks of their announced word count): item k + 1 starts where item k ends.
// Every word position p gets next(p) in parallel: the position after an item
// starting at p, or where the parser stops (an item it rejects, the end, fewer
// than 8 bytes left). Three doubling passes give next^8; one thread follows it
// from 0 (one shared-memory load per 8 items), and one thread per item lists
// and summarises it (next^1, ^2 and ^4 lead there from its anchor). Packets
// whose items share one sequence number (every packet of a frame) need no walk
// at all: the parser's state change has a closed form. Other packets are walked
// item by item.
//
// Bound by latency: a chain of memory round trips, barriers of the CTA and the
// chase, with one CTA per packet. So words are classified straight from the
// loads, the summary is taken while listing, and 16-bit positions leave room
// for two CTAs per SM: 43.8 -> 42.7 us for a 1080p 4:2:0 frame in 51 packets of
// 8 KiB with its decode, 40.2 -> 39.5 with one thread per item instead of one
// per anchor that followed eight links (the graph with the decode lies between).
constexpr int kFastWords = 8192;  // packets up to 32 KiB take this path
// Codes of next(p) that are not positions.
constexpr uint32_t kLeft = 0xfffdu; // fewer than 8 bytes left: not an item
constexpr uint32_t kStop = 0xfffeu; // the parser rejects the item
constexpr uint32_t kDone = 0xffffu; // the item ends the packet exactly
constexpr int kPacketThreads = 1024;
constexpr int kAnchorRounds = 3; // the chase follows next^8
constexpr int kAnchorStep = 1 << kAnchorRounds;

struct PacketSmem
{
	uint32_t words[kFastWords];
	uint16_t next[kAnchorRounds + 1][kFastWords];         // next^(2^r), a code (>= kLeft) where the chain stops first
	uint16_t anchors[kFastWords / (2 * kAnchorStep) + 2]; // every kAnchorStep-th item
};
constexpr size_t kPacketSmemBytes = sizeof(PacketSmem);

struct ItemSummary // also the per-packet record in PacketParams::summaries (8 words)
{
	uint32_t nitems;
	uint32_t error;         // first rejected item << 2 | kind (1: before the sequence check, 2: after it); ~0u: none
	uint32_t trailing;      // 1: bytes left over after the last item (the parser's size != 0)
	uint32_t seq_min, seq_max;
	uint32_t fast;                  // 1: the items were listed (the packet fits kFastWords)
	unsigned long long last_header; // (item + 1) << 32 | announced blocks, of the last accepted header; 0: none
};
static_assert(sizeof(ItemSummary) == 32, "per-packet record");

// Classification of an item starting at word p (rem >= 8 bytes left).
struct ItemInfo
{
	bool header;
	uint32_t seq, words, block, total;
	uint32_t error; // 0, 1 (before the sequence check), 2 (after it)
};

__device__ __forceinline__ ItemInfo classify(uint32_t w0, uint32_t w1, uint32_t rem, const PacketParams &pp)
{
	ItemInfo it;
	it.header = (w0 >> 31) & 1u;
	it.seq = (w0 >> 28) & 7u;
	it.total = w1 & 0xffffffu;
	it.block = (w1 >> 8) & 0xffffffu;
	it.error = 0;
	if (it.header)
	{
		it.words = 2;
		if (((w1 >> 26) & 1u) != uint32_t(pp.chroma444))
			it.error = 1;
		else if (((w1 >> 24) & 3u) != 0 || int(w0 & 0x3fffu) + 1 != pp.width || int((w0 >> 14) & 0x3fffu) + 1 != pp.height)
			it.error = 2;
	}
	else
	{
		it.words = (w0 >> 16) & 0xfffu;
		if (it.words * 4u > rem)
			it.error = 1;
		else if (it.block >= uint32_t(pp.block_count) || it.words < 2)
			it.error = 2;
	}
	return it;
}

// A listed item in one word, so that its parts stay together: its position, its
// number in the packet and its block. Packets whose byte ranges overlap share
// slots of the list; a slot that holds another number than its reader's was
// stored for a packet that starts elsewhere (with the same number, for one that
// starts at the same word, where the items are the same).
__device__ __forceinline__ unsigned long long item_record(uint32_t pos, uint32_t k, uint32_t block)
{
	return (unsigned long long)block << 32 | (k << 16 | pos);
}
static_assert(kFastWords <= 0x10000, "positions and item numbers in 16 bits");

// Stages the packet (nwords <= kFastWords), lists its items in pp.items and
// fills the item summary. Every thread of the CTA calls it.
__device__ void discover_items(PacketSmem &sm, ItemSummary &sum, const PacketParams &pp, uint32_t first,
                               uint32_t size, uint32_t nwords)
{
	const int t = threadIdx.x;
	constexpr int kLoads = 4; // words in flight per thread, each with its successor
	for (uint32_t base = t; base < nwords; base += kLoads * kPacketThreads)
	{
		uint32_t w0[kLoads], w1[kLoads];
#pragma unroll
		for (int u = 0; u < kLoads; u++)
		{
			const uint32_t p = base + u * kPacketThreads;
			w0[u] = p < nwords ? __ldg(pp.data + first + p) : 0u;
			w1[u] = p + 1 < nwords ? __ldg(pp.data + first + p + 1) : 0u;
		}
#pragma unroll
		for (int u = 0; u < kLoads; u++)
		{
			const uint32_t p = base + u * kPacketThreads;
			if (p >= nwords)
				break;
			sm.words[p] = w0[u];
			const uint32_t rem = size - 4 * p;
			uint32_t nxt = kLeft;
			if (rem >= 8)
			{
				const ItemInfo it = classify(w0[u], w1[u], rem, pp);
				nxt = it.error ? kStop : (p + it.words < nwords ? p + it.words : kDone);
			}
			sm.next[0][p] = uint16_t(nxt);
		}
	}
	if (t == 0)
	{
		sum.nitems = 0;
		sum.error = ~0u;
		sum.trailing = 0;
		sum.seq_min = 7;
		sum.seq_max = 0;
		sum.last_header = 0;
	}
	__syncthreads();
#pragma unroll
	for (int r = 0; r < kAnchorRounds; r++)
	{
		for (uint32_t p = t; p < nwords; p += kPacketThreads)
		{
			const uint32_t j = sm.next[r][p];
			sm.next[r + 1][p] = j >= kLeft ? uint16_t(j) : sm.next[r][j];
		}
		__syncthreads();
	}
	__shared__ uint32_t s_anchors;
	if (t == 0)
	{
		uint32_t m = 0, p = 0;
		while (nwords > 0)
		{
			sm.anchors[m++] = uint16_t(p);
			p = sm.next[kAnchorRounds][p];
			if (p >= kLeft)
				break;
		}
		s_anchors = m;
	}
	__syncthreads();
	// Item k is k % 8 steps after its anchor. The sequence range covers the
	// items whose sequence number the parser looks at. Only the last item can be
	// rejected.
	const uint32_t slots = s_anchors * kAnchorStep;
	uint32_t smin = 7, smax = 0;
	for (uint32_t k = t; k < slots; k += kPacketThreads)
	{
		uint32_t q = sm.anchors[k / kAnchorStep];
#pragma unroll
		for (int r = 0; r < kAnchorRounds; r++)
			if ((k >> r & 1u) && q < kLeft)
				q = sm.next[r][q];
		if (q >= kLeft)
			continue; // the chain stops before
		const uint32_t nx = sm.next[0][q];
		if (nx == kLeft)
		{
			sum.trailing = 1; // q is not an item: fewer than 8 bytes were left
			sum.nitems = k;
			continue;
		}
		const ItemInfo it = classify(sm.words[q], sm.words[q + 1], size - 4 * q, pp);
		pp.items[first + k] = item_record(q, k, it.header ? kNoBlock : it.block);
		if (it.error)
			sum.error = k << 2 | it.error;
		else if (it.header)
			atomicMax(&sum.last_header, (unsigned long long)(k + 1) << 32 | it.total);
		if (it.error != 1)
		{
			smin = min(smin, it.seq);
			smax = max(smax, it.seq);
		}
		if (nx >= kLeft)
			sum.nitems = k + 1;
	}
	if (uint32_t(t & ~31) < slots) // uniform over the warp
	{
		smin = __reduce_min_sync(0xffffffffu, smin);
		smax = __reduce_max_sync(0xffffffffu, smax);
		if ((t & 31) == 0 && smin <= smax)
		{
			atomicMin(&sum.seq_min, smin);
			atomicMax(&sum.seq_max, smax);
		}
	}
	__syncthreads();
}

// The parser's pass over a packet whose items share one sequence number, in
// closed form (see walk_packet for the item-by-item rules).
__device__ __forceinline__ WalkResult uniform_walk(const ItemSummary &sum, uint32_t state, bool &accepts_blocks)
{
	WalkResult r{state, kNoPos, kNoTotal, false};
	accepts_blocks = false;
	const uint32_t err_item = sum.error == ~0u ? ~0u : sum.error >> 2;
	const uint32_t err_kind = sum.error == ~0u ? 0u : sum.error & 3u;
	if (sum.nitems == 0)
	{
		r.error = sum.trailing != 0;
		return r;
	}
	if (err_item == 0 && err_kind == 1)
	{
		r.error = true; // rejected before its sequence number is looked at
		return r;
	}
	const uint32_t s = sum.seq_min;
	const bool fresh = state == kNoneState;
	const uint32_t diff = fresh ? 0u : ((s - (state - 1)) & 7u);
	if (!fresh && diff > 3)
		return r; // an older sequence: the packet is ignored
	if (fresh || diff != 0)
	{
		r.state = 1 + s;
		r.restart = 0;
	}
	if (sum.last_header)
		r.total = uint32_t(sum.last_header & 0xffffffffull);
	r.error = err_item != ~0u || sum.trailing != 0;
	accepts_blocks = true;
	return r;
}

// State maps as 9 nibbles: nibble x = state after the packet(s) from state x.
__device__ __forceinline__ uint32_t map_at(unsigned long long m, uint32_t x)
{
	return x < 8 ? (uint32_t(m) >> (4 * x)) & 0xfu : uint32_t(m >> 32) & 0xfu;
}

__device__ __forceinline__ unsigned long long compose(unsigned long long a, unsigned long long b)
{
	// a first, then b
	uint32_t lo = 0;
#pragma unroll
	for (int x = 0; x < 8; x++)
		lo |= map_at(b, map_at(a, x)) << (4 * x);
	return (unsigned long long)map_at(b, map_at(a, 8)) << 32 | lo;
}

constexpr unsigned long long kIdentityMap = 0x876543210ull; // nibble x = x

__device__ __forceinline__ unsigned long long packet_map(const PacketParams &pp, int p)
{
	unsigned long long m = 0;
	for (int x = 0; x < 9; x++)
		m |= (unsigned long long)(__ldcg(pp.tables + (size_t(p) * 9 + x) * 2) & 0xfu) << (4 * x);
	return m;
}

// Run by the last CTA of the table pass (1024 threads), once every packet's
// table is written.
__device__ void scan_packets(const PacketParams &pp)
{
	__shared__ unsigned long long s_warp[32];
	__shared__ unsigned long long s_last_restart, s_last_total;
	__shared__ uint32_t s_invalid;
	const int t = threadIdx.x, n = pp.count, lane = t & 31, warp = t >> 5;
	const int per = (n + 1023) / 1024;
	const int p0 = min(t * per, n), p1 = min(p0 + per, n);
	if (t == 0)
	{
		s_last_restart = 0;
		s_last_total = 0;
		s_invalid = 0;
	}
	// This thread's packets composed.
	const bool active = warp * 32 * per < n; // uniform over the warp
	const int warps = (n + 32 * per - 1) / (32 * per);
	unsigned long long incl = kIdentityMap;
	for (int p = p0; p < p1; p++)
		incl = compose(incl, packet_map(pp, p));
	// The packets of one frame have one map, which changes nothing the second
	// time: no scan (1080p in 51 packets: 40.5 -> 40.1 us with the decode).
	const unsigned long long one = packet_map(pp, 0);
	const bool alike = __syncthreads_and(per == 1 && (t >= n || incl == one) && compose(one, one) == one);
	unsigned long long before = t == 0 ? kIdentityMap : one, all = one;
	if (!alike)
	{
		// A scan over threads: within each warp by shuffles, then over the warp
		// totals. Warps past the last packet hold the identity.
		if (active)
		{
#pragma unroll
			for (int off = 1; off < 32; off *= 2)
			{
				const unsigned long long other = __shfl_up_sync(0xffffffffu, incl, off);
				if (lane >= off)
					incl = compose(other, incl);
			}
		}
		if (lane == 31)
			s_warp[warp] = incl;
		__syncthreads();
		if (warp == 0)
		{
			unsigned long long w = s_warp[lane];
			for (int off = 1; off < warps; off *= 2)
			{
				const unsigned long long other = __shfl_up_sync(0xffffffffu, w, off);
				if (lane >= off)
					w = compose(other, w);
			}
			s_warp[lane] = w; // inclusive over the active warps
		}
		__syncthreads();
		unsigned long long excl = active ? __shfl_up_sync(0xffffffffu, incl, 1) : kIdentityMap;
		if (lane == 0)
			excl = kIdentityMap;
		before = compose(warp == 0 ? kIdentityMap : s_warp[warp - 1], excl);
		all = s_warp[warps - 1];
	}
	// State before each of this thread's packets (the maps applied to "no
	// sequence"); the last restart and the last accepted header (ordered by
	// packet, then item: 1 + packet << 16 | item).
	uint32_t state = map_at(before, kNoneState);
	unsigned long long last_restart = 0, last_total = 0;
	uint32_t invalid = 0;
	for (int p = p0; p < p1; p++)
	{
		pp.state_before[p] = uint8_t(state);
		const uint32_t a = __ldcg(pp.tables + (size_t(p) * 9 + state) * 2);
		const uint32_t total = __ldcg(pp.tables + (size_t(p) * 9 + state) * 2 + 1);
		const uint32_t restart = a >> 8;
		if (restart != kNoPos)
			last_restart = 1ull + ((unsigned long long)p << 16 | restart);
		if (total != kNoTotal)
			last_total = 1ull + ((unsigned long long)p << 32 | total);
		invalid += (a >> 4) & 1u;
		state = a & 0xfu;
	}
	if (last_restart)
		atomicMax(&s_last_restart, last_restart);
	if (last_total)
		atomicMax(&s_last_total, last_total);
	if (invalid)
		atomicAdd(&s_invalid, invalid);
	__syncthreads();
	if (t == 0)
	{
		PacketStatus st = {};
		const uint32_t final_state = map_at(all, kNoneState);
		st.sequence = final_state == kNoneState ? 0xffffffffu : final_state - 1;
		st.invalid_packets = s_invalid;
		const unsigned long long lr = s_last_restart;
		st.restart_packet = lr ? uint32_t((lr - 1) >> 16) : 0u;
		st.restart_item = lr ? uint32_t((lr - 1) & 0xffffu) : 0u;
		// The block total: the last header at or after the last restart, else
		// the frame's block count (clear() in the reference parser).
		const unsigned long long lt = s_last_total;
		const uint32_t total_packet = lt ? uint32_t((lt - 1) >> 32) : 0u;
		st.total_blocks = (lt && lr && total_packet >= st.restart_packet) ? uint32_t((lt - 1) & 0xffffffffu)
		                                                                  : uint32_t(pp.block_count);
		st.decoded_blocks = 0;
		*pp.status = st;
	}
}

__global__ void __launch_bounds__(kPacketThreads, 2) packet_tables_kernel(const PacketParams pp)
{
	extern __shared__ __align__(16) unsigned char s_raw[];
	PacketSmem &sm = *reinterpret_cast<PacketSmem *>(s_raw);
	__shared__ ItemSummary sum;
	const int p = blockIdx.x;
	uint32_t first = 0, size = 0;
	const bool ok = packet_span(pp, p, first, size);
	const uint32_t nwords = (size + 3) / 4;
	const bool fast = ok && nwords <= uint32_t(kFastWords);
	pdl_trigger(); // the block pass may launch meanwhile
	for (int b = p * kPacketThreads + int(threadIdx.x); b < pp.block_count; b += pp.count * kPacketThreads)
		pp.first[b] = kNoKey;
	if (fast)
		discover_items(sm, sum, pp, first, size, nwords);
	if (threadIdx.x == 0)
	{
		ItemSummary rec = fast ? sum : ItemSummary{};
		rec.fast = fast ? 1u : 0u;
		reinterpret_cast<ItemSummary *>(pp.summaries)[p] = rec;
	}
	if (threadIdx.x < 9)
	{
		const uint32_t init = threadIdx.x;
		WalkResult r;
		bool acc;
		if (!ok)
			r = WalkResult{init, kNoPos, kNoTotal, true};
		else if (fast && sum.seq_min == sum.seq_max)
			r = uniform_walk(sum, init, acc);
		else if (fast)
			r = walk_packet([&](uint32_t i) { return i < nwords ? sm.words[i] : 0u; }, size, init, pp,
			                [](uint32_t, uint32_t, uint32_t) {});
		else
			r = walk_packet([&](uint32_t i) { return i < nwords ? __ldg(pp.data + first + i) : 0u; }, size, init, pp,
			                [](uint32_t, uint32_t, uint32_t) {});
		pp.tables[(size_t(p) * 9 + init) * 2 + 0] = r.state | (r.error ? 16u : 0u) | (r.restart << 8);
		pp.tables[(size_t(p) * 9 + init) * 2 + 1] = r.total;
	}
	// The last CTA to finish scans every packet's table (no CTA waits for
	// another). The tables are the first warp's stores, so its first thread's
	// release covers them; the rest is for the next kernel.
	__shared__ uint32_t s_ticket;
	if (threadIdx.x < 32)
	{
		__syncwarp();
		if (threadIdx.x == 0)
			s_ticket = atom_acq_rel_add(pp.counter, 1u);
	}
	__syncthreads();
	if (s_ticket != uint32_t(pp.count) - 1)
		return;
	if (threadIdx.x == 0)
		*pp.counter = 0; // ready for the next call
	scan_packets(pp);
}

__global__ void __launch_bounds__(256) packet_blocks_kernel(const PacketParams pp)
{
	const int p = blockIdx.x;
	uint32_t first = 0, size = 0;
	const bool ok = packet_span(pp, p, first, size);
	const uint32_t nwords = (size + 3) / 4;
	pdl_trigger(); // the dequantiser may launch meanwhile
	pdl_wait();
	// One round trip: the state, the summary and the thread's first item (which
	// need not exist, but its place does) are read before they are known to count.
	const uint32_t rp = __ldcg(&pp.status->restart_packet), ri = __ldcg(&pp.status->restart_item);
	const uint32_t seq = __ldcg(&pp.status->sequence);
	const uint32_t state = pp.state_before[p];
	const ItemSummary sum = reinterpret_cast<const ItemSummary *>(pp.summaries)[p];
	unsigned long long rec = 0;
	if (ok && threadIdx.x < nwords)
		rec = __ldcg(pp.items + first + threadIdx.x);
	if (!ok || seq == 0xffffffffu || uint32_t(p) < rp)
		return; // uniform over the CTA
	uint32_t fresh = 0; // blocks this thread saw first
	auto keep = [&](uint32_t b, uint32_t word, uint32_t item) {
		if (uint32_t(p) == rp && item < ri)
			return; // before the last restart: cleared
		const unsigned long long key = (unsigned long long)p << 44 | (unsigned long long)item << 30 | (first + word);
		if (atomicMin(pp.first + b, key) == kNoKey)
			fresh++;
	};
	bool walk = true;
	if (sum.fast && sum.seq_min == sum.seq_max)
	{
		bool accepts;
		(void)uniform_walk(sum, state, accepts);
		const uint32_t err_item = sum.error == ~0u ? ~0u : sum.error >> 2;
		const uint32_t n = accepts ? min(sum.nitems, err_item) : 0u;
		bool lost = false;
		for (uint32_t k = threadIdx.x; k < n; k += blockDim.x)
		{
			if (k >= blockDim.x)
				rec = __ldcg(pp.items + first + k);
			const uint32_t pos = uint32_t(rec) & 0xffffu, block = uint32_t(rec >> 32);
			if (((uint32_t(rec) >> 16) & 0xffffu) != k)
				lost = true;
			else if (pos + 1 < nwords && block < uint32_t(pp.block_count)) // not a sequence header
				keep(block, pos, k);
		}
		walk = __syncthreads_or(lost);
	}
	// Item by item (proposing a block a second time changes nothing).
	if (walk && threadIdx.x == 0)
		walk_packet([&](uint32_t i) { return i < nwords ? __ldg(pp.data + first + i) : 0u; }, size, state, pp, keep);
	fresh = __reduce_add_sync(0xffffffffu, fresh);
	if ((threadIdx.x & 31) == 0 && fresh)
		atomicAdd(&pp.status->decoded_blocks, fresh);
}

} // namespace

void launch_packet_tables(const PacketParams &pp, cudaStream_t stream)
{
	cudaFuncSetAttribute(packet_tables_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kPacketSmemBytes));
	LaunchConfig lc(dim3(pp.count), dim3(kPacketThreads), stream, false);
	lc.cfg.dynamicSmemBytes = kPacketSmemBytes;
	cudaLaunchKernelEx(&lc.cfg, packet_tables_kernel, pp);
}

void launch_packet_blocks(const PacketParams &pp, cudaStream_t stream)
{
	LaunchConfig lc(dim3(pp.count), dim3(256), stream, true);
	cudaLaunchKernelEx(&lc.cfg, packet_blocks_kernel, pp);
}
} // namespace pw
