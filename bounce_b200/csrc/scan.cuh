#pragma once
// One-pass exclusive scan of u32 (decoupled look-back, as the one-sweep sort):
// a block takes the next tile through a counter, reduces its SC_TILE entries,
// publishes the tile's sum, adds up the sums of the tiles before it (walking
// back until a tile that already published its inclusive prefix; bounded wait)
// and writes its entries' offsets.

#include "b3g_internal.cuh"

constexpr int SC_THREADS = 256;
constexpr int SC_ITEMS = 8;
constexpr uint32_t SC_TILE = SC_THREADS * SC_ITEMS;
constexpr unsigned long long SC_AGG = 1ull << 62;
constexpr unsigned long long SC_INC = 2ull << 62;
constexpr uint32_t SC_SPIN = 1u << 22;

inline uint32_t scan_tiles(uint32_t n) { return (n + SC_TILE - 1) / SC_TILE; }

// One block's part of the scan of n entries; every block of SC_THREADS threads
// takes one tile, and as many blocks take part as there are tiles, or more.
// load(first, v): entries [first, first + SC_ITEMS) into v, 0 from n on.
// state: the tile counter, then one word per tile (flag in bits 62-63, sum in
// bits 0-31), zeroed before the launch. The tile holding the last entry writes
// the total (0 for an empty scan).
template <class Load>
__device__ __forceinline__ void scan_tile(const Load& load, uint32_t* out, uint32_t n, unsigned long long* state,
	uint32_t* total, uint32_t* err)
{
	__shared__ uint32_t sTile, sPrefix;
	__shared__ uint32_t warpSums[SC_THREADS / 32];
	const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
	if (t == 0)
		sTile = atomicAdd(reinterpret_cast<unsigned int*>(state), 1u);
	__syncthreads();
	const uint32_t tile = sTile;
	const uint32_t numTiles = (n + SC_TILE - 1) / SC_TILE;
	if (tile >= numTiles)
	{
		if (tile == 0 && t == 0 && total)
			*total = 0u;
		return;
	}
	// Thread t owns entries [t * SC_ITEMS, t * SC_ITEMS + SC_ITEMS) of the tile.
	const uint32_t first = tile * SC_TILE + t * SC_ITEMS;
	uint32_t v[SC_ITEMS];
	load(first, v);
	uint32_t sum = 0;
#pragma unroll
	for (int r = 0; r < SC_ITEMS; ++r)
		sum += v[r];
	uint32_t incl = sum;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1)
	{
		uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
		if (lane >= (uint32_t)o)
			incl += y;
	}
	if (lane == 31)
		warpSums[warp] = incl;
	__syncthreads();
	if (warp == 0)
	{
		uint32_t w = lane < SC_THREADS / 32 ? warpSums[lane] : 0u;
		uint32_t wi = w;
#pragma unroll
		for (int o = 1; o < SC_THREADS / 32; o <<= 1)
		{
			uint32_t y = __shfl_up_sync(0xFFFFFFFFu, wi, o);
			if (lane >= (uint32_t)o)
				wi += y;
		}
		const uint32_t agg = __shfl_sync(0xFFFFFFFFu, wi, SC_THREADS / 32 - 1);
		if (lane < SC_THREADS / 32)
			warpSums[lane] = wi - w;
		// Look-back by the whole warp: lane k reads the tile k + 1 places
		// back, so a round trip covers 32 tiles. A window is taken once every
		// tile in it has published; the nearest inclusive prefix in it ends
		// the walk (tiles before the first one count as an inclusive 0).
		volatile unsigned long long* st = state + 1;
		if (lane == 0)
			st[tile] = (tile == 0 ? SC_INC : SC_AGG) | agg;
		uint32_t prefix = 0;
		int32_t look = (int32_t)tile - 1;
		uint32_t spins = 0;
		while (tile > 0)
		{
			const int32_t idx = look - (int32_t)lane;
			unsigned long long w8 = 2ull << 62; // before tile 0: an inclusive 0
			if (idx >= 0)
				w8 = st[idx];
			if (!__all_sync(0xFFFFFFFFu, (w8 >> 62) != 0ull))
			{
				if (++spins > SC_SPIN)
				{
					if (lane == 0)
						atomicOr(err, B3G_ST_WAIT_TIMEOUT);
					break;
				}
				continue;
			}
			const uint32_t inc = __ballot_sync(0xFFFFFFFFu, (w8 & SC_INC) != 0ull);
			const uint32_t last = inc ? (uint32_t)(__ffs(inc) - 1) : 31u;
			uint32_t v = lane <= last ? (uint32_t)w8 : 0u;
#pragma unroll
			for (int o = 16; o > 0; o >>= 1)
				v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
			prefix += v;
			if (inc)
				break;
			look -= 32;
		}
		if (lane == 0)
		{
			if (tile > 0)
			{
				__threadfence();
				st[tile] = SC_INC | (uint32_t)(prefix + agg);
			}
			sPrefix = prefix;
			if (tile == numTiles - 1 && total)
				*total = prefix + agg;
		}
	}
	__syncthreads();
	uint32_t run = sPrefix + warpSums[warp] + incl - sum;
#pragma unroll
	for (int r = 0; r < SC_ITEMS; ++r)
	{
		if (first + r < n)
			out[first + r] = run;
		run += v[r];
	}
}

// The same over pairs of counts packed in a u64 (the first in bits 32 and up,
// below 2^30). Tile status words: state in bits 62-63, the pair below.
constexpr unsigned long long SC_PAIR = SC_AGG - 1ull;

// Block-wide exclusive scan of one u64 per thread; returns the thread's
// exclusive prefix and leaves the block total in *total.
__device__ __forceinline__ unsigned long long block_scan(unsigned long long v, unsigned long long* total)
{
	__shared__ unsigned long long warpSum[SC_THREADS / 32];
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	unsigned long long x = v;
	for (int off = 1; off < 32; off <<= 1)
	{
		unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, x, off);
		if (lane >= (uint32_t)off)
			x += y;
	}
	if (lane == 31)
		warpSum[warp] = x;
	__syncthreads();
	if (warp == 0)
	{
		unsigned long long w = lane < SC_THREADS / 32 ? warpSum[lane] : 0ull;
		for (int off = 1; off < 32; off <<= 1)
		{
			unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, w, off);
			if (lane >= (uint32_t)off)
				w += y;
		}
		if (lane < SC_THREADS / 32)
			warpSum[lane] = w;
	}
	__syncthreads();
	unsigned long long before = warp ? warpSum[warp - 1] : 0ull;
	*total = warpSum[SC_THREADS / 32 - 1];
	return before + x - v;
}

// Called by the first warp of a block: publishes tile's total and returns the
// sum of the tiles before it; st: the status words, 0 before the launch.
__device__ __forceinline__ unsigned long long look_back_pairs(volatile unsigned long long* st, uint32_t tile,
	unsigned long long total, bool& timedOut)
{
	const uint32_t lane = threadIdx.x & 31u;
	unsigned long long prefix = 0;
	if (tile == 0)
	{
		if (lane == 0)
			st[0] = SC_INC | total;
		return prefix;
	}
	if (lane == 0)
		st[tile] = SC_AGG | total;
	int32_t hi = (int32_t)tile - 1;
	uint32_t spins = 0;
	while (true)
	{
		const int32_t idx = hi - (int32_t)lane;
		const unsigned long long v = idx >= 0 ? (unsigned long long)st[idx] : (unsigned long long)SC_INC;
		const uint32_t notReady = __ballot_sync(0xFFFFFFFFu, (v & ~SC_PAIR) == 0ull);
		const uint32_t inc = __ballot_sync(0xFFFFFFFFu, (v & SC_INC) != 0ull);
		const uint32_t last = inc ? (uint32_t)__ffs(inc) - 1u : 31u;
		const uint32_t need = last == 31u ? 0xFFFFFFFFu : (2u << last) - 1u;
		if (notReady & need)
		{
			if (++spins > SC_SPIN)
			{
				timedOut = true;
				break;
			}
			continue;
		}
		unsigned long long part = lane <= last ? (v & SC_PAIR) : 0ull;
		for (int off = 16; off > 0; off >>= 1)
			part += __shfl_xor_sync(0xFFFFFFFFu, part, off);
		prefix += part;
		if (inc)
			break;
		hi -= 32;
	}
	if (lane == 0)
	{
		__threadfence();
		st[tile] = SC_INC | (prefix + total);
	}
	return prefix;
}
