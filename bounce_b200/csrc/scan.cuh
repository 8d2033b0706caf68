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
