// Fat-AABB update and broadphase of one collision pass.
//
//  k_sync        per proxy: swept AABB of the fixture over [xf0, xf1] and the
//                b3DynamicTree::MoveProxy keep-or-reinsert rule
//                (fixture.cpp:120-132, dynamic_tree.cpp:139-207), or the
//                CreateProxy fattening on a creation pass (dynamic_tree.cpp:108-128)
//  k_bounds / k_morton / radix sort
//                world-major 64-bit keys: world index << 32 | 30-bit Morton code
//                of the fat-AABB centre, sorted by an LSD radix sort
//  k_build       Karras (2012) radix tree over the sorted keys, with ropes
//                (the next node in depth-first order after a subtree)
//  k_refit       bottom-up node AABBs
//  k_traverse    each leaf's search of the subtrees after it in sorted order,
//                so each overlapping pair is met once; the AddPair filters
//                (contact_manager.cpp:98-160) and the b3Contact::Create A/B
//                order (contact.cpp:290-322) are applied per pair
//
// The overlap set found this way is the set of pairs the reference has a
// contact for after FindNewContacts (pairs are created when either proxy
// moves); order.cu turns it into the contact list, which also keeps the
// contacts UpdateContacts skips because neither body is active.

#include <cuda/atomic>

#include "collide_common.cuh"
#include "scan.cuh"

namespace {

constexpr uint32_t SENT = 0xFFFFFFFFu;


// Lanes per fixture in k_sync: a hull's vertex loop is split across them.
constexpr uint32_t SYNC_LANES = 8;

__device__ __forceinline__ V3 shfl_xor3(uint32_t mask, V3 v, int o)
{
	return V3{__shfl_xor_sync(mask, v.x, o), __shfl_xor_sync(mask, v.y, o), __shfl_xor_sync(mask, v.z, o)};
}

// b3Shape::ComputeAABB at two transforms for the lanes of one group, from
// the fixture's preloaded type and params (compute_aabbs's arithmetic): a
// hull's vertices are strided over the lanes and the boxes combined by min /
// max, which are exact, so the result is the serial loop's
// (b3HullShape::ComputeAABB, hull_shape.cpp:160-164). Every lane of the
// group ends with the same boxes.
__device__ __forceinline__ void group_aabbs(const DevScene& S, uint32_t type, float4 p0, float4 p1, float4 p2,
	uint32_t hullIndex, const XF& xa, const XF& xb, bool two, AABB& a, AABB& b, uint32_t lane, uint32_t mask)
{
	if (type == B3G_SHAPE_SPHERE)
	{
		V3 c = V3{p0.x, p0.y, p0.z};
		V3 rv = V3{p0.w, p0.w, p0.w};
		V3 ca = xmul(xa, c);
		a.lo = ca - rv;
		a.hi = ca + rv;
		V3 cb = two ? xmul(xb, c) : ca;
		b.lo = cb - rv;
		b.hi = cb + rv;
		return;
	}
	if (type == B3G_SHAPE_CAPSULE)
	{
		V3 v1 = V3{p0.x, p0.y, p0.z};
		V3 v2 = V3{p0.w, p1.x, p1.y};
		V3 rv = V3{p1.z, p1.z, p1.z};
		V3 c1 = xmul(xa, v1), c2 = xmul(xa, v2);
		a.lo = vmin(c1, c2) - rv;
		a.hi = vmax(c1, c2) + rv;
		if (two)
		{
			c1 = xmul(xb, v1);
			c2 = xmul(xb, v2);
		}
		b.lo = vmin(c1, c2) - rv;
		b.hi = vmax(c1, c2) + rv;
		return;
	}
	if (type == B3G_SHAPE_TRIANGLE)
	{
		// The reference ignores the transform here (triangle_shape.cpp:59-67).
		V3 v1 = V3{p0.x, p0.y, p0.z};
		V3 v2 = V3{p0.w, p1.x, p1.y};
		V3 v3_ = V3{p1.z, p1.w, p2.x};
		V3 rv = V3{p2.y, p2.y, p2.y};
		a.lo = vmin(v1, vmin(v2, v3_)) - rv;
		a.hi = vmax(v1, vmax(v2, v3_)) + rv;
		b = a;
		return;
	}
	const HullDesc h = S.hulls[hullIndex];
	const float4* hv = S.hverts + h.vOff;
	float4 w = hv[0];
	V3 v0 = V3{w.x, w.y, w.z};
	V3 ta = xmul(xa, v0), tb = two ? xmul(xb, v0) : ta;
	a.lo = a.hi = ta;
	b.lo = b.hi = tb;
	for (uint32_t k = 1 + lane; k < h.vCnt; k += SYNC_LANES)
	{
		w = hv[k];
		V3 v = V3{w.x, w.y, w.z};
		ta = xmul(xa, v);
		a.lo = vmin(a.lo, ta);
		a.hi = vmax(a.hi, ta);
		if (two)
		{
			tb = xmul(xb, v);
			b.lo = vmin(b.lo, tb);
			b.hi = vmax(b.hi, tb);
		}
	}
	for (int o = SYNC_LANES / 2; o > 0; o >>= 1)
	{
		a.lo = vmin(a.lo, shfl_xor3(mask, a.lo, o));
		a.hi = vmax(a.hi, shfl_xor3(mask, a.hi, o));
		if (two)
		{
			b.lo = vmin(b.lo, shfl_xor3(mask, b.lo, o));
			b.hi = vmax(b.hi, shfl_xor3(mask, b.hi, o));
		}
	}
	float r = p0.x;
	aabb_extend(a, r);
	if (two)
		aabb_extend(b, r);
}

// Atomic min / max of IEEE floats (no NaN): non-negative floats order like
// their bits as signed integers, negative ones in reverse as unsigned.
__device__ __forceinline__ void atomic_min_float(float* a, float v)
{
	if (v >= 0.0f)
		atomicMin(reinterpret_cast<int*>(a), __float_as_int(v));
	else
		atomicMax(reinterpret_cast<unsigned int*>(a), __float_as_uint(v));
}
__device__ __forceinline__ void atomic_max_float(float* a, float v)
{
	if (v >= 0.0f)
		atomicMax(reinterpret_cast<int*>(a), __float_as_int(v));
	else
		atomicMin(reinterpret_cast<unsigned int*>(a), __float_as_uint(v));
}

// Refit of a reused tree (the passes between rebuilds): only the proxies
// whose fat AABB was re-inserted (moved) changed, and a walk needs every
// node to contain its leaves, not to be tight. k_sync writes a moved proxy's
// new box into its leaf and grows the leaf's ancestors by it (atomic min /
// max per coordinate), stopping at the first that already contains it (every
// node above contains that one). Nodes only grow until the next rebuild makes
// them tight again; an unmoved leaf's box is contained already.
__device__ __forceinline__ void grow_leaf(Buffers& B, uint32_t nLeaves, uint32_t proxy, V3 lo, V3 hi)
{
	const uint32_t leaf = nLeaves - 1u + B.leafOf[proxy];
	float* llo = reinterpret_cast<float*>(&B.nodeLo[leaf]);
	float* lhi = reinterpret_cast<float*>(&B.nodeHi[leaf]);
	llo[0] = lo.x;
	llo[1] = lo.y;
	llo[2] = lo.z;
	lhi[0] = hi.x;
	lhi[1] = hi.y;
	lhi[2] = hi.z;
	if (nLeaves < 2)
		return;
	uint32_t p = B.nodeParent[leaf];
	while (true)
	{
		const float4 cl = __ldcg(&B.nodeLo[p]), ch = __ldcg(&B.nodeHi[p]);
		if (cl.x <= lo.x && cl.y <= lo.y && cl.z <= lo.z && ch.x >= hi.x && ch.y >= hi.y && ch.z >= hi.z)
			return;
		float* plo = reinterpret_cast<float*>(&B.nodeLo[p]);
		float* phi = reinterpret_cast<float*>(&B.nodeHi[p]);
		atomic_min_float(plo + 0, lo.x);
		atomic_min_float(plo + 1, lo.y);
		atomic_min_float(plo + 2, lo.z);
		atomic_max_float(phi + 0, hi.x);
		atomic_max_float(phi + 1, hi.y);
		atomic_max_float(phi + 2, hi.z);
		if (p == 0)
			return;
		p = B.nodeParent[p];
	}
}

// One group of SYNC_LANES lanes per fixture; lane 0 writes. All lanes of a
// group take the same branches, so the group mask is exact for the shuffles.
// The per-body transforms of the pass (m_xf and b3Sweep::GetTransform(0),
// sweep.h:43-63, two float4 each, read by the later stages) are written by
// lane 1 of group b for body b. The fixture's records are loaded before any
// branch so that their loads overlap.
__global__ void k_sync(DevScene S, Buffers B, uint32_t nf, uint32_t nb, int creation, int grow)
{
	const uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) / SYNC_LANES;
	const uint32_t lane = threadIdx.x % SYNC_LANES;
	const uint32_t mask = ((1u << SYNC_LANES) - 1u) << ((threadIdx.x & 31u) & ~(SYNC_LANES - 1u));
	if (lane == 1 && g < nb)
	{
		pack_xf(S.bodyXf, g, load_xf(S.bodyState + 17 * (size_t)g));
		pack_xf(S.bodyXf0, g, sweep_xf0(S, g));
	}
	if (g >= nf)
		return;
	const uint32_t i = g;
	const bool w0 = lane == 0;
	const uint8_t life = S.fixLife[i];
	const uint32_t type = S.fixType[i];
	const uint32_t body = S.fixBody[i];
	const uint32_t hullIndex = S.fixHull[i];
	const float4 p0 = S.fixParams[3 * i + 0], p1 = S.fixParams[3 * i + 1], p2 = S.fixParams[3 * i + 2];
	const float4 tl = B.fatLo[i], th = B.fatHi[i];
	const float* st = S.bodyState + 17 * (size_t)body;
	float sv[17];
#pragma unroll
	for (int k = 0; k < 17; ++k)
		sv[k] = st[k];
	const uint32_t btype = S.bodyType[body];
	// The walk's filter reads one word per proxy (pair_filter).
	if (w0)
		B.proxyInfo[i] = (body & 0x0FFFFFFFu) | (btype == B3G_BODY_DYNAMIC ? 1u << 28 : 0u) | (type << 29);
	if (life == FIX_DEAD)
	{
		// No proxy: an empty box (lower > upper) that overlaps nothing.
		if (w0)
		{
			B.fatLo[i] = make_float4(B3G_MAX_SCALAR, B3G_MAX_SCALAR, B3G_MAX_SCALAR, 0.0f);
			B.fatHi[i] = make_float4(-B3G_MAX_SCALAR, -B3G_MAX_SCALAR, -B3G_MAX_SCALAR, 0.0f);
			B.moved[i] = 0;
		}
		return;
	}
	if (type == B3G_SHAPE_MESH)
	{
		// Meshes sit on static bodies: their proxy is created once (k_mesh_fat
		// on a creation pass) and never moves.
		if (w0)
			B.moved[i] = 0;
		return;
	}
	XF xf1 = load_xf(sv);
	if (creation || life == FIX_FRESH)
	{
		// b3DynamicTree::CreateProxy (dynamic_tree.cpp:108-128).
		AABB a, unused;
		group_aabbs(S, type, p0, p1, p2, hullIndex, xf1, xf1, false, a, unused, lane, mask);
		if (w0)
		{
			V3 r = V3{B3G_AABB_EXTENSION, B3G_AABB_EXTENSION, B3G_AABB_EXTENSION};
			V3 lo = a.lo - r, hi = a.hi + r;
			B.fatLo[i] = make_float4(lo.x, lo.y, lo.z, 0.0f);
			B.fatHi[i] = make_float4(hi.x, hi.y, hi.z, 0.0f);
			B.moved[i] = 1;
		}
		return;
	}
	// Every non-static body is synchronised, whatever its awake flag:
	// b3World::Solve synchronises each body of a solved island
	// (world.cpp:424-449), including those the island put to sleep in that
	// step (island.cpp:297-305). A body asleep since its last move keeps its
	// sweep, so synchronising it again finds its AABB inside the fat AABB it
	// got then and moves nothing: the result is the reference's, which skips it.
	if (btype == B3G_BODY_STATIC)
	{
		if (w0)
			B.moved[i] = 0;
		return;
	}
	// b3Body::SynchronizeFixtures (body.cpp:216-229): xf0 from the sweep start.
	XF xf0;
	xf0.q = Q4{V3{sv[10], sv[11], sv[12]}, sv[13]};
	V3 c0 = V3{sv[7], sv[8], sv[9]};
	V3 lc = V3{sv[14], sv[15], sv[16]};
	xf0.p = c0 - rot(xf0.q, lc);

	// b3Fixture::Synchronize (fixture.cpp:120-132).
	AABB a1, a2;
	group_aabbs(S, type, p0, p1, p2, hullIndex, xf0, xf1, true, a1, a2, lane, mask);
	if (!w0)
		return;
	AABB aabb;
	aabb.lo = vmin(a1.lo, a2.lo);
	aabb.hi = vmax(a1.hi, a2.hi);
	V3 disp = aabb_center(a2) - aabb_center(a1);

	// b3DynamicTree::MoveProxy (dynamic_tree.cpp:139-207).
	AABB fat = aabb;
	aabb_extend(fat, B3G_AABB_EXTENSION);
	V3 d = B3G_AABB_MULTIPLIER * disp;
	if (d.x < 0.0f)
		fat.lo.x += d.x;
	else
		fat.hi.x += d.x;
	if (d.y < 0.0f)
		fat.lo.y += d.y;
	else
		fat.hi.y += d.y;
	if (d.z < 0.0f)
		fat.lo.z += d.z;
	else
		fat.hi.z += d.z;

	AABB tree;
	tree.lo = V3{tl.x, tl.y, tl.z};
	tree.hi = V3{th.x, th.y, th.z};
	if (aabb_contains(tree, aabb))
	{
		AABB huge = fat;
		aabb_extend(huge, 4.0f * B3G_AABB_EXTENSION);
		if (aabb_contains(huge, tree))
		{
			B.moved[i] = 0;
			return;
		}
	}
	B.fatLo[i] = make_float4(fat.lo.x, fat.lo.y, fat.lo.z, 0.0f);
	B.fatHi[i] = make_float4(fat.hi.x, fat.hi.y, fat.hi.z, 0.0f);
	B.moved[i] = 1;
	if (grow)
		grow_leaf(B, nf, i, fat.lo, fat.hi);
}

// ---------------------------------------------------------------------------
// Scene bounds of the fat-AABB centres (for Morton quantisation).

__device__ __forceinline__ int f2o(float f)
{
	int i = __float_as_int(f);
	return i >= 0 ? i : i ^ 0x7FFFFFFF;
}
__device__ __forceinline__ float o2f(int i)
{
	return __int_as_float(i >= 0 ? i : i ^ 0x7FFFFFFF);
}

__global__ void k_bounds_init(int* bnd)
{
	if (threadIdx.x < 3)
		bnd[threadIdx.x] = 0x7FFFFFFF;
	else if (threadIdx.x < 6)
		bnd[threadIdx.x] = (int)0x80000000;
}

__global__ void k_bounds(DevScene S, Buffers B, uint32_t n, int* bnd)
{
	__shared__ int s[6][8];
	float mn[3] = {B3G_MAX_SCALAR, B3G_MAX_SCALAR, B3G_MAX_SCALAR};
	float mx[3] = {-B3G_MAX_SCALAR, -B3G_MAX_SCALAR, -B3G_MAX_SCALAR};
	for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
	{
		if (S.fixLife[i] == FIX_DEAD)
			continue;
		float4 lo = B.fatLo[i], hi = B.fatHi[i];
		float c[3] = {0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z)};
		for (int k = 0; k < 3; ++k)
		{
			mn[k] = fminf(mn[k], c[k]);
			mx[k] = fmaxf(mx[k], c[k]);
		}
	}
	for (int k = 0; k < 3; ++k)
	{
		for (int o = 16; o > 0; o >>= 1)
		{
			mn[k] = fminf(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], o));
			mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
		}
	}
	int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	if (lane == 0)
	{
		for (int k = 0; k < 3; ++k)
		{
			s[k][warp] = f2o(mn[k]);
			s[3 + k][warp] = f2o(mx[k]);
		}
	}
	__syncthreads();
	if (threadIdx.x < 6)
	{
		int nw = blockDim.x >> 5;
		int v = s[threadIdx.x][0];
		for (int w = 1; w < nw; ++w)
			v = threadIdx.x < 3 ? min(v, s[threadIdx.x][w]) : max(v, s[threadIdx.x][w]);
		if (threadIdx.x < 3)
			atomicMin(bnd + threadIdx.x, v);
		else
			atomicMax(bnd + threadIdx.x, v);
	}
}

__device__ __forceinline__ uint32_t expand10(uint32_t v)
{
	v = (v * 0x00010001u) & 0xFF0000FFu;
	v = (v * 0x00000101u) & 0x0F00F00Fu;
	v = (v * 0x00000011u) & 0xC30C30C3u;
	v = (v * 0x00000005u) & 0x49249249u;
	return v;
}

__global__ void k_morton(DevScene S, Buffers B, uint32_t n, const int* bnd)
{
	uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n)
		return;
	float lo[3] = {o2f(bnd[0]), o2f(bnd[1]), o2f(bnd[2])};
	float hi[3] = {o2f(bnd[3]), o2f(bnd[4]), o2f(bnd[5])};
	float4 a = B.fatLo[i], b = B.fatHi[i];
	float c[3] = {0.5f * (a.x + b.x), 0.5f * (a.y + b.y), 0.5f * (a.z + b.z)};
	uint32_t q[3];
	for (int k = 0; k < 3; ++k)
	{
		float ext = hi[k] - lo[k];
		float t = ext > 0.0f ? (c[k] - lo[k]) / ext : 0.0f;
		t = fminf(fmaxf(t, 0.0f), 1.0f);
		q[k] = min((uint32_t)(t * 1024.0f), 1023u);
	}
	uint32_t code = (expand10(q[0]) << 2) | (expand10(q[1]) << 1) | expand10(q[2]);
	// A proxy wider than a quarter of the scene's longest side (a ground box, a
	// mesh) sorts after the other proxies of its world: its pairs are then
	// found by the many short walks of the leaves before it instead of by one
	// long walk of its own. The longest side and not each axis's own, since a
	// flat or narrow world is not wide on every axis: bodies spread over a
	// 40 m terrain but 5 m high would nearly all count as wide. The wide ones
	// keep their Morton order among themselves. Only the traversal order
	// changes. Measured on 3,001 bodies over a terrain mesh: walk 746 -> 41 us.
	float side = 0.0f, wide = 0.0f;
	const float e[3] = {b.x - a.x, b.y - a.y, b.z - a.z};
	for (int k = 0; k < 3; ++k)
	{
		side = fmaxf(side, hi[k] - lo[k]);
		wide = fmaxf(wide, e[k]);
	}
	if (side > 0.0f && wide > 0.25f * side)
		code |= 1u << 30;
	uint32_t world = S.bodyWorld[S.fixBody[i]];
	// Dead proxies sort after every live one.
	B.keysA[i] = S.fixLife[i] == FIX_DEAD ? ~0ull : ((unsigned long long)world << 32) | code;
	B.valsA[i] = i;
}

// ---------------------------------------------------------------------------
// Scans.

// One-sweep LSD radix sort (Merrill & Garland's decoupled look-back): one
// histogram kernel for every digit pass up front, then one kernel per pass.
// A block ranks its tile's keys per digit in shared memory (stable: element
// order within the tile), publishes the tile's digit counts, adds up the
// counts of the tiles before it (walking back until a tile that already
// published an inclusive prefix) and scatters. Tiles are taken in launch
// order through a counter, so a tile only waits for tiles of blocks that
// started before it; the waits are bounded all the same.
constexpr int OS_THREADS = 256;
constexpr int OS_ITEMS = 4;
constexpr uint32_t OS_TILE = OS_THREADS * OS_ITEMS;
constexpr uint32_t OS_AGG = 1u << 30;     // the tile's own count is published
constexpr uint32_t OS_INC = 2u << 30;     // the count through this tile is published
constexpr uint32_t OS_MASK = OS_AGG - 1u; // counts below 2^30
constexpr uint32_t OS_SPIN = 1u << 22;

struct SortShifts
{
	int s[8];
	int n;
};

__global__ void k_os_hist(const unsigned long long* keys, uint32_t n, SortShifts sh, uint32_t* ghist)
{
	__shared__ uint32_t h[8][256];
	for (int p = 0; p < sh.n; ++p)
		h[p][threadIdx.x] = 0;
	__syncthreads();
	for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
	{
		unsigned long long k = keys[i];
		for (int p = 0; p < sh.n; ++p)
			atomicAdd(&h[p][(uint32_t)(k >> sh.s[p]) & 0xFFu], 1u);
	}
	__syncthreads();
	for (int p = 0; p < sh.n; ++p)
		if (h[p][threadIdx.x])
			atomicAdd(&ghist[p * 256 + threadIdx.x], h[p][threadIdx.x]);
}

// Exclusive scan of each pass's 256 digit counts (one block of 256 per pass).
__global__ void k_os_scan(uint32_t* ghist)
{
	__shared__ uint32_t v[256];
	uint32_t* g = ghist + blockIdx.x * 256;
	uint32_t x = g[threadIdx.x];
	v[threadIdx.x] = x;
	__syncthreads();
	for (uint32_t off = 1; off < 256; off <<= 1)
	{
		uint32_t y = threadIdx.x >= off ? v[threadIdx.x - off] : 0u;
		__syncthreads();
		v[threadIdx.x] += y;
		__syncthreads();
	}
	g[threadIdx.x] = v[threadIdx.x] - x;
}

__global__ void __launch_bounds__(OS_THREADS) k_onesweep(const unsigned long long* kin, const uint32_t* vin,
	unsigned long long* kout, uint32_t* vout, uint32_t n, int shift, const uint32_t* gOffset, uint32_t* status,
	uint32_t* tileCounter, uint32_t* err)
{
	__shared__ uint32_t sTile;
	__shared__ uint32_t run[256];
	__shared__ uint32_t wc[OS_THREADS / 32][256];
	__shared__ uint32_t base[256];
	const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
	if (t == 0)
		sTile = atomicAdd(tileCounter, 1u);
	run[t] = 0;
	for (int w = 0; w < OS_THREADS / 32; ++w)
		wc[w][t] = 0;
	__syncthreads();
	const uint32_t tile = sTile;
	const uint32_t lt = (1u << lane) - 1u;
	unsigned long long key[OS_ITEMS];
	uint32_t val[OS_ITEMS], dig[OS_ITEMS], rank[OS_ITEMS];
	for (int r = 0; r < OS_ITEMS; ++r)
	{
		uint32_t idx = tile * OS_TILE + r * OS_THREADS + t;
		bool valid = idx < n;
		key[r] = valid ? kin[idx] : 0ull;
		val[r] = valid ? vin[idx] : 0u;
		uint32_t d = valid ? ((uint32_t)(key[r] >> shift) & 0xFFu) : 0x100u;
		dig[r] = d;
		uint32_t peers = __match_any_sync(0xffffffffu, d);
		uint32_t pr = __popc(peers & lt);
		if (valid && pr == 0)
			wc[warp][d] = __popc(peers);
		__syncthreads();
		{
			uint32_t sum = run[t];
			for (int w = 0; w < OS_THREADS / 32; ++w)
			{
				uint32_t cnt = wc[w][t];
				wc[w][t] = sum;
				sum += cnt;
			}
			run[t] = sum;
		}
		__syncthreads();
		rank[r] = valid ? wc[warp][d] + pr : 0u;
		__syncthreads();
		for (int w = 0; w < OS_THREADS / 32; ++w)
			wc[w][t] = 0;
		__syncthreads();
	}
	// Thread t owns digit t: publish, look back, publish the inclusive prefix.
	{
		const uint32_t mine = run[t];
		volatile uint32_t* st = status;
		if (tile == 0)
			st[t] = OS_INC | mine;
		else
		{
			st[(size_t)tile * 256 + t] = OS_AGG | mine;
			uint32_t prefix = 0;
			int32_t look = (int32_t)tile - 1;
			uint32_t spins = 0;
			while (look >= 0)
			{
				uint32_t v = st[(size_t)look * 256 + t];
				if ((v & ~OS_MASK) == 0u)
				{
					if (++spins > OS_SPIN)
					{
						atomicOr(err, B3G_ST_WAIT_TIMEOUT);
						break;
					}
					continue;
				}
				prefix += v & OS_MASK;
				if (v & OS_INC)
					break;
				--look;
			}
			__threadfence();
			st[(size_t)tile * 256 + t] = OS_INC | (prefix + mine);
			base[t] = gOffset[t] + prefix;
		}
		if (tile == 0)
			base[t] = gOffset[t];
	}
	__syncthreads();
	for (int r = 0; r < OS_ITEMS; ++r)
	{
		if (dig[r] > 0xFFu)
			continue;
		uint32_t pos = base[dig[r]] + rank[r];
		if (pos < n)
		{
			kout[pos] = key[r];
			vout[pos] = val[r];
		}
	}
}

// ---------------------------------------------------------------------------
// Karras radix tree.

__device__ __forceinline__ int delta(const unsigned long long* k, int n, int i, int j)
{
	if (j < 0 || j >= n)
		return -1;
	unsigned long long a = k[i], b = k[j];
	if (a == b)
		return 64 + __clz((uint32_t)i ^ (uint32_t)j);
	return __clzll(a ^ b);
}

__global__ void k_build(Buffers B, int n)
{
	int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n - 1)
		return;
	const unsigned long long* k = B.keysA;
	int d = (delta(k, n, i, i + 1) - delta(k, n, i, i - 1)) >= 0 ? 1 : -1;
	int dmin = delta(k, n, i, i - d);
	int lmax = 2;
	while (delta(k, n, i, i + lmax * d) > dmin)
		lmax <<= 1;
	int l = 0;
	for (int t = lmax >> 1; t >= 1; t >>= 1)
		if (delta(k, n, i, i + (l + t) * d) > dmin)
			l += t;
	int j = i + l * d;
	int dnode = delta(k, n, i, j);
	int s = 0;
	int t = l;
	do
	{
		t = (t + 1) >> 1;
		if (delta(k, n, i, i + (s + t) * d) > dnode)
			s += t;
	} while (t > 1);
	int gamma = i + s * d + min(d, 0);
	int first = min(i, j), last = max(i, j);
	uint32_t left = (first == gamma) ? (uint32_t)(n - 1 + gamma) : (uint32_t)gamma;
	uint32_t right = (last == gamma + 1) ? (uint32_t)(n - 1 + gamma + 1) : (uint32_t)(gamma + 1);
	B.nodeLeft[i] = left;
	B.nodeRight[i] = right;
	B.nodeParent[left] = i;
	B.nodeParent[right] = i;
	B.nodeFirst[i] = first;
	B.nodeEnd[i] = last;
	B.splitRight[gamma] = right;
}

__global__ void k_leaves(DevScene S, Buffers B, int n)
{
	int j = blockIdx.x * blockDim.x + threadIdx.x;
	if (j >= n)
		return;
	uint32_t node = n - 1 + j;
	uint32_t proxy = B.valsA[j];
	uint32_t rope = (j == n - 1) ? SENT : B.splitRight[j];
	B.nodeLeft[node] = proxy;
	B.nodeFirst[node] = j;
	B.leafOf[proxy] = j;
	// Traversal reads a node as two float4: (lower, left child or proxy) and
	// (upper, rope).
	float4 lo = B.fatLo[proxy], hi = B.fatHi[proxy];
	B.nodeLo[node] = make_float4(lo.x, lo.y, lo.z, __uint_as_float(proxy));
	B.nodeHi[node] = make_float4(hi.x, hi.y, hi.z, __uint_as_float(rope));
	B.nodeRope[node] = rope;
	// What the walk's filter and contact order need of the proxy, addressed
	// by the leaf's position so it loads beside the node.
	B.leafData[j] = make_uint2(B.proxyInfo[proxy], S.fixKey[proxy]);
	if (j < n - 1)
	{
		B.nodeRope[j] = (B.nodeEnd[j] == (uint32_t)(n - 1)) ? SENT : B.splitRight[B.nodeEnd[j]];
		B.refitFlag[j] = 0;
	}
	// Last sorted leaf of each world (dead proxies, sorted last, belong to none).
	if (S.fixLife[proxy] != FIX_DEAD)
	{
		uint32_t w = S.bodyWorld[S.fixBody[proxy]];
		uint32_t nx = j == n - 1 ? SENT : B.valsA[j + 1];
		if (nx == SENT || S.fixLife[nx] == FIX_DEAD || S.bodyWorld[S.fixBody[nx]] != w)
			B.worldEnd[w] = j;
	}
}

// A climb is one dependent step per level: the second child to arrive takes
// its sibling's box and goes on. The child's own box stays in registers, and
// the parent's links load while the atomic is on its way: 70,000
// leaves 40 -> 30 us, 370,000 69 -> 55.
__global__ void k_refit(Buffers B, int n)
{
	int j = blockIdx.x * blockDim.x + threadIdx.x;
	if (j >= n || n < 2)
		return;
	uint32_t node = n - 1 + j;
	float4 lo = B.nodeLo[node], hi = B.nodeHi[node];
	uint32_t p = B.nodeParent[node];
	while (true)
	{
		// Release this child's box, acquire the sibling's: one acq_rel atomic
		// per level instead of two full fences.
		cuda::atomic_ref<uint32_t, cuda::thread_scope_device> flag(B.refitFlag[p]);
		const uint32_t l = B.nodeLeft[p], r = B.nodeRight[p], rope = B.nodeRope[p];
		const uint32_t up = p == 0 ? 0u : B.nodeParent[p];
		const uint32_t old = flag.fetch_add(1u, cuda::memory_order_acq_rel);
		if (old == 0)
			return;
		const uint32_t other = node == l ? r : l;
		const float4 ol = __ldcg(&B.nodeLo[other]), oh = __ldcg(&B.nodeHi[other]);
		lo = make_float4(fminf(lo.x, ol.x), fminf(lo.y, ol.y), fminf(lo.z, ol.z), __uint_as_float(l));
		hi = make_float4(fmaxf(hi.x, oh.x), fmaxf(hi.y, oh.y), fmaxf(hi.z, oh.z), __uint_as_float(rope));
		B.nodeLo[p] = lo;
		B.nodeHi[p] = hi;
		if (p == 0)
			return;
		node = p;
		p = up;
	}
}

// ---------------------------------------------------------------------------
// Pair search.

// b3Contact::s_registers (contact.cpp:253-288): registered type pairs, and
// whether (t1, t2) is the primary order (fixture A keeps type t1).
__device__ __forceinline__ bool registered(uint32_t a, uint32_t b)
{
	// bit (a * 5 + b)
	const uint32_t mask =
		(1u << (0 * 5 + 0)) | (1u << (1 * 5 + 0)) | (1u << (0 * 5 + 1)) | (1u << (1 * 5 + 1)) |
		(1u << (2 * 5 + 0)) | (1u << (0 * 5 + 2)) | (1u << (2 * 5 + 1)) | (1u << (1 * 5 + 2)) |
		(1u << (3 * 5 + 0)) | (1u << (0 * 5 + 3)) | (1u << (3 * 5 + 1)) | (1u << (1 * 5 + 3)) |
		(1u << (3 * 5 + 2)) | (1u << (2 * 5 + 3)) | (1u << (3 * 5 + 3)) |
		(1u << (3 * 5 + 4)) | (1u << (4 * 5 + 3)) | (1u << (4 * 5 + 0)) | (1u << (0 * 5 + 4)) |
		(1u << (4 * 5 + 1)) | (1u << (1 * 5 + 4));
	return (mask >> (a * 5 + b)) & 1u;
}
__device__ __forceinline__ bool primary(uint32_t a, uint32_t b)
{
	const uint32_t mask = (1u << (0 * 5 + 0)) | (1u << (1 * 5 + 0)) | (1u << (1 * 5 + 1)) |
		(1u << (2 * 5 + 0)) | (1u << (2 * 5 + 1)) | (1u << (3 * 5 + 0)) | (1u << (3 * 5 + 1)) |
		(1u << (3 * 5 + 2)) | (1u << (3 * 5 + 3)) | (1u << (3 * 5 + 4)) | (1u << (4 * 5 + 0)) |
		(1u << (4 * 5 + 1));
	return (mask >> (a * 5 + b)) & 1u;
}

// AddPair filters: same body (contact_manager.cpp:104-108), b3Body::ShouldCollide
// (at least one dynamic body, body.cpp:240-246) and a registered shape pair
// (b3Contact::Create returns nullptr otherwise, contact.cpp:318-321).
__device__ __forceinline__ bool pair_filter(uint32_t infoA, uint32_t infoB)
{
	if (((infoA ^ infoB) & 0x0FFFFFFFu) == 0u)
		return false;
	if (((infoA | infoB) & (1u << 28)) == 0u)
		return false;
	return registered(infoA >> 29, infoB >> 29);
}

// The contact record of overlapping proxies pa, pb (keys keyA, keyB, shape
// types typeA, typeB): the broadphase order (min, max) of proxy ids
// (b3BroadPhase::Report, broad_phase.cpp:341-342) followed by the factory's
// primary-type swap (b3Contact::Create, contact.cpp:306-317). x = fixture A,
// y = fixture B.
__device__ __forceinline__ uint2 canon_pair_keys(uint32_t pa, uint32_t keyA, uint32_t typeA, uint32_t pb,
	uint32_t keyB, uint32_t typeB)
{
	const bool aFirst = keyA < keyB;
	uint32_t f1 = aFirst ? pa : pb, f2 = aFirst ? pb : pa;
	uint32_t t1 = aFirst ? typeA : typeB, t2 = aFirst ? typeB : typeA;
	if (!primary(t1, t2))
		return make_uint2(f2, f1);
	return make_uint2(f1, f2);
}

// The leaves' walks. Every pair is found once, from the leaf that comes first
// in the tree: the subtrees after leaf j are the right siblings on its path to
// the root, a chain of ropes (a leaf's rope, that node's rope, ...), and a
// subtree is searched downwards from there.
//
// A warp takes `leaves` leaves. A lane follows its leaf's chain only while the
// warp's stack holds fewer than 32 nodes; otherwise each lane pops a node that
// some leaf's box overlaps, tests both of its children and pushes those that
// overlap in turn, so the lanes stay busy however uneven the leaves' searches
// are. Overlapping leaves go to a list, filtered and written to the pair list
// (rawA, rawB) 32 at a time (the order of the pairs is free: the contact order
// follows the proxy keys). With a lane per leaf walking the ropes, 10
// of 32 lanes were active: 86 us for 65,536 mixed bodies, now 50; 3,001 bodies on
// a terrain 40 -> 16; 370,000 proxies in 512 worlds 130 -> 104. What bounds it
// now is the dependent loads of a step, 50 steps a warp.
//
// MW: several worlds share the tree. They are contiguous in its order, so a
// right child past the last leaf of the query's world is not entered; its
// first leaf is its own index (a left child begins where its parent does).
constexpr uint32_t WALK_STACK = 128; // 256: 1 % longer, for the shared memory it takes from the others
struct WalkWarp
{
	uint32_t left[WALK_STACK], right[WALK_STACK]; // children of the nodes to search
	uint32_t hitLeaf[96], hitProxy[96];
	float box[6][32];                                     // per leaf of the warp: fat AABB,
	uint32_t info[32], key[32], proxy[32], last[32];      // proxyInfo, key, proxy, its world's last leaf,
	uint32_t visits[32], found[32];                       // nodes tested, pairs found
	uint8_t query[WALK_STACK], hitQuery[96];          // whose
};

struct WalkBox
{
	V3 lo, hi;
	__device__ __forceinline__ WalkBox(const WalkWarp& W, uint32_t q)
		: lo{W.box[0][q], W.box[1][q], W.box[2][q]}, hi{W.box[3][q], W.box[4][q], W.box[5][q]}
	{
	}
	__device__ __forceinline__ bool overlaps(float4 l, float4 h) const
	{
		return !(h.x < lo.x || l.x > hi.x || h.y < lo.y || l.y > hi.y || h.z < lo.z || l.z > hi.z);
	}
};

// Whether leaf q's walk may test one more node (LIMIT: b3g_set_walk_limit).
template <bool LIMIT>
__device__ __forceinline__ bool walk_visit(WalkWarp& W, Buffers& B, uint32_t q, uint32_t limit)
{
	if (!LIMIT || atomicAdd(&W.visits[q], 1u) < limit)
		return true;
	atomicOr(&B.counters[CTR_STATUS], B3G_ST_WAIT_TIMEOUT);
	return false;
}

// The lanes' pairs (query q's leaf with the leaf at `leaf`, proxy pb) to the
// pair list; CTR_TRAV_OVERFLOW counts a leaf's pairs past B3G_TRAV_SLOTS.
__device__ __forceinline__ void walk_record(WalkWarp& W, Buffers& B, uint32_t cap, bool any, uint32_t q,
	uint32_t leaf, uint32_t pb)
{
	const uint32_t lane = threadIdx.x & 31u;
	uint2 p = make_uint2(0u, 0u);
	bool over = false;
	if (any)
	{
		const uint2 db = __ldg(B.leafData + leaf);
		any = pair_filter(W.info[q], db.x);
		if (any)
		{
			p = canon_pair_keys(W.proxy[q], W.key[q], W.info[q] >> 29, pb, db.y, db.x >> 29);
			over = atomicAdd(&W.found[q], 1u) >= B3G_TRAV_SLOTS;
		}
	}
	const uint32_t m = __ballot_sync(0xffffffffu, any), om = __ballot_sync(0xffffffffu, over);
	uint32_t base = 0;
	if (lane == 0)
	{
		if (m)
			base = atomicAdd(&B.counters[CTR_RAW], (uint32_t)__popc(m));
		if (om)
			atomicAdd(&B.counters[CTR_TRAV_OVERFLOW], (uint32_t)__popc(om));
	}
	const uint32_t slot = __shfl_sync(0xffffffffu, base, 0) + __popc(m & ((1u << lane) - 1u));
	if (any && slot < cap)
	{
		B.rawA[slot] = p.x;
		B.rawB[slot] = p.y;
	}
}

// The subtrees under l and r for query q along the ropes, a lane on its own:
// where the stack has no room. Pairs are left to the whole warp, one node a
// step.
template <bool MW, bool LIMIT>
__device__ __forceinline__ void walk_ropes(WalkWarp& W, Buffers& B, uint32_t n, uint32_t cap, uint32_t limit, bool on,
	uint32_t l, uint32_t r, uint32_t q)
{
	const uint32_t inner = n - 1;
	uint32_t node = on ? l : SENT;
	const uint32_t stop = on ? __float_as_uint(__ldg(B.nodeHi + r).w) : SENT;
	// A depth-first walk meets each node at most once.
	for (uint32_t steps = 0; steps < 2u * n && __any_sync(0xffffffffu, node != stop); ++steps)
	{
		bool hit = false;
		uint32_t leaf = 0, pb = 0;
		if (node != stop)
		{
			if ((MW && B.nodeFirst[node] > W.last[q]) || !walk_visit<LIMIT>(W, B, q, limit))
				node = stop;
			else
			{
				const float4 lo = __ldg(B.nodeLo + node), hi = __ldg(B.nodeHi + node);
				const bool overlap = WalkBox(W, q).overlaps(lo, hi);
				hit = overlap && node >= inner;
				leaf = node - inner;
				pb = __float_as_uint(lo.w);
				node = __float_as_uint(overlap && !hit ? lo.w : hi.w);
			}
		}
		walk_record(W, B, cap, hit, q, leaf, pb);
	}
}

template <bool MW, bool LIMIT>
__global__ void k_traverse(DevScene S, Buffers B, uint32_t n, uint32_t leaves, uint32_t cap, uint32_t limit)
{
	extern __shared__ float4 walkShared[];
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	WalkWarp& W = reinterpret_cast<WalkWarp*>(walkShared)[warp];
	const uint32_t j = (blockIdx.x * (blockDim.x >> 5) + warp) * leaves + lane;
	const uint32_t inner = n - 1, nodes = 2u * n - 1u;
	const uint32_t below = (1u << lane) - 1u;
	uint32_t node = SENT;
	if (lane < leaves && j < n)
	{
		const float4 ql = __ldg(B.nodeLo + inner + j), qh = __ldg(B.nodeHi + inner + j);
		const uint32_t pa = __float_as_uint(ql.w);
		const uint2 da = __ldg(B.leafData + j);
		W.box[0][lane] = ql.x;
		W.box[1][lane] = ql.y;
		W.box[2][lane] = ql.z;
		W.box[3][lane] = qh.x;
		W.box[4][lane] = qh.y;
		W.box[5][lane] = qh.z;
		W.info[lane] = da.x;
		W.key[lane] = da.y;
		W.proxy[lane] = pa;
		if (S.fixLife[pa] != FIX_DEAD)
		{
			node = __float_as_uint(qh.w);
			W.last[lane] = MW ? B.worldEnd[S.bodyWorld[S.fixBody[pa]]] : 0xFFFFFFFFu;
		}
	}
	W.visits[lane] = W.found[lane] = 0;
	__syncwarp();
	const WalkBox box(W, lane);
	const uint32_t last = MW ? W.last[lane] : 0xFFFFFFFFu;
	uint32_t size = 0, hits = 0;
	auto push = [&](bool on, uint32_t l, uint32_t r, uint32_t q) {
		const uint32_t m = __ballot_sync(0xffffffffu, on);
		if (on)
		{
			const uint32_t at = size + __popc(m & below);
			W.left[at] = l;
			W.right[at] = r;
			W.query[at] = (uint8_t)q;
		}
		size += __popc(m);
	};
	auto found = [&](bool on, uint32_t leaf, uint32_t proxy, uint32_t q) {
		const uint32_t m = __ballot_sync(0xffffffffu, on);
		if (on)
		{
			const uint32_t at = hits + __popc(m & below);
			W.hitLeaf[at] = leaf;
			W.hitProxy[at] = proxy;
			W.hitQuery[at] = (uint8_t)q;
		}
		hits += __popc(m);
	};
	// The warp's leaves meet each node at most once each.
	const uint32_t most = nodes < (1u << 26) ? 64u * nodes : 0xFFFFFFFFu;
	for (uint32_t steps = 0;; ++steps)
	{
		if (steps > most)
		{
			if (lane == 0)
				atomicOr(&B.counters[CTR_STATUS], B3G_ST_WAIT_TIMEOUT);
			break;
		}
		if (size < 32u && __any_sync(0xffffffffu, node != SENT))
		{
			bool hit = false, enter = false;
			uint32_t x = 0, left = 0, right = 0;
			if (node != SENT)
			{
				x = node;
				if (x >= nodes)
				{
					atomicOr(&B.counters[CTR_STATUS], B3G_ST_WAIT_TIMEOUT);
					node = SENT;
				}
				else if ((MW && (x >= inner ? x - inner : x) > last) || !walk_visit<LIMIT>(W, B, lane, limit))
					node = SENT;
				else
				{
					const float4 lo = __ldg(B.nodeLo + x), hi = __ldg(B.nodeHi + x);
					if (x < inner)
						right = __ldg(B.nodeRight + x);
					const bool overlap = box.overlaps(lo, hi);
					hit = overlap && x >= inner;
					enter = overlap && x < inner;
					left = __float_as_uint(lo.w);
					node = __float_as_uint(hi.w);
				}
			}
			push(enter, left, right, lane);
			found(hit, x - inner, left, lane);
		}
		else if (size > 0)
		{
			const uint32_t take = min(size, 32u);
			const bool on = lane < take;
			size -= take;
			uint32_t l = 0, r = 0, q = 0;
			if (on)
			{
				l = W.left[size + lane];
				r = W.right[size + lane];
				q = W.query[size + lane];
			}
			__syncwarp();
			if (size + 64u > WALK_STACK)
			{
				walk_ropes<MW, LIMIT>(W, B, n, cap, limit, on, l, r, q);
				continue;
			}
			bool hitL = false, hitR = false, enterL = false, enterR = false;
			uint32_t ll = 0, lr = 0, rl = 0, rr = 0;
			if (on)
			{
				const float4 ll4 = __ldg(B.nodeLo + l), lh4 = __ldg(B.nodeHi + l);
				const float4 rl4 = __ldg(B.nodeLo + r), rh4 = __ldg(B.nodeHi + r);
				if (l < inner)
					lr = __ldg(B.nodeRight + l);
				if (r < inner)
					rr = __ldg(B.nodeRight + r);
				ll = __float_as_uint(ll4.w);
				rl = __float_as_uint(rl4.w);
				const WalkBox box(W, q);
				const bool okL = walk_visit<LIMIT>(W, B, q, limit) && box.overlaps(ll4, lh4);
				const bool okR = (!MW || (r >= inner ? r - inner : r) <= W.last[q]) && walk_visit<LIMIT>(W, B, q, limit) &&
					box.overlaps(rl4, rh4);
				hitL = okL && l >= inner;
				hitR = okR && r >= inner;
				enterL = okL && l < inner;
				enterR = okR && r < inner;
			}
			push(enterL, ll, lr, q);
			push(enterR, rl, rr, q);
			found(hitL, l - inner, ll, q);
			found(hitR, r - inner, rl, q);
		}
		else
			break;
		__syncwarp();
		while (hits >= 32u)
		{
			hits -= 32u;
			walk_record(W, B, cap, true, W.hitQuery[hits + lane], W.hitLeaf[hits + lane], W.hitProxy[hits + lane]);
			__syncwarp();
		}
	}
	const bool on = lane < hits;
	walk_record(W, B, cap, on, on ? W.hitQuery[lane] : 0u, on ? W.hitLeaf[lane] : 0u, on ? W.hitProxy[lane] : 0u);
}

// Scan in place.
__global__ void __launch_bounds__(SC_THREADS) k_scan_tiles(uint32_t* data, uint32_t n, unsigned long long* state,
	uint32_t* total, uint32_t* err)
{
	scan_tile(
		[=](uint32_t first, uint32_t* v) {
#pragma unroll
			for (int r = 0; r < SC_ITEMS; ++r)
				v[r] = first + r < n ? data[first + r] : 0u;
		},
		data, n, state, total, err);
}

} // namespace

// Words of scan state (u32) a scan of up to n entries needs in aux.
uint32_t scan_aux_words(uint32_t n)
{
	return 2u * (scan_tiles(n) + 1u);
}

void scan_exclusive(uint32_t* data, uint32_t n, uint32_t* aux, uint32_t* total, uint32_t* err, cudaStream_t s)
{
	const uint32_t tiles = scan_tiles(n);
	cudaMemsetAsync(aux, 0, sizeof(unsigned long long) * (tiles + 1u), s);
	k_scan_tiles<<<tiles ? tiles : 1u, SC_THREADS, 0, s>>>(data, n, reinterpret_cast<unsigned long long*>(aux), total, err);
}

// Stable sort of n (key, value) records by the low `bits` bits of the keys
// (the one-sweep passes of the broadphase sort). scratch holds
// radix_sort_scratch_words(n, bits) words. Returns the buffer pair holding
// the result: (keys, vals) or (keysTmp, valsTmp).
uint32_t radix_sort_scratch_words(uint32_t n, int bits)
{
	uint32_t passes = (uint32_t)(bits + 7) / 8;
	return 256u * (9u + passes * ((n + OS_TILE - 1) / OS_TILE));
}

bool radix_sort_pairs(unsigned long long* keys, uint32_t* vals, unsigned long long* keysTmp, uint32_t* valsTmp,
	uint32_t n, int bits, uint32_t* scratch, uint32_t* err, cudaStream_t s)
{
	SortShifts sh;
	sh.n = 0;
	for (int sft = 0; sft < bits && sh.n < 8; sft += 8)
		sh.s[sh.n++] = sft;
	if (n == 0 || sh.n == 0)
		return false;
	const uint32_t numTiles = (n + OS_TILE - 1) / OS_TILE;
	cudaMemsetAsync(scratch, 0, sizeof(uint32_t) * (9 * 256 + (size_t)sh.n * numTiles * 256), s);
	k_os_hist<<<min((n + 255) / 256, 148u * 4u), 256, 0, s>>>(keys, n, sh, scratch);
	k_os_scan<<<sh.n, 256, 0, s>>>(scratch);
	unsigned long long *kin = keys, *kout = keysTmp;
	uint32_t *vin = vals, *vout = valsTmp;
	for (int p = 0; p < sh.n; ++p)
	{
		k_onesweep<<<numTiles, OS_THREADS, 0, s>>>(kin, vin, kout, vout, n, sh.s[p], scratch + 256 * p,
			scratch + 9 * 256 + (size_t)p * numTiles * 256, scratch + 8 * 256 + p, err);
		std::swap(kin, kout);
		std::swap(vin, vout);
	}
	return kin != keys;
}

void launch_sync(b3g_ctx* c, cudaStream_t s)
{
	uint32_t n = c->nFixtures;
	if (n == 0)
		return;
	const size_t groups = std::max<size_t>(n, c->nBodies);
	// A pass that reuses the LBVH refits it from here (grow_leaf).
	const int grow = !c->treeRebuild && c->treeLeaves == n ? 1 : 0;
	k_sync<<<(uint32_t)((groups * SYNC_LANES + 127) / 128), 128, 0, s>>>(c->scene, c->buf, n, c->nBodies,
		c->creationPass ? 1 : 0, grow);
	if (c->creationPass)
		launch_mesh_fat(c, s);
}

// Kernels launched by launch_broadphase for the current scene (kept next to
// the launcher so the count follows its structure).
uint32_t broadphase_launches(const b3g_ctx* c)
{
	uint32_t n = c->nFixtures;
	if (n == 0)
		return 0;
	uint32_t wb = 0;
	while ((1u << wb) < c->nWorlds)
		++wb;
	uint32_t passes = 4 + (wb + 7) / 8;
	if (!c->treeRebuild)
		return 1; // the walk; the tree is refit by the sync kernel
	// bounds init, bounds, Morton; sort: histogram, scan, one kernel per
	// pass; build; leaves, refit; walk
	return 3 + (passes + 2) + (n > 1 ? 1 : 0) + 2 + 1;
}

void launch_broadphase(b3g_ctx* c, cudaStream_t s)
{
	Buffers& B = c->buf;
	int n = (int)c->nFixtures;
	c->treeLeaves = (uint32_t)n;
	if (n == 0)
		return;
	if (!c->treeRebuild)
	{
		// Same tree as the last pass, refit by k_sync (grow_leaf): walk.
		prof_mark(c, PM_SORTED, s);
		prof_mark(c, PM_BUILT, s);
		launch_traverse(c, s);
		prof_mark(c, PM_TRAVERSED, s);
		return;
	}
	int* bnd = (int*)B.sceneBounds;
	k_bounds_init<<<1, 32, 0, s>>>(bnd);
	k_bounds<<<min((n + 255) / 256, 148 * 4), 256, 0, s>>>(c->scene, B, (uint32_t)n, bnd);
	k_morton<<<(n + 255) / 256, 256, 0, s>>>(c->scene, B, (uint32_t)n, bnd);

	// Radix sort over the Morton bits and, for several worlds, the world bits.
	SortShifts sh;
	sh.n = 0;
	for (int sft = 0; sft < 32; sft += 8)
		sh.s[sh.n++] = sft;
	uint32_t wb = 0;
	while ((1u << wb) < c->nWorlds)
		++wb;
	for (uint32_t sft = 0; sft < wb; sft += 8)
		sh.s[sh.n++] = 32 + (int)sft;
	const uint32_t numTiles = ((uint32_t)n + OS_TILE - 1) / OS_TILE;
	// sortHist: digit counts (8 x 256), tile counters (256), tile status (8 x tiles x 256)
	uint32_t* ghist = B.sortHist;
	uint32_t* tileCounters = B.sortHist + 8 * 256;
	uint32_t* status = B.sortHist + 9 * 256;
	cudaMemsetAsync(B.sortHist, 0, sizeof(uint32_t) * (9 * 256 + (size_t)sh.n * numTiles * 256), s);
	k_os_hist<<<min((n + 255) / 256, 148 * 4), 256, 0, s>>>(B.keysA, (uint32_t)n, sh, ghist);
	k_os_scan<<<sh.n, 256, 0, s>>>(ghist);
	unsigned long long *kin = B.keysA, *kout = B.keysB;
	uint32_t *vin = B.valsA, *vout = B.valsB;
	for (int p = 0; p < sh.n; ++p)
	{
		k_onesweep<<<numTiles, OS_THREADS, 0, s>>>(kin, vin, kout, vout, (uint32_t)n, sh.s[p], ghist + 256 * p,
			status + (size_t)p * numTiles * 256, tileCounters + p, B.counters + CTR_STATUS);
		std::swap(kin, kout);
		std::swap(vin, vout);
	}
	if (kin != B.keysA)
	{
		cudaMemcpyAsync(B.keysA, kin, sizeof(unsigned long long) * n, cudaMemcpyDeviceToDevice, s);
		cudaMemcpyAsync(B.valsA, vin, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, s);
	}
	prof_mark(c, PM_SORTED, s);

	if (n > 1)
		k_build<<<(n - 1 + 255) / 256, 256, 0, s>>>(B, n);
	k_leaves<<<(n + 255) / 256, 256, 0, s>>>(c->scene, B, n);
	k_refit<<<(n + 255) / 256, 256, 0, s>>>(B, n);
	prof_mark(c, PM_BUILT, s);

	launch_traverse(c, s);
	prof_mark(c, PM_TRAVERSED, s);
}

// LBVH traversal of the tree built by this pass, with the tuned block size;
// CTR_RAW and CTR_TRAV_OVERFLOW start at 0. Re-running it on the same tree
// writes the same pairs.
void launch_traverse(b3g_ctx* c, cudaStream_t s)
{
	Buffers& B = c->buf;
	int n = (int)c->nFixtures;
	if (n == 0)
		return;
	const int tb = (int)c->tune.v[B3G_TUNE_TRAVERSE];
	// As few leaves a warp as leave the GPU 16 warps an SM, down to 4: 454
	// leaves take 15 us with 4 a warp and 26 with 16, 65,536 take 54 with 16
	// and 78 with 32; 370,000 take 104 with 32, 98 with 16 and 132 with 8.
	uint32_t leaves = 32;
	while (leaves > 4u && (uint32_t)n / leaves < 148u * 16u)
		leaves >>= 1;
	const uint32_t perBlock = leaves * (uint32_t)(tb / 32);
	const uint32_t blocks = ((uint32_t)n + perBlock - 1) / perBlock;
	const size_t smem = (size_t)(tb / 32) * sizeof(WalkWarp);
	auto* walk = c->nWorlds > 1 ? (c->walkLimit ? k_traverse<true, true> : k_traverse<true, false>)
								: (c->walkLimit ? k_traverse<false, true> : k_traverse<false, false>);
	walk<<<blocks, tb, smem, s>>>(c->scene, B, (uint32_t)n, leaves, c->cfg.max_contacts, c->walkLimit);
}

void carveout_broadphase()
{
	set_carveout({
		(const void*)k_sync, (const void*)k_bounds_init, (const void*)k_bounds, (const void*)k_morton,
		(const void*)k_os_hist, (const void*)k_os_scan, (const void*)k_onesweep, (const void*)k_build,
		(const void*)k_leaves, (const void*)k_refit, (const void*)k_traverse<false, false>,
		(const void*)k_traverse<false, true>, (const void*)k_traverse<true, false>,
		(const void*)k_traverse<true, true>, (const void*)k_scan_tiles});
}
