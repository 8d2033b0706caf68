// Warp-per-pair hull-hull narrowphase: b3CollideHulls with the feature cache
// (collide_hulls.cpp:355-534) and without it (collide_hulls.cpp:189-264).
//
// The 32 lanes of a warp share one contact. The separating-axis queries are
// spread over the lanes: face queries (sat.cpp:33-58) put faces on lanes and
// loop over the other hull's vertices for the support point; the edge query
// (sat.cpp:111-174) flattens the (edge1, edge2) double loop onto lanes after
// the per-edge data (both endpoints, edge vector and length, the two adjacent
// face normals of the Gauss map) is precomputed into shared memory. Every
// argmax is reduced with warp shuffles on (value, flattened index), keeping
// the larger value and, on equal values, the lower index - which is exactly
// the first maximum the reference's sequential "if (s > max)" loops select.
// The serial remainder (incident face clipping, polygon reduction, the cache
// decision tree) runs on lane 0.

#include "collide_common.cuh"

namespace {


struct EdgeRec
{
	float4 P; // xyz endpoint, w = |E|
	float4 E; // xyz edge vector
	float4 U; // xyz normal of the edge's face
	float4 V; // xyz normal of the twin's face
};

__device__ __forceinline__ V3 f3(float4 a) { return V3{a.x, a.y, a.z}; }

// First-maximum reduction across the warp on (value, index).
__device__ __forceinline__ void warp_argmax(float& v, uint32_t& idx)
{
	for (int o = 16; o > 0; o >>= 1)
	{
		float ov = __shfl_xor_sync(0xffffffffu, v, o);
		uint32_t oi = __shfl_xor_sync(0xffffffffu, idx, o);
		if (ov > v || (ov == v && oi < idx))
		{
			v = ov;
			idx = oi;
		}
	}
}

// b3QueryFaceSeparation(hull, hull) (sat.cpp:33-58).
__device__ void warp_query_faces(const XF& xf1, const HullRef& h1, const XF& xf2, const HullRef& h2,
	uint32_t lane, uint32_t& index, float& sep)
{
	XF xf = xmult(xf2, xf1);
	float best = -B3G_MAX_SCALAR;
	uint32_t bi = 0xFFFFFFFFu;
	// Few faces against many vertices (a triangle's two against a hull): the
	// vertices go on the lanes instead, one face after the other. A face costs
	// about 25 instructions of reduction then, and 12 per 32 vertices, where
	// a lane per face costs 12 per vertex: it pays from 3 faces and 12
	// vertices down and up. Measured on 13,870 items of 64-vertex hulls
	// against triangles, with the launch shape below: 140 -> 130 us.
	if (h1.fCnt <= 3 && h2.vCnt >= 12)
	{
		for (uint32_t i = 0; i < h1.fCnt; ++i)
		{
			PL plane = pmul(xf, hp(h1, i));
			V3 d = -plane.n;
			float sp = -INFINITY;
			uint32_t si = 0xFFFFFFFFu;
			for (uint32_t k = lane; k < h2.vCnt; k += 32)
			{
				float proj = dot(d, hv(h2, k));
				if (si == 0xFFFFFFFFu || proj > sp)
				{
					si = k;
					sp = proj;
				}
			}
			warp_argmax(sp, si);
			float s = pdist(hv(h2, si), plane);
			if (s > best)
			{
				best = s;
				bi = i;
			}
		}
		index = bi == 0xFFFFFFFFu ? 0u : bi;
		sep = best;
		return;
	}
	for (uint32_t i = lane; i < h1.fCnt; i += 32)
	{
		PL plane = pmul(xf, hp(h1, i));
		V3 d = -plane.n;
		uint32_t si = 0;
		float sp = dot(d, hv(h2, 0));
		for (uint32_t k = 1; k < h2.vCnt; ++k)
		{
			float proj = dot(d, hv(h2, k));
			if (proj > sp)
			{
				si = k;
				sp = proj;
			}
		}
		float s = pdist(hv(h2, si), plane);
		if (s > best)
		{
			best = s;
			bi = i;
		}
	}
	warp_argmax(best, bi);
	index = bi == 0xFFFFFFFFu ? 0u : bi;
	sep = best;
}

// b3IsMinkowskiFace (sat.cpp:60-71).
__device__ __forceinline__ bool is_minkowski_face(V3 A, V3 B, V3 BxA, V3 C, V3 D, V3 DxC)
{
	float ADC = dot(A, DxC);
	float BDC = dot(B, DxC);
	float CBA = dot(C, BxA);
	float DBA = dot(D, BxA);
	return CBA * DBA < 0.0f && ADC * BDC < 0.0f && CBA * BDC > 0.0f;
}

// b3Project(P1, Q1, E1, P2, E2, C1) (sat.cpp:73-109); L1 = |E1|, L2 = |E2|.
__device__ __forceinline__ float project_edges(V3 P1, V3 E1, float L1, V3 P2, V3 E2, float L2, V3 C1)
{
	if (L1 < B3G_LINEAR_SLOP)
		return -B3G_MAX_SCALAR;
	if (L2 < B3G_LINEAR_SLOP)
		return -B3G_MAX_SCALAR;
	const float kTol = 0.005f;
	V3 E1_x_E2 = cross(E1, E2);
	float L = len(E1_x_E2);
	if (L < (kTol * L1) * L2)
		return -B3G_MAX_SCALAR;
	V3 N = (1.0f / L) * E1_x_E2;
	if (dot(N, P1 - C1) < 0.0f)
		N = -N;
	return dot(N, P2 - P1);
}

__device__ __forceinline__ void edge_rec_1(EdgeRec& r, const XF& xf, const HullRef& h1, uint32_t i)
{
	uint4 e1 = h1.e[i], t1 = h1.e[i + 1];
	V3 P1 = xmul(xf, hv(h1, e1.x));
	V3 Q1 = xmul(xf, hv(h1, t1.x));
	V3 E1 = Q1 - P1;
	V3 U1 = rot(xf.q, hp(h1, e1.y).n);
	V3 V1 = rot(xf.q, hp(h1, t1.y).n);
	r.P = make_float4(P1.x, P1.y, P1.z, len(E1));
	r.E = make_float4(E1.x, E1.y, E1.z, 0.0f);
	r.U = make_float4(U1.x, U1.y, U1.z, 0.0f);
	r.V = make_float4(V1.x, V1.y, V1.z, 0.0f);
}

__device__ __forceinline__ void edge_rec_2(EdgeRec& r, const HullRef& h2, uint32_t j)
{
	uint4 e2 = h2.e[j], t2 = h2.e[j + 1];
	V3 P2 = hv(h2, e2.x);
	V3 Q2 = hv(h2, t2.x);
	V3 E2 = Q2 - P2;
	V3 U2 = hp(h2, e2.y).n;
	V3 V2 = hp(h2, t2.y).n;
	r.P = make_float4(P2.x, P2.y, P2.z, len(E2));
	r.E = make_float4(E2.x, E2.y, E2.z, 0.0f);
	r.U = make_float4(U2.x, U2.y, U2.z, 0.0f);
	r.V = make_float4(V2.x, V2.y, V2.z, 0.0f);
}

__device__ __forceinline__ float edge_pair_sep(const EdgeRec& a, const EdgeRec& b, V3 C1)
{
	V3 U1 = f3(a.U), V1 = f3(a.V), E1 = f3(a.E);
	V3 U2 = f3(b.U), V2 = f3(b.V), E2 = f3(b.E);
	if (!is_minkowski_face(U1, V1, -E1, -U2, -V2, -E2))
		return -INFINITY; // not a Minkowski face: never a candidate
	return project_edges(f3(a.P), E1, a.P.w, f3(b.P), E2, b.P.w, C1);
}

// Hulls with fewer unique edges than this on both sides share the pairs out
// flat over the lanes (both edge sets staged); otherwise the larger set sits
// on the lanes and only the smaller one is staged.
constexpr uint32_t SAT_FLAT_EDGES = 48;

// Edge records of shared memory one warp needs (maxUE: the most unique
// edges of any hull): both sets of a flat query (at most 2 maxUE, and at
// most 2 (SAT_FLAT_EDGES - 1)), or the smaller set of a broadcast one (at
// most maxUE).
__host__ __device__ __forceinline__ uint32_t sat_warp_recs(uint32_t maxUE)
{
	if (maxUE < SAT_FLAT_EDGES)
		return 2 * maxUE;
	return maxUE > 2 * (SAT_FLAT_EDGES - 1) ? maxUE : 2 * (SAT_FLAT_EDGES - 1);
}

// The warps that share one hull pair's edge query: this one is `part` of
// `parts`, they meet at barrier `bar` of their block, and slot[] holds one
// (separation, pair) per part in shared memory. The barrier has no limit: every
// warp of the pair comes to it or none does, since they run the same queries on
// the same values up to it.
struct EdgeParts
{
	uint32_t part, parts, bar;
	float2* slot;
};

// b3QueryEdgeSeparation(hull, hull) (sat.cpp:111-174). recs holds
// sat_warp_recs(maxUE) records.
__device__ void warp_query_edges(const XF& xf1, const HullRef& h1, const XF& xf2, const HullRef& h2,
	uint32_t lane, EdgeRec* recs, uint32_t maxUE, const EdgeParts& P, uint32_t& index1, uint32_t& index2, float& sep)
{
	XF xf = xmult(xf2, xf1);
	V3 C1 = xmul(xf, h1.centroid);
	uint32_t n1 = h1.eCnt / 2, n2 = h2.eCnt / 2;
	const bool flat = n1 < SAT_FLAT_EDGES && n2 < SAT_FLAT_EDGES;
	EdgeRec* r1 = recs;
	EdgeRec* r2 = recs + (flat ? n1 : 0);
	bool staged = n1 <= maxUE && n2 <= maxUE;
	if (staged && flat)
	{
		for (uint32_t i = lane; i < n1; i += 32)
			edge_rec_1(r1[i], xf, h1, 2 * i);
		for (uint32_t j = lane; j < n2; j += 32)
			edge_rec_2(r2[j], h2, 2 * j);
		__syncwarp();
	}
	float best = -B3G_MAX_SCALAR;
	uint32_t bk = 0xFFFFFFFFu;
	uint32_t total = n1 * n2;
	// Each lane keeps the first maximum in k = i n2 + j among the pairs it
	// tests (larger value, or equal value and smaller k; nothing at or below
	// the start value, as the serial loop's strict test), and warp_argmax
	// picks the first maximum over the lanes: the serial loop's answer,
	// whatever pairs a lane is given.
	auto keep = [&](float s, uint32_t k) {
		if (s > best || (s == best && bk != 0xFFFFFFFFu && k < bk))
		{
			best = s;
			bk = k;
		}
	};
	if (staged && !flat)
	{
		// Larger hull's edges on the lanes, held in registers; the other
		// hull's edges staged and read by all lanes at once (shared-memory
		// broadcast).
		const bool rows1 = n1 >= n2;
		const uint32_t nl = rows1 ? n1 : n2, nb = rows1 ? n2 : n1;
		EdgeRec* rb = recs;
		const uint32_t b0 = nb * P.part / P.parts, b1 = nb * (P.part + 1) / P.parts;
		for (uint32_t b = b0 + lane; b < b1; b += 32)
		{
			if (rows1)
				edge_rec_2(rb[b], h2, 2 * b);
			else
				edge_rec_1(rb[b], xf, h1, 2 * b);
		}
		__syncwarp();
		for (uint32_t base = 0; base < nl; base += 32)
		{
			const uint32_t l = base + lane;
			const bool valid = l < nl;
			EdgeRec mine;
			const uint32_t le = 2 * (valid ? l : 0);
			if (rows1)
				edge_rec_1(mine, xf, h1, le);
			else
				edge_rec_2(mine, h2, le);
			for (uint32_t b = b0; b < b1; ++b)
			{
				const EdgeRec other = rb[b];
				if (!valid)
					continue;
				const uint32_t i = rows1 ? l : b, j = rows1 ? b : l;
				keep(rows1 ? edge_pair_sep(mine, other, C1) : edge_pair_sep(other, mine, C1), i * n2 + j);
			}
		}
	}
	else
	{
		// (i, j) of k = i n2 + j, stepped without a division per pair.
		const uint32_t k0 = lane + 32 * P.part, step = 32 * P.parts;
		uint32_t i = n2 ? k0 / n2 : 0u, j = k0 - i * n2;
		for (uint32_t k = k0; k < total; k += step, j += step)
		{
			while (j >= n2)
			{
				j -= n2;
				++i;
			}
			float s;
			if (staged)
			{
				s = edge_pair_sep(r1[i], r2[j], C1);
			}
			else
			{
				EdgeRec a, b;
				edge_rec_1(a, xf, h1, 2 * i);
				edge_rec_2(b, h2, 2 * j);
				s = edge_pair_sep(a, b, C1);
			}
			keep(s, k);
		}
	}
	warp_argmax(best, bk);
	if (P.parts > 1)
	{
		// First maximum over the parts: as over the lanes.
		if (lane == 0)
			P.slot[P.part] = make_float2(best, __uint_as_float(bk));
		asm volatile("bar.sync %0, %1;" ::"r"(P.bar), "r"(32u * P.parts) : "memory");
		for (uint32_t q = 0; q < P.parts; ++q)
		{
			const float2 o = P.slot[q];
			const uint32_t ok = __float_as_uint(o.y);
			if (o.x > best || (o.x == best && ok < bk))
			{
				best = o.x;
				bk = ok;
			}
		}
	}
	if (bk == 0xFFFFFFFFu)
	{
		index1 = 0;
		index2 = 0;
	}
	else
	{
		index1 = 2 * (bk / n2);
		index2 = 2 * (bk % n2);
	}
	sep = best;
	__syncwarp();
}

// b3BuildEdgeContact (collide_hulls.cpp:30-73).
__device__ void build_edge_contact(DevManifold& m, const XF& xf1, uint32_t index1, const HullRef& h1,
	const XF& xf2, uint32_t index2, const HullRef& h2)
{
	uint4 e1 = h1.e[index1], t1 = h1.e[index1 + 1];
	V3 C1 = xmul(xf1, h1.centroid);
	V3 P1 = xmul(xf1, hv(h1, e1.x));
	V3 Q1 = xmul(xf1, hv(h1, t1.x));
	V3 E1 = Q1 - P1;
	uint4 e2 = h2.e[index2], t2 = h2.e[index2 + 1];
	V3 P2 = xmul(xf2, hv(h2, e2.x));
	V3 Q2 = xmul(xf2, hv(h2, t2.x));
	V3 E2 = Q2 - P2;
	V3 N = cross(E1, E2);
	normalize_inplace(N);
	if (dot(N, P1 - C1) < 0.0f)
		N = -N;
	V3 point1, point2;
	closest_on_segments(point1, point2, P1, Q1, P2, Q2);
	m.pointCount = 1;
	set_point(m.points[0], rotc(xf1.q, N), xmult(xf1, point1), xmult(xf2, point2));
	set_id(m.points[0], mkpair(index1, index1 + 1, index2, index2 + 1));
	m.points[0].edgeContact = 1;
}

// b3BuildFaceContact (collide_hulls.cpp:75-187) on one thread.
__device__ void build_face_contact(DevManifold& m, const XF& xf1, uint32_t index1, const HullRef& h1, float r1,
	const XF& xf2, const HullRef& h2, float r2, bool flipNormal, uint32_t* status)
{
	float totalRadius = r1 + r2;
	PL localPlane1 = hp(h1, index1);
	PL plane1 = pmul(xf1, localPlane1);
	V3 normal1 = rotc(xf2.q, plane1.n);
	uint32_t index2 = hull_support_face(h2, -normal1);
	Poly pa, pb;
	if (!build_polygon(pa, xf2, index2, h2))
	{
		atomicOr(status, B3G_ST_POLY_OVERFLOW);
		return;
	}
	bool ok;
	Poly* clip = clip_polygon_to_face_side_planes(pa, pb, xf1, totalRadius, index1, h1, ok);
	if (!ok)
	{
		atomicOr(status, B3G_ST_POLY_OVERFLOW);
		return;
	}
	if (clip->n == 0)
		return;
	CV poly1[B3G_MAX_POLY];
	uint32_t n1 = 0;
	uint32_t minIndex = 0;
	float minSep = B3G_MAX_SCALAR;
	for (uint32_t i = 0; i < clip->n; ++i)
	{
		V3 p = clip->v[i].pos;
		float s = pdist(p, plane1);
		if (s <= totalRadius)
		{
			if (s < minSep)
			{
				minIndex = n1;
				minSep = s;
			}
			poly1[n1].pos = pclosest(p, plane1);
			poly1[n1].clipIndex = i;
			++n1;
		}
	}
	if (n1 == 0)
		return;
	V3 normal = plane1.n;
	V3 oriented = flipNormal ? -normal : normal;
	CV red[4];
	uint32_t cnt = reduce_polygon(red, poly1, n1, oriented, minIndex);
	for (uint32_t i = 0; i < cnt; ++i)
	{
		const ClipV& v2 = clip->v[red[i].clipIndex];
		V3 v1 = pclosest(v2.pos, plane1);
		DevPoint& mp = m.points[i];
		if (flipNormal)
		{
			set_point(mp, rotc(xf2.q, oriented), xmult(xf2, v2.pos), xmult(xf1, v1));
			set_id(mp, mkpair(v2.pair.inEdge2, v2.pair.outEdge2, v2.pair.inEdge1, v2.pair.outEdge1));
		}
		else
		{
			set_point(mp, rotc(xf1.q, oriented), xmult(xf1, v1), xmult(xf2, v2.pos));
			set_id(mp, v2.pair);
		}
		mp.edgeContact = 0;
	}
	m.pointCount = cnt;
}

// Shared-memory buffers of one warp for warp_build_face_contact: two clip
// polygons (ping-pong) and the kept points of the reference face.
struct WarpClip
{
	ClipV a[B3G_MAX_POLY];
	ClipV b[B3G_MAX_POLY];
	CV kept[B3G_MAX_POLY];
};

// Shared memory of one warp in the hull kernels: the edge records of the edge
// query, then (the query done) the clip buffers of the face contact.
__host__ __device__ __forceinline__ size_t sat_warp_bytes(uint32_t maxUE)
{
	size_t recs = (size_t)sat_warp_recs(maxUE) * sizeof(EdgeRec);
	return recs > sizeof(WarpClip) ? recs : sizeof(WarpClip);
}

// The same where the second hull is a triangle: it has 3 edges, so a flat edge
// query holds at most SAT_FLAT_EDGES - 1 + 3 records and a broadcast one 3,
// however large the hulls are.
__host__ __device__ __forceinline__ size_t sat_triangle_warp_bytes()
{
	size_t recs = (SAT_FLAT_EDGES + 2) * sizeof(EdgeRec);
	return recs > sizeof(WarpClip) ? recs : sizeof(WarpClip);
}

// Exclusive prefix sum of v over the warp; *total receives the sum.
__device__ __forceinline__ uint32_t warp_excl_scan(uint32_t v, uint32_t lane, uint32_t& total)
{
	uint32_t x = v;
	for (int o = 1; o < 32; o <<= 1)
	{
		uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
		if (lane >= (uint32_t)o)
			x += y;
	}
	total = __shfl_sync(0xffffffffu, x, 31);
	return x - v;
}

// b3ClipPolygonToPlane (clip.cpp:101-150) on the warp: vertex i (lanes take i
// and i + 32) emits what the sequential loop emits at step i — v2, the
// intersection, or both — at the place a prefix sum of the emit counts gives,
// so out holds the sequential loop's polygon, same values, same order. d1 of
// step i is the distance of vertex i - 1 (n - 1 for step 0), the value the
// loop carries over. Returns the new vertex count, or B3G_MAX_POLY + 1 when
// the polygon would outgrow the buffer (the loop fails there too).
__device__ uint32_t warp_clip_polygon_to_plane(ClipV* out, const ClipV* in, uint32_t n, PL plane, uint32_t edge,
	uint32_t lane)
{
	uint32_t base = 0;
	for (uint32_t i0 = 0; i0 < n; i0 += 32)
	{
		const uint32_t i = i0 + lane;
		uint32_t cnt = 0;
		ClipV v1, v2;
		float d1 = 0.0f, d2 = 0.0f;
		if (i < n)
		{
			v2 = in[i];
			v1 = in[i == 0 ? n - 1 : i - 1];
			d2 = pdist(v2.pos, plane);
			d1 = pdist(v1.pos, plane);
			if (d1 <= 0.0f && d2 <= 0.0f)
				cnt = 1;
			else if (d1 <= 0.0f && d2 > 0.0f)
				cnt = 1;
			else if (d1 > 0.0f && d2 <= 0.0f)
				cnt = 2;
		}
		uint32_t total;
		const uint32_t o = base + warp_excl_scan(cnt, lane, total);
		base += total;
		// Writes past the buffer are skipped; the count reports the overflow.
		if (cnt != 0 && o + cnt <= B3G_MAX_POLY)
		{
			if (d1 <= 0.0f && d2 <= 0.0f)
				out[o] = v2;
			else if (d1 <= 0.0f && d2 > 0.0f)
			{
				float fraction = d1 / (d1 - d2);
				out[o].pos = v1.pos + fraction * (v2.pos - v1.pos);
				out[o].pair = mkpair(edge, B3G_NULL_EDGE, v1.pair.outEdge2, B3G_NULL_EDGE);
			}
			else
			{
				float fraction = d1 / (d1 - d2);
				out[o].pos = v1.pos + fraction * (v2.pos - v1.pos);
				out[o].pair = mkpair(B3G_NULL_EDGE, edge, B3G_NULL_EDGE, v2.pair.inEdge2);
				out[o + 1] = v2;
			}
		}
	}
	__syncwarp();
	return base > B3G_MAX_POLY ? B3G_MAX_POLY + 1 : base;
}

// b3BuildFaceContact (collide_hulls.cpp:75-187) on the warp, with W in
// shared memory: the incident polygon (lane 0 walks the face loop), the
// clipping against the reference face's side planes (warp_clip_polygon_to_
// plane), the kept points and the deepest of them (first minimum: smaller
// separation, on ties the earlier point), then the reduction to four points
// and the manifold on lane 0. Same operations and order as build_face_contact;
// returns the point count on every lane.
__device__ __noinline__ uint32_t warp_build_face_contact(DevManifold& m, const XF& xf1, uint32_t index1, const HullRef& h1,
	float r1, const XF& xf2, const HullRef& h2, float r2, bool flipNormal, uint32_t* status, uint32_t lane,
	WarpClip& W)
{
	float totalRadius = r1 + r2;
	PL localPlane1 = hp(h1, index1);
	PL plane1 = pmul(xf1, localPlane1);
	V3 normal1 = rotc(xf2.q, plane1.n);
	uint32_t index2 = hull_support_face(h2, -normal1);
	uint32_t n = 0;
	if (lane == 0)
	{
		uint32_t begin = h2.f[index2];
		uint32_t edge = begin;
		do
		{
			if (n >= B3G_MAX_POLY)
			{
				n = B3G_MAX_POLY + 1;
				break;
			}
			ClipV& cv = W.a[n++];
			cv.pos = xmul(xf2, hv(h2, he_origin(h2, edge)));
			cv.pair = mkpair(B3G_NULL_EDGE, B3G_NULL_EDGE, he_prev(h2, edge), edge);
			edge = he_next(h2, edge);
		} while (edge != begin);
	}
	n = __shfl_sync(0xffffffffu, n, 0);
	__syncwarp();
	bool ok = n <= B3G_MAX_POLY;
	ClipV* in = W.a;
	ClipV* out = W.b;
	if (ok)
	{
		uint32_t begin = h1.f[index1];
		uint32_t edge = begin;
		uint32_t guard = 0;
		do
		{
			if (++guard > h1.eCnt)
			{
				ok = false;
				break;
			}
			PL plane = hull_edge_side_plane(h1, edge);
			plane.d += totalRadius;
			PL cp = pmul(xf1, plane);
			uint32_t nn = warp_clip_polygon_to_plane(out, in, n, cp, edge, lane);
			if (nn > B3G_MAX_POLY)
			{
				ok = false;
				break;
			}
			ClipV* t = in;
			in = out;
			out = t;
			n = nn;
			if (n == 0)
				break;
			edge = he_next(h1, edge);
		} while (edge != begin);
	}
	if (!ok)
	{
		if (lane == 0)
			atomicOr(status, B3G_ST_POLY_OVERFLOW);
		return 0;
	}
	if (n == 0)
		return 0;
	// Kept points (separation within the radius), projected on the reference
	// plane, in order; the first of the smallest separation.
	uint32_t base = 0;
	float bestS = B3G_MAX_SCALAR;
	uint32_t bestK = 0xFFFFFFFFu;
	for (uint32_t i0 = 0; i0 < n; i0 += 32)
	{
		const uint32_t i = i0 + lane;
		bool keep = false;
		V3 p{0.0f, 0.0f, 0.0f};
		float sep = 0.0f;
		if (i < n)
		{
			p = in[i].pos;
			sep = pdist(p, plane1);
			keep = sep <= totalRadius;
		}
		uint32_t total;
		const uint32_t k = base + warp_excl_scan(keep ? 1u : 0u, lane, total);
		if (keep)
		{
			W.kept[k].pos = pclosest(p, plane1);
			W.kept[k].clipIndex = i;
			if (sep < bestS || (sep == bestS && k < bestK))
			{
				bestS = sep;
				bestK = k;
			}
		}
		base += total;
	}
	const uint32_t n1 = base;
	if (n1 == 0)
		return 0;
	for (int o = 16; o > 0; o >>= 1)
	{
		float os = __shfl_xor_sync(0xffffffffu, bestS, o);
		uint32_t ok2 = __shfl_xor_sync(0xffffffffu, bestK, o);
		if (os < bestS || (os == bestS && ok2 < bestK))
		{
			bestS = os;
			bestK = ok2;
		}
	}
	__syncwarp();
	uint32_t cnt = 0;
	if (lane == 0)
	{
		V3 normal = plane1.n;
		V3 oriented = flipNormal ? -normal : normal;
		CV red[4];
		cnt = reduce_polygon(red, W.kept, n1, oriented, bestK);
		for (uint32_t i = 0; i < cnt; ++i)
		{
			const ClipV& v2 = in[red[i].clipIndex];
			V3 v1 = pclosest(v2.pos, plane1);
			DevPoint& mp = m.points[i];
			if (flipNormal)
			{
				set_point(mp, rotc(xf2.q, oriented), xmult(xf2, v2.pos), xmult(xf1, v1));
				set_id(mp, mkpair(v2.pair.inEdge2, v2.pair.outEdge2, v2.pair.inEdge1, v2.pair.outEdge1));
			}
			else
			{
				set_point(mp, rotc(xf1.q, oriented), xmult(xf1, v1), xmult(xf2, v2.pos));
				set_id(mp, v2.pair);
			}
			mp.edgeContact = 0;
		}
		m.pointCount = cnt;
	}
	cnt = __shfl_sync(0xffffffffu, cnt, 0);
	__syncwarp();
	return cnt;
}

// b3RebuildEdgeContact (collide_hulls.cpp:266-321).
__device__ void rebuild_edge_contact(DevManifold& m, const XF& xf1, uint32_t index1, const HullRef& h1,
	const XF& xf2, uint32_t index2, const HullRef& h2)
{
	uint4 e1 = h1.e[index1], t1 = h1.e[index1 + 1];
	V3 C1 = xmul(xf1, h1.centroid);
	V3 P1 = xmul(xf1, hv(h1, e1.x));
	V3 Q1 = xmul(xf1, hv(h1, t1.x));
	V3 E1 = Q1 - P1;
	uint4 e2 = h2.e[index2], t2 = h2.e[index2 + 1];
	V3 P2 = xmul(xf2, hv(h2, e2.x));
	V3 Q2 = xmul(xf2, hv(h2, t2.x));
	V3 E2 = Q2 - P2;
	V3 point1, point2;
	closest_on_segments(point1, point2, P1, Q1, P2, Q2);
	float w1[3], w2[3];
	barycentric_segment(w1, P2, Q2, point1);
	barycentric_segment(w2, P1, Q1, point2);
	if (w1[1] > 0.0f && w1[1] <= w1[2] && w2[1] > 0.0f && w2[1] <= w2[2])
	{
		V3 N = cross(E1, E2);
		normalize_inplace(N);
		if (dot(N, P1 - C1) < 0.0f)
			N = -N;
		m.pointCount = 1;
		set_point(m.points[0], rotc(xf1.q, N), xmult(xf1, point1), xmult(xf2, point2));
		set_id(m.points[0], mkpair(index1, index1 + 1, index2, index2 + 1));
		m.points[0].edgeContact = 1;
	}
}

// The orientation test of b3RebuildFaceContact (collide_hulls.cpp:323-353).
__device__ __forceinline__ bool face_contact_persists(const XF& xf1, const XF& xf2, const XF& xf01, const XF& xf02)
{
	Q4 q01 = xf01.q, q1 = xf1.q;
	Q4 q02 = xf02.q, q2 = xf2.q;
	Q4 dq0 = qmul(conj(q01), q02);
	Q4 dq = qmul(conj(q1), q2);
	Q4 q = qmul(conj(dq0), dq);
	const float kCosTol = 0.995f;
	return fabsr(q.s) > kCosTol;
}

enum
{
	CT_EMPTY = 0,
	CT_SEPARATION = 1,
	CT_OVERLAP = 2
};
enum
{
	FT_EDGES = 0,
	FT_FACE1 = 1,
	FT_FACE2 = 2
};

// b3FeatureCache::ReadEdges (sat.cpp:226-281).
__device__ uint32_t read_edges(const XF& xf1, const HullRef& h1, const XF& xf2, const HullRef& h2, uint32_t i,
	uint32_t j, float totalRadius)
{
	XF xf = xmult(xf2, xf1);
	V3 C1 = xmul(xf, h1.centroid);
	EdgeRec a, b;
	edge_rec_1(a, xf, h1, i);
	edge_rec_2(b, h2, j);
	V3 U1 = f3(a.U), V1 = f3(a.V), E1 = f3(a.E);
	V3 U2 = f3(b.U), V2 = f3(b.V), E2 = f3(b.E);
	if (is_minkowski_face(U1, V1, -E1, -U2, -V2, -E2))
	{
		float s = project_edges(f3(a.P), E1, a.P.w, f3(b.P), E2, b.P.w, C1);
		return s > totalRadius ? CT_SEPARATION : CT_OVERLAP;
	}
	return CT_EMPTY;
}

struct HullCtx
{
	XF xf1, xf2, xf01, xf02;
	HullRef h1, h2;
	float r1, r2;
	EdgeRec* recs;
	uint32_t maxUE;
	uint32_t* status;
	WarpClip* clip; // the warp's shared clip buffers
	EdgeParts parts;
};

// Lane 0 builds, the warp learns the point count.
// Face contact on the warp (H.clip: the warp's shared clip buffers); every
// lane learns the point count.
__device__ uint32_t face_contact_all(DevManifold& m, const HullCtx& H, bool flip, uint32_t index, uint32_t lane)
{
	if (flip)
		return warp_build_face_contact(m, H.xf2, index, H.h2, H.r2, H.xf1, H.h1, H.r1, true, H.status, lane, *H.clip);
	return warp_build_face_contact(m, H.xf1, index, H.h1, H.r1, H.xf2, H.h2, H.r2, false, H.status, lane, *H.clip);
}

// b3CollideHulls without cache (collide_hulls.cpp:189-264).
__device__ void collide_hulls_nocache(DevManifold& m, const HullCtx& H, uint32_t lane)
{
	float totalRadius = H.r1 + H.r2;
	uint32_t fi1, fi2, ei1, ei2;
	float fs1, fs2, es;
	warp_query_faces(H.xf1, H.h1, H.xf2, H.h2, lane, fi1, fs1);
	if (fs1 > totalRadius)
		return;
	warp_query_faces(H.xf2, H.h2, H.xf1, H.h1, lane, fi2, fs2);
	if (fs2 > totalRadius)
		return;
	warp_query_edges(H.xf1, H.h1, H.xf2, H.h2, lane, H.recs, H.maxUE, H.parts, ei1, ei2, es);
	if (es > totalRadius)
		return;
	const float kRelEdgeTol = 0.90f;
	const float kRelFaceTol = 0.98f;
	const float kAbsTol = 0.5f * B3G_LINEAR_SLOP;
	uint32_t pc;
	if (es > kRelEdgeTol * fmaxr(fs1, fs2) + kAbsTol)
	{
		if (lane == 0)
			build_edge_contact(m, H.xf1, ei1, H.h1, H.xf2, ei2, H.h2);
		pc = 1;
	}
	else if (fs2 > kRelFaceTol * fs1 + kAbsTol)
		pc = face_contact_all(m, H, true, fi2, lane);
	else
		pc = face_contact_all(m, H, false, fi1, lane);
	if (pc > 0)
		return;
	if (es > fmaxr(fs1, fs2))
	{
		if (lane == 0)
			build_edge_contact(m, H.xf1, ei1, H.h1, H.xf2, ei2, H.h2);
	}
	else if (fs2 > fs1)
		face_contact_all(m, H, true, fi2, lane);
	else
		face_contact_all(m, H, false, fi1, lane);
}

// Thread-level b3FeatureCache::ReadFace (sat.cpp:209-224).
__device__ uint32_t read_face_thread(const XF& xf1, const HullRef& h1, const XF& xf2, const HullRef& h2,
	uint32_t index1, float totalRadius)
{
	XF xf = xmult(xf2, xf1);
	PL plane = pmul(xf, hp(h1, index1));
	uint32_t si = hull_support_vertex(h2, -plane.n);
	float s = pdist(hv(h2, si), plane);
	return s > totalRadius ? CT_SEPARATION : CT_OVERLAP;
}

// Warp-aggregated append of c to a list (the calling lanes of the warp).
__device__ __forceinline__ void warp_append(uint32_t* list, uint32_t* count, uint32_t c)
{
	uint32_t mask = __activemask();
	uint32_t lane = threadIdx.x & 31;
	uint32_t leader = __ffs(mask) - 1;
	uint32_t base = 0;
	if (lane == leader)
		base = atomicAdd(count, (uint32_t)__popc(mask));
	base = __shfl_sync(mask, base, leader);
	list[base + __popc(mask & ((1u << lane) - 1u))] = c;
}

// The SAT half of b3CollideHullsCache (collide_hulls.cpp:417-515), one warp
// per contact. cache is uniform across the warp; m is written by lane 0.
__device__ void sat_after_miss(DevManifold& m, const HullCtx& H, uint4& cache, uint32_t lane)
{
	float totalRadius = H.r1 + H.r2;
	uint32_t fi1, fi2, ei1, ei2;
	float fs1, fs2, es;
	warp_query_faces(H.xf1, H.h1, H.xf2, H.h2, lane, fi1, fs1);
	if (fs1 > totalRadius)
	{
		cache = make_uint4(CT_SEPARATION, FT_FACE1, fi1, fi1);
		return;
	}
	warp_query_faces(H.xf2, H.h2, H.xf1, H.h1, lane, fi2, fs2);
	if (fs2 > totalRadius)
	{
		cache = make_uint4(CT_SEPARATION, FT_FACE2, fi2, fi2);
		return;
	}
	warp_query_edges(H.xf1, H.h1, H.xf2, H.h2, lane, H.recs, H.maxUE, H.parts, ei1, ei2, es);
	if (es > totalRadius)
	{
		cache = make_uint4(CT_SEPARATION, FT_EDGES, ei1, ei2);
		return;
	}
	if (H.parts.part != 0)
		return; // the contact is the first part's
	const float kRelEdgeTol = 0.90f;
	const float kRelFaceTol = 0.98f;
	const float kAbsTol = 0.5f * B3G_LINEAR_SLOP;
	if (es > kRelEdgeTol * fmaxr(fs1, fs2) + kAbsTol)
	{
		if (lane == 0)
			build_edge_contact(m, H.xf1, ei1, H.h1, H.xf2, ei2, H.h2);
		cache = make_uint4(CT_OVERLAP, FT_EDGES, ei1, ei2);
		return;
	}
	if (fs2 > kRelFaceTol * fs1 + kAbsTol)
	{
		if (face_contact_all(m, H, true, fi2, lane) > 0)
		{
			cache = make_uint4(CT_OVERLAP, FT_FACE2, fi2, fi2);
			return;
		}
	}
	else
	{
		if (face_contact_all(m, H, false, fi1, lane) > 0)
		{
			cache = make_uint4(CT_OVERLAP, FT_FACE1, fi1, fi1);
			return;
		}
	}
	// Heuristic failed. Fallback.
	if (es > fmaxr(fs1, fs2))
	{
		if (lane == 0)
			build_edge_contact(m, H.xf1, ei1, H.h1, H.xf2, ei2, H.h2);
		cache = make_uint4(CT_OVERLAP, FT_EDGES, ei1, ei2);
		return;
	}
	if (fs2 > fs1)
	{
		if (face_contact_all(m, H, true, fi2, lane) > 0)
			cache = make_uint4(CT_OVERLAP, FT_FACE2, fi2, fi2);
	}
	else
	{
		if (face_contact_all(m, H, false, fi1, lane) > 0)
			cache = make_uint4(CT_OVERLAP, FT_FACE1, fi1, fi1);
	}
}

__device__ __forceinline__ void load_hull_ctx(const NPArgs& a, uint32_t c, HullCtx& H)
{
	uint32_t fa = a.pairA[c], fb = a.pairB[c];
	uint32_t ba = a.S.fixBody[fa], bb = a.S.fixBody[fb];
	H.xf1 = a.exA ? load_xf7(a.exA + 7 * (size_t)c) : body_xf(a.S, ba);
	H.xf2 = a.exB ? load_xf7(a.exB + 7 * (size_t)c) : body_xf(a.S, bb);
	H.xf01 = a.ex0A ? load_xf7(a.ex0A + 7 * (size_t)c) : body_xf0(a.S, ba);
	H.xf02 = a.ex0B ? load_xf7(a.ex0B + 7 * (size_t)c) : body_xf0(a.S, bb);
	H.h1 = hull_ref(a.S, a.S.fixHull[fa]);
	H.h2 = hull_ref(a.S, a.S.fixHull[fb]);
	H.r1 = a.S.fixParams[3 * fa].x;
	H.r2 = a.S.fixParams[3 * fb].x;
	H.status = a.status;
	H.recs = nullptr;
	H.maxUE = 0;
	H.clip = nullptr;
	H.parts = EdgeParts{0, 1, 0, nullptr};
}

constexpr int PROBE_THREADS = 128;
constexpr int PROBE_BLOCKS = 4;
static_assert(CLIP_SLOTS == 8, "with 16 slots the rings fill the SM's shared memory: three contexts at once took 415 us a "
	"pass of 65,536 mixed bodies and 879 of 512 worlds, with 8 they take 392 and 831");

// A thread's clip polygon: a ring of vertices in shared memory, one column of
// words per thread. A vertex's edge pair takes two words of two 16-bit edges
// (0xFFFF: none).
struct ClipRings
{
	float x[CLIP_SLOTS][PROBE_THREADS], y[CLIP_SLOTS][PROBE_THREADS], z[CLIP_SLOTS][PROBE_THREADS];
	uint32_t pair1[CLIP_SLOTS][PROBE_THREADS], pair2[CLIP_SLOTS][PROBE_THREADS];

	__device__ __forceinline__ V3 pos(uint32_t i) const
	{
		const uint32_t s = i % CLIP_SLOTS, t = threadIdx.x;
		return V3{x[s][t], y[s][t], z[s][t]};
	}
	__device__ __forceinline__ void put(uint32_t i, V3 p, uint32_t p1, uint32_t p2)
	{
		const uint32_t s = i % CLIP_SLOTS, t = threadIdx.x;
		x[s][t] = p.x;
		y[s][t] = p.y;
		z[s][t] = p.z;
		pair1[s][t] = p1;
		pair2[s][t] = p2;
	}
};
__device__ __forceinline__ uint32_t ring_edges(uint32_t in, uint32_t out) { return in | out << 16; }
__device__ __forceinline__ uint32_t ring_edge(uint32_t e) { return e == 0xFFFFu ? B3G_NULL_EDGE : e; }

// Leaves a contact that its cache does not resolve to the SAT kernel.
__device__ __forceinline__ void probe_miss(const NPArgs& a, uint32_t c, uint4 cache)
{
	a.cache[c] = cache;
	warp_append(a.missList, a.missCount, c);
}
// ... flushed: the feature fields stay as ReadState left them.
__device__ __forceinline__ void probe_flush(const NPArgs& a, uint32_t c, uint4 cache)
{
	cache.x = CT_EMPTY;
	probe_miss(a, c, cache);
}

// b3BuildFaceContact (collide_hulls.cpp:75-187) of a cached face, a contact
// per lane; live: the lane's contact is its own (the others repeat one of
// them and write nothing). The warp takes each side plane and each vertex in
// step, over the largest polygon of its lanes.
__device__ void rebuild_faces(const NPArgs& a, uint32_t c, bool live, ClipRings& R)
{
	uint4 cache = a.prevCache[a.prevIndex[c]];
	HullCtx H;
	load_hull_ctx(a, c, H);
	const bool flip = cache.y == FT_FACE2;
	const XF xf1 = flip ? H.xf2 : H.xf1, xf2 = flip ? H.xf1 : H.xf2;
	const HullRef h1 = flip ? H.h2 : H.h1, h2 = flip ? H.h1 : H.h2;
	const float totalRadius = (flip ? H.r2 : H.r1) + (flip ? H.r1 : H.r2);
	const uint32_t index1 = cache.z;
	const PL plane1 = pmul(xf1, hp(h1, index1));
	uint32_t head = 0, cnt = 0;
	bool failed = false; // the polygon outgrows the ring: not with hulls that ring_holds
	{
		// b3BuildPolygon (clip.cpp:33-58).
		V3 normal1 = rotc(xf2.q, plane1.n);
		const uint32_t begin = h2.f[hull_support_face(h2, -normal1)];
		uint32_t edge = begin;
		do
		{
			failed = cnt == CLIP_SLOTS;
			if (failed)
				break;
			const uint4 e = h2.e[edge];
			R.put(cnt++, xmul(xf2, hv(h2, e.x)), ~0u, ring_edges(e.z, edge));
			edge = e.w;
		} while (edge != begin);
	}
	__syncwarp();
	// b3ClipPolygonToFaceSidePlanes (clip.cpp:244-281), b3ClipPolygonToPlane
	// (clip.cpp:101-150): vertices leave the ring's head and the clipped
	// polygon grows behind its tail.
	const uint32_t begin = h1.f[index1];
	uint32_t edge = begin, guard = 0;
	bool run = !failed;
	while (__any_sync(0xffffffffu, run))
	{
		PL cp = plane1;
		V3 p1 = plane1.n;
		float d1 = 0.0f;
		uint32_t out1 = 0, n = 0, outN = 0;
		const uint32_t tail = head + cnt;
		if (run && ++guard > h1.eCnt)
		{
			failed = true; // face loops are validated on upload; never loop forever
			run = false;
		}
		if (run)
		{
			PL plane = hull_edge_side_plane(h1, edge);
			plane.d += totalRadius;
			cp = pmul(xf1, plane);
			n = cnt;
			p1 = R.pos(tail - 1);
			out1 = R.pair2[(tail - 1) % CLIP_SLOTS][threadIdx.x] >> 16;
			d1 = pdist(p1, cp);
		}
		const uint32_t most = __reduce_max_sync(0xffffffffu, n);
		for (uint32_t i = 0; i < most; ++i)
		{
			if (i < n)
			{
				const uint32_t s = (head + i) % CLIP_SLOTS;
				const V3 p2 = R.pos(s);
				const uint32_t e1 = R.pair1[s][threadIdx.x], e2 = R.pair2[s][threadIdx.x];
				const float d2 = pdist(p2, cp);
				const bool leaves = d1 <= 0.0f && d2 > 0.0f, enters = d1 > 0.0f && d2 <= 0.0f;
				const bool stays = d1 <= 0.0f && d2 <= 0.0f;
				const uint32_t adds = (leaves || enters ? 1u : 0u) + (enters || stays ? 1u : 0u);
				if (outN + adds + (n - i - 1) > CLIP_SLOTS)
				{
					failed = true;
					run = false;
					n = 0;
				}
				else
				{
					if (leaves || enters)
					{
						const float fraction = d1 / (d1 - d2);
						R.put(tail + outN++, p1 + fraction * (p2 - p1),
							leaves ? ring_edges(edge, 0xFFFFu) : ring_edges(0xFFFFu, edge),
							leaves ? ring_edges(out1, 0xFFFFu) : ring_edges(0xFFFFu, e2 & 0xFFFFu));
					}
					if (enters || stays)
						R.put(tail + outN++, p2, e1, e2);
				}
				p1 = p2;
				d1 = d2;
				out1 = e2 >> 16;
			}
			__syncwarp();
		}
		if (run)
		{
			head = tail;
			cnt = outN;
			edge = he_next(h1, edge);
			run = cnt > 0 && edge != begin;
		}
	}
	if (failed)
		cnt = 0;
	// The vertices on or behind the reference face, moved up to the head.
	uint32_t n1 = 0, minIndex = 0;
	float minSep = B3G_MAX_SCALAR;
	for (uint32_t i = 0; i < cnt; ++i)
	{
		const uint32_t s = (head + i) % CLIP_SLOTS;
		const V3 p = R.pos(s);
		const float sep = pdist(p, plane1);
		if (sep <= totalRadius)
		{
			if (sep < minSep)
			{
				minIndex = n1;
				minSep = sep;
			}
			R.put(head + n1, p, R.pair1[s][threadIdx.x], R.pair2[s][threadIdx.x]);
			++n1;
		}
	}
	__syncwarp();
	// b3ReducePolygon (cluster.cpp:59-200) of their projections on the face:
	// o[k] is the projection of vertex at[k].
	auto get = [&](uint32_t k) { return pclosest(R.pos(head + k), plane1); };
	const V3 oriented = flip ? -plane1.n : plane1.n;
	V3 o[4];
	uint32_t at[4];
	uint32_t pc, sorted;
	if (n1 <= 4)
	{
#pragma unroll
		for (uint32_t k = 0; k < 4; ++k)
		{
			at[k] = k;
			o[k] = k < n1 ? get(k) : oriented;
		}
		pc = sorted = n1;
	}
	else
	{
		pc = 1;
		sorted = 0;
		at[0] = minIndex;
		at[1] = at[2] = at[3] = 0;
		o[0] = get(minIndex);
		o[1] = o[2] = o[3] = o[0];
		float mx = -B3G_MAX_SCALAR;
		for (uint32_t i = 0; i < n1; ++i)
		{
			if (i == at[0])
				continue;
			const V3 v = get(i) - o[0];
			const float dd = dot(v, v);
			if (dd > mx)
			{
				mx = dd;
				at[1] = i;
			}
		}
		if (!(mx < B3G_EPSILON * B3G_EPSILON))
		{
			pc = 2;
			o[1] = get(at[1]);
			mx = -B3G_MAX_SCALAR;
			for (uint32_t i = 0; i < n1; ++i)
			{
				if (i == at[0] || i == at[1])
					continue;
				const V3 nn = cross(o[1] - o[0], get(i) - o[0]);
				const float a2 = fabsr(dot(nn, oriented));
				if (a2 > mx)
				{
					mx = a2;
					at[2] = i;
				}
			}
			const float kAreaTol = 0.01f;
			if (!(mx < 2.0f * kAreaTol))
			{
				pc = 3;
				o[2] = get(at[2]);
				const uint32_t c0 = at[0], c1 = at[1];
				if (!is_ccw(o[0], o[1], o[2], oriented))
				{
					const V3 v = o[0];
					o[0] = o[1];
					o[1] = v;
					at[0] = c1;
					at[1] = c0;
				}
				float mn = B3G_MAX_SCALAR;
				for (uint32_t i = 0; i < n1; ++i)
				{
					if (i == c0 || i == c1 || i == at[2])
						continue;
					const V3 nn = cross(o[1] - o[0], get(i) - o[0]);
					const float sa2 = dot(nn, oriented);
					if (sa2 < mn)
					{
						mn = sa2;
						at[3] = i;
					}
				}
				if (!(fabsr(mn) < 2.0f * kAreaTol))
				{
					pc = sorted = 4;
					o[3] = get(at[3]);
				}
			}
		}
	}
	__syncwarp();
	// b3SortPolygon (cluster.cpp:34-57).
#pragma unroll
	for (uint32_t i = 1; i < 4; ++i)
	{
		const V3 B = o[i];
#pragma unroll
		for (uint32_t j = i + 1; j < 4; ++j)
			if (j < sorted && !is_ccw(o[0], B, o[j], oriented))
			{
				const V3 v = o[i];
				o[i] = o[j];
				o[j] = v;
				const uint32_t k = at[i];
				at[i] = at[j];
				at[j] = k;
			}
	}
	if (!live)
		return;
	DevManifold& m = a.man[c];
	if (failed)
		atomicOr(a.status, B3G_ST_POLY_OVERFLOW);
	const XF xm1 = flip ? xf2 : xf1, xm2 = flip ? xf1 : xf2;
	const V3 normal = rotc(xm1.q, oriented);
#pragma unroll
	for (uint32_t i = 0; i < 4; ++i)
	{
		if (i >= pc)
			break;
		const uint32_t s = (head + at[i]) % CLIP_SLOTS;
		const V3 v2 = R.pos(s);
		const uint32_t e1 = R.pair1[s][threadIdx.x], e2 = R.pair2[s][threadIdx.x];
		const uint32_t q1 = flip ? e2 : e1, q2 = flip ? e1 : e2;
		set_point(m.points[i], normal, xmult(xm1, flip ? v2 : o[i]), xmult(xm2, flip ? o[i] : v2));
		set_id(m.points[i], mkpair(ring_edge(q1 & 0xFFFFu), ring_edge(q1 >> 16), ring_edge(q2 & 0xFFFFu),
			ring_edge(q2 >> 16)));
	}
	m.pointCount = pc;
	if (pc > 0)
	{
		a.cache[c] = cache; // overlap cache hit
		finish_convex(a, c, m);
	}
	else
		probe_flush(a, c, cache);
}

// Whether the contact is one for k_hulls_probe_large.
__device__ __forceinline__ bool probe_large(const NPArgs& a, uint32_t c)
{
	return !ring_holds(a.S.hulls[a.S.fixHull[a.pairA[c]]], a.S.hulls[a.S.fixHull[a.pairB[c]]]);
}

// Pass 1, the cache half of b3CollideHullsCache (collide_hulls.cpp:367-415):
// b3FeatureCache::ReadState (sat.cpp:178-207), then the separation hit, or the
// overlap hit that rebuilds the cached edge or face contact. What a cache does
// not resolve goes to the SAT kernel.
//
// A block takes a tile of contacts and sorts them by what their caches hold,
// so that a warp reads faces or edges and not some of each; the face contacts
// to rebuild queue up until the block is full of them (or the contacts run
// out) and rebuild on a lane each, in step, their polygons in shared memory.
// With everything on the contact's own thread, 5.6 lanes of a warp were active
// and the polygons lived in local memory: a pass of 512 worlds with 572,000 hull
// pairs took 1,288 us, now 1,113. Blocks of 64 threads, or 5 blocks an SM
// with 96 registers, take 10 % of that longer.
//
// LARGE: the scene has hulls for k_hulls_probe_large, whose contacts are not
// this kernel's.
template <bool LARGE>
__global__ void __launch_bounds__(PROBE_THREADS, PROBE_BLOCKS) k_hulls_probe(NPArgs a)
{
	__shared__ ClipRings rings;
	__shared__ uint32_t sRead[PROBE_THREADS], sFace[2 * PROBE_THREADS];
	__shared__ uint32_t sFaces, sEdges, sQueue;
	const uint32_t n = *a.listCount;
	const uint32_t tid = threadIdx.x, lane = tid & 31u;
	if (tid == 0)
		sQueue = 0;
	for (uint32_t base = blockIdx.x * PROBE_THREADS;; base += gridDim.x * PROBE_THREADS)
	{
		const bool more = base < n;
		if (more)
		{
			if (tid == 0)
				sFaces = sEdges = 0;
			__syncthreads();
			uint32_t c = 0;
			bool face = false, edges = false;
			if (base + tid < n)
				c = a.list[base + tid];
			if (base + tid < n && !(LARGE && probe_large(a, c)))
			{
				const int32_t prev = a.prevIndex[c];
				const uint4 cache = prev >= 0 ? a.prevCache[prev] : make_uint4(CT_EMPTY, FT_FACE1, 0, 0);
				man_clear(a.man[c]);
				const bool hit = a.convexCache && (cache.x == CT_SEPARATION || cache.x == CT_OVERLAP);
				face = hit && (cache.y == FT_FACE1 || cache.y == FT_FACE2);
				edges = hit && cache.y == FT_EDGES;
				if (!a.convexCache)
					probe_miss(a, c, cache);
				else if (cache.x == CT_EMPTY)
					probe_miss(a, c, make_uint4(CT_EMPTY, FT_FACE1, 0, 0));
				else if (!face && !edges)
					probe_flush(a, c, cache);
			}
			__syncwarp();
			const uint32_t below = (1u << lane) - 1u;
			const uint32_t fm = __ballot_sync(0xffffffffu, face), em = __ballot_sync(0xffffffffu, edges);
			uint32_t f0 = 0, e0 = 0;
			if (lane == 0)
			{
				f0 = fm ? atomicAdd(&sFaces, (uint32_t)__popc(fm)) : 0u;
				e0 = em ? atomicAdd(&sEdges, (uint32_t)__popc(em)) : 0u;
			}
			f0 = __shfl_sync(0xffffffffu, f0, 0);
			e0 = __shfl_sync(0xffffffffu, e0, 0);
			// Faces from the front, edges from the back.
			if (face)
				sRead[f0 + __popc(fm & below)] = c;
			if (edges)
				sRead[PROBE_THREADS - 1 - (e0 + __popc(em & below))] = c;
			__syncthreads();
			if (tid < sFaces)
			{
				// A face of either hull is read with the hulls in the face's order.
				c = sRead[tid];
				const uint4 cache = a.prevCache[a.prevIndex[c]];
				HullCtx H;
				load_hull_ctx(a, c, H);
				const bool f2 = cache.y == FT_FACE2;
				const uint32_t state = read_face_thread(f2 ? H.xf2 : H.xf1, f2 ? H.h2 : H.h1, f2 ? H.xf1 : H.xf2,
					f2 ? H.h1 : H.h2, cache.z, H.r1 + H.r2);
				if (cache.x == CT_SEPARATION && state == CT_SEPARATION)
				{
					a.cache[c] = cache; // separation cache hit
					finish_convex(a, c, a.man[c]);
				}
				else if (cache.x == CT_OVERLAP && state == CT_OVERLAP &&
					face_contact_persists(f2 ? H.xf2 : H.xf1, f2 ? H.xf1 : H.xf2, f2 ? H.xf02 : H.xf01,
						f2 ? H.xf01 : H.xf02))
					sFace[atomicAdd(&sQueue, 1u)] = c;
				else
					probe_flush(a, c, cache);
			}
			else if (tid >= PROBE_THREADS - sEdges)
			{
				c = sRead[tid];
				const uint4 cache = a.prevCache[a.prevIndex[c]];
				HullCtx H;
				load_hull_ctx(a, c, H);
				const uint32_t state = read_edges(H.xf1, H.h1, H.xf2, H.h2, cache.z, cache.w, H.r1 + H.r2);
				DevManifold& m = a.man[c];
				bool done = cache.x == CT_SEPARATION && state == CT_SEPARATION;
				if (cache.x == CT_OVERLAP && state == CT_OVERLAP)
				{
					rebuild_edge_contact(m, H.xf1, cache.z, H.h1, H.xf2, cache.w, H.h2);
					done = m.pointCount > 0;
				}
				if (done)
				{
					a.cache[c] = cache;
					finish_convex(a, c, m);
				}
				else
					probe_flush(a, c, cache);
			}
		}
		__syncthreads();
		const uint32_t queued = sQueue;
		const uint32_t take = more && queued < PROBE_THREADS ? 0u : min(queued, (uint32_t)PROBE_THREADS);
		if ((tid & ~31u) < take)
			rebuild_faces(a, sFace[queued - take + min(tid, take - 1u)], tid < take, rings);
		__syncthreads();
		if (tid == 0)
			sQueue = queued - take;
		if (!more && queued == take)
			break;
	}
}

// The same for hulls whose polygons may outgrow the rings, a contact per thread
// from its cache to its manifold: the polygons are in local memory, and without
// the rings' shared memory more of them stay in L1. Contacts of 20,000 pairs of
// 6, 8, 12 and 16-sided prisms take 83, 99, 143 and 206 us so (with the launch of
// the other kernel), 93, 116, 174 and 246 built so in k_hulls_probe, and 104, 137,
// 174 and 248 clipped in the ring there until they outgrew it.
__global__ void __launch_bounds__(PROBE_THREADS) k_hulls_probe_large(NPArgs a)
{
	const uint32_t n = *a.listCount;
	for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
	{
		const uint32_t c = a.list[t];
		if (!probe_large(a, c))
			continue;
		const int32_t prev = a.prevIndex[c];
		uint4 cache = prev >= 0 ? a.prevCache[prev] : make_uint4(CT_EMPTY, FT_FACE1, 0, 0);
		DevManifold& m = a.man[c];
		man_clear(m);
		if (!a.convexCache)
		{
			probe_miss(a, c, cache);
			continue;
		}
		bool done = false;
		if (cache.x == CT_EMPTY)
			cache = make_uint4(CT_EMPTY, FT_FACE1, 0, 0);
		else
		{
			HullCtx H;
			load_hull_ctx(a, c, H);
			const bool face = cache.y == FT_FACE1 || cache.y == FT_FACE2;
			// A face of either hull with the hulls in the face's order.
			const bool f2 = cache.y == FT_FACE2;
			const XF xa = f2 ? H.xf2 : H.xf1, xb = f2 ? H.xf1 : H.xf2;
			const HullRef ha = f2 ? H.h2 : H.h1, hb = f2 ? H.h1 : H.h2;
			uint32_t state = CT_EMPTY;
			if (cache.y == FT_EDGES)
				state = read_edges(H.xf1, H.h1, H.xf2, H.h2, cache.z, cache.w, H.r1 + H.r2);
			else if (face)
				state = read_face_thread(xa, ha, xb, hb, cache.z, H.r1 + H.r2);
			done = cache.x == CT_SEPARATION && state == CT_SEPARATION;
			if (cache.x == CT_OVERLAP && state == CT_OVERLAP)
			{
				if (!face)
					rebuild_edge_contact(m, H.xf1, cache.z, H.h1, H.xf2, cache.w, H.h2);
				else if (face_contact_persists(xa, xb, f2 ? H.xf02 : H.xf01, f2 ? H.xf01 : H.xf02))
					build_face_contact(m, xa, cache.z, ha, f2 ? H.r2 : H.r1, xb, hb, f2 ? H.r1 : H.r2, f2, a.status);
				done = m.pointCount > 0;
			}
		}
		if (done)
		{
			a.cache[c] = cache;
			finish_convex(a, c, m);
		}
		else
			probe_flush(a, c, cache);
	}
}

// Bulk copies from global into shared memory (the TMA engine without a
// tensor map: cp.async.bulk, 16-byte aligned addresses, sizes multiples of 16
// bytes) that complete on a shared-memory barrier. Sources are this GPU's
// own memory; no multicast.
__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
	return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long* bar, uint32_t arrivals)
{
	asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(arrivals) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* bar, uint32_t bytes)
{
	asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
				 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, uint32_t phase)
{
	uint32_t done;
	asm volatile("{\n\t.reg .pred p;\n\t"
				 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
				 "selp.u32 %0, 1, 0, p;\n\t}"
				 : "=r"(done)
				 : "r"(smem_addr(bar)), "r"(phase)
				 : "memory");
	return done != 0;
}
__device__ __forceinline__ void bulk_to_shared(void* dst, const void* src, uint32_t bytes, unsigned long long* bar)
{
	asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
					 smem_addr(dst)),
				 "l"(src), "r"(bytes), "r"(smem_addr(bar))
				 : "memory");
}

// Bytes of one warp's staging area: vertices and planes of two hulls of the
// scene's largest sizes.
__host__ __device__ __forceinline__ size_t sat_stage_bytes(uint32_t maxV, uint32_t maxF)
{
	return 2 * 16 * ((size_t)maxV + maxF);
}

// Waits at most STAGE_SPIN polls for the barrier's phase; every lane polls.
constexpr uint32_t STAGE_SPIN = 1u << 22;
__device__ __forceinline__ bool stage_wait(unsigned long long* bar, uint32_t phase)
{
	for (uint32_t k = 0; k < STAGE_SPIN; ++k)
		if (mbar_try_wait(bar, phase))
			return true;
	return false;
}

// What the bulk copies bring in, by the warp's lanes. Out of line: it hardly
// ever runs.
__device__ __noinline__ void stage_by_lanes(float4* to, const HullRef& h1, const HullRef& h2, uint32_t lane)
{
	auto copy = [&](const float4* from, uint32_t n) {
		for (uint32_t i = lane; i < n; i += 32)
			to[i] = from[i];
		to += n;
	};
	copy(h1.v, h1.vCnt);
	copy(h1.p, h1.fCnt);
	copy(h2.v, h2.vCnt);
	copy(h2.p, h2.fCnt);
	__syncwarp();
}

// Pass 2: one warp per contact the cache did not resolve (W warps per block).
// With STAGE, each pair's hull vertices and planes are brought into the warp's
// shared memory by bulk copies (lane 0 issues four, the warp waits on its
// barrier), and the face and edge queries and the face contact read them there
// instead of from global memory, where every lane's loop over the other hull's
// vertices waited on each load. The half-edges, twice as much, stay there: each
// is read once, a lane an edge, and without them two blocks fit beside the other
// kernels' (three contexts at once, 512 worlds: 830 -> 814 us, a pile of 24,064
// hulls: 198 -> 194). Shared memory per block:
// W barriers (16-byte rounded), then per warp its query / clip area
// (sat_warp_bytes), then per warp its staging area (sat_stage_bytes).
//
// With fewer pairs than half (a quarter) of the warps, 2 (4) warps of a block
// share a pair: each runs the face queries and its part of the edge pairs (93
// x 93 of them between two 64-vertex hulls, most of the time), and the first
// goes on with the contact. Measured on 77 pairs of 12-64-vertex hulls: 158 us
// with a warp each, 62 us with 4.
template <int W, bool STAGE>
__global__ void __launch_bounds__(W * 32) k_hulls_sat(NPArgs a, uint32_t maxUE)
{
	extern __shared__ float4 smem[];
	const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const size_t barBytes = STAGE ? ((W * 8 + 15) & ~15) : 0;
	char* base = reinterpret_cast<char*>(smem) + barBytes;
	char* wsm = base + (size_t)warp * sat_warp_bytes(maxUE);
	EdgeRec* recs = reinterpret_cast<EdgeRec*>(wsm);
	unsigned long long* bar = reinterpret_cast<unsigned long long*>(smem) + warp;
	const size_t stageBytes = sat_stage_bytes(a.S.hullMaxV, a.S.hullMaxF);
	char* stage = base + (size_t)W * sat_warp_bytes(maxUE) + (size_t)warp * stageBytes;
	uint32_t phase = 0;
	if (STAGE)
	{
		if (lane == 0)
		{
			mbar_init(bar, 1);
			asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
		}
		__syncwarp();
	}
	__shared__ float2 partBest[W];
	uint32_t n = *a.missCount;
	uint32_t nw = gridDim.x * W;
	const uint32_t parts = !a.convexCache ? 1u : (W >= 4 && 4u * n <= nw ? 4u : (2u * n <= nw ? 2u : 1u));
	// Warps that share have one pair each: parts * n <= nw.
	for (uint32_t t = (blockIdx.x * W + warp) / parts; t < n; t += nw / parts)
	{
		uint32_t c = a.missList[t];
		HullCtx H;
		load_hull_ctx(a, c, H);
		H.parts = EdgeParts{warp % parts, parts, 1u + warp / parts, &partBest[warp / parts * parts]};
		H.recs = recs;
		H.clip = reinterpret_cast<WarpClip*>(wsm);
		H.maxUE = maxUE;
		if (STAGE)
		{
			float4* v1 = reinterpret_cast<float4*>(stage);
			float4* p1 = v1 + H.h1.vCnt;
			float4* v2 = p1 + H.h1.fCnt;
			float4* p2 = v2 + H.h2.vCnt;
			if (lane == 0)
			{
				// The warp's reads of the previous pair (generic proxy) come
				// before these writes (async proxy).
				asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
				const uint32_t bytes = 16u * (H.h1.vCnt + H.h1.fCnt + H.h2.vCnt + H.h2.fCnt);
				mbar_arrive_expect_tx(bar, bytes);
				bulk_to_shared(v1, H.h1.v, 16u * H.h1.vCnt, bar);
				bulk_to_shared(p1, H.h1.p, 16u * H.h1.fCnt, bar);
				bulk_to_shared(v2, H.h2.v, 16u * H.h2.vCnt, bar);
				bulk_to_shared(p2, H.h2.p, 16u * H.h2.fCnt, bar);
			}
			const bool ok = stage_wait(bar, phase);
			if (!__all_sync(0xffffffffu, ok))
			{
				// The copies did not land in time: report it, wait (bounded)
				// for them before the shared memory goes away, and stop. A warp
				// that shares its pair brings the hulls in itself (the same
				// values) and goes on: the others wait for it where their edge
				// queries meet.
				if (lane == 0)
					atomicOr(a.status, B3G_ST_WAIT_TIMEOUT);
				stage_wait(bar, phase);
				if (parts == 1)
					return;
				stage_by_lanes(v1, H.h1, H.h2, lane);
			}
			phase ^= 1u;
			H.h1.v = v1;
			H.h1.p = p1;
			H.h2.v = v2;
			H.h2.p = p2;
		}
		uint4 cache = a.cache[c];
		DevManifold& m = a.man[c];
		if (a.convexCache)
			sat_after_miss(m, H, cache, lane);
		else
			collide_hulls_nocache(m, H, lane);
		__syncwarp();
		if (lane == 0 && H.parts.part == 0)
		{
			finish_convex(a, c, m);
			a.cache[c] = cache;
		}
		__syncwarp();
	}
}

// b3CollideHullAndTriangle (collide_hull_triangle.cpp:24-124) after the
// hull-hull SAT: points on a triangle edge that has a coplanar wing take the
// triangle's face normal (oriented from the hull to the triangle) so bodies
// slide over mesh edges. Lane 0 only.
__device__ void triangle_wing_normals(DevManifold& m, const float4 w4[3], const XF& xf1, const HullRef& h1,
	const XF& xf2, const HullRef& h2)
{
	PL plane2 = pmul(xf2, hp(h2, 0));
	V3 centroid1 = xmul(xf1, h1.centroid);
	V3 centroid2 = xmul(xf2, h2.centroid);
	for (uint32_t i = 0; i < m.pointCount; ++i)
	{
		DevPoint& mp = m.points[i];
		uint32_t inEdge2 = mp.key[2], outEdge2 = mp.key[3];
		uint32_t e2;
		if (mp.edgeContact)
			e2 = inEdge2;
		else
		{
			e2 = inEdge2 == B3G_NULL_EDGE ? outEdge2 : inEdge2;
			if (e2 == B3G_NULL_EDGE)
				continue;
		}
		uint32_t edgeIndex = e2 >> 1; // half-edges 2k, 2k + 1 lie on triangle edge k
		if (edgeIndex > 2 || w4[edgeIndex].w == 0.0f)
			continue;
		uint32_t ev1 = edgeIndex;
		uint32_t ev2 = edgeIndex + 1 < 3 ? edgeIndex + 1 : 0;
		V3 A = V3{w4[edgeIndex].x, w4[edgeIndex].y, w4[edgeIndex].z};
		V3 B = hv(h2, ev2);
		V3 C = hv(h2, ev1);
		V3 center = ((A + B) + C) / 3.0f;
		float distance = pdist(center, hp(h2, 0));
		const float kCoplanarTol = 0.005f;
		if (distance > -kCoplanarTol && distance < kCoplanarTol)
		{
			V3 localN1 = V3{mp.n[0], mp.n[1], mp.n[2]};
			V3 localC1 = V3{mp.p1[0], mp.p1[1], mp.p1[2]};
			V3 localC2 = V3{mp.p2[0], mp.p2[1], mp.p2[2]};
			V3 n1 = rot(xf1.q, localN1);
			V3 c1 = xmul(xf1, localC1);
			V3 c2 = xmul(xf2, localC2);
			float sep = dot(c2 - c1, n1);
			V3 n = plane2.n;
			if (dot(n, centroid2 - centroid1) < 0.0f)
				n = -n;
			V3 nc1 = c2 - sep * n;
			V3 ln = rotc(xf1.q, n);
			V3 lp = xmult(xf1, nc1);
			mp.n[0] = ln.x, mp.n[1] = ln.y, mp.n[2] = ln.z;
			mp.p1[0] = lp.x, mp.p1[1] = lp.y, mp.p1[2] = lp.z;
		}
	}
}

// Hull (A) against triangle (B): one warp per contact, the full SAT of
// b3CollideHulls without a feature cache (b3HullAndTriangleContact keeps
// none), on the triangle's two-faced hull.
template <int W>
__global__ void __launch_bounds__(W * 32) k_hull_triangle(NPArgs a, uint32_t maxUE)
{
	extern __shared__ float4 smem[];
	const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	char* wsm = reinterpret_cast<char*>(smem) + (size_t)warp * sat_warp_bytes(maxUE);
	EdgeRec* recs = reinterpret_cast<EdgeRec*>(wsm);
	uint32_t n = *a.listCount;
	for (uint32_t t = blockIdx.x * W + warp; t < n; t += gridDim.x * W)
	{
		uint32_t c = a.list[t];
		uint32_t fa = a.pairA[c], fb = a.pairB[c];
		HullCtx H;
		H.xf1 = a.exA ? load_xf7(a.exA + 7 * (size_t)c) : body_xf(a.S, a.S.fixBody[fa]);
		H.xf2 = a.exB ? load_xf7(a.exB + 7 * (size_t)c) : body_xf(a.S, a.S.fixBody[fb]);
		H.h1 = hull_ref(a.S, a.S.fixHull[fa]);
		H.h2 = tri_ref(a.S, fb);
		H.r1 = a.S.fixParams[3 * fa].x;
		H.r2 = a.S.fixParams[3 * fb + 2].y;
		H.status = a.status;
		H.recs = recs;
		H.clip = reinterpret_cast<WarpClip*>(wsm);
		H.maxUE = maxUE;
		H.parts = EdgeParts{0, 1, 0, nullptr};
		DevManifold& m = a.man[c];
		if (lane == 0)
			man_clear(m);
		__syncwarp();
		collide_hulls_nocache(m, H, lane);
		__syncwarp();
		if (lane == 0)
		{
			float4 w4[3];
			for (int k = 0; k < 3; ++k)
				w4[k] = a.S.fixWing[3 * (size_t)fb + k];
			triangle_wing_normals(m, w4, H.xf1, H.h1, H.xf2, H.h2);
			finish_convex(a, c, m);
			a.cache[c] = make_uint4(B3G_NULL, B3G_NULL, B3G_NULL, B3G_NULL);
		}
		__syncwarp();
	}
}

// Mesh work items of hull-mesh contacts (hull A, mesh B): one warp per
// triangle, b3CollideHullAndTriangle on the child triangle
// (hull_mesh_contact.cpp:42-50), points tagged with the triangle. Sensor
// contacts record the triangle's overlap in pointCount.
template <int W>
__global__ void __launch_bounds__(W * 32, 4) k_mesh_items_hull(NPArgs a, Buffers B, uint32_t maxUE)
{
	extern __shared__ float4 smem[];
	const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	char* wsm = reinterpret_cast<char*>(smem) + (size_t)warp * sat_triangle_warp_bytes();
	EdgeRec* recs = reinterpret_cast<EdgeRec*>(wsm);
	uint32_t n = min(B.counters[CTR_MESH_PAIRS], B.meshPairCap);
	for (uint32_t i = blockIdx.x * W + warp; i < n; i += gridDim.x * W)
	{
		uint32_t c = B.meshPairC[i], t = B.meshPairT[i];
		uint32_t fa = a.pairA[c], fb = a.pairB[c];
		if (a.S.fixType[fa] != B3G_SHAPE_HULL || a.S.fixType[fb] != B3G_SHAPE_MESH)
			continue;
		MeshTri tri;
		mesh_triangle(a.S, fb, t, tri);
		HullCtx H;
		H.xf1 = body_xf(a.S, a.S.fixBody[fa]);
		H.xf2 = body_xf(a.S, a.S.fixBody[fb]);
		H.h1 = hull_ref(a.S, a.S.fixHull[fa]);
		H.h2 = mesh_tri_ref(tri);
		H.r1 = a.S.fixParams[3 * fa].x;
		H.r2 = tri.radius;
		H.status = a.status;
		H.recs = recs;
		H.clip = reinterpret_cast<WarpClip*>(wsm);
		H.maxUE = maxUE;
		H.parts = EdgeParts{0, 1, 0, nullptr};
		DevManifold& m = B.meshPairMan[i];
		if (lane == 0)
			man_clear(m);
		__syncwarp();
		if ((a.S.fixFlags[fa] | a.S.fixFlags[fb]) & B3G_FIXTURE_SENSOR)
		{
			if (lane == 0)
			{
				GProxy pb;
				pb.gv = nullptr;
				pb.lv[0] = tri.v[0];
				pb.lv[1] = tri.v[1];
				pb.lv[2] = tri.v[2];
				pb.count = 3;
				pb.radius = tri.radius;
				GProxy pa;
				pa.gv = H.h1.v;
				pa.count = H.h1.vCnt;
				pa.radius = H.r1;
				GJKOut q = gjk(H.xf1, pa, H.xf2, pb, true);
				m.pointCount = q.distance <= 10.0f * B3G_EPSILON ? 1u : 0u;
			}
			__syncwarp();
			continue;
		}
		collide_hulls_nocache(m, H, lane);
		__syncwarp();
		if (lane == 0)
		{
			triangle_wing_normals(m, tri.wing, H.xf1, H.h1, H.xf2, H.h2);
			for (uint32_t j = 0; j < m.pointCount; ++j)
				m.points[j].triangleKey = t;
		}
		__syncwarp();
	}
}

} // namespace

void launch_hulls_sat(const NPArgs& a, uint32_t maxUE, const Tune& tune, cudaStream_t s);
size_t hull_sat_smem(int warps, uint32_t maxUE);

// Hull-triangle contacts (bucket BK_HULL_TRIANGLE), with the SAT kernel's
// warps per block.
void launch_hull_triangles(const NPArgs& base, const uint32_t* list, const uint32_t* count, uint32_t maxUE,
	const Tune& tune, cudaStream_t s)
{
	NPArgs a = base;
	a.list = list;
	a.listCount = count;
	uint32_t ue = maxUE > 3 ? maxUE : 3;
	const int bps = (int)tune.v[B3G_TUNE_SAT_BLOCKS];
	size_t smem;
	switch (tune.v[B3G_TUNE_SAT_WARPS])
	{
	case 2:
		smem = hull_sat_smem(2, ue);
		if (smem > 48 * 1024)
			cudaFuncSetAttribute(k_hull_triangle<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
		k_hull_triangle<2><<<persistent_blocks(bps), 64, smem, s>>>(a, ue);
		break;
	case 8:
		smem = hull_sat_smem(8, ue);
		if (smem > 48 * 1024)
			cudaFuncSetAttribute(k_hull_triangle<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
		k_hull_triangle<8><<<persistent_blocks(bps), 256, smem, s>>>(a, ue);
		break;
	default:
		smem = hull_sat_smem(4, ue);
		if (smem > 48 * 1024)
			cudaFuncSetAttribute(k_hull_triangle<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
		k_hull_triangle<4><<<persistent_blocks(bps), 128, smem, s>>>(a, ue);
		break;
	}
}

template <int W, bool STAGE>
void launch_sat_kernel(const NPArgs& a, uint32_t maxUE, int blocksPerSM, size_t smem, cudaStream_t s)
{
	static size_t configured = 0;
	if (smem > 48 * 1024 && smem > configured)
	{
		cudaFuncSetAttribute(k_hulls_sat<W, STAGE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
		configured = smem;
	}
	// Up to 4 warps share a pair.
	k_hulls_sat<W, STAGE><<<work_blocks(4ull * a.hcPostCap, W, blocksPerSM), W * 32, smem, s>>>(a, maxUE);
}

// The staged kernel when its shared memory fits a block, else the kernel
// that reads the hulls from global memory.
template <int W>
void launch_sat(const NPArgs& a, uint32_t maxUE, int blocksPerSM, cudaStream_t s)
{
	const size_t plain = (size_t)W * sat_warp_bytes(maxUE);
	const size_t staged = ((W * 8 + 15) & ~(size_t)15) + plain +
		(size_t)W * sat_stage_bytes(a.S.hullMaxV, a.S.hullMaxF);
	static int optin = -1;
	if (optin < 0)
	{
		int dev = 0;
		cudaGetDevice(&dev);
		if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
			optin = 48 * 1024;
	}
	if (staged <= (size_t)optin && a.S.hullMaxV > 0)
		launch_sat_kernel<W, true>(a, maxUE, blocksPerSM, staged, s);
	else
		launch_sat_kernel<W, false>(a, maxUE, blocksPerSM, plain, s);
}

void launch_hulls(const NPArgs& base, const uint32_t* list, const uint32_t* count, uint32_t maxUE, const Tune& tune,
	cudaStream_t s)
{
	NPArgs a = base;
	a.list = list;
	a.listCount = count;
	launch_hulls_probe(a, a.list, a.listCount, tune, s);
	launch_hulls_sat(a, maxUE, tune, s);
}

void launch_hulls_sat(const NPArgs& a, uint32_t maxUE, const Tune& tune, cudaStream_t s)
{
	const int bps = (int)tune.v[B3G_TUNE_SAT_BLOCKS];
	switch (tune.v[B3G_TUNE_SAT_WARPS])
	{
	case 2:
		launch_sat<2>(a, maxUE, bps, s);
		break;
	case 8:
		launch_sat<8>(a, maxUE, bps, s);
		break;
	default:
		launch_sat<4>(a, maxUE, bps, s);
		break;
	}
}

void launch_hulls_probe(const NPArgs& base, const uint32_t* list, const uint32_t* count, const Tune& tune,
	cudaStream_t s)
{
	NPArgs a = base;
	a.list = list;
	a.listCount = count;
	const int blocks = work_blocks(a.hcPostCap, PROBE_THREADS, (int)tune.v[B3G_TUNE_PROBE]);
	if (!a.S.hullsLarge)
	{
		k_hulls_probe<false><<<blocks, PROBE_THREADS, 0, s>>>(a);
		return;
	}
	k_hulls_probe<true><<<blocks, PROBE_THREADS, 0, s>>>(a);
	k_hulls_probe_large<<<blocks, PROBE_THREADS, 0, s>>>(a);
}

// Dynamic shared memory of the SAT kernel with `warps` warps per block.
size_t hull_sat_smem(int warps, uint32_t maxUE)
{
	return (size_t)warps * sat_warp_bytes(maxUE);
}

void launch_mesh_items_hull(const NPArgs& a, const Buffers& B, uint32_t maxUE, const Tune& tune, cudaStream_t s)
{
	uint32_t ue = maxUE > 3 ? maxUE : 3;
	// As many blocks as 128 registers allow (with 80 or 255 it takes longer).
	k_mesh_items_hull<4><<<persistent_blocks(4), 128, 4 * sat_triangle_warp_bytes(), s>>>(a, B, ue);
}

void carveout_narrow_hulls()
{
	set_carveout({
		(const void*)k_hulls_probe<false>, (const void*)k_hulls_probe<true>, (const void*)k_hulls_sat<2, true>, (const void*)k_hulls_sat<4, true>,
		(const void*)k_hulls_sat<8, true>, (const void*)k_hulls_sat<2, false>, (const void*)k_hulls_sat<4, false>,
		(const void*)k_hulls_sat<8, false>, (const void*)k_hull_triangle<2>, (const void*)k_hull_triangle<4>,
		(const void*)k_hull_triangle<8>, (const void*)k_mesh_items_hull<4>});
}
