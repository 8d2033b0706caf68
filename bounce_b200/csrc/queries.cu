// World queries on the device: b3World::QueryAABB, RayCast, RayCastSingle,
// ShapeCast and ShapeCastSingle (world.cpp:452-878) over the LBVH and fat
// AABBs of the last pass, with each shape's own ray cast:
//   b3SphereShape::RayCast    sphere_shape.cpp:69-122
//   b3CapsuleShape::RayCast   capsule_shape.cpp:180-322
//   b3HullShape::RayCast      hull_shape.cpp:189-275
//   b3TriangleShape::RayCast  triangle_shape.cpp:95-180
//   b3MeshShape::RayCast      mesh_shape.cpp:81-146, over b3StaticTree::RayCast
//                             (static_tree.h:150-292)
//
// The calls that report every hit walk the LBVH from the root along its ropes,
// a thread per query; those that report one meet its boxes nearest first, the
// lanes of a warp in step. The reference walks its dynamic tree instead; the
// set of proxies a query meets is the same (fat AABBs overlapping the box, or
// the segment), only the order differs: QueryAABB and RayCast (every hit) are returned per query in LBVH
// order, and RayCastSingle keeps the smallest fraction, the smaller fixture
// index on an exact tie (the reference keeps the first one its tree meets).

#include <algorithm>
#include <vector>

#include "lane_gjk.cuh"

namespace {

constexpr uint32_t SENT = 0xFFFFFFFFu;

struct RayIn
{
	V3 p1, p2;
	float maxFraction;
};

struct RayOut
{
	float fraction;
	V3 normal;
};

__device__ __forceinline__ V3 vabs(V3 v) { return V3{fabsf(v.x), fabsf(v.y), fabsf(v.z)}; }

// The segment tests of b3DynamicTree::RayCast / b3StaticTree::RayCast
// (static_tree.h:185-262): the segment's AABB overlaps the node's, and no
// axis of the box or of cross(e_i, r) separates them.
struct SegTest
{
	V3 p1, q2, r;
	AABB box;

	__device__ void init(V3 a, V3 b, float maxFraction)
	{
		p1 = a;
		r = b - a;
		normalize_inplace(r);
		q2 = a + maxFraction * (b - a);
		box.lo = vmin(a, q2);
		box.hi = vmax(a, q2);
	}

	// Shortens the segment to [p1, p1 + f (b - p1)].
	__device__ void clip(V3 b, float f)
	{
		q2 = p1 + f * (b - p1);
		box.lo = vmin(p1, q2);
		box.hi = vmax(p1, q2);
	}

	__device__ bool pass(V3 lo, V3 hi) const
	{
		if (box.hi.x < lo.x || box.lo.x > hi.x || box.hi.y < lo.y || box.lo.y > hi.y || box.hi.z < lo.z ||
			box.lo.z > hi.z)
			return false;
		V3 c = 0.5f * (lo + hi);
		V3 h = 0.5f * (hi - lo);
		V3 s = p1 - c;
		V3 t = q2 - c;
		if (fabsf(s.x + t.x) - (fabsf(s.x - t.x) + 2.0f * h.x) > 0.0f)
			return false;
		if (fabsf(s.y + t.y) - (fabsf(s.y - t.y) + 2.0f * h.y) > 0.0f)
			return false;
		if (fabsf(s.z + t.z) - (fabsf(s.z - t.z) + 2.0f * h.z) > 0.0f)
			return false;
		V3 v1 = cross(V3{1.0f, 0.0f, 0.0f}, r);
		if (fabsf(dot(v1, s)) - dot(vabs(v1), h) > 0.0f)
			return false;
		V3 v2 = cross(V3{0.0f, 1.0f, 0.0f}, r);
		if (fabsf(dot(v2, s)) - dot(vabs(v2), h) > 0.0f)
			return false;
		V3 v3 = cross(V3{0.0f, 0.0f, 1.0f}, r);
		if (fabsf(dot(v3, s)) - dot(vabs(v3), h) > 0.0f)
			return false;
		return true;
	}
};

// Ray against a sphere of radius `radius` around m = p1 - centre.
__device__ __forceinline__ bool ray_sphere_at(RayOut& o, V3 m, V3 d, float a, float radius, float maxFraction)
{
	float b = dot(m, d);
	float c = dot(m, m) - radius * radius;
	float disc = b * b - a * c;
	if (disc < 0.0f)
		return false;
	float t = -b - sqrtf(disc);
	if (t > 0.0f && t <= maxFraction * a)
	{
		t /= a;
		o.fraction = t;
		o.normal = normalized(m + t * d);
		return true;
	}
	return false;
}

// c: the centre in the world.
__device__ __forceinline__ bool ray_sphere_world(RayOut& o, const RayIn& in, V3 c, float radius)
{
	V3 d = in.p2 - in.p1;
	float a = dot(d, d);
	if (a < B3G_EPSILON * B3G_EPSILON)
		return false;
	V3 m = in.p1 - c;
	return ray_sphere_at(o, m, d, a, radius, in.maxFraction);
}

// P, Q: the segment in the world.
__device__ __forceinline__ bool ray_capsule_world(RayOut& o, const RayIn& in, V3 P, V3 Q, float radius)
{
	V3 A = in.p1, B = in.p2;
	V3 n = B - A;
	float nn = dot(n, n);
	if (nn < B3G_EPSILON * B3G_EPSILON)
		return false;
	V3 d = Q - P;
	float dd = dot(d, d);
	if (dd < B3G_EPSILON * B3G_EPSILON)
		return ray_sphere_at(o, A - P, n, nn, radius, in.maxFraction);
	V3 m = A - P;
	float nd = dot(n, d);
	float mm = dot(m, m);
	float md = dot(m, d);
	float mn = dot(m, n);
	float a = dd * nn - nd * nd;
	if (fabsf(a) < 2.0f * (B3G_EPSILON * B3G_EPSILON))
		return false;
	float b = dd * mn - nd * md;
	float c = dd * (mm - radius * radius) - md * md;
	float disc = b * b - a * c;
	if (disc < 0.0f)
		return false;
	float t = -b - sqrtf(disc);
	t /= a;
	if (t < 0.0f || t > 1.0f)
		return false;
	// Which part of the capsule the cylinder hit lies on.
	float tp = md + t * nd;
	V3 C;
	if (tp < 0.0f)
		C = P;
	else if (tp > dd)
		C = Q;
	else
	{
		V3 X = (1.0f - t) * A + t * B;
		V3 e2 = cross(d, X - P);
		V3 e3 = cross(e2, d);
		normalize_inplace(e3);
		o.fraction = t;
		o.normal = e3;
		return true;
	}
	// Hemisphere at C.
	return ray_sphere_at(o, A - C, n, nn, radius, in.maxFraction);
}

// A hull of `count` planes.
__device__ __forceinline__ bool ray_planes(RayOut& o, const RayIn& in, const XF& xf, const float4* planes, uint32_t count)
{
	auto plane = [&](uint32_t i) {
		const float4 w = __ldg(planes + i);
		return PL{V3{w.x, w.y, w.z}, w.w};
	};
	V3 p1 = rotc(xf.q, in.p1 - xf.p);
	V3 p2 = rotc(xf.q, in.p2 - xf.p);
	V3 d = p2 - p1;
	float lower = 0.0f, upper = in.maxFraction;
	uint32_t index = B3G_NULL;
	// Four planes load together: the test of one may end the loop, so the
	// compiler does not load ahead by itself.
	for (uint32_t i0 = 0; i0 < count; i0 += 4)
	{
		PL pl4[4];
#pragma unroll
		for (uint32_t k = 0; k < 4; ++k)
			pl4[k] = plane(min(i0 + k, count - 1u));
#pragma unroll
		for (uint32_t k = 0; k < 4; ++k)
		{
			const uint32_t i = i0 + k;
			if (i >= count)
				break;
			const PL pl = pl4[k];
			float numerator = pl.d - dot(pl.n, p1);
			float denominator = dot(pl.n, d);
			if (denominator == 0.0f)
			{
				if (numerator < 0.0f)
					return false;
			}
			else
			{
				if (denominator < 0.0f)
				{
					if (numerator < lower * denominator)
					{
						lower = numerator / denominator;
						index = i;
					}
				}
				else if (numerator < upper * denominator)
					upper = numerator / denominator;
				if (upper < lower)
					return false;
			}
		}
	}
	if (index != B3G_NULL)
	{
		o.fraction = lower;
		o.normal = rot(xf.q, plane(index).n);
		return true;
	}
	return false;
}

__device__ bool ray_triangle(RayOut& o, const RayIn& in, const XF& xf, V3 v1, V3 v2, V3 v3)
{
	V3 p1 = xmult(xf, in.p1);
	V3 p2 = xmult(xf, in.p2);
	V3 d = p2 - p1;
	if (dot(d, d) < B3G_EPSILON * B3G_EPSILON)
		return false;
	V3 n = cross(v2 - v1, v3 - v1);
	float l = len(n);
	if (l == 0.0f)
		return false;
	float inv = 1.0f / l; // b3Vec3::operator/= scales by the reciprocal
	n = inv * n;
	float num = dot(n, v1 - p1);
	float den = dot(n, d);
	if (den == 0.0f)
		return false;
	float fraction = num / den;
	if (fraction < 0.0f || in.maxFraction < fraction)
		return false;
	V3 Q = p1 + fraction * d;
	V3 AB = v2 - v1, AC = v3 - v1;
	V3 QA = v1 - Q, QB = v2 - Q, QC = v3 - Q;
	V3 QB_x_QC = cross(QB, QC);
	V3 QC_x_QA = cross(QC, QA);
	V3 QA_x_QB = cross(QA, QB);
	V3 AB_x_AC = cross(AB, AC);
	float u = dot(QB_x_QC, AB_x_AC);
	float v = dot(QC_x_QA, AB_x_AC);
	float w = dot(QA_x_QB, AB_x_AC);
	if (u >= 0.0f && v >= 0.0f && w >= 0.0f)
	{
		o.fraction = fraction;
		o.normal = num > 0.0f ? rot(xf.q, -n) : rot(xf.q, n);
		return true;
	}
	return false;
}

// b3MeshShape::RayCast: the segment in the mesh's unscaled frame walks the
// static tree (depth first, child2 first, as b3StaticTree::RayCast's stack);
// each leaf's triangle (scaled) is ray cast with the original segment; the
// first smallest fraction wins.
__device__ bool ray_mesh(RayOut& o, const RayIn& in, const XF& xf, const DevScene& S, uint32_t fix, uint32_t* status)
{
	const MeshDesc md = S.meshes[S.fixHull[fix]];
	float4 sp = S.fixParams[3 * fix];
	V3 sc = V3{sp.x, sp.y, sp.z};
	V3 inv = V3{1.0f / sc.x, 1.0f / sc.y, 1.0f / sc.z};
	SegTest seg;
	seg.init(vmul(inv, xmult(xf, in.p1)), vmul(inv, xmult(xf, in.p2)), in.maxFraction);
	bool hit = false;
	o.fraction = B3G_MAX_SCALAR;
	constexpr uint32_t STACK = 64;
	uint32_t stack[STACK];
	uint32_t sp_ = 0;
	stack[sp_++] = md.root;
	while (sp_ > 0)
	{
		uint32_t id = stack[--sp_];
		if (id == B3G_NULL_NODE)
			continue;
		float4 lo = S.meshNodes[2 * (size_t)(md.nOff + id)], hi = S.meshNodes[2 * (size_t)(md.nOff + id) + 1];
		if (!seg.pass(V3{lo.x, lo.y, lo.z}, V3{hi.x, hi.y, hi.z}))
			continue;
		uint32_t child1 = __float_as_uint(lo.w), other = __float_as_uint(hi.w);
		if (child1 == B3G_NULL_NODE)
		{
			uint4 t = S.meshTris[md.tOff + other];
			auto vert = [&](uint32_t i) {
				float4 a = S.meshVerts[md.vOff + i];
				return vmul(sc, V3{a.x, a.y, a.z});
			};
			RayOut r;
			if (ray_triangle(r, in, xf, vert(t.x), vert(t.y), vert(t.z)) && r.fraction < o.fraction)
			{
				hit = true;
				o = r;
				// Triangle boxes are grown by B3_LINEAR_SLOP: a triangle hit no
				// later than this one is met by the shortened segment too.
				seg.clip(vmul(inv, xmult(xf, in.p2)), r.fraction);
			}
		}
		else
		{
			if (sp_ + 2 > STACK)
			{
				atomicOr(status, B3G_ST_POLY_OVERFLOW);
				return hit;
			}
			stack[sp_++] = child1;
			stack[sp_++] = other;
		}
	}
	return hit;
}

// b3Fixture::RayCast (fixture.h) at the body's transform of the last pass.
// Out of line: the ordered walks come here for triangles and meshes only.
__device__ __noinline__ bool ray_fixture(RayOut& o, const RayIn& in, const DevScene& S, uint32_t f, uint32_t* status)
{
	XF xf = body_xf(S, S.fixBody[f]);
	float4 p0 = S.fixParams[3 * f], p1 = S.fixParams[3 * f + 1], p2 = S.fixParams[3 * f + 2];
	switch (S.fixType[f])
	{
	case B3G_SHAPE_SPHERE:
		return ray_sphere_world(o, in, xmul(xf, V3{p0.x, p0.y, p0.z}), p0.w);
	case B3G_SHAPE_CAPSULE:
		return ray_capsule_world(o, in, xmul(xf, V3{p0.x, p0.y, p0.z}), xmul(xf, V3{p0.w, p1.x, p1.y}), p1.z);
	case B3G_SHAPE_TRIANGLE:
		return ray_triangle(o, in, xf, V3{p0.x, p0.y, p0.z}, V3{p0.w, p1.x, p1.y}, V3{p1.z, p1.w, p2.x});
	case B3G_SHAPE_HULL:
	{
		const HullDesc h = S.hulls[S.fixHull[f]];
		return ray_planes(o, in, xf, S.hplanes + h.fOff, h.fCnt);
	}
	case B3G_SHAPE_MESH:
		return ray_mesh(o, in, xf, S, f, status);
	default:
		return false;
	}
}

struct QueryCtx
{
	DevScene S;
	const float4* nodeLo;
	const float4* nodeHi;
	const uint32_t* nodeRight;
	const float4* fatLo;
	const float4* fatHi;
	uint32_t leaves;
	uint32_t* status;
};

__device__ __forceinline__ bool query_takes(const QueryCtx& q, uint32_t f, uint32_t world)
{
	return q.S.fixLife[f] != FIX_DEAD && q.S.bodyWorld[q.S.fixBody[f]] == world;
}

// Rope walk of the LBVH from the root; visit(proxy) for every leaf `accept`
// lets through (internal nodes are descended when `accept` passes them).
template <class Accept, class Visit>
__device__ __forceinline__ void lbvh_walk(const QueryCtx& q, Accept&& accept, Visit&& visit)
{
	const uint32_t nodes = 2u * q.leaves - 1u;
	uint32_t node = 0;
	uint32_t steps = 0;
	while (node != SENT)
	{
		if (++steps > nodes + 1u || node >= nodes)
		{
			atomicOr(q.status, B3G_ST_WAIT_TIMEOUT);
			return;
		}
		float4 lo = q.nodeLo[node], hi = q.nodeHi[node];
		bool pass = accept(V3{lo.x, lo.y, lo.z}, V3{hi.x, hi.y, hi.z});
		if (pass && node < q.leaves - 1u)
		{
			node = __float_as_uint(lo.w);
			continue;
		}
		if (pass)
			visit(__float_as_uint(lo.w));
		node = __float_as_uint(hi.w);
	}
}

// b3World::QueryAABB: fat AABBs overlapping the box (b3TestOverlap, closed).
template <int MODE>
__global__ void k_query_aabb(QueryCtx q, const float* boxes, const uint32_t* worlds, uint32_t n, uint32_t* counts,
	uint2* out, uint32_t capacity)
{
	uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n)
		return;
	AABB b;
	b.lo = V3{boxes[6 * i], boxes[6 * i + 1], boxes[6 * i + 2]};
	b.hi = V3{boxes[6 * i + 3], boxes[6 * i + 4], boxes[6 * i + 5]};
	uint32_t world = worlds ? worlds[i] : 0u;
	uint32_t k = MODE == 0 ? 0u : counts[i];
	auto overlap = [&](V3 lo, V3 hi) {
		return !(hi.x < b.lo.x || lo.x > b.hi.x || hi.y < b.lo.y || lo.y > b.hi.y || hi.z < b.lo.z || lo.z > b.hi.z);
	};
	lbvh_walk(q, overlap, [&](uint32_t f) {
		float4 lo = q.fatLo[f], hi = q.fatHi[f];
		if (!overlap(V3{lo.x, lo.y, lo.z}, V3{hi.x, hi.y, hi.z}) || !query_takes(q, f, world))
			return;
		if (MODE == 1 && k < capacity)
			out[k] = make_uint2(i, f);
		++k;
	});
	if (MODE == 0)
		counts[i] = k;
}

// b3World::RayCast with a listener that keeps every hit (MODE 0 counts,
// MODE 1 writes fixture + (point, normal, fraction)).
template <int MODE>
__global__ void k_ray_cast(QueryCtx q, const float* rays, const uint32_t* worlds, uint32_t n, uint32_t* counts,
	uint2* outIdx, float* outHit, uint32_t capacity)
{
	uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n)
		return;
	RayIn in;
	in.p1 = V3{rays[6 * i], rays[6 * i + 1], rays[6 * i + 2]};
	in.p2 = V3{rays[6 * i + 3], rays[6 * i + 4], rays[6 * i + 5]};
	in.maxFraction = 1.0f;
	uint32_t world = worlds ? worlds[i] : 0u;
	uint32_t k = MODE == 1 ? counts[i] : 0u;
	if (dot(in.p2 - in.p1, in.p2 - in.p1) > 0.0f)
	{
		SegTest seg;
		seg.init(in.p1, in.p2, in.maxFraction);
		lbvh_walk(q, [&](V3 lo, V3 hi) { return seg.pass(lo, hi); }, [&](uint32_t f) {
			if (!query_takes(q, f, world))
				return;
			RayOut o;
			if (!ray_fixture(o, in, q.S, f, q.status))
				return;
			if (MODE == 1 && k < capacity)
			{
				V3 p = (1.0f - o.fraction) * in.p1 + o.fraction * in.p2;
				outIdx[k] = make_uint2(i, f);
				float* h = outHit + 7 * (size_t)k;
				h[0] = p.x, h[1] = p.y, h[2] = p.z;
				h[3] = o.normal.x, h[4] = o.normal.y, h[5] = o.normal.z;
				h[6] = o.fraction;
			}
			++k;
		});
	}
	if (MODE == 0)
		counts[i] = k;
}

// Entry of a moving point or box into the boxes of the ordered walks: the
// fraction of the motion d at which it meets a box, by the three slabs, each
// plane one multiply-add. The boxes are grown by `pad` (many times the
// rounding of these few operations at the query's coordinates), so a box that
// the exact tests at the leaves let through is never cut here.
struct SlabTest
{
	V3 inv;  // 1 / d, finite: a zero component becomes a huge one
	V3 a, b; // box plane * inv + a (lower planes) or + b (upper planes)

	__device__ void init(V3 lo, V3 hi, V3 d, float pad)
	{
		auto recip = [](float v) { return fabsf(v) > 1e-30f ? 1.0f / v : copysignf(1e30f, v); };
		inv = V3{recip(d.x), recip(d.y), recip(d.z)};
		a = V3{-(hi.x + pad) * inv.x, -(hi.y + pad) * inv.y, -(hi.z + pad) * inv.z};
		b = V3{-(lo.x - pad) * inv.x, -(lo.y - pad) * inv.y, -(lo.z - pad) * inv.z};
	}

	// Whether the box is met at a fraction in [0, limit], and the first such.
	// An empty box (lower above upper: a dead proxy's) is never met.
	__device__ __forceinline__ bool enter(V3 lo, V3 hi, float limit, float& t) const
	{
		const float ax = __fmaf_rn(lo.x, inv.x, a.x), bx = __fmaf_rn(hi.x, inv.x, b.x);
		const float ay = __fmaf_rn(lo.y, inv.y, a.y), by = __fmaf_rn(hi.y, inv.y, b.y);
		const float az = __fmaf_rn(lo.z, inv.z, a.z), bz = __fmaf_rn(hi.z, inv.z, b.z);
		t = fmaxf(fmaxf(fminf(ax, bx), fminf(ay, by)), fmaxf(fminf(az, bz), 0.0f));
		const float u = fminf(fminf(fmaxf(ax, bx), fmaxf(ay, by)), fminf(fmaxf(az, bz), limit));
		return t <= u && lo.x <= hi.x;
	}
};

// Largest coordinate of a query, for the slack of its box tests.
__device__ __forceinline__ float coord_mag(V3 a, V3 b)
{
	return fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fabsf(a.z)), fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fabsf(b.z)));
}

// ---------------------------------------------------------------------------
// Ordered walks.
//
// The walks below visit the tree in the order a query meets its boxes: of a
// node's two children the nearer is taken next, the other goes on a stack with
// the fraction at which it is met and is dropped there if something nearer
// was found meanwhile. Such a walk is a chain of dependent loads, so each call
// first lays the tree out for it (k_walk_tree): one 64-byte record per inner
// node with both children's boxes and references, and one per leaf with all
// that its tests read but a hull's planes. The layout is made by every call,
// for the boxes and transforms of the last pass; 65,536 leaves take 4 us,
// where walking the pass's own arrays takes six loads from four arrays a level
// and a chain of fixture, body and transform loads a leaf.

// Child references: an inner node's index, or a leaf's with this bit.
constexpr uint32_t WALK_LEAF = 1u << 31;

// Leaf kinds: the shape types, and leaves that are never met.
constexpr uint32_t LEAF_NONE = 7u;

// turned (when set): receives 1 if a live triangle fixture sits on a body away
// from the identity transform. The reference ignores the transform in a
// triangle's AABB (triangle_shape.cpp:59-67), so such a fixture lies outside
// its box: a hit on it says nothing of where the box is met, no box that a ray
// meets is skipped for a hit before it, and a shape cast may not skip boxes its
// motion does not meet.
__global__ void k_walk_tree(QueryCtx q, float4* nodes, float4* leaves, uint32_t* turned)
{
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	const uint32_t inner = q.leaves - 1u;
	if (i < inner)
	{
		const uint32_t l = __float_as_uint(q.nodeLo[i].w), r = q.nodeRight[i];
		const float4 l0 = q.nodeLo[l], l1 = q.nodeHi[l], r0 = q.nodeLo[r], r1 = q.nodeHi[r];
		auto ref = [&](uint32_t c) { return __uint_as_float(c < inner ? c : (c - inner) | WALK_LEAF); };
		float4* n = nodes + 4 * (size_t)i;
		n[0] = make_float4(l0.x, l0.y, l0.z, l1.x);
		n[1] = make_float4(l1.y, l1.z, r0.x, r0.y);
		n[2] = make_float4(r0.z, r1.x, r1.y, r1.z);
		n[3] = make_float4(ref(l), ref(r), 0.0f, 0.0f);
	}
	if (i >= q.leaves)
		return;
	const DevScene& S = q.S;
	const uint32_t f = __float_as_uint(q.nodeLo[inner + i].w);
	const uint32_t body = S.fixBody[f], type = S.fixType[f];
	const XF xf = body_xf(S, body);
	const float4 bound = S.fixBound[f];
	const V3 c = xmul(xf, V3{bound.x, bound.y, bound.z});
	const float4 p0 = S.fixParams[3 * f], p1 = S.fixParams[3 * f + 1];
	uint32_t kind = S.fixLife[f] == FIX_DEAD ? LEAF_NONE : type, off = 0, blunt = 0;
	if (turned && kind == B3G_SHAPE_TRIANGLE &&
		!(xf.p.x == 0.0f && xf.p.y == 0.0f && xf.p.z == 0.0f && xf.q.v.x == 0.0f && xf.q.v.y == 0.0f && xf.q.v.z == 0.0f))
		*turned = 1u;
	float4 s0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), s1 = s0;
	if (type == B3G_SHAPE_SPHERE)
	{
		const V3 m = xmul(xf, V3{p0.x, p0.y, p0.z});
		s0 = make_float4(m.x, m.y, m.z, p0.w);
	}
	else if (type == B3G_SHAPE_CAPSULE)
	{
		const V3 a = xmul(xf, V3{p0.x, p0.y, p0.z}), e = xmul(xf, V3{p0.w, p1.x, p1.y});
		s0 = make_float4(a.x, a.y, a.z, p1.z);
		s1 = make_float4(e.x, e.y, e.z, 0.0f);
	}
	else if (type == B3G_SHAPE_HULL)
	{
		const HullDesc h = S.hulls[S.fixHull[f]];
		off = h.fOff;
		blunt = h.blunt;
		kind |= h.fCnt << 3;
		s0 = make_float4(xf.p.x, xf.p.y, xf.p.z, xf.q.s);
		s1 = make_float4(xf.q.v.x, xf.q.v.y, xf.q.v.z, 0.0f);
	}
	// Only the hulls of which a bounding sphere says enough are tested against
	// it (ray_reaches).
	float4* o = leaves + 4 * (size_t)i;
	o[0] = make_float4(c.x, c.y, c.z, blunt ? bound.w : INFINITY);
	o[1] = make_float4(__uint_as_float(f), __uint_as_float(kind), __uint_as_float(S.bodyWorld[body]), __uint_as_float(off));
	o[2] = s0;
	o[3] = s1;
}

struct WalkTree
{
	const float4* nodes;
	const float4* leaves;
	const uint32_t* turned; // see k_walk_tree; nullptr: no triangles
	uint32_t count;         // leaves
	bool own;               // the records are this call's alone
};

// A path's keys share one bit more at every level (64 key bits, then 32 index
// bits), so a depth-first stack never holds more than 96 entries.
constexpr uint32_t WALK_STACK = 96;

__device__ __forceinline__ uint32_t walk_root(const WalkTree& t) { return t.count > 1u ? 0u : WALK_LEAF; }

// The children of inner node `node` met within limit, the nearer in a (with
// its entry fraction ta); returns their number.
__device__ __forceinline__ uint32_t walk_expand(const WalkTree& t, const SlabTest& slab, uint32_t node, float limit,
	uint32_t& a, float& ta, uint32_t& b, float& tb)
{
	const float4* n = t.nodes + 4 * (size_t)node;
	const float4 n0 = __ldg(n), n1 = __ldg(n + 1), n2 = __ldg(n + 2);
	const float2 ref = __ldg(reinterpret_cast<const float2*>(n + 3));
	float tl, tr;
	const bool hl = slab.enter(V3{n0.x, n0.y, n0.z}, V3{n0.w, n1.x, n1.y}, limit, tl);
	const bool hr = slab.enter(V3{n1.z, n1.w, n2.x}, V3{n2.y, n2.z, n2.w}, limit, tr);
	const uint32_t l = __float_as_uint(ref.x), r = __float_as_uint(ref.y);
	const bool leftFirst = hl && (!hr || tl <= tr);
	a = leftFirst ? l : r;
	b = leftFirst ? r : l;
	ta = leftFirst ? tl : tr;
	tb = leftFirst ? tr : tl;
	return (hl ? 1u : 0u) + (hr ? 1u : 0u);
}

// b3Fixture::RayCast of the fixture of a leaf record: the shape casts of
// ray_fixture from the record's world-space data (the same expressions).
__device__ __forceinline__ bool ray_leaf(RayOut& o, const RayIn& in, const QueryCtx& q, const float4* rec, uint32_t kind,
	uint32_t f, uint32_t off)
{
	const uint32_t type = kind & 7u;
	const float4 s0 = __ldg(rec + 2), s1 = __ldg(rec + 3);
	if (type == B3G_SHAPE_SPHERE)
		return ray_sphere_world(o, in, V3{s0.x, s0.y, s0.z}, s0.w);
	if (type == B3G_SHAPE_CAPSULE)
		return ray_capsule_world(o, in, V3{s0.x, s0.y, s0.z}, V3{s1.x, s1.y, s1.z}, s0.w);
	if (type == B3G_SHAPE_HULL)
	{
		XF xf;
		xf.p = V3{s0.x, s0.y, s0.z};
		xf.q = Q4{V3{s1.x, s1.y, s1.z}, s0.w};
		return ray_planes(o, in, xf, q.S.hplanes + off, kind >> 3);
	}
	return ray_fixture(o, in, q.S, f, q.status);
}

// Whether leaf `leaf` is to be cast: live, in the ray's world, and, for a
// blunt hull, its bounding sphere within reach of the segment.
//
// A cast accepts rays that pass its shape at a distance, by its rounding, and
// such a hit counts like any other. A hull's cast, some 30 roundings in a row
// of lengths up to 3.5 M (M: the largest coordinate), is off by less than 32
// eps/2 of that, e = 7e-6 M, at each plane: the ray meets the hull with its
// planes moved out by e, which reaches e R / r past the hull, where R is its
// radius around the centroid and r the centroid's distance from the nearest
// plane. Blunt is R <= 16 r, so 2e-4 M covers it. A sphere's or a capsule's
// discriminant is off by what grows with the square of the length over the
// radius (at 100 m and 0.1 m rays 16 mm outside are hits), and a triangle has
// no inside; they are always cast. 524,288 rays of 10 m among 65,536 bodies,
// all shapes tested against their spheres: 1.06 ms, hulls alone 1.05 ms.
__device__ __forceinline__ bool ray_reaches(const WalkTree& t, const RayIn& in, uint32_t world, uint32_t leaf,
	uint32_t& kind)
{
	const float4* rec = t.leaves + 4 * (size_t)leaf;
	const float4 bound = __ldg(rec), id = __ldg(rec + 1);
	kind = __float_as_uint(id.y);
	if ((kind & 7u) == LEAF_NONE || __float_as_uint(id.z) != world)
		return false;
	const V3 c = V3{bound.x, bound.y, bound.z};
	const V3 d = in.p2 - in.p1, m = c - in.p1;
	const float s = fminf(fmaxf(dot(m, d) / dot(d, d), 0.0f), 1.0f);
	const V3 e = m - s * d;
	const float reach = bound.w + (1e-3f + 2e-4f * fmaxf(coord_mag(in.p1, in.p2), coord_mag(c, c)));
	return !(dot(e, e) > reach * reach);
}

// The cast of such a leaf: a hit is the shape's, where the whole segment also
// passes the reference's own test of the leaf's box.
__device__ __forceinline__ bool ray_hits(RayOut& o, uint32_t& f, const QueryCtx& q, const WalkTree& t, const RayIn& in,
	uint32_t leaf)
{
	const float4* rec = t.leaves + 4 * (size_t)leaf;
	const float4 id = __ldg(rec + 1);
	f = __float_as_uint(id.x);
	if (!ray_leaf(o, in, q, rec, __float_as_uint(id.y), f, __float_as_uint(id.w)))
		return false;
	const float4 lo = __ldg(q.nodeLo + (t.count - 1u + leaf)), hi = __ldg(q.nodeHi + (t.count - 1u + leaf));
	SegTest seg;
	seg.init(in.p1, in.p2, in.maxFraction);
	return seg.pass(V3{lo.x, lo.y, lo.z}, V3{hi.x, hi.y, hi.z});
}

// The entry fraction from which boxes are left out once a hit at `fraction` is
// known. A hit lies in its fixture's fat box but for the rounding of its
// fraction, at most the root of a discriminant's: sqrt(16 eps/2) = 1e-3 of the
// distance to the shape over the length, 3e-3 for shapes up to the ray's length.
constexpr float RAY_SLACK = 0x1p-8f;
// turned: see k_walk_tree.
__device__ __forceinline__ float ray_limit(float fraction, bool turned)
{
	return turned ? 1.0f : fminf(fraction + RAY_SLACK, 1.0f);
}

__device__ __forceinline__ void ray_slab(SlabTest& slab, const RayIn& in)
{
	slab.init(in.p1, in.p1, in.p2 - in.p1, 1e-5f * coord_mag(in.p1, in.p2) + 1e-6f);
}

__device__ __forceinline__ void ray_write(uint32_t* outFix, float* outHit, uint32_t i, const RayIn& in, uint32_t best,
	float fraction, V3 normal)
{
	const bool hit = best != B3G_NULL;
	outFix[i] = best;
	float* h = outHit + 7 * (size_t)i;
	V3 p = hit ? (1.0f - fraction) * in.p1 + fraction * in.p2 : V3{0.0f, 0.0f, 0.0f};
	h[0] = p.x, h[1] = p.y, h[2] = p.z;
	h[3] = hit ? normal.x : 0.0f, h[4] = hit ? normal.y : 0.0f, h[5] = hit ? normal.z : 0.0f;
	h[6] = hit ? fraction : 0.0f;
}

__device__ __forceinline__ RayIn load_ray(const float* rays, uint32_t i)
{
	RayIn in;
	in.p1 = V3{rays[6 * (size_t)i], rays[6 * (size_t)i + 1], rays[6 * (size_t)i + 2]};
	in.p2 = V3{rays[6 * (size_t)i + 3], rays[6 * (size_t)i + 4], rays[6 * (size_t)i + 5]};
	in.maxFraction = 1.0f;
	return in;
}

// b3World::RayCastSingle (the smallest fraction, the smaller fixture on an
// exact tie), many rays: a lane walks its ray, and the warp moves in step
// (every lane one level or one stack entry further, then all meet again:
// written as a plain loop per ray the lanes never met before their rays' ends
// and ran nearly one after the other, 4 of 32 active). Walking, the tests of
// a leaf and the shape casts diverge differently, so they are kept apart: a
// lane that reaches a leaf puts it on its warp's queue and walks on; a full
// queue is taken by the whole warp, one leaf per lane, and the leaves to cast
// go on a queue per shape type, which a full warp empties in turn. A lane has
// two rays' places: it starts the next ray while the queues still hold leaves
// of the one before. Each warp has a fixed share of the rays. Measured,
// 524,288 rays of 10 m in the 65,536-body world: 6.2 ms with one thread per
// ray on a walk without order, 1.15 ms now (62 levels and 11 leaves a
// ray, at 14 of 32 lanes: issue of those and the waits for their loads bound
// it, not the 46 MB read and written).
constexpr int RAY_WARPS = 4;
constexpr int RAY_BLOCKS = 8;       // per SM: 6 took 1.21 ms, 4 took 1.34 ms
constexpr int RAY_STEPS = 4;        // levels between two looks at the queues: 2 took 1.28 ms
constexpr uint32_t RAY_LOW = 4;     // lanes walking below which part-filled queues are emptied
constexpr int RAY_TYPES = 4; // sphere, capsule, hull, the rest
constexpr uint32_t WALK_POP = SENT - 1u; // take the next stack entry

struct RayWarp
{
	unsigned long long best[64]; // per ray place: fraction bits, fixture; ~0: none
	float p[6][64];
	float fraction[64], normal[3][64]; // of the best
	uint32_t world[64];
	uint32_t pending[64];         // queued leaves of the place's ray
	uint32_t leaf[64];            // leaves reached
	uint32_t cast[RAY_TYPES][64]; // leaves to cast
	uint8_t leafOwner[64];        // their rays' places
	uint8_t owner[RAY_TYPES][64];
};

__device__ __forceinline__ RayIn warp_ray(const RayWarp& W, uint32_t place)
{
	RayIn in;
	in.p1 = V3{W.p[0][place], W.p[1][place], W.p[2][place]};
	in.p2 = V3{W.p[3][place], W.p[4][place], W.p[5][place]};
	in.maxFraction = 1.0f;
	return in;
}

__global__ void __launch_bounds__(RAY_WARPS * 32, RAY_BLOCKS) k_ray_first(QueryCtx q, WalkTree tree, const float* rays,
	const uint32_t* worlds, uint32_t n, uint32_t share, uint32_t* outFix, float* outHit)
{
	__shared__ RayWarp shared[RAY_WARPS];
	const bool turned = tree.turned && *tree.turned;
	const uint32_t lane = threadIdx.x & 31u;
	RayWarp& W = shared[threadIdx.x >> 5];
	const uint32_t warp = blockIdx.x * RAY_WARPS + (threadIdx.x >> 5);
	uint32_t next = min(warp * share, n);
	const uint32_t end = min(next + share, n);
	const uint32_t lt = (1u << lane) - 1u;
	uint2 stack[WALK_STACK]; // reference, entry fraction (float bits)
	uint32_t sp = 0, steps = 0, node = SENT;
	uint32_t cur = lane;                            // the place of the ray being walked
	uint32_t rayCur = B3G_NULL, rayOther = B3G_NULL; // the rays in places cur and cur ^ 32
	SlabTest slab;
	slab.inv = slab.a = slab.b = V3{0.0f, 0.0f, 0.0f};
	uint32_t leaves = 0, qn[RAY_TYPES] = {0, 0, 0, 0};
	W.pending[lane] = W.pending[lane + 32u] = 0;
	W.best[lane] = W.best[lane + 32u] = ~0ull;
	__syncwarp();
	auto finish = [&](uint32_t place, uint32_t& r) {
		const unsigned long long key = W.best[place];
		ray_write(outFix, outHit, r, warp_ray(W, place), key == ~0ull ? B3G_NULL : (uint32_t)key, W.fraction[place],
			V3{W.normal[0][place], W.normal[1][place], W.normal[2][place]});
		r = B3G_NULL;
	};
	for (;;)
	{
		// Rays whose leaves are all done are written; a lane whose walk is over
		// goes on with its other place once that is free.
		if (rayOther != B3G_NULL && W.pending[cur ^ 32u] == 0)
			finish(cur ^ 32u, rayOther);
		__syncwarp();
		if (node == SENT && rayCur != B3G_NULL && rayOther == B3G_NULL)
		{
			rayOther = rayCur;
			rayCur = B3G_NULL;
			cur ^= 32u;
		}
		const bool idle = rayCur == B3G_NULL;
		const uint32_t want = __ballot_sync(0xFFFFFFFFu, idle);
		if (want != 0u && next < end)
		{
			const uint32_t mine = next + __popc(want & lt);
			if (idle && mine < end)
			{
				rayCur = mine;
				const RayIn in = load_ray(rays, mine);
				W.p[0][cur] = in.p1.x, W.p[1][cur] = in.p1.y, W.p[2][cur] = in.p1.z;
				W.p[3][cur] = in.p2.x, W.p[4][cur] = in.p2.y, W.p[5][cur] = in.p2.z;
				W.world[cur] = worlds ? worlds[mine] : 0u;
				W.best[cur] = ~0ull;
				sp = 0;
				steps = 0;
				const V3 d = in.p2 - in.p1;
				if (dot(d, d) > 0.0f)
				{
					ray_slab(slab, in);
					node = walk_root(tree);
				}
			}
			next = min(next + (uint32_t)__popc(want), end);
		}
		__syncwarp();
		// Walk toward the next leaf, a few levels at a time.
		const unsigned long long key = W.best[cur];
		const float limit = key == ~0ull ? 1.0f : ray_limit(__uint_as_float((uint32_t)(key >> 32)), turned);
#pragma unroll 1
		for (int k = 0; k < RAY_STEPS; ++k)
		{
			bool popNow = node == WALK_POP;
			if (node < WALK_LEAF)
			{
				uint32_t a, b;
				float ta, tb;
				const uint32_t hits = walk_expand(tree, slab, node, limit, a, ta, b, tb);
				if (hits == 2u)
					stack[min(sp, WALK_STACK - 1u)] = make_uint2(b, __float_as_uint(tb));
				sp += hits == 2u ? 1u : 0u;
				node = a;
				popNow = hits == 0u;
				if (++steps > 2u * tree.count || sp > WALK_STACK)
				{
					atomicOr(q.status, B3G_ST_WAIT_TIMEOUT);
					popNow = true;
					sp = 0;
				}
			}
			if (popNow)
			{
				node = SENT;
				if (sp > 0)
				{
					const uint2 e = stack[--sp];
					node = __uint_as_float(e.y) <= limit ? e.x : WALK_POP;
				}
			}
			__syncwarp();
		}
		const bool reached = node >= WALK_LEAF && node < WALK_POP;
		const uint32_t m = __ballot_sync(0xFFFFFFFFu, reached);
		if (reached)
		{
			const uint32_t pos = leaves + __popc(m & lt);
			W.leaf[pos] = node & ~WALK_LEAF;
			W.leafOwner[pos] = (uint8_t)cur;
			++W.pending[cur];
			node = sp > 0 ? WALK_POP : SENT;
		}
		leaves += __popc(m);
		// The queues are emptied by full warps, and as far as they go when few
		// lanes are left walking.
		const uint32_t walking = __popc(__ballot_sync(0xFFFFFFFFu, node != SENT));
		const bool low = walking < RAY_LOW;
		if (leaves < 32u && !low)
			continue;
		__syncwarp();
		if (leaves > 0u)
		{
			const uint32_t take = min(leaves, 32u);
			leaves -= take;
			uint32_t type = RAY_TYPES, leaf = 0, owner = 0;
			if (lane < take)
			{
				owner = W.leafOwner[leaves + lane];
				leaf = W.leaf[leaves + lane];
				uint32_t kind;
				if (ray_reaches(tree, warp_ray(W, owner), W.world[owner], leaf, kind))
				{
					const uint32_t shape = kind & 7u;
					type = shape == B3G_SHAPE_SPHERE ? 0u
													 : (shape == B3G_SHAPE_CAPSULE ? 1u : (shape == B3G_SHAPE_HULL ? 2u : 3u));
				}
				else
					atomicSub(&W.pending[owner], 1u);
			}
#pragma unroll
			for (uint32_t k = 0; k < RAY_TYPES; ++k)
			{
				const uint32_t mk = __ballot_sync(0xFFFFFFFFu, type == k);
				if (type == k)
				{
					const uint32_t pos = qn[k] + __popc(mk & lt);
					W.cast[k][pos] = leaf;
					W.owner[k][pos] = (uint8_t)owner;
				}
				qn[k] += __popc(mk);
			}
			__syncwarp();
		}
		const bool drain = low && leaves == 0u;
#pragma unroll 1
		for (uint32_t k = 0; k < RAY_TYPES; ++k)
		{
			const uint32_t have = k == 0u ? qn[0] : (k == 1u ? qn[1] : (k == 2u ? qn[2] : qn[3]));
			if (have < 32u && !(drain && have > 0u))
				continue;
			const uint32_t take = min(have, 32u);
			const uint32_t left = have - take;
			qn[0] = k == 0u ? left : qn[0];
			qn[1] = k == 1u ? left : qn[1];
			qn[2] = k == 2u ? left : qn[2];
			qn[3] = k == 3u ? left : qn[3];
			unsigned long long mine = ~0ull;
			uint32_t owner = 0;
			RayOut o;
			if (lane < take)
			{
				owner = W.owner[k][left + lane];
				uint32_t f;
				// A NaN fraction is below no other and never the first. The bits of
				// the others order as the fractions do, but for -0 (a ray that starts
				// in a triangle's plane): the key takes it as +0.
				if (ray_hits(o, f, q, tree, warp_ray(W, owner), W.cast[k][left + lane]) && o.fraction < B3G_MAX_SCALAR)
				{
					mine = ((unsigned long long)__float_as_uint(o.fraction + 0.0f) << 32) | f;
					atomicMin(&W.best[owner], mine);
				}
				atomicSub(&W.pending[owner], 1u);
			}
			__syncwarp();
			// A fixture is one leaf, so a key has one lane.
			if (mine != ~0ull && W.best[owner] == mine)
			{
				W.fraction[owner] = o.fraction;
				W.normal[0][owner] = o.normal.x, W.normal[1][owner] = o.normal.y, W.normal[2][owner] = o.normal.z;
			}
			__syncwarp();
		}
		if (walking == 0u && next >= end && leaves + qn[0] + qn[1] + qn[2] + qn[3] == 0u)
		{
			// Only results are left to write, if any.
			if (rayOther != B3G_NULL)
				finish(cur ^ 32u, rayOther);
			if (rayCur != B3G_NULL)
				finish(cur, rayCur);
			break;
		}
	}
}

// The same for few rays: a warp per ray. The warp's stack in shared memory
// holds the nodes still to visit; up to 32 are taken at a time (the nearer
// children are pushed last, so they come first), inner nodes push their
// children, leaves cast their shapes, and the best fraction so far drops the
// rest. A ray takes about as many rounds as the tree is deep, where one lane
// would wait for every node and shape in turn. Bound by the latency of those
// rounds. Measured, 100 rays of 10 m in a 5,000-body world, host copies and
// all: 680 us with one thread per ray on a walk without order, 97 us now.
constexpr uint32_t RAY_FRONT = 1024; // stack entries per warp

__global__ void __launch_bounds__(32) k_ray_first_warp(QueryCtx q, WalkTree tree, const float* rays,
	const uint32_t* worlds, uint32_t n, uint32_t* outFix, float* outHit)
{
	__shared__ uint2 stack[RAY_FRONT]; // reference, entry fraction (float bits)
	const bool turned = tree.turned && *tree.turned;
	const uint32_t lane = threadIdx.x;
	const uint32_t lt = (1u << lane) - 1u;
	const uint32_t i = blockIdx.x;
	const RayIn in = load_ray(rays, i);
	const uint32_t world = worlds ? worlds[i] : 0u;
	uint32_t best = B3G_NULL;
	RayOut bestOut;
	bestOut.fraction = B3G_MAX_SCALAR;
	bestOut.normal = V3{0.0f, 0.0f, 0.0f};
	const V3 d = in.p2 - in.p1;
	uint32_t size = 0, steps = 0;
	SlabTest slab;
	if (dot(d, d) > 0.0f)
	{
		ray_slab(slab, in);
		if (lane == 0)
			stack[0] = make_uint2(walk_root(tree), 0u);
		size = 1;
	}
	float limit = 1.0f;
	__syncwarp();
	while (size > 0)
	{
		// Near the end of the stack one node at a time: depth first, which
		// adds at most WALK_STACK entries.
		const uint32_t take = size > RAY_FRONT - 64u - WALK_STACK ? 1u : min(size, 32u);
		steps += take;
		if (steps > 4u * tree.count)
		{
			if (lane == 0)
				atomicOr(q.status, B3G_ST_WAIT_TIMEOUT);
			break;
		}
		uint2 e = make_uint2(SENT, 0u);
		if (lane < take)
			e = stack[size - 1u - lane];
		size -= take;
		__syncwarp();
		uint32_t hits = 0, a = 0, b = 0;
		float ta = 0.0f, tb = 0.0f;
		if (e.x != SENT && __uint_as_float(e.y) <= limit)
		{
			if (e.x < WALK_LEAF)
				hits = walk_expand(tree, slab, e.x, limit, a, ta, b, tb);
			else
			{
				const uint32_t leaf = e.x & ~WALK_LEAF;
				uint32_t kind, f;
				RayOut o;
				if (ray_reaches(tree, in, world, leaf, kind) && ray_hits(o, f, q, tree, in, leaf) &&
					(o.fraction < bestOut.fraction || (o.fraction == bestOut.fraction && f < best)))
				{
					best = f;
					bestOut = o;
				}
			}
		}
		// Far children below the near ones; the first lane took the top of the
		// stack, so its child goes back on top.
		const uint32_t two = __ballot_sync(0xFFFFFFFFu, hits == 2u), one = __ballot_sync(0xFFFFFFFFu, hits >= 1u);
		if (hits == 2u)
			stack[size + __popc(two & ~lt) - 1u] = make_uint2(b, __float_as_uint(tb));
		size += __popc(two);
		if (hits >= 1u)
			stack[size + __popc(one & ~lt) - 1u] = make_uint2(a, __float_as_uint(ta));
		size += __popc(one);
		float least = fminf(limit, ray_limit(bestOut.fraction, turned));
		for (int o = 16; o > 0; o >>= 1)
			least = fminf(least, __shfl_xor_sync(0xFFFFFFFFu, least, o));
		limit = least;
		__syncwarp();
	}
	float least = bestOut.fraction;
	uint32_t first = best;
	for (int o = 16; o > 0; o >>= 1)
	{
		const float of = __shfl_xor_sync(0xFFFFFFFFu, least, o);
		const uint32_t ob = __shfl_xor_sync(0xFFFFFFFFu, first, o);
		if (of < least || (of == least && ob < first))
		{
			least = of;
			first = ob;
		}
	}
	if (first == B3G_NULL ? lane == 0 : best == first)
		ray_write(outFix, outHit, i, in, first, bestOut.fraction, bestOut.normal);
}

// Rays up to this many go a warp each. Both kernels' times at 12,000 rays:
// 124 and 286 us; at 40,000: 459 and 317 us. In worlds of 300, 5,000 and 65,536
// bodies, with rays of 1, 10, 100 and 1,000 m, a warp each takes time by their
// number and a lane each hardly more from one to 48,000; the lines cross between
// 17,000 and 26,000.
constexpr uint32_t RAY_WARP_MAX = 148u * 160u;

// The tree laid out for the ordered walks, in records that no other call writes
// while this one's walk reads them (as read-only memory). They are the
// context's, and a call waits for the last one's walk where that ran on another
// stream. A captured call, whose replays the host does not see, has records of
// its own, as nodes of its graph.
cudaError_t launch_walk_tree(b3g_ctx* c, const QueryCtx& q, WalkTree& t, cudaStream_t s)
{
	float4* nodes = c->buf.walkTree;
	t.own = s != c->stream && in_capture(s);
	cudaError_t e = cudaSuccess;
	if (t.own)
		e = cudaMallocAsync((void**)&nodes, sizeof(float4) * walk_tree_words(c->cfg.max_proxies), s);
	else if (s != c->stream || c->walkBeside)
	{
		// A walk on a caller's stream was recorded there. The stream may be gone
		// by now and another have its handle, so a caller's always waits.
		if (!c->walkBeside)
			e = cudaEventRecord(c->walkDone, c->stream);
		if (e == cudaSuccess)
			e = cudaStreamWaitEvent(s, c->walkDone, 0);
		c->walkBeside = s != c->stream;
	}
	if (e != cudaSuccess)
	{
		cudaGetLastError();
		return e;
	}
	float4* leaves = nodes + 4 * (size_t)c->cfg.max_proxies;
	uint32_t* turned = c->anyTriangle ? reinterpret_cast<uint32_t*>(nodes + 8 * (size_t)c->cfg.max_proxies) : nullptr;
	if (turned)
		e = cudaMemsetAsync(turned, 0, sizeof(uint32_t), s);
	t.nodes = nodes;
	t.leaves = leaves;
	t.turned = turned;
	t.count = q.leaves;
	k_walk_tree<<<(q.leaves + 127) / 128, 128, 0, s>>>(q, nodes, leaves, turned);
	return e;
}

// The call's walk is launched.
cudaError_t end_walk(b3g_ctx* c, const WalkTree& t, cudaStream_t s)
{
	if (t.own)
		return cudaFreeAsync(const_cast<float4*>(t.nodes), s);
	return s == c->stream ? cudaSuccess : cudaEventRecord(c->walkDone, s);
}

cudaError_t launch_ray_first(b3g_ctx* c, const QueryCtx& q, const float* rays, const uint32_t* worlds, uint32_t n, uint32_t* fix,
	float* hit, cudaStream_t s)
{
	WalkTree t;
	cudaError_t e = launch_walk_tree(c, q, t, s);
	if (e != cudaSuccess)
		return e;
	if (n <= RAY_WARP_MAX)
		k_ray_first_warp<<<n, 32, 0, s>>>(q, t, rays, worlds, n, fix, hit);
	else
	{
		// Resident warps, each with an equal share of at least a warp's rays.
		const uint32_t warps = std::min((n + 31u) / 32u, 148u * RAY_BLOCKS * RAY_WARPS);
		const uint32_t share = (n + warps - 1u) / warps;
		k_ray_first<<<(warps + RAY_WARPS - 1u) / RAY_WARPS, RAY_WARPS * 32, 0, s>>>(q, t, rays, worlds, n, share, fix, hit);
	}
	return end_walk(c, t, s);
}

// ---------------------------------------------------------------------------
// Shape casts: b3World::ShapeCast / ShapeCastSingle (world.cpp:568-851), each
// candidate fixture (fat AABB overlapping the swept AABB of the cast shape)
// tested with the translational b3TimeOfImpact (time_of_impact.cpp:666-776)
// and the touching ones evaluated with b3GJK at the time of impact.

// b3TOIOutput::State (time_of_impact.h:40-47).
enum : uint32_t
{
	TOI_UNKNOWN = 0,
	TOI_FAILED,
	TOI_OVERLAPPED,
	TOI_TOUCHING,
	TOI_SEPARATED
};

struct TOIOut
{
	uint32_t state;
	float t;
};

// b3TimeOfImpact(xf1, proxy1, d1, xf2, proxy2, d2) (time_of_impact.cpp:666-776):
// Mirtich's conservative advancement along the translations, the GJK simplex
// carried from one iteration to the next, at most 20 iterations.
__device__ __noinline__ TOIOut toi_translate(const XF& xf1, const GProxy& p1, V3 d1, const XF& xf2, const GProxy& p2,
	V3 d2)
{
	const float totalRadius = p1.radius + p2.radius;
	const float target = fmaxr(B3G_LINEAR_SLOP, totalRadius - 3.0f * B3G_LINEAR_SLOP);
	const float tolerance = 0.25f * B3G_LINEAR_SLOP;
	GJKCache cache;
	cache.count = 0;
	cache.metric = 0.0f;
	for (int i = 0; i < 4; ++i)
		cache.index1[i] = cache.index2[i] = 0u;
	float t = 0.0f;
	XF xf1t = xf1, xf2t = xf2;
	for (uint32_t iteration = 0; iteration < 20u; ++iteration)
	{
		GJKOut q = gjk_cached(xf1t, p1, xf2t, p2, cache);
		if (q.distance == 0.0f)
			return TOIOut{TOI_OVERLAPPED, 0.0f};
		if (q.distance < target + tolerance)
			return TOIOut{TOI_TOUCHING, t};
		V3 n = (q.point2 - q.point1) / q.distance;
		float denominator = dot(d2 - d1, n);
		if (denominator >= 0.0f)
			return TOIOut{TOI_SEPARATED, 1.0f};
		float dt = (target - q.distance) / denominator;
		t += dt;
		if (t >= 1.0f)
			return TOIOut{TOI_SEPARATED, 1.0f};
		xf1t.p = xf1.p + t * d1;
		xf2t.p = xf2.p + t * d2;
	}
	return TOIOut{TOI_UNKNOWN, t};
}

// The proxy of a mesh fixture's triangle (gjk.cpp:75-89): its vertices
// scaled by the mesh scale, the mesh radius.
__device__ GProxy mesh_triangle_proxy(const DevScene& S, uint32_t fix, uint32_t tri)
{
	const MeshDesc md = S.meshes[S.fixHull[fix]];
	const float4 sp = S.fixParams[3 * fix];
	const V3 sc = V3{sp.x, sp.y, sp.z};
	const uint4 t = S.meshTris[md.tOff + tri];
	auto vert = [&](uint32_t i) {
		float4 a = S.meshVerts[md.vOff + i];
		return vmul(sc, V3{a.x, a.y, a.z});
	};
	GProxy g;
	g.gv = nullptr;
	g.lv[0] = vert(t.x);
	g.lv[1] = vert(t.y);
	g.lv[2] = vert(t.z);
	g.count = 3;
	g.radius = sp.w;
	return g;
}

// b3WorldShapeCastQueryWrapper::Evaluate (world.cpp:719-731).
__device__ __noinline__ void cast_evaluate(V3& point, V3& normal, const XF& xA, const GProxy& pA, const XF& xB,
	const GProxy& pB)
{
	GJKOut q = gjk(xA, pA, xB, pB, false);
	normal = normalized(q.point1 - q.point2);
	point = q.point2 + pB.radius * normal;
}

struct CastIn
{
	uint32_t type, hull, world;
	float4 p0, p1, p2;
	XF xf;
	V3 d;
};

// b3g_shape_cast_input: type, hull, world, pad, params[12], position[3],
// rotation[4], displacement[3], pad[2].
__device__ __forceinline__ CastIn load_cast(const float* in, uint32_t i)
{
	const float* r = in + 28 * (size_t)i;
	CastIn c;
	c.type = __float_as_uint(r[0]);
	c.hull = __float_as_uint(r[1]);
	c.world = __float_as_uint(r[2]);
	c.p0 = make_float4(r[4], r[5], r[6], r[7]);
	c.p1 = make_float4(r[8], r[9], r[10], r[11]);
	c.p2 = make_float4(r[12], r[13], r[14], r[15]);
	c.xf.p = V3{r[16], r[17], r[18]};
	c.xf.q = Q4{V3{r[19], r[20], r[21]}, r[22]};
	c.d = V3{r[23], r[24], r[25]};
	return c;
}

// The cast's end transform and swept AABB (world.cpp:759-768).
__device__ __forceinline__ AABB cast_sweep(const DevScene& S, const CastIn& in, XF& xf2)
{
	xf2 = in.xf;
	xf2.p = in.xf.p + in.d;
	AABB a1, a2;
	compute_shape_aabbs(S, in.type, in.p0, in.p1, in.p2, in.hull, in.xf, xf2, true, a1, a2);
	AABB sw;
	sw.lo = vmin(a1.lo, a2.lo);
	sw.hi = vmax(a1.hi, a2.hi);
	return sw;
}

__device__ __forceinline__ bool box_overlap(const AABB& b, float4 lo, float4 hi)
{
	return !(hi.x < b.lo.x || lo.x > b.hi.x || hi.y < b.lo.y || lo.y > b.hi.y || hi.z < b.lo.z || lo.z > b.hi.z);
}

// Mesh fixture f against cast `in`: the triangles under the swept box in the
// unscaled mesh frame (world.cpp:638-664), in the static tree's depth-first
// order; visit(triangle, toi, proxy) for each touching one.
template <class Visit>
__device__ __forceinline__ void cast_mesh(const QueryCtx& q, const CastIn& in, const GProxy& pA, const XF& xf2,
	uint32_t f, const XF& xfB, Visit&& visit)
{
	const DevScene& S = q.S;
	const MeshDesc md = S.meshes[S.fixHull[f]];
	const float4 sp = S.fixParams[3 * f];
	const V3 inv = V3{1.0f / sp.x, 1.0f / sp.y, 1.0f / sp.z};
	AABB m1, m2;
	compute_shape_aabbs(S, in.type, in.p0, in.p1, in.p2, in.hull, xmult(xfB, in.xf), xmult(xfB, xf2), true, m1, m2);
	m1 = aabb_scaled(m1, inv);
	m2 = aabb_scaled(m2, inv);
	AABB box;
	box.lo = vmin(m1.lo, m2.lo);
	box.hi = vmax(m1.hi, m2.hi);
	const V3 zero = V3{0.0f, 0.0f, 0.0f};
	constexpr uint32_t STACK = 64;
	uint32_t stack[STACK];
	uint32_t sp_ = 0;
	stack[sp_++] = md.root;
	while (sp_ > 0)
	{
		uint32_t id = stack[--sp_];
		if (id == B3G_NULL_NODE)
			continue;
		float4 nlo = S.meshNodes[2 * (size_t)(md.nOff + id)], nhi = S.meshNodes[2 * (size_t)(md.nOff + id) + 1];
		if (!box_overlap(box, nlo, nhi))
			continue;
		uint32_t child1 = __float_as_uint(nlo.w), other = __float_as_uint(nhi.w);
		if (child1 == B3G_NULL_NODE)
		{
			const GProxy pB = mesh_triangle_proxy(S, f, other);
			TOIOut r = toi_translate(in.xf, pA, in.d, xfB, pB, zero);
			if (r.state == TOI_TOUCHING)
				visit(other, r.t, pB);
		}
		else
		{
			if (sp_ + 2 > STACK)
			{
				atomicOr(q.status, B3G_ST_POLY_OVERFLOW);
				return;
			}
			stack[sp_++] = child1;
			stack[sp_++] = other;
		}
	}
}

// One (cast, fixture) candidate on one lane: the time of impact against a
// convex fixture, or against each triangle of a mesh fixture. MODE 0 counts
// the touching results in *count, MODE 1 writes them (slot base + a count
// taken from *count), MODE 2 lowers *best to (fraction bits, fixture).
template <int MODE>
__device__ __noinline__ void cast_candidate(const QueryCtx& q, const float* casts, uint32_t i, uint32_t f,
	uint32_t* count, uint32_t base, uint32_t* outIdx, float* outHit, uint32_t capacity, unsigned long long* best)
{
	const DevScene& S = q.S;
	const CastIn in = load_cast(casts, i);
	const GProxy pA = convex_proxy(S, in.type, in.p0, in.p1, in.p2, in.hull);
	const XF xfB = body_xf(S, S.fixBody[f]);
	auto act = [&](uint32_t child, float t, const GProxy& pB) {
		if (MODE == 2)
		{
			atomicMin(best, ((unsigned long long)__float_as_uint(t) << 32) | f);
			return;
		}
		const uint32_t slot = atomicAdd(count, 1u);
		if (MODE == 1 && base + slot < capacity)
		{
			XF xt;
			xt.q = in.xf.q;
			xt.p = in.xf.p + t * in.d;
			V3 point, normal;
			cast_evaluate(point, normal, xt, pA, xfB, pB);
			uint32_t* o = outIdx + 3 * (size_t)(base + slot);
			o[0] = i;
			o[1] = f;
			o[2] = child;
			float* h = outHit + 7 * (size_t)(base + slot);
			h[0] = point.x, h[1] = point.y, h[2] = point.z;
			h[3] = normal.x, h[4] = normal.y, h[5] = normal.z;
			h[6] = t;
		}
	};
	if (S.fixType[f] != B3G_SHAPE_MESH)
	{
		const GProxy pB =
			convex_proxy(S, S.fixType[f], S.fixParams[3 * f], S.fixParams[3 * f + 1], S.fixParams[3 * f + 2], S.fixHull[f]);
		TOIOut r = toi_translate(in.xf, pA, in.d, xfB, pB, V3{0.0f, 0.0f, 0.0f});
		if (r.state == TOI_TOUCHING)
			act(0u, r.t, pB);
		return;
	}
	XF xf2;
	cast_sweep(S, in, xf2);
	cast_mesh(q, in, pA, xf2, f, xfB, act);
}

// b3World::ShapeCast with a listener that returns 1 for every fixture
// (MODE 0 counts, MODE 1 writes (cast, fixture, triangle) + (point, normal,
// fraction), in no particular order within a cast).
//
// A warp holds 32 casts. Its lanes walk their casts' LBVH paths only until
// each finds its next candidate fixture (fat AABB overlapping the swept box)
// and push it into the warp's queue in shared memory; whenever 32 candidates
// are queued (or the walks are over) every lane takes one and runs its time
// of impact, so the lanes run the same GJK code on different candidates
// instead of each walking and testing its own cast alone. Per-cast counts
// meet in shared memory.
template <int MODE>
__global__ void __launch_bounds__(128) k_shape_cast(QueryCtx q, const float* casts, const uint32_t* order, uint32_t n,
	uint32_t* counts, uint32_t* outIdx, float* outHit, uint32_t capacity)
{
	constexpr int WARPS = 4;
	__shared__ uint32_t qLane[WARPS][64], qFix[WARPS][64];
	__shared__ uint32_t sCount[WARPS][32];
	const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
	const uint32_t warpBase = blockIdx.x * blockDim.x + w * 32u;
	const uint32_t t = warpBase + lane;
	const bool active = t < n;
	// Casts are taken in the order of their Morton keys, so the lanes of a
	// warp walk neighbouring parts of the tree; results go to their own slots.
	const uint32_t i = active ? (order ? order[t] : t) : 0u;
	sCount[w][lane] = 0;
	__syncwarp();
	const DevScene& S = q.S;
	bool walking = false;
	uint32_t world = 0;
	AABB sw;
	sw.lo = sw.hi = V3{0.0f, 0.0f, 0.0f};
	if (active)
	{
		const CastIn in = load_cast(casts, i);
		// A mesh cannot be cast (world.cpp:755-760).
		walking = in.type != B3G_SHAPE_MESH;
		world = in.world;
		XF xf2;
		sw = cast_sweep(S, in, xf2);
	}
	const uint32_t nodes = 2u * q.leaves - 1u;
	uint32_t node = 0, steps = 0, qn = 0;
	for (;;)
	{
		uint32_t f = 0;
		bool got = false;
		while (walking && node != SENT)
		{
			if (++steps > nodes + 1u || node >= nodes)
			{
				atomicOr(q.status, B3G_ST_WAIT_TIMEOUT);
				node = SENT;
				break;
			}
			const float4 lo = q.nodeLo[node], hi = q.nodeHi[node];
			const bool pass = box_overlap(sw, lo, hi);
			if (pass && node < q.leaves - 1u)
			{
				node = __float_as_uint(lo.w);
				continue;
			}
			node = __float_as_uint(hi.w);
			if (pass)
			{
				const uint32_t proxy = __float_as_uint(lo.w);
				if (box_overlap(sw, q.fatLo[proxy], q.fatHi[proxy]) && query_takes(q, proxy, world))
				{
					f = proxy;
					got = true;
					break;
				}
			}
		}
		if (!got)
			walking = false;
		const uint32_t m = __ballot_sync(0xFFFFFFFFu, got);
		if (got)
		{
			const uint32_t pos = qn + __popc(m & ((1u << lane) - 1u));
			qLane[w][pos] = lane;
			qFix[w][pos] = f;
		}
		qn += __popc(m);
		const bool more = __any_sync(0xFFFFFFFFu, walking);
		if (qn >= 32u || (!more && qn > 0u))
		{
			__syncwarp();
			const uint32_t take = min(qn, 32u);
			if (lane < take)
			{
				const uint32_t e = qn - take + lane;
				const uint32_t cl = qLane[w][e];
				const uint32_t ci = order ? order[warpBase + cl] : warpBase + cl;
				cast_candidate<MODE>(q, casts, ci, qFix[w][e], &sCount[w][cl], MODE == 1 ? counts[ci] : 0u, outIdx,
					outHit, capacity, nullptr);
			}
			qn -= take;
			__syncwarp();
		}
		if (!more && qn == 0u)
			break;
	}
	__syncwarp();
	if (!active)
		return;
	if (MODE == 0)
		counts[i] = sCount[w][lane];
}

// The winner of a single cast that is a mesh: its smallest triangle at the
// winning fraction, evaluated there (world.cpp:828-848).
__device__ __noinline__ void cast_mesh_winner(const QueryCtx& q, const float* casts, uint32_t i, uint32_t f, float t,
	uint32_t* outSingle, float* outHit)
{
	const DevScene& S = q.S;
	const CastIn in = load_cast(casts, i);
	const GProxy pA = convex_proxy(S, in.type, in.p0, in.p1, in.p2, in.hull);
	const XF xfB = body_xf(S, S.fixBody[f]);
	GProxy pB;
	pB.gv = nullptr;
	pB.lv[0] = pB.lv[1] = pB.lv[2] = V3{0.0f, 0.0f, 0.0f};
	pB.count = 1;
	pB.radius = 0.0f;
	uint32_t child = B3G_NULL;
	XF xf2;
	cast_sweep(S, in, xf2);
	cast_mesh(q, in, pA, xf2, f, xfB, [&](uint32_t tri, float tt, const GProxy& pt) {
		if (tt == t && tri < child)
		{
			child = tri;
			pB = pt;
		}
	});
	XF xt;
	xt.q = in.xf.q;
	xt.p = in.xf.p + t * in.d;
	V3 point, normal;
	cast_evaluate(point, normal, xt, pA, xfB, pB);
	float* h = outHit + 7 * (size_t)i;
	h[0] = point.x, h[1] = point.y, h[2] = point.z;
	h[3] = normal.x, h[4] = normal.y, h[5] = normal.z;
	h[6] = t;
	outSingle[2 * (size_t)i] = f;
	outSingle[2 * (size_t)i + 1] = child;
}

// b3World::ShapeCastSingle: the smallest fraction, then the smaller fixture and
// triangle on an exact tie. A warp holds `casts per warp` casts, 32 / that many
// lanes each. The first lane of a cast walks the tree in the order the cast
// shape's moving box meets the boxes and gathers the next candidates (fixtures
// whose fat AABB overlaps the swept box, as the reference takes them), one for
// each lane of the cast; then every lane runs the time of impact of its
// candidate, the warp in step; the best fraction drops what the box meets only
// later. A touching result has the shapes within 1.25 slop of each other, so
// their boxes (the fixture's inside its fat AABB) meet at that fraction up to
// the slack added here. Few casts get a warp each, so that a cast's
// candidates are tested side by side; many share one. Bound by the latency of
// the GJK steps and by lanes whose candidate is done before their warp's
// others. Measured, 16,384 casts of 1-4 m in a 20,001-body world: 5.06 ms with
// every candidate under the swept box tested, 1.17 ms now; 700 casts in 3,000 bodies: 3.95 -> 0.19 ms.
constexpr int CAST_WARPS = 2;
constexpr int CAST_BLOCKS = 6; // per SM: 8 took 1.21 ms, 12 took 1.43 ms

__global__ void __launch_bounds__(CAST_WARPS * 32, CAST_BLOCKS) k_shape_cast_first(QueryCtx q, WalkTree tree,
	const float* casts, uint32_t n, uint32_t lanesPerCast, uint32_t* outSingle, float* outHit)
{
	__shared__ float simplex[CAST_WARPS][LANE_SIMPLEX_WORDS * LANE_ROW];
	__shared__ uint32_t candFix[CAST_WARPS][32];
	__shared__ float candEntry[CAST_WARPS][32];
	__shared__ unsigned long long sBest[CAST_WARPS][32]; // per cast of the warp: fraction bits, fixture
	const DevScene& S = q.S;
	const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
	const uint32_t mine = lane / lanesPerCast, slot = lane % lanesPerCast; // cast of the warp, candidate of the cast
	const uint32_t i = (blockIdx.x * CAST_WARPS + w) * (32u / lanesPerCast) + mine;
	const bool valid = i < n;
	const bool walker = valid && slot == 0u;
	CastIn in = load_cast(casts, valid ? i : 0u);
	sBest[w][lane] = ~0ull;
	// A mesh cannot be cast (world.cpp:755-760).
	uint2 stack[WALK_STACK]; // reference, entry fraction (float bits)
	uint32_t sp = 0, steps = 0, node = SENT;
	AABB sw;
	sw.lo = sw.hi = V3{0.0f, 0.0f, 0.0f};
	SlabTest slab;
	slab.inv = slab.a = slab.b = V3{0.0f, 0.0f, 0.0f};
	bool prune = false;
	float entry = 0.0f; // of node
	if (walker && in.type != B3G_SHAPE_MESH)
	{
		XF xf2 = in.xf;
		xf2.p = in.xf.p + in.d;
		AABB a1, a2;
		compute_shape_aabbs(S, in.type, in.p0, in.p1, in.p2, in.hull, in.xf, xf2, true, a1, a2);
		sw.lo = vmin(a1.lo, a2.lo);
		sw.hi = vmax(a1.hi, a2.hi);
		// A cast triangle's box does not move with it (the reference's quirk
		// above): the swept box is then met as a whole, at fraction 0.
		prune = in.type != B3G_SHAPE_TRIANGLE && !(tree.turned && *tree.turned);
		const float pad = 4.0f * B3G_LINEAR_SLOP + 1e-5f * coord_mag(sw.lo, sw.hi);
		if (prune)
			slab.init(a1.lo, a1.hi, in.d, pad);
		else
			slab.init(sw.lo, sw.hi, V3{0.0f, 0.0f, 0.0f}, pad);
		node = walk_root(tree);
	}
	prune = __shfl_sync(0xFFFFFFFFu, prune ? 1 : 0, lane - slot) != 0;
	LaneProxy<1> pA, pB;
	const float* record = casts + 28 * (size_t)(valid ? i : 0u);
	pB.gv = nullptr;
	pB.lv = record + 4;
	pB.count = 1;
	float rA = 0.0f;
	if (in.type < B3G_SHAPE_MESH)
		rA = pA.set(S, in.type, in.hull, record + 4);
	else
		pA = pB;
	LaneSimplex sx;
	sx.mine = simplex[w] + lane;
	sx.count = sx.steps = sx.saveCount = 0;
	sx.metric = 0.0f;
	__syncwarp();
	for (;;)
	{
		// Walk on to as many candidates as the cast has lanes.
		unsigned long long key = sBest[w][mine];
		const float limit = prune && key != ~0ull ? __uint_as_float((uint32_t)(key >> 32)) : 1.0f;
		uint32_t found = 0;
		while (__any_sync(0xFFFFFFFFu, node != SENT && found < lanesPerCast))
		{
			if (node != SENT && found < lanesPerCast)
			{
				bool popNow = node == WALK_POP;
				if (node < WALK_LEAF)
				{
					uint32_t a, b;
					float ta, tb;
					const uint32_t hits = walk_expand(tree, slab, node, limit, a, ta, b, tb);
					if (hits == 2u)
						stack[min(sp, WALK_STACK - 1u)] = make_uint2(b, __float_as_uint(tb));
					sp += hits == 2u ? 1u : 0u;
					node = a;
					entry = ta;
					popNow = hits == 0u;
					if (++steps > 2u * tree.count || sp > WALK_STACK)
					{
						atomicOr(q.status, B3G_ST_WAIT_TIMEOUT);
						popNow = true;
						sp = 0;
					}
				}
				else if (!popNow)
				{
					const uint32_t leaf = node & ~WALK_LEAF;
					const float4 id = __ldg(tree.leaves + 4 * (size_t)leaf + 1);
					const float4 lo = __ldg(q.nodeLo + (tree.count - 1u + leaf)), hi = __ldg(q.nodeHi + (tree.count - 1u + leaf));
					if (box_overlap(sw, lo, hi) && (__float_as_uint(id.y) & 7u) != LEAF_NONE && __float_as_uint(id.z) == in.world)
					{
						candFix[w][lane + found] = __float_as_uint(id.x);
						candEntry[w][lane + found] = entry;
						++found;
					}
					popNow = true;
				}
				if (popNow)
				{
					node = SENT;
					if (sp > 0)
					{
						const uint2 e = stack[--sp];
						entry = __uint_as_float(e.y);
						node = entry <= limit ? e.x : WALK_POP;
					}
				}
			}
			__syncwarp();
		}
		const uint32_t have = __shfl_sync(0xFFFFFFFFu, found, lane - slot);
		// With nothing gathered anywhere the walks are over: the last round
		// evaluates the winners at their fractions.
		const bool last = !__any_sync(0xFFFFFFFFu, have > 0u);
		uint32_t f = 0;
		bool run = false;
		if (!last)
		{
			run = slot < have;
			if (run)
			{
				f = candFix[w][lane];
				run = !(prune && candEntry[w][lane] > limit);
			}
		}
		else if (walker && key != ~0ull)
		{
			f = (uint32_t)key;
			run = true;
		}
		float t = last && run ? __uint_as_float((uint32_t)(key >> 32)) : 0.0f;
		XF xfA = in.xf, xfB = in.xf;
		float rB = 0.0f;
		const bool mesh = run && S.fixType[f] == B3G_SHAPE_MESH;
		if (run)
			xfB = body_xf(S, S.fixBody[f]);
		if (mesh)
		{
			if (!last)
				cast_candidate<2>(q, casts, i, f, nullptr, 0u, nullptr, nullptr, 0u, &sBest[w][mine]);
			else
				cast_mesh_winner(q, casts, i, f, t, outSingle, outHit);
			run = false;
		}
		if (run)
		{
			rB = pB.set(S, S.fixType[f], S.fixHull[f], reinterpret_cast<const float*>(S.fixParams + 3 * (size_t)f));
			if (last)
				xfA.p = in.xf.p + t * in.d;
		}
		const V3 pB0 = xfB.p;
		// b3TimeOfImpact (time_of_impact.cpp:666-776), as toi_translate: the
		// warp runs each GJK together.
		const float target = fmaxr(B3G_LINEAR_SLOP, (rA + rB) - 3.0f * B3G_LINEAR_SLOP);
		const float tolerance = 0.25f * B3G_LINEAR_SLOP;
		sx.count = 0;
		sx.metric = 0.0f;
		for (uint32_t iteration = 0; iteration < 20u && __any_sync(0xFFFFFFFFu, run); ++iteration)
		{
			if (run)
				sx.start(pA, pB, xfA, xfB);
			__syncwarp();
			bool gjk = run;
			while (__any_sync(0xFFFFFFFFu, gjk))
			{
				V3 dA, dB;
				if (gjk)
					gjk = sx.directions(xfA, xfB, dA, dB);
				__syncwarp();
				uint32_t ia = 0, ib = 0;
				if (gjk)
					ia = pA.support(dA);
				__syncwarp();
				if (gjk)
					ib = pB.support(dB);
				__syncwarp();
				if (gjk)
					gjk = sx.add(pA, pB, xfA, xfB, ia, ib);
				__syncwarp();
			}
			if (run)
			{
				V3 P1, P2;
				sx.end(pA, pB, xfA, xfB, P1, P2);
				if (last)
				{
					// b3WorldShapeCastQueryWrapper::Evaluate (world.cpp:719-731).
					const V3 normal = normalized(P1 - P2);
					const V3 point = P2 + rB * normal;
					float* h = outHit + 7 * (size_t)i;
					h[0] = point.x, h[1] = point.y, h[2] = point.z;
					h[3] = normal.x, h[4] = normal.y, h[5] = normal.z;
					h[6] = t;
					outSingle[2 * (size_t)i] = f;
					outSingle[2 * (size_t)i + 1] = 0u;
					run = false;
				}
				else
				{
					const float distance = len(P1 - P2);
					if (distance == 0.0f)
						run = false;
					else if (distance < target + tolerance)
					{
						atomicMin(&sBest[w][mine], ((unsigned long long)__float_as_uint(t) << 32) | f);
						run = false;
					}
					else
					{
						const V3 zero = V3{0.0f, 0.0f, 0.0f};
						const V3 nrm = (P2 - P1) / distance;
						const float denominator = dot(zero - in.d, nrm);
						if (denominator >= 0.0f)
							run = false;
						else
						{
							t += (target - distance) / denominator;
							run = !(t >= 1.0f);
							xfA.p = in.xf.p + t * in.d;
							xfB.p = pB0 + t * zero;
						}
					}
				}
			}
			__syncwarp();
		}
		if (last)
			break;
	}
	if (walker && sBest[w][mine] == ~0ull)
	{
		float* h = outHit + 7 * (size_t)i;
		for (int e = 0; e < 7; ++e)
			h[e] = 0.0f;
		outSingle[2 * (size_t)i] = B3G_NULL;
		outSingle[2 * (size_t)i + 1] = B3G_NULL;
	}
}

cudaError_t launch_shape_cast_first(b3g_ctx* c, const QueryCtx& q, const float* casts, uint32_t n, uint32_t* fix,
	float* hit, cudaStream_t s)
{
	WalkTree t;
	cudaError_t e = launch_walk_tree(c, q, t, s);
	if (e != cudaSuccess)
		return e;
	// As many lanes to a cast as leave the GPU about 16 warps per SM: 16,384
	// casts took 1.17 ms with 4 lanes each, 1.23 ms with 16.
	uint32_t lanes = 32;
	while (lanes > 1u && (unsigned long long)n * lanes > 32ull * 148ull * 16ull)
		lanes >>= 1;
	const uint32_t perBlock = CAST_WARPS * (32u / lanes);
	k_shape_cast_first<<<(n + perBlock - 1) / perBlock, CAST_WARPS * 32, 0, s>>>(q, t, casts, n, lanes, fix, hit);
	return end_walk(c, t, s);
}

__device__ __forceinline__ uint32_t cast_expand10(uint32_t v)
{
	v = (v * 0x00010001u) & 0xFF0000FFu;
	v = (v * 0x00000101u) & 0x0F00F00Fu;
	v = (v * 0x00000011u) & 0xC30C30C3u;
	v = (v * 0x00000005u) & 0x49249249u;
	return v;
}

// Sort keys of the casts: world, then the 30-bit Morton code of the middle of
// the sweep within the tree's root box.
__global__ void k_cast_keys(const float* casts, uint32_t n, const float4* nodeLo, const float4* nodeHi,
	unsigned long long* keys, uint32_t* vals)
{
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n)
		return;
	const float* r = casts + 28 * (size_t)i;
	const float4 lo = nodeLo[0], hi = nodeHi[0];
	const float c[3] = {r[16] + 0.5f * r[23], r[17] + 0.5f * r[24], r[18] + 0.5f * r[25]};
	const float l[3] = {lo.x, lo.y, lo.z}, h[3] = {hi.x, hi.y, hi.z};
	uint32_t qv[3];
	for (int k = 0; k < 3; ++k)
	{
		float ext = h[k] - l[k];
		float t = ext > 0.0f ? (c[k] - l[k]) / ext : 0.0f;
		t = fminf(fmaxf(t, 0.0f), 1.0f);
		qv[k] = min((uint32_t)(t * 1024.0f), 1023u);
	}
	const uint32_t code = (cast_expand10(qv[0]) << 2) | (cast_expand10(qv[1]) << 1) | cast_expand10(qv[2]);
	keys[i] = ((unsigned long long)__float_as_uint(r[2]) << 30) | code;
	vals[i] = i;
}

int qfail(b3g_ctx* c, int code, const char* msg)
{
	c->err = msg;
	return code;
}

// Device scratch of the query calls, grown on demand.
bool q_reserve(b3g_ctx* c, size_t bytes)
{
	if (c->qScratchBytes >= bytes)
		return true;
	if (c->qScratch)
		cudaFree(c->qScratch);
	c->qScratch = nullptr;
	c->qScratchBytes = 0;
	size_t want = bytes < ((size_t)1 << 20) ? ((size_t)1 << 20) : bytes;
	if (cudaMalloc(&c->qScratch, want) != cudaSuccess)
		return false;
	c->qScratchBytes = want;
	return true;
}

int q_begin(b3g_ctx* c, uint32_t n, const void* in, size_t inBytes, const uint32_t* worlds, QueryCtx& q,
	size_t extraBytes, char*& base, const uint32_t*& dWorlds, const void*& dIn)
{
	if (!c->havePass || c->treeLeaves == 0)
		return qfail(c, B3G_E_STATE, "world query: no collision pass yet");
	if (n > std::max(c->cfg.max_proxies, c->cfg.max_contacts))
		return qfail(c, B3G_E_CAPACITY, "world query: more queries than max(max_proxies, max_contacts) per call");
	if (cudaSetDevice(c->device) != cudaSuccess)
		return qfail(c, B3G_E_CUDA, "world query: device");
	auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
	size_t need = al(inBytes) + al(4 * (size_t)n) + extraBytes;
	if (!q_reserve(c, need))
		return qfail(c, B3G_E_CUDA, "world query: device allocation failed");
	base = (char*)c->qScratch;
	dIn = base;
	if (cudaMemcpyAsync(base, in, inBytes, cudaMemcpyHostToDevice, c->stream) != cudaSuccess)
		return qfail(c, B3G_E_CUDA, "world query: copy");
	base += al(inBytes);
	dWorlds = nullptr;
	if (worlds)
	{
		if (cudaMemcpyAsync(base, worlds, 4 * (size_t)n, cudaMemcpyHostToDevice, c->stream) != cudaSuccess)
			return qfail(c, B3G_E_CUDA, "world query: copy");
		dWorlds = (const uint32_t*)base;
	}
	base += al(4 * (size_t)n);
	q.S = c->scene;
	q.nodeLo = c->buf.nodeLo;
	q.nodeHi = c->buf.nodeHi;
	q.nodeRight = c->buf.nodeRight;
	q.fatLo = c->buf.fatLo;
	q.fatHi = c->buf.fatHi;
	q.leaves = c->treeLeaves;
	q.status = c->buf.counters + CTR_SCRATCH;
	return B3G_OK;
}

int q_status(b3g_ctx* c)
{
	uint32_t st = 0;
	if (cudaMemcpyAsync(&st, c->buf.counters + CTR_SCRATCH, 4, cudaMemcpyDeviceToHost, c->stream) != cudaSuccess ||
		cudaStreamSynchronize(c->stream) != cudaSuccess)
		return qfail(c, B3G_E_CUDA, "world query: kernel failed");
	if (st)
		return qfail(c, st & B3G_ST_WAIT_TIMEOUT ? B3G_E_TIMEOUT : B3G_E_CAPACITY,
			"world query: tree walk stopped (stack or step limit)");
	return B3G_OK;
}

} // namespace

extern "C" int b3g_query_aabb(b3g_ctx* c, uint32_t n, const float* boxes, const uint32_t* worlds, uint32_t* out,
	uint32_t capacity)
{
	if (!c || (n && (!boxes || (!out && capacity))))
		return c ? qfail(c, B3G_E_INVALID, "b3g_query_aabb: null argument") : B3G_E_INVALID;
	if (n == 0)
		return 0;
	QueryCtx q;
	char* base;
	const uint32_t* dWorlds;
	const void* dIn;
	const size_t cntBytes = ((4 * (size_t)n + 4 + 255) & ~(size_t)255);
	const size_t outBytes = 8 * (size_t)capacity;
	int rc = q_begin(c, n, boxes, 24 * (size_t)n, worlds, q, cntBytes + outBytes + 256, base, dWorlds, dIn);
	if (rc)
		return rc;
	uint32_t* counts = (uint32_t*)base;
	uint2* dOut = (uint2*)(base + cntBytes);
	cudaStream_t s = c->stream;
	cudaMemsetAsync(c->buf.counters + CTR_SCRATCH, 0, 4, s);
	const uint32_t blocks = (n + 127) / 128;
	k_query_aabb<0><<<blocks, 128, 0, s>>>(q, (const float*)dIn, dWorlds, n, counts, dOut, capacity);
	scan_exclusive(counts, n, c->buf.scanAux, counts + n, c->buf.counters + CTR_STATUS, s);
	k_query_aabb<1><<<blocks, 128, 0, s>>>(q, (const float*)dIn, dWorlds, n, counts, dOut, capacity);
	uint32_t total = 0;
	if (cudaMemcpyAsync(&total, counts + n, 4, cudaMemcpyDeviceToHost, s) != cudaSuccess)
		return qfail(c, B3G_E_CUDA, "b3g_query_aabb: copy");
	rc = q_status(c);
	if (rc)
		return rc;
	uint32_t m = total < capacity ? total : capacity;
	if (m && cudaMemcpy(out, dOut, 8 * (size_t)m, cudaMemcpyDeviceToHost) != cudaSuccess)
		return qfail(c, B3G_E_CUDA, "b3g_query_aabb: copy");
	return (int)total;
}

extern "C" int b3g_ray_cast(b3g_ctx* c, uint32_t n, const float* rays, const uint32_t* worlds, uint32_t* index,
	float* hits, uint32_t capacity)
{
	if (!c || (n && (!rays || ((!index || !hits) && capacity))))
		return c ? qfail(c, B3G_E_INVALID, "b3g_ray_cast: null argument") : B3G_E_INVALID;
	if (n == 0)
		return 0;
	QueryCtx q;
	char* base;
	const uint32_t* dWorlds;
	const void* dIn;
	const size_t cntBytes = ((4 * (size_t)n + 4 + 255) & ~(size_t)255);
	const size_t idxBytes = ((8 * (size_t)capacity + 255) & ~(size_t)255);
	int rc = q_begin(c, n, rays, 24 * (size_t)n, worlds, q, cntBytes + idxBytes + 28 * (size_t)capacity + 256, base,
		dWorlds, dIn);
	if (rc)
		return rc;
	uint32_t* counts = (uint32_t*)base;
	uint2* dIdx = (uint2*)(base + cntBytes);
	float* dHit = (float*)(base + cntBytes + idxBytes);
	cudaStream_t s = c->stream;
	cudaMemsetAsync(c->buf.counters + CTR_SCRATCH, 0, 4, s);
	const uint32_t blocks = (n + 127) / 128;
	k_ray_cast<0><<<blocks, 128, 0, s>>>(q, (const float*)dIn, dWorlds, n, counts, dIdx, dHit, capacity);
	scan_exclusive(counts, n, c->buf.scanAux, counts + n, c->buf.counters + CTR_STATUS, s);
	k_ray_cast<1><<<blocks, 128, 0, s>>>(q, (const float*)dIn, dWorlds, n, counts, dIdx, dHit, capacity);
	uint32_t total = 0;
	if (cudaMemcpyAsync(&total, counts + n, 4, cudaMemcpyDeviceToHost, s) != cudaSuccess)
		return qfail(c, B3G_E_CUDA, "b3g_ray_cast: copy");
	rc = q_status(c);
	if (rc)
		return rc;
	uint32_t m = total < capacity ? total : capacity;
	if (m && (cudaMemcpy(index, dIdx, 8 * (size_t)m, cudaMemcpyDeviceToHost) != cudaSuccess ||
				 cudaMemcpy(hits, dHit, 28 * (size_t)m, cudaMemcpyDeviceToHost) != cudaSuccess))
		return qfail(c, B3G_E_CUDA, "b3g_ray_cast: copy");
	return (int)total;
}

extern "C" int b3g_ray_cast_single(b3g_ctx* c, uint32_t n, const float* rays, const uint32_t* worlds,
	uint32_t* fixture, float* hit)
{
	if (!c || (n && (!rays || !fixture || !hit)))
		return c ? qfail(c, B3G_E_INVALID, "b3g_ray_cast_single: null argument") : B3G_E_INVALID;
	if (n == 0)
		return 0;
	QueryCtx q;
	char* base;
	const uint32_t* dWorlds;
	const void* dIn;
	const size_t fixBytes = ((4 * (size_t)n + 255) & ~(size_t)255);
	int rc = q_begin(c, n, rays, 24 * (size_t)n, worlds, q, fixBytes + 28 * (size_t)n + 256, base, dWorlds, dIn);
	if (rc)
		return rc;
	uint32_t* dFix = (uint32_t*)base;
	float* dHit = (float*)(base + fixBytes);
	cudaStream_t s = c->stream;
	cudaMemsetAsync(c->buf.counters + CTR_SCRATCH, 0, 4, s);
	if (launch_ray_first(c, q, (const float*)dIn, dWorlds, n, dFix, dHit, s) != cudaSuccess)
		return qfail(c, B3G_E_CUDA, "b3g_ray_cast_single: launch");
	rc = q_status(c);
	if (rc)
		return rc;
	if (cudaMemcpy(fixture, dFix, 4 * (size_t)n, cudaMemcpyDeviceToHost) != cudaSuccess ||
		cudaMemcpy(hit, dHit, 28 * (size_t)n, cudaMemcpyDeviceToHost) != cudaSuccess)
		return qfail(c, B3G_E_CUDA, "b3g_ray_cast_single: copy");
	int hits = 0;
	for (uint32_t i = 0; i < n; ++i)
		hits += fixture[i] != B3G_NULL ? 1 : 0;
	return hits;
}

extern "C" int b3g_ray_cast_single_device(b3g_ctx* c, uint32_t n, const float* rays, const uint32_t* worlds,
	uint32_t* fixture, float* hit, void* stream)
{
	if (!c || (n && (!rays || !fixture || !hit)))
		return c ? qfail(c, B3G_E_INVALID, "b3g_ray_cast_single_device: null argument") : B3G_E_INVALID;
	if (!c->havePass || c->treeLeaves == 0)
		return qfail(c, B3G_E_STATE, "world query: no collision pass yet");
	if (n == 0)
		return B3G_OK;
	QueryCtx q;
	q.S = c->scene;
	q.nodeLo = c->buf.nodeLo;
	q.nodeHi = c->buf.nodeHi;
	q.nodeRight = c->buf.nodeRight;
	q.fatLo = c->buf.fatLo;
	q.fatHi = c->buf.fatHi;
	q.leaves = c->treeLeaves;
	q.status = c->buf.counters + CTR_SCRATCH;
	cudaStream_t s = stream ? (cudaStream_t)stream : c->stream;
	if (launch_ray_first(c, q, rays, worlds, n, fixture, hit, s) != cudaSuccess || cudaGetLastError() != cudaSuccess)
		return qfail(c, B3G_E_CUDA, "b3g_ray_cast_single_device: launch");
	return B3G_OK;
}

// Host check of the casts: the shape types a cast may have and their hulls.
static_assert(sizeof(b3g_shape_cast_input) == 112, "b3g_shape_cast_input: 28 words");

// Scratch bytes of cast_order for n casts.
static size_t cast_order_bytes(uint32_t n)
{
	auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
	return 2 * al(8 * (size_t)n) + 2 * al(4 * (size_t)n) + al(4 * (size_t)radix_sort_scratch_words(n, 48));
}

// The casts' processing order (sorted by world and Morton key) in scratch
// at p; returns the order array.
static const uint32_t* cast_order(b3g_ctx* c, const float* dCasts, uint32_t n, char* p, uint32_t worldBits,
	cudaStream_t s)
{
	auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
	unsigned long long* keys = (unsigned long long*)p;
	p += al(8 * (size_t)n);
	unsigned long long* keysTmp = (unsigned long long*)p;
	p += al(8 * (size_t)n);
	uint32_t* vals = (uint32_t*)p;
	p += al(4 * (size_t)n);
	uint32_t* valsTmp = (uint32_t*)p;
	p += al(4 * (size_t)n);
	uint32_t* scratch = (uint32_t*)p;
	k_cast_keys<<<(n + 255) / 256, 256, 0, s>>>(dCasts, n, c->buf.nodeLo, c->buf.nodeHi, keys, vals);
	bool swapped = radix_sort_pairs(keys, vals, keysTmp, valsTmp, n, 30 + (int)worldBits, scratch,
		c->buf.counters + CTR_SCRATCH, s);
	return swapped ? valsTmp : vals;
}

static uint32_t world_bits(const b3g_ctx* c)
{
	uint32_t b = 0;
	while (b < 18 && (1u << b) < c->nWorlds)
		++b;
	return b;
}

static int cast_check(b3g_ctx* c, uint32_t n, const b3g_shape_cast_input* casts)
{
	for (uint32_t i = 0; i < n; ++i)
	{
		const uint32_t t = casts[i].shape_type;
		if (t > B3G_SHAPE_MESH)
			return qfail(c, B3G_E_INVALID, "shape cast: unknown shape type");
		if (t == B3G_SHAPE_HULL && casts[i].hull >= c->nHulls)
			return qfail(c, B3G_E_INVALID, "shape cast: hull out of range");
	}
	return B3G_OK;
}

extern "C" int b3g_shape_cast(b3g_ctx* c, uint32_t n, const b3g_shape_cast_input* casts, uint32_t* index,
	float* hits, uint32_t capacity)
{
	if (!c || (n && (!casts || ((!index || !hits) && capacity))))
		return c ? qfail(c, B3G_E_INVALID, "b3g_shape_cast: null argument") : B3G_E_INVALID;
	if (n == 0)
		return 0;
	int rc = cast_check(c, n, casts);
	if (rc)
		return rc;
	QueryCtx q;
	char* base;
	const uint32_t* dWorlds;
	const void* dIn;
	const size_t cntBytes = ((4 * (size_t)n + 4 + 255) & ~(size_t)255);
	const size_t idxBytes = ((12 * (size_t)capacity + 255) & ~(size_t)255);
	const size_t hitBytes = ((28 * (size_t)capacity + 255) & ~(size_t)255);
	rc = q_begin(c, n, casts, sizeof(b3g_shape_cast_input) * (size_t)n, nullptr, q,
		cntBytes + idxBytes + hitBytes + cast_order_bytes(n) + 256, base, dWorlds, dIn);
	if (rc)
		return rc;
	uint32_t* counts = (uint32_t*)base;
	uint32_t* dIdx = (uint32_t*)(base + cntBytes);
	float* dHit = (float*)(base + cntBytes + idxBytes);
	cudaStream_t s = c->stream;
	cudaMemsetAsync(c->buf.counters + CTR_SCRATCH, 0, 4, s);
	const uint32_t* order =
		cast_order(c, (const float*)dIn, n, base + cntBytes + idxBytes + hitBytes, world_bits(c), s);
	const uint32_t blocks = (n + 127) / 128;
	k_shape_cast<0><<<blocks, 128, 0, s>>>(q, (const float*)dIn, order, n, counts, dIdx, dHit, capacity);
	scan_exclusive(counts, n, c->buf.scanAux, counts + n, c->buf.counters + CTR_STATUS, s);
	k_shape_cast<1><<<blocks, 128, 0, s>>>(q, (const float*)dIn, order, n, counts, dIdx, dHit, capacity);
	uint32_t total = 0;
	if (cudaMemcpyAsync(&total, counts + n, 4, cudaMemcpyDeviceToHost, s) != cudaSuccess)
		return qfail(c, B3G_E_CUDA, "b3g_shape_cast: copy");
	rc = q_status(c);
	if (rc)
		return rc;
	uint32_t m = total < capacity ? total : capacity;
	if (m && (cudaMemcpy(index, dIdx, 12 * (size_t)m, cudaMemcpyDeviceToHost) != cudaSuccess ||
				 cudaMemcpy(hits, dHit, 28 * (size_t)m, cudaMemcpyDeviceToHost) != cudaSuccess))
		return qfail(c, B3G_E_CUDA, "b3g_shape_cast: copy");
	return (int)total;
}

extern "C" int b3g_shape_cast_single(b3g_ctx* c, uint32_t n, const b3g_shape_cast_input* casts, uint32_t* fixture,
	float* hit)
{
	if (!c || (n && (!casts || !fixture || !hit)))
		return c ? qfail(c, B3G_E_INVALID, "b3g_shape_cast_single: null argument") : B3G_E_INVALID;
	if (n == 0)
		return 0;
	int rc = cast_check(c, n, casts);
	if (rc)
		return rc;
	QueryCtx q;
	char* base;
	const uint32_t* dWorlds;
	const void* dIn;
	const size_t fixBytes = ((8 * (size_t)n + 255) & ~(size_t)255);
	const size_t hitBytes = ((28 * (size_t)n + 255) & ~(size_t)255);
	rc = q_begin(c, n, casts, sizeof(b3g_shape_cast_input) * (size_t)n, nullptr, q,
		fixBytes + hitBytes + 256, base, dWorlds, dIn);
	if (rc)
		return rc;
	uint32_t* dFix = (uint32_t*)base;
	float* dHit = (float*)(base + fixBytes);
	cudaStream_t s = c->stream;
	cudaMemsetAsync(c->buf.counters + CTR_SCRATCH, 0, 4, s);
	if (launch_shape_cast_first(c, q, (const float*)dIn, n, dFix, dHit, s) != cudaSuccess)
		return qfail(c, B3G_E_CUDA, "b3g_shape_cast_single: launch");
	rc = q_status(c);
	if (rc)
		return rc;
	if (cudaMemcpy(fixture, dFix, 8 * (size_t)n, cudaMemcpyDeviceToHost) != cudaSuccess ||
		cudaMemcpy(hit, dHit, 28 * (size_t)n, cudaMemcpyDeviceToHost) != cudaSuccess)
		return qfail(c, B3G_E_CUDA, "b3g_shape_cast_single: copy");
	int hits = 0;
	for (uint32_t i = 0; i < n; ++i)
		hits += fixture[2 * i] != B3G_NULL ? 1 : 0;
	return hits;
}

extern "C" int b3g_shape_cast_single_device(b3g_ctx* c, uint32_t n, const b3g_shape_cast_input* casts,
	uint32_t* fixture, float* hit, void* stream)
{
	if (!c || (n && (!casts || !fixture || !hit)))
		return c ? qfail(c, B3G_E_INVALID, "b3g_shape_cast_single_device: null argument") : B3G_E_INVALID;
	if (!c->havePass || c->treeLeaves == 0)
		return qfail(c, B3G_E_STATE, "world query: no collision pass yet");
	if (n == 0)
		return B3G_OK;
	QueryCtx q;
	q.S = c->scene;
	q.nodeLo = c->buf.nodeLo;
	q.nodeHi = c->buf.nodeHi;
	q.nodeRight = c->buf.nodeRight;
	q.fatLo = c->buf.fatLo;
	q.fatHi = c->buf.fatHi;
	q.leaves = c->treeLeaves;
	q.status = c->buf.counters + CTR_SCRATCH;
	cudaStream_t s = stream ? (cudaStream_t)stream : c->stream;
	if (n > std::max(c->cfg.max_proxies, c->cfg.max_contacts))
		return qfail(c, B3G_E_CAPACITY, "world query: more queries than max(max_proxies, max_contacts) per call");
	if (launch_shape_cast_first(c, q, (const float*)casts, n, fixture, hit, s) != cudaSuccess ||
		cudaGetLastError() != cudaSuccess)
		return qfail(c, B3G_E_CUDA, "b3g_shape_cast_single_device: launch");
	return B3G_OK;
}

void free_queries(b3g_ctx* c)
{
	if (c->qScratch)
		cudaFree(c->qScratch);
	c->qScratch = nullptr;
	c->qScratchBytes = 0;
}
