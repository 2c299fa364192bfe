/* bvh_host.cc -- binned surface-area-heuristic hierarchy over a mesh's
 * triangles (host side).
 *
 * The reference finds triangle candidates with a per-mesh octree
 * (src/octree.inl, built in Mesh::build_octree, src/mesh.cc); the octree stays
 * the definition of which hit a ray gets.  Its leaves follow the mesh's
 * bounding box, so a thin, wide mesh (a terrain) gets leaves that are thin
 * slabs, lists each triangle in many of them and spreads over far more
 * memory than the L2 cache holds.  This hierarchy has one entry per triangle
 * and tight boxes; the GPU traversal uses it to find the closest candidate
 * and then confirms that candidate against the octree.
 *
 * Boxes are the exact float bounds of the float vertices the triangle test
 * reads; the traversal widens them by a per-ray margin, so the hierarchy
 * never loses a triangle that the test would accept.
 */
#include <math.h>
#include <float.h>
#include <string.h>
#include <algorithm>
#include <numeric>
#include "scene_host.h"

namespace sray {

namespace {

struct Bounds {
	float mn[3], mx[3];
	void clear()
	{
		for(int a = 0; a < 3; a++) { mn[a] = FLT_MAX; mx[a] = -FLT_MAX; }
	}
	void grow(const Bounds &b)
	{
		for(int a = 0; a < 3; a++) {
			mn[a] = std::min(mn[a], b.mn[a]);
			mx[a] = std::max(mx[a], b.mx[a]);
		}
	}
	double area() const
	{
		double e[3];
		for(int a = 0; a < 3; a++) e[a] = mx[a] > mn[a] ? (double)mx[a] - (double)mn[a] : 0.0;
		return e[0] * e[1] + e[1] * e[2] + e[2] * e[0];
	}
};

enum { NBINS = 16, LEAF_MIN = 4, LEAF_MAX = 8, MEDIAN_DEPTH = 36 };

struct Builder {
	const std::vector<Bounds> *tb;
	const std::vector<float> *cen;   /* 3 per face */
	std::vector<int> *order;
	std::vector<DevBvhNode> *nodes;
	int max_depth = 0;
	int leaf_min = LEAF_MIN, leaf_max = LEAF_MAX;

	Bounds range_bounds(int b, int e) const
	{
		Bounds r;
		r.clear();
		for(int i = b; i < e; i++) r.grow((*tb)[(*order)[i]]);
		return r;
	}

	static int leaf_ref(int b, int e) { return ~((b << 4) | (e - b)); }

	int bin_of(int f, int a, float from, double scale) const
	{
		const int k = (int)(((double)(*cen)[(size_t)f * 3 + a] - (double)from) * scale);
		return k < 0 ? 0 : (k >= NBINS ? NBINS - 1 : k);
	}

	/* reference to a subtree over order[b, e), whose boxes' bounds are pb.
	 * A node reads its items three times: the centroids' bounds, the bins of
	 * all three axes, and the partition by the best split, whose sides'
	 * bounds are those of its bins.  (2,000 objects with boxes of their own
	 * 1.6 ms with a pass per axis, all bins cleared and the bounds taken
	 * anew, 1.2 this way, 20,000 18.3 and 13.9; over the octree leaves'
	 * unions, many of which coincide and need no bins, 1.1 and 13.8 before.) */
	int build(int b, int e, int depth, const Bounds &pb)
	{
		max_depth = std::max(max_depth, depth);
		int n = e - b;
		if(n <= leaf_min) return leaf_ref(b, e);
		Bounds cb;
		cb.clear();
		for(int i = b; i < e; i++) {
			const float *c = &(*cen)[(size_t)(*order)[i] * 3];
			for(int a = 0; a < 3; a++) {
				cb.mn[a] = std::min(cb.mn[a], c[a]);
				cb.mx[a] = std::max(cb.mx[a], c[a]);
			}
		}
		int axis = -1, split = -1;
		double best = DBL_MAX;
		Bounds lb, rbx;
		if(depth < MEDIAN_DEPTH) {
			/* only bins with items are cleared and looked at: a split after an
			 * empty bin is the one before it */
			const double parea = pb.area();
			Bounds bin[3][NBINS];
			int cnt[3][NBINS];
			unsigned used[3] = {0, 0, 0};
			double sc[3];
			for(int a = 0; a < 3; a++) {
				const double ext = (double)cb.mx[a] - (double)cb.mn[a];
				sc[a] = ext > 0.0 ? NBINS / ext : 0.0;
			}
			for(int i = b; i < e; i++) {
				const int f = (*order)[i];
				const Bounds &fb = (*tb)[f];
				for(int a = 0; a < 3; a++) {
					if(sc[a] == 0.0) continue;
					const int k = bin_of(f, a, cb.mn[a], sc[a]);
					if((used[a] >> k) & 1u) {
						cnt[a][k]++;
						bin[a][k].grow(fb);
					} else {
						used[a] |= 1u << k;
						cnt[a][k] = 1;
						bin[a][k] = fb;
					}
				}
			}
			for(int a = 0; a < 3; a++) {
				if(sc[a] == 0.0) continue;
				int at[NBINS], m = 0;
				for(int k = 0; k < NBINS; k++) if((used[a] >> k) & 1u) at[m++] = k;
				if(m < 2) continue;
				Bounds right[NBINS];
				int rn[NBINS];
				right[m - 1] = bin[a][at[m - 1]];
				rn[m - 1] = cnt[a][at[m - 1]];
				for(int j = m - 2; j > 0; j--) {
					right[j] = right[j + 1];
					right[j].grow(bin[a][at[j]]);
					rn[j] = rn[j + 1] + cnt[a][at[j]];
				}
				Bounds acc = bin[a][at[0]];
				int accn = cnt[a][at[0]];
				for(int j = 0; j < m - 1; j++) {
					if(j > 0) {
						acc.grow(bin[a][at[j]]);
						accn += cnt[a][at[j]];
					}
					double cost = 1.0 + (acc.area() * accn + right[j + 1].area() * rn[j + 1]) / (parea > 0.0 ? parea : 1.0);
					if(cost < best) {
						best = cost;
						axis = a;
						split = at[j];
						lb = acc;
						rbx = right[j + 1];
					}
				}
			}
			if(n <= leaf_max && (axis < 0 || best >= (double)n)) return leaf_ref(b, e);
		}
		int mid = b;
		if(axis >= 0) {
			const double sc = NBINS / ((double)cb.mx[axis] - (double)cb.mn[axis]);
			int *m = std::partition(order->data() + b, order->data() + e, [&](int f) { return bin_of(f, axis, cb.mn[axis], sc) <= split; });
			mid = (int)(m - order->data());
		}
		if(mid <= b || mid >= e) {
			/* no useful split (coincident centroids or the depth cap): halve
			 * the range along the widest centroid axis */
			int a = 0;
			for(int k = 1; k < 3; k++) if(cb.mx[k] - cb.mn[k] > cb.mx[a] - cb.mn[a]) a = k;
			mid = b + n / 2;
			std::nth_element(order->begin() + b, order->begin() + mid, order->begin() + e,
					[&](int x, int y) { return (*cen)[(size_t)x * 3 + a] < (*cen)[(size_t)y * 3 + a]; });
			lb = range_bounds(b, mid);
			rbx = range_bounds(mid, e);
		}
		int id = (int)nodes->size();
		nodes->push_back(DevBvhNode());
		int l = build(b, mid, depth + 1, lb);
		int r = build(mid, e, depth + 1, rbx);
		DevBvhNode &nd = (*nodes)[id];
		memset(&nd, 0, sizeof nd);
		for(int a = 0; a < 3; a++) {
			nd.lmn[a] = lb.mn[a];
			nd.lmx[a] = lb.mx[a];
			nd.rmn[a] = rbx.mn[a];
			nd.rmx[a] = rbx.mx[a];
		}
		nd.left = l;
		nd.right = r;
		return id;
	}
};

}  // namespace

void MeshBvh::build_items(const float *mn, const float *mx, size_t n, int leaf_max)
{
	nodes.clear();
	order.clear();
	depth = 0;
	/* leaf references hold a 27-bit start: larger item sets use the octree alone */
	if(n == 0 || n >= ((size_t)1 << 27)) return;
	std::vector<Bounds> tb(n);
	std::vector<float> cen(n * 3);
	for(size_t i = 0; i < n; i++) {
		for(int a = 0; a < 3; a++) {
			tb[i].mn[a] = mn[i * 3 + a];
			tb[i].mx[a] = mx[i * 3 + a];
			cen[i * 3 + a] = (float)(((double)mn[i * 3 + a] + (double)mx[i * 3 + a]) * 0.5);
		}
	}
	order.resize(n);
	std::iota(order.begin(), order.end(), 0);
	Builder B;
	B.tb = &tb;
	B.cen = &cen;
	B.order = &order;
	B.nodes = &nodes;
	B.leaf_min = leaf_max < LEAF_MIN ? leaf_max : LEAF_MIN;
	B.leaf_max = leaf_max;
	nodes.reserve(leaf_max < 2 ? n : n / 2 + 1);
	int ref = B.build(0, (int)n, 1, B.range_bounds(0, (int)n));
	if(ref < 0) {
		/* at most leaf_min items: a root node with one leaf */
		DevBvhNode nd;
		memset(&nd, 0, sizeof nd);
		Bounds bb;
		bb.clear();
		for(size_t i = 0; i < n; i++) bb.grow(tb[i]);
		for(int a = 0; a < 3; a++) {
			nd.lmn[a] = bb.mn[a];
			nd.lmx[a] = bb.mx[a];
			nd.rmn[a] = FLT_MAX;
			nd.rmx[a] = -FLT_MAX;
		}
		nd.left = ref;
		nd.right = BVH_NONE;
		nodes.push_back(nd);
	}
	/* otherwise build() created the root first: it is node 0 */
	depth = B.max_depth;
}

namespace {
struct Entry {
	int ref;
	float mn[3], mx[3];
	double area() const
	{
		if(ref == BVH_NONE) return -1.0;
		double e[3];
		for(int a = 0; a < 3; a++) e[a] = mx[a] > mn[a] ? (double)mx[a] - (double)mn[a] : 0.0;
		return e[0] * e[1] + e[1] * e[2] + e[2] * e[0];
	}
};

void children_of(const DevBvhNode &n, Entry *e)
{
	e[0].ref = n.left;
	e[1].ref = n.right;
	for(int a = 0; a < 3; a++) {
		e[0].mn[a] = n.lmn[a];
		e[0].mx[a] = n.lmx[a];
		e[1].mn[a] = n.rmn[a];
		e[1].mx[a] = n.rmx[a];
	}
}

int collapse_node(const std::vector<DevBvhNode> &b2, int n2, std::vector<DevBvh4> &out)
{
	Entry c[4];
	int nc = 2;
	children_of(b2[n2], c);
	while(nc < 4) {
		int best = -1;
		double ba = -1.0;
		for(int k = 0; k < nc; k++) {
			if(c[k].ref < 0 || c[k].ref == BVH_NONE) continue;
			double a = c[k].area();
			if(a > ba) { ba = a; best = k; }
		}
		if(best < 0) break;
		Entry two[2];
		children_of(b2[c[best].ref], two);
		c[best] = two[0];
		c[nc++] = two[1];
	}
	int id = (int)out.size();
	out.push_back(DevBvh4());
	int refs[4];
	for(int k = 0; k < 4; k++) {
		if(k >= nc || c[k].ref == BVH_NONE) refs[k] = BVH_NONE;
		else if(c[k].ref >= 0) refs[k] = collapse_node(b2, c[k].ref, out);
		else refs[k] = c[k].ref;
	}
	DevBvh4 &d = out[id];
	memset(&d, 0, sizeof d);
	for(int k = 0; k < 4; k++) {
		bool ok = k < nc && refs[k] != BVH_NONE;
		d.lox[k] = ok ? c[k].mn[0] : FLT_MAX;
		d.loy[k] = ok ? c[k].mn[1] : FLT_MAX;
		d.loz[k] = ok ? c[k].mn[2] : FLT_MAX;
		d.hix[k] = ok ? c[k].mx[0] : -FLT_MAX;
		d.hiy[k] = ok ? c[k].mx[1] : -FLT_MAX;
		d.hiz[k] = ok ? c[k].mx[2] : -FLT_MAX;
		d.child[k] = refs[k];
	}
	return id;
}
}  // namespace

void MeshBvh::collapse4(std::vector<DevBvh4> &out) const
{
	out.clear();
	if(nodes.empty()) return;
	out.reserve(nodes.size() / 2 + 1);
	collapse_node(nodes, 0, out);
}

void MeshBvh::build(const std::vector<float> &pos)
{
	size_t nf = pos.size() / 9;
	std::vector<float> mn(nf * 3), mx(nf * 3);
	for(size_t i = 0; i < nf; i++) {
		for(int a = 0; a < 3; a++) {
			float lo = pos[i * 9 + a], hi = lo;
			for(int v = 1; v < 3; v++) {
				float c = pos[i * 9 + v * 3 + a];
				lo = std::min(lo, c);
				hi = std::max(hi, c);
			}
			mn[i * 3 + a] = lo;
			mx[i * 3 + a] = hi;
		}
	}
	build_items(mn.data(), mx.data(), nf, LEAF_MAX);
}

}  // namespace sray
