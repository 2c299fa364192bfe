/* photon.cu -- photon emission and tracing, and the device photon map.
 *
 *   k_proj_*        the lights' projection maps (src/projmap.cc:60-190)
 *   k_photon_emit   Light::gen_photon (src/light.cc:111-148) with ProjMap::gen_dir
 *                   (src/projmap.cc:193-209), each photon on its own Philox
 *                   stream, so photon j of light i is the same photon the CPU
 *                   oracle shoots
 *   k_photon_bounce Scene::trace_caustics_photon / trace_global_photon
 *                   (src/scene.cc:571-760), one interaction per pass; the
 *                   renderer's k_trace finds the hits in between
 *   compaction      keeps stored photons in emission order
 *   k_rs_*          stable LSD radix sort of the photons by their grid cell
 *   k_starts*       the photons before every cell
 * PhotonMap::add_photon / scale_photon_power (src/pmap.cc:73-100) become the
 * per-light power scale applied at store time.  The kd-tree of the reference
 * (kd_insert3f, kd_nearest_range3f) is replaced by the grid: a range
 * query visits the rows of cells that its sphere reaches and tests every
 * photon in them with the kd-tree's distance rule, so the photon set of each
 * gather is the same.
 */
#include <math.h>
#include <string.h>
#include <algorithm>
#include <cooperative_groups.h>
#include "renderer.h"

namespace cg = cooperative_groups;

namespace sray {

enum { CAUST_PHOTON = 1, GI_PHOTON = 2, DIRECT_PHOTON = 0 };

struct PRay {
	V3 o, d;
	int time, iter;
	IorStack st;
};

struct PState {
	float col[3];
	int type;
	V3 pos, dir, norm;
};

/* outcome of one photon-surface interaction */
enum { P_DROP = 0, P_STORE = 1, P_CONT = 2, P_TO_CAUST = 3 };

__device__ __forceinline__ void refract_ray(PRay &r, V3 n, float mat_ior, bool entering, float ray_mag)
{
	float ior = r.st.calc_ior(entering, mat_ior);
	if(entering) r.st.enter(mat_ior);
	else r.st.leave();
	r.d = refraction(r.d / ray_mag, n, ior) * ray_mag;
	if(dot(r.d, n) > 0.0f) {
		if(entering) r.st.leave();
		else r.st.enter(mat_ior);
	}
}

/* one iteration of Scene::trace_caustics_photon (src/scene.cc:571-647) at
 * the hit h: reflect or refract (P_CONT) or absorb and store (P_STORE) */
__device__ int caust_step(const DScene &S, PRay &r, PState &ph, const Hit &h, sray_rng *s)
{
	const DevMat &m = mat_of(S, h.obj);
	Surf sp;
	surface_point(S, h, r.o, r.d, r.time, sp, m.textured, m.textured && m.tex[TA_NORMAL] >= 0);
	MatVals mv;
	mat_values(S, m, sp.tex, mv);
	float refl = mv.refl, refr = mv.refr, mat_ior = mv.ior;
	bool entering;
	V3 normal;
	float ray_mag = len(r.d);
	if(dot(r.d, sp.normal) > 0.0f) { normal = -sp.normal; entering = false; }
	else { normal = sp.normal; entering = true; }
	float ior = r.st.calc_ior(entering, mat_ior);
	/* a normal map replaces the normal after the index of refraction is
	 * known (src/scene.cc:600-605) */
	if(m.have_normal) normal = bump_normal(S, m, sp);
	float ray_dot_n = dot(-r.d / ray_mag, normal);
	float sf0 = refr > 0.0f ? (ior - 1.0f) / (ior + 1.0f) : 1.0f;
	float fres = fresnel(sf0 * sf0, ray_dot_n);
	refl = fres * refl;
	refr = (1.0f - fres) * refr;
	float rnum = frand(s, 1.0f);
	if(rnum < refl) {
		r.d = reflection(r.d, normal);
		r.iter--;
		r.o = sp.pos;
		ph.type = CAUST_PHOTON;
		for(int k = 0; k < 3; k++) ph.col[k] = ph.col[k] * mv.ks[k];
		return P_CONT;
	}
	if(rnum < refr) {
		refract_ray(r, normal, mat_ior, entering, ray_mag);
		r.o = sp.pos;
		ph.type = CAUST_PHOTON;
		for(int k = 0; k < 3; k++) ph.col[k] = ph.col[k] * mv.ks[k];
		return P_CONT;
	}
	ph.dir = normalized(r.d);
	ph.pos = sp.pos;
	ph.norm = normal;
	return P_STORE;
}

/* one iteration of Scene::trace_global_photon (src/scene.cc:650-760) at the
 * hit h: diffuse bounce (P_CONT), specular bounce that hands the photon to
 * the caustic rules (P_TO_CAUST), absorption (P_DROP) or storage (P_STORE) */
__device__ int global_step(const DScene &S, PRay &r, PState &ph, const Hit &h, sray_rng *s)
{
	V3 incident = normalized(r.d);
	const DevMat &m = mat_of(S, h.obj);
	Surf sp;
	surface_point(S, h, r.o, r.d, r.time, sp, m.textured);
	V3 normal;
	bool entering;
	float ray_mag = len(r.d);
	if(dot(r.d, sp.normal) > 0.0f) { normal = -sp.normal; entering = false; }
	else { normal = sp.normal; entering = true; }
	MatVals mv;
	mat_values(S, m, sp.tex, mv);
	float diff_avg = (mv.kd[0] + mv.kd[1] + mv.kd[2]) / 3.0f;
	float spec_avg = (mv.ks[0] + mv.ks[1] + mv.ks[2]) / 3.0f;
	float rnum = frand(s, 1.0f);
	if(rnum < diff_avg) {
		V3 dir = sphrand(s, 1.0f);
		if(dot(dir, normal) < 0.0f) dir = -dir;
		float ndotl = dot(-incident, normal);
		r.d = dir * (float)SRAY_RAY_MAGNITUDE;
		r.iter--;
		r.o = sp.pos;
		ph.type = GI_PHOTON;
		for(int k = 0; k < 3; k++) ph.col[k] = ph.col[k] * (ndotl * (mv.kd[k] / diff_avg));
		return P_CONT;
	}
	if(rnum < diff_avg + spec_avg) {
		float refl = mv.refl, refr = mv.refr, mat_ior = mv.ior;
		float ior = r.st.calc_ior(entering, mat_ior);
		float ray_dot_n = dot(-r.d / ray_mag, normal);
		float sf0 = refr > 0.0f ? (ior - 1.0f) / (ior + 1.0f) : 1.0f;
		float fres = fresnel(sf0 * sf0, ray_dot_n);
		refl = fres * refl;
		refr = (1.0f - fres) * refr;
		float rn2 = frand(s, 1.0f);
		if(rn2 < refl) {
			r.d = reflection(r.d, normal);
			r.iter--;
			r.o = sp.pos;
			ph.type = CAUST_PHOTON;
			for(int k = 0; k < 3; k++) ph.col[k] = ph.col[k] * mv.ks[k];
			return P_TO_CAUST;
		}
		if(rn2 < refr) {
			refract_ray(r, normal, mat_ior, entering, ray_mag);
			r.o = sp.pos;
			ph.type = CAUST_PHOTON;
			for(int k = 0; k < 3; k++) ph.col[k] = ph.col[k] * mv.ks[k];
			return P_TO_CAUST;
		}
		return P_DROP;
	}
	ph.dir = incident;
	ph.pos = sp.pos;
	ph.norm = normal;
	return P_STORE;
}

/* One try of ProjMap::gen_dir(true): the direction drawn after n draws of the
 * stream s, and whether its cell is set (cell_from_dir in deterministic float
 * math) */
__device__ __forceinline__ bool try_dir(const uint32_t *bits, sray_rng s, uint32_t n, V3 &v)
{
	sray_rng_seek(&s, n);
	v = sphrand(&s, 1.0f);
	float theta = sray_atan2_f(v.z, v.x);
	float phi = sray_atan2_f(sqrtf(v.x * v.x + v.z * v.z), v.y);
	if(theta < 0.0f) theta = SRAY_TWO_PI_F + theta;
	float u = theta / SRAY_TWO_PI_F, w = phi / SRAY_PI_F;
	int uc = (int)(u * 64.0f), vc = (int)(w * 32.0f);
	uc = uc < 0 ? 0 : (uc > 63 ? 63 : uc);
	vc = vc < 0 ? 0 : (vc > 31 ? 31 : vc);
	int idx = vc * 64 + uc;
	return (bits[idx >> 5] >> (idx & 31)) & 1u;
}

/* The directions of up to 32 photons (one per lane with need set, from its
 * stream s after s.n draws, through its map's bits) by the whole warp.  A
 * photon takes the first direction of its stream whose cell is set; a stream
 * is addressed by its draw count, so its tries can be made in any order: each
 * round deals the lanes out over the photons still without a direction, a
 * run of tries each, and a photon takes the first that succeeds.  (A thread
 * per photon, one try after the other, left a warp waiting for its unluckiest
 * photon: 176 us for the 20,000 caustic photons of a scene whose specular
 * objects cover a few percent of the sphere.)  Returns false where 2^20 tries
 * found none. */
#define GEN_DIR_TRIES (1 << 20)
__device__ __forceinline__ bool gen_dirs(bool need, const uint32_t *bits, sray_rng &s, V3 &out, int *list)
{
	const unsigned FULL = 0xffffffffu;
	const int lane = threadIdx.x & 31;
	const unsigned lt = (1u << lane) - 1u;
	unsigned open = __ballot_sync(FULL, need);
	bool found = false;
	uint32_t tried = 0;
	while(open) {
		const int m = __popc(open), per = 32 / m, rank = __popc(open & lt);
		const bool mine = (open >> lane) & 1u;
		if(mine) list[rank] = lane;
		__syncwarp();
		const int g = lane / per, src = g < m ? list[g] : lane;
		sray_rng t;
		t.k0 = s.k0;
		t.k1 = s.k1;
		t.c1 = __shfl_sync(FULL, s.c1, src);
		t.c2 = __shfl_sync(FULL, s.c2, src);
		t.c3 = __shfl_sync(FULL, s.c3, src);
		t.buf[0] = t.buf[1] = t.buf[2] = t.buf[3] = 0;
		const uint32_t n = __shfl_sync(FULL, s.n + 2 * tried, src) + 2 * (uint32_t)(lane - g * per);
		const uint32_t *b = (const uint32_t *)__shfl_sync(FULL, (unsigned long long)bits, src);
		V3 v = mk(0.0f, 0.0f, 0.0f);
		const bool hit = g < m && try_dir(b, t, n, v);
		const unsigned hits = __ballot_sync(FULL, hit);
		int w = lane;
		bool got = false;
		if(mine) {
			const unsigned run = (hits >> (rank * per)) & (per == 32 ? FULL : (1u << per) - 1u);
			got = run != 0;
			const int k = got ? __ffs(run) - 1 : per;
			w = rank * per + (got ? k : 0);
			tried += got ? k + 1 : per;
		}
		const V3 d = mk(__shfl_sync(FULL, v.x, w), __shfl_sync(FULL, v.y, w), __shfl_sync(FULL, v.z, w));
		if(got) {
			out = d;
			found = true;
			s.n += 2 * tried;
		}
		open = __ballot_sync(FULL, mine && !got && tried < GEN_DIR_TRIES);
	}
	return found;
}

/* ---------------- projection maps ----------------
 * Light::build_proj_intern and ::build_projmap (src/light.cc:151-200,
 * 392-432): from each sample point of a light, every object's box becomes a
 * sphere around its centre, and a cell of the 64 x 32 direction grid is set
 * when a corner of it, taken to the centre's distance, lies in the sphere, or
 * when it holds the centre's direction; a light inside a box sets the whole
 * map.  The coverage is the sum of the set cells' shares of the sphere in the
 * order in which they were set (samples, boxes, the centre's cell, then rows)
 * -- a sum in double, whose rounding depends on that order.
 *
 * k_proj_view takes a thread per (sample, box), k_proj_mark a block: the
 * corners' tests (33 rows of 65, a warp per row) and, per cell they set, the
 * smallest (sample, box, place) over all blocks.  k_proj_cover, a block per
 * map, gives the bits and the sum.  On the host, a thread per light, this
 * took 1.9 ms for three lights over 201 objects before the first photon left
 * (1.4 ms for six frames of 25 objects); here under 50 us (80 us). */
struct ProjSample {
	double lp[3];
	int box0, nbox;       /* the boxes it sees */
	int slot;             /* the light of the job */
	unsigned order;       /* among the light's samples */
};

struct ProjBox {
	double mn[3], mx[3];
	int caustic, pad;     /* also in the caustic map */
};

#define PROJ_CELLS 2048
#define PROJ_SLOT (PROJ_CELLS + 1)   /* a map's cells, and 0 when the light is inside a box */
#define PROJ_NONE 0xffffffffffffffffull

/* one box as one sample sees it */
struct ProjView {
	double c[3], dist, rad_sq;    /* the box's centre, its distance, the sphere's squared radius */
	float u[3];                   /* the centre's direction */
	float lo, hi;                 /* cosines below / above which a corner is out / in the sphere for certain */
	float phi, cap;               /* its colatitude; the angle beyond which a row holds no corner in the sphere */
	int live;                     /* 0: the light is inside the box (or no such box) */
};

/* The angles of a direction (x, y, z), as the cell it lies in needs them:
 * |atan2(z, x)|, and acos of c = y / length, correctly rounded where a cell
 * ends.  There the last bit decides the cell: the host's functions round
 * correctly but for a few per cent of the last place, the device's are up to
 * two places off (acos put 72 of the 117,648 directions of integers up to 24,
 * all at 45 degrees' elevation, into the row before theirs).  Near an edge B
 * the angle is B plus the small rest sin(a - B) = (z cos B - x sin B) / r,
 * taken without cancellation from B's sine and cosine in two doubles. */
__device__ __forceinline__ const ProjAngle &proj_edge(const ProjAngle *edge, double a)
{
	/* (no number, of a light at the very centre of a flat box, becomes INT_MIN) */
	const int k = (int)rint(a * (32.0 / 3.14159265358979323846));
	return edge[k < 0 ? 0 : (k > 32 ? 32 : k)];
}

__device__ __forceinline__ double proj_theta(const ProjAngle *edge, double x, double z)
{
	const double a = atan2(fabs(z), x);
	const ProjAngle &e = proj_edge(edge, a);
	if(!(fabs(a - e.hi) < 1e-13) || e.hi == 0.0) return a;
	const double w = fabs(z), p = w * e.cos_hi, q = x * e.sin_hi;
	const double s = (p - q) + ((fma(w, e.cos_hi, -p) - fma(x, e.sin_hi, -q)) + (w * e.cos_lo - x * e.sin_lo));
	return e.hi + (e.lo + s / sqrt(x * x + z * z));
}

__device__ __forceinline__ double proj_phi(const ProjAngle *edge, double c)
{
	const double a = acos(c);
	const ProjAngle &e = proj_edge(edge, a);
	if(!(fabs(a - e.hi) < 1e-13) || e.sin_hi == 0.0) return a;
	return e.hi + (e.lo + ((e.cos_hi - c) + e.cos_lo) / e.sin_hi);
}

/* a thread per (sample, box): the double arithmetic, of which this GPU does
 * little at once, with every lane at work; a light inside a box, and the
 * cell of the centre's direction, go straight into the maps */
__global__ void __launch_bounds__(128) k_proj_view(const ProjSample *samples, int nsamples, int most, const ProjBox *boxes, ProjView *views,
		const ProjTables *tables, unsigned long long *first)
{
	for(long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < (long long)nsamples * most; i += (long long)gridDim.x * blockDim.x) {
		const int si = (int)(i / most), bi = (int)(i - (long long)si * most);
		const ProjSample &S = samples[si];
		ProjView &V = views[i];
		V.live = 0;
		if(bi >= S.nbox) continue;
		const ProjBox &B = boxes[S.box0 + bi];
		unsigned long long *map = first + (size_t)S.slot * 2 * PROJ_SLOT;
		const double lx = S.lp[0], ly = S.lp[1], lz = S.lp[2];
		if(lx >= B.mn[0] && ly >= B.mn[1] && lz >= B.mn[2] && lx < B.mx[0] && ly < B.mx[1] && lz < B.mx[2]) {
			map[PROJ_CELLS] = 0;
			if(B.caustic) map[PROJ_SLOT + PROJ_CELLS] = 0;
			continue;
		}
		const double cx = (B.mn[0] + B.mx[0]) / 2.0, cy = (B.mn[1] + B.mx[1]) / 2.0, cz = (B.mn[2] + B.mx[2]) / 2.0;
		const double ex = B.mn[0] - cx, ey = B.mn[1] - cy, ez = B.mn[2] - cz;
		const double rad_sq = ex * ex + ey * ey + ez * ez;
		const double vx = cx - lx, vy = cy - ly, vz = cz - lz;
		const double dist = sqrt(vx * vx + vy * vy + vz * vz);
		V.c[0] = cx; V.c[1] = cy; V.c[2] = cz;
		V.dist = dist;
		V.rad_sq = rad_sq;
		/* a corner direction c is in the sphere when c . v / dist >= 1 -
		 * rad_sq / (2 dist^2): decided in float outside a margin of its
		 * rounding (and of the double test's where the light is far from the
		 * origin), by the reference's own test in double within it */
		const float fd = (float)dist, cos_t = (float)(1.0 - rad_sq / (2.0 * dist * dist));
		const float far = (float)fmax(fmax(fabs(lx), fabs(ly)), fabs(lz)) / fd;
		const float margin = 4e-6f + 1e-12f * far * (1.0f + far);
		V.u[0] = (float)vx / fd;
		V.u[1] = (float)vy / fd;
		V.u[2] = (float)vz / fd;
		V.lo = cos_t - margin;
		V.hi = cos_t + margin;
		V.phi = acosf(fminf(fmaxf(V.u[1], -1.0f), 1.0f));
		V.cap = V.lo > -1.0f ? acosf(fminf(V.lo, 1.0f)) + 2e-3f : 4.0f;
		V.live = 1;
		double theta = proj_theta(tables->edge, vx, vz);
		const double ph = proj_phi(tables->edge, vy / dist);
		if(vz < 0.0) theta = 3.14159265358979323846 * 2.0 - theta;
		double u = theta / (3.14159265358979323846 * 2.0), v = ph / 3.14159265358979323846;
		int a = (int)(u * 64), b = (int)(v * 32);
		a = a < 0 ? 0 : (a >= 64 ? 63 : a);
		b = b < 0 ? 0 : (b >= 32 ? 31 : b);
		const int cell = b * 64 + a;
		const unsigned long long key = (((unsigned long long)S.order * (unsigned)S.nbox + bi) * 2ull) * PROJ_CELLS + cell;
		atomicMin(map + cell, key);
		if(B.caustic) atomicMin(map + PROJ_SLOT + cell, key);
	}
}

__global__ void __launch_bounds__(128) k_proj_mark(const ProjSample *samples, int nsamples, int most, const ProjBox *boxes,
		const ProjView *views, const ProjTables *tables, unsigned long long *first)
{
	__shared__ unsigned in[33][3];      /* the corners in the sphere */
	const unsigned FULL = 0xffffffffu;
	const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
	for(int si = blockIdx.y; si < nsamples; si += gridDim.y) {
		const ProjView &V = views[(size_t)si * most + blockIdx.x];
		if(!V.live) continue;
		const ProjSample &S = samples[si];
		unsigned long long *map = first + (size_t)S.slot * 2 * PROJ_SLOT;
		const bool caustic = boxes[S.box0 + blockIdx.x].caustic != 0;
		const float ux = V.u[0], uy = V.u[1], uz = V.u[2], lo = V.lo, hi = V.hi, phi = V.phi, cap = V.cap;
		__syncthreads();
		for(int r = w; r < 33; r += 4) {
			if(fabsf((float)r * (3.14159265f / 32.0f) - phi) > cap) {
				if(lane < 3) in[r][lane] = 0;
				continue;
			}
			#pragma unroll
			for(int k = 0; k < 3; k++) {
				const int u = k * 32 + lane;
				bool hit = false;
				if(u < 65) {
					const float4 c = *reinterpret_cast<const float4 *>(tables->cornerf[r * 65 + u]);
					const float s = c.x * ux + c.y * uy + c.z * uz;
					hit = s > hi;
					if(!hit && !(s < lo)) {
						const double *cd = tables->corner[r * 65 + u];
						double px = S.lp[0] + cd[0] * V.dist, py = S.lp[1] + cd[1] * V.dist, pz = S.lp[2] + cd[2] * V.dist;
						double dx = px - V.c[0], dy = py - V.c[1], dz = pz - V.c[2];
						hit = dx * dx + dy * dy + dz * dz <= V.rad_sq;
					}
				}
				const unsigned b = __ballot_sync(FULL, hit);
				if(lane == 0) in[r][k] = b;
			}
		}
		__syncthreads();
		/* after the centre's own cell, the others by rows */
		const unsigned long long order = ((unsigned long long)S.order * (unsigned)S.nbox + blockIdx.x) * 2ull + 1ull;
		for(int cell = tid; cell < PROJ_CELLS; cell += 128) {
			const int uc = cell & 63, vc = cell >> 6;
			const unsigned *a = in[vc], *b = in[vc + 1];
			const int k0 = uc >> 5, k1 = (uc + 1) >> 5;
			const unsigned m0 = 1u << (uc & 31), m1 = 1u << ((uc + 1) & 31);
			if(!((a[k0] | b[k0]) & m0) && !((a[k1] | b[k1]) & m1)) continue;
			const unsigned long long key = order * PROJ_CELLS + cell;
			if(map[cell] > key) atomicMin(map + cell, key);
			if(caustic && map[PROJ_SLOT + cell] > key) atomicMin(map + PROJ_SLOT + cell, key);
		}
	}
}

/* A block per map: its bits and its coverage.  The coverage that counts is the
 * ordered double sum rounded to float.  Any order of summation is within
 * 2^-41 of it (2,048 terms, each addition within 2^-53), so a sum in parallel
 * gives that float unless it lies within margin = 2^-40 of where floats round;
 * then (once in some 30,000 maps) the cells are sorted by the order in which they
 * were set and added one by one, 2,048 dependent additions taking 65 us. */
__global__ void __launch_bounds__(1024) k_proj_cover(const unsigned long long *first, const ProjTables *tables, double margin,
		uint32_t *bits, float *cov)
{
	__shared__ unsigned long long key[PROJ_CELLS];
	__shared__ double part[32];
	__shared__ int nset, unsure;
	const unsigned FULL = 0xffffffffu;
	const int t = threadIdx.x, lane = t & 31;
	const unsigned long long *map = first + (size_t)blockIdx.x * PROJ_SLOT;
	const bool whole = map[PROJ_CELLS] == 0;
	if(t == 0) nset = 0;
	__syncthreads();
	double c = 0.0;
	for(int k = 0; k < 2; k++) {
		const int cell = k * 1024 + t;
		const unsigned long long v = map[cell];
		const bool set = whole || v != PROJ_NONE;
		const unsigned b = __ballot_sync(FULL, set);
		if(lane == 0) {
			bits[(size_t)blockIdx.x * 64 + (cell >> 5)] = b;
			atomicAdd(&nset, __popc(b));
		}
		key[cell] = v;
		if(set) c += tables->share[cell];
	}
	for(int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(FULL, c, o);
	if(lane == 0) part[t >> 5] = c;
	__syncthreads();
	if(t < 32) {
		c = part[lane];
		for(int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(FULL, c, o);
		if(t == 0) {
			const float f = whole ? 1.0f : (nset == 0 ? 0.0f : (float)fmin(c, 1.0));
			const double lo = c * (1.0 - margin), hi = c * (1.0 + margin);
			unsure = !whole && nset > 0 && ((float)fmin(lo, 1.0) != f || (float)fmin(hi, 1.0) != f);
			cov[blockIdx.x] = f;
		}
	}
	__syncthreads();
	if(!unsure) return;
	/* bitonic sort (unset cells last); a key's low bits are its cell */
	for(int size = 2; size <= PROJ_CELLS; size <<= 1) {
		for(int step = size >> 1; step > 0; step >>= 1) {
			const int i = 2 * t - (t & (step - 1));
			const bool up = (i & size) == 0;
			const unsigned long long a = key[i], b = key[i + step];
			if((a > b) == up) {
				key[i] = b;
				key[i + step] = a;
			}
			__syncthreads();
		}
	}
	if(t == 0) {
		c = 0.0;
		for(int i = 0; i < nset; i++) c += tables->share[key[i] & (PROJ_CELLS - 1)];
		cov[blockIdx.x] = (float)(c < 0.0 ? 0.0 : (c > 1.0 ? 1.0 : c));
	}
}

/* The reference traces one photon to its end with recursive calls, one map
 * after the other.  Here the photons of both maps advance together, one
 * surface interaction per pass, over ray queues that the renderer's
 * closest-hit kernel traces:
 *   k_photon_emit    Light::gen_photon (src/light.cc:111-148) with
 *                    ProjMap::gen_dir (src/projmap.cc:193-209) -> queue
 *   k_trace          closest hits of the queue (render.cu)
 *   k_photon_bounce  one trace_caustics_photon / trace_global_photon step
 *                    per photon -> stored photon, next queue, or loss
 *   k_photon_finish  the last photons, each traced to its end
 * A photon keeps its own Philox stream: the queue carries its stream address
 * (map, light, index) and draw count, so photon j of light i takes the same
 * draws and the same path as the CPU oracle's recursive tracer.
 *
 * Photon queue entry (RayQueue fields):
 *   o = origin, colour r     d = direction, colour g
 *   w = colour b, ior, interactions in this phase, photon index in its map
 *   meta = light, iter, phase | type << 4 | map << 8, time
 *   stk = ior stack          ext = draws taken, stack depth
 * Phase 0 follows the global rules, phase 1 the caustic rules; map 0 is the
 * caustic map, map 1 the global one. */

#define PHOTON_GUARD 4096   /* interactions per phase (loop bound of the oracle's tracer) */
#define PHOTON_SORT_MIN (1 << 20)   /* an emission pass of at least this many photons is sorted before it is traced */

/* A job of the photon wavefront: one frame's two maps (a batch traces the
 * maps of all its jobs in one wavefront).  Its photons are the global
 * indices [base, base + total[0]) (caustic map) and then total[1] more
 * (global map); each keeps the stream address of its frame's own photon
 * (map, light within the scene, index within the light). */
struct PJob {
	int base;
	int total[2];
	int light0, nlights;  /* its scene's lights in the light table */
	int prefix0;          /* per-light prefix sums at prefix + prefix0: the caustic
	                         map's nlights + 1, then the global map's */
	int scale0;           /* per-light power scales at scale + scale0: caustic, then global */
	int proj0;            /* its first light's projection maps (128 words) and coverages (2) */
	int t0, t1;           /* the frame's interval */
};

struct PhotonSet {
	int njobs, total;
	const PJob *jobs;
	const int *prefix;
	const float *scale;
	const uint32_t *projbits;
	const float *coverage;
	DevPhoton *out;       /* per global index: the stored photon and its flag */
	int *valid;
};

__device__ __forceinline__ int pjob_of(const PhotonSet &P, int id)
{
	int lo = 0, hi = P.njobs - 1;
	while(lo < hi) {
		int mid = (lo + hi + 1) >> 1;
		if(P.jobs[mid].base <= id) lo = mid;
		else hi = mid - 1;
	}
	return lo;
}

__device__ __forceinline__ void push_photon(const RayQueue &q, int slot, const PRay &r, const PState &ph, int guard, int gid,
		int li, int job, int phase, int map, uint32_t draws)
{
	q.o[slot] = make_float4(r.o.x, r.o.y, r.o.z, ph.col[0]);
	q.d[slot] = make_float4(r.d.x, r.d.y, r.d.z, ph.col[1]);
	q.w[slot] = make_float4(ph.col[2], r.st.ior, __int_as_float(guard), __int_as_float(gid));
	q.meta[slot] = make_int4(li | (job << 16), r.iter, phase | (ph.type << 4) | (map << 8), r.time);
	q.stk[slot] = make_float4(r.st.stk[0], r.st.stk[1], r.st.stk[2], r.st.stk[3]);
	q.ext[slot] = make_int2((int)draws, r.st.sp);
}

static __device__ __forceinline__ int photon_slot(int *counter)
{
	cg::coalesced_group g = cg::coalesced_threads();
	int base = 0;
	if(g.thread_rank() == 0) base = atomicAdd(counter, (int)g.size());
	return g.shfl(base, 0) + (int)g.thread_rank();
}

/* emission: `per` photons per warp (32, or fewer where there are too few
 * photons to fill the GPU with a lane each: their tries then take the lanes) */
__global__ void __launch_bounds__(128) k_photon_emit(DScene S, PhotonSet P, int per, RayQueue q, DevCounters *ctr)
{
	__shared__ int list[4][32];
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	const long long id64 = ((long long)blockIdx.x * 4 + w) * per + lane;
	const bool here = lane < per && id64 < P.total;
	const int id = here ? (int)id64 : 0;
	int job = pjob_of(P, id);
	const PJob &J = P.jobs[job];
	int local = id - J.base;
	int map = local >= J.total[0] ? 1 : 0;
	int gid = map ? local - J.total[0] : local;
	int global = map;
	const int *prefix = P.prefix + J.prefix0 + map * (J.nlights + 1);
	int li = 0;
	while(li + 1 < J.nlights && prefix[li + 1] <= gid) li++;
	int j = gid - prefix[li];
	sray_rng s;
	sray_rng_init(&s, S.seed, global ? SRAY_DOM_GLOBAL : SRAY_DOM_CAUST, (uint32_t)j, (uint32_t)li);
	int ms = J.t0 == J.t1 ? J.t0 : (sray_rng_int(&s) % (J.t1 - J.t0) + J.t0);
	int lg = J.light0 + li;
	const DevLight &L = S.lights[lg];
	PState ph;
	V3 pos = light_point(S, lg, ms, &s);
	float cov = P.coverage[(J.proj0 + li) * 2 + (global ? 0 : 1)];
	const uint32_t *bits = P.projbits + (size_t)(J.proj0 + li) * 128 + (global ? 0 : 64);
	for(int k = 0; k < 3; k++) ph.col[k] = L.col[k] * S.photon_energy;
	for(int k = 0; k < 3; k++) ph.col[k] = ph.col[k] * cov;
	ph.type = DIRECT_PHOTON;
	const bool proj = cov != 0.0f;
	V3 dir = mk(0.0f, 0.0f, 0.0f);
	bool ok = gen_dirs(here && proj, bits, s, dir, list[w]);
	if(!here) return;
	if(!proj) {
		for(int k = 0; k < 3; k++) ph.col[k] = L.col[k] * S.photon_energy;
		dir = sphrand(&s, 1.0f);
		ok = true;
	}
	if(!ok) atomicOr(&ctr->gen_dir_fail, 1);
	P.valid[id] = 0;
	if(ok && S.iter > 0) {
		PRay r;
		r.o = pos;
		r.d = dir * (float)SRAY_RAY_MAGNITUDE;
		r.time = ms;
		r.iter = S.iter;
		r.st.ior = 1.0f;
		r.st.sp = 0;
		for(int k = 0; k < 4; k++) r.st.stk[k] = 0.0f;
		int slot = photon_slot(q.count);
		push_photon(q, slot, r, ph, 0, id, li, job, global ? 0 : 1, map, s.n);
	}
}

/* a photon in flight, as the queue entry holds it */
struct PFlight {
	PRay r;
	PState ph;
	int li, job, gid, phase, guard, map;   /* gid: the photon's global index */
	uint32_t draws;
};

__device__ __forceinline__ void load_photon(const RayQueue &q, int i, PFlight &f)
{
	float4 o4 = q.o[i], d4 = q.d[i], w4 = q.w[i], k4 = q.stk[i];
	int4 meta = q.meta[i];
	int2 ext = q.ext[i];
	f.li = meta.x & 0xffff;
	f.job = meta.x >> 16;
	f.phase = meta.z & 15;
	f.map = (meta.z >> 8) & 1;
	f.guard = __float_as_int(w4.z);
	f.gid = __float_as_int(w4.w);
	f.r.o = mk(o4.x, o4.y, o4.z);
	f.r.d = mk(d4.x, d4.y, d4.z);
	f.r.time = meta.w;
	f.r.iter = meta.y;
	f.r.st.ior = w4.y;
	f.r.st.stk[0] = k4.x; f.r.st.stk[1] = k4.y; f.r.st.stk[2] = k4.z; f.r.st.stk[3] = k4.w;
	f.r.st.sp = ext.y;
	f.ph.col[0] = o4.w; f.ph.col[1] = d4.w; f.ph.col[2] = w4.x;
	f.ph.type = (meta.z >> 4) & 15;
	f.draws = (uint32_t)ext.x;
}

/* one surface interaction of a photon at hit h (h.obj >= 0): stores it
 * (returns 1), loses it (0) or leaves it ready for its next trace (2) */
__device__ __forceinline__ int photon_interact(const DScene &S, const PhotonSet &P, PFlight &f, const Hit &h)
{
	int global = f.map;
	const PJob &J = P.jobs[f.job];
	int gid = f.gid - J.base - (f.map ? J.total[0] : 0);   /* within its frame's map */
	sray_rng s;
	sray_rng_init(&s, S.seed, global ? SRAY_DOM_GLOBAL : SRAY_DOM_CAUST,
			(uint32_t)(gid - P.prefix[J.prefix0 + f.map * (J.nlights + 1) + f.li]), (uint32_t)f.li);
	sray_rng_seek(&s, f.draws);
	int res = f.phase == 0 ? global_step(S, f.r, f.ph, h, &s) : caust_step(S, f.r, f.ph, h, &s);
	f.draws = s.n;
	if(res == P_STORE) {
		if(!global && f.ph.type != CAUST_PHOTON) return 0;
		float sc = P.scale[J.scale0 + f.map * J.nlights + f.li];
		DevPhoton p;
		p.p[0] = f.ph.pos.x; p.p[1] = f.ph.pos.y; p.p[2] = f.ph.pos.z; p.p[3] = f.ph.col[0] * sc;
		p.d[0] = f.ph.dir.x; p.d[1] = f.ph.dir.y; p.d[2] = f.ph.dir.z; p.d[3] = f.ph.col[1] * sc;
		p.n[0] = f.ph.norm.x; p.n[1] = f.ph.norm.y; p.n[2] = f.ph.norm.z; p.n[3] = f.ph.col[2] * sc;
		P.out[f.gid] = p;
		P.valid[f.gid] = 1;
		return 1;
	}
	if(res == P_DROP) return 0;
	if(res == P_TO_CAUST) {
		f.phase = 1;
		f.guard = 0;
	} else if(++f.guard >= PHOTON_GUARD) {
		return 0;
	}
	return f.r.iter <= 0 ? 0 : 2;
}

__global__ void __launch_bounds__(128) k_photon_bounce(DScene S, PhotonSet P, RayQueue qi, const int4 *hits, RayQueue qo)
{
	int n = *qi.count;
	for(int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
		const int i = qi.order ? (int)qi.order[k] : k;
		int4 hv = hits[i];
		if(hv.y < 0) continue;                       /* photon left the scene */
		Hit h;
		h.t = __int_as_float(hv.x);
		h.obj = hv.y;
		h.prim = hv.z;
		h.tie = hv.w;
		PFlight f;
		load_photon(qi, i, f);
		if(photon_interact(S, P, f, h) != 2) continue;
		int slot = photon_slot(qo.count);
		if(slot >= qo.cap) continue;                 /* cannot happen: a photon has one successor */
		push_photon(qo, slot, f.r, f.ph, f.guard, f.gid, f.li, f.job, f.phase, f.map, f.draws);
	}
}

/* The tail of the photon maps: once few photons are left, each thread takes
 * photons from the queue (through a shared counter) and traces every one to
 * its end, instead of one interaction per pass; a pass costs as much as its
 * slowest ray, and the tail is made of few photons on long paths.  Photons
 * whose hit the octrees must decide are handed back, before that trace, to
 * the pending queue, which the pass-wise loop finishes. */
__global__ void __launch_bounds__(128) k_photon_finish(DScene S, PhotonSet P, RayQueue qi, int *next, RayQueue qpend,
		DevCounters *ctr)
{
	int n = *qi.count;
	int overflow = 0;
	for(;;) {
		int i = atomicAdd(next, 1);
		if(i >= n) break;
		PFlight f;
		load_photon(qi, i, f);
		for(int step = 0; step < 2 * PHOTON_GUARD + 2; step++) {
			Hit h;
			if(!trace_two_level<false, false>(S, f.r.o, f.r.d, f.r.time, h, nullptr, &overflow, pixel_scene(S, f.gid))) {
				int slot = photon_slot(qpend.count);
				if(slot < qpend.cap) push_photon(qpend, slot, f.r, f.ph, f.guard, f.gid, f.li, f.job, f.phase, f.map, f.draws);
				break;
			}
			if(h.obj < 0) break;
			if(photon_interact(S, P, f, h) != 2) break;
		}
	}
	if(overflow) atomicOr(&ctr->overflow, 1);
}

/* ---------------- scan / compaction ---------------- */
#define TILE 2048

__global__ void k_count_valid(const int *valid, int n, unsigned *bcount)
{
	__shared__ int s;
	if(threadIdx.x == 0) s = 0;
	__syncthreads();
	int base = blockIdx.x * TILE, c = 0;
	for(int i = base + threadIdx.x; i < base + TILE && i < n; i += blockDim.x) c += valid[i];
	atomicAdd(&s, c);
	__syncthreads();
	if(threadIdx.x == 0) bcount[blockIdx.x] = s;
}

/* exclusive scan of m entries by one block of 1024 threads; total -> *total */
__global__ void k_scan_excl(unsigned *data, int m, unsigned *total)
{
	__shared__ unsigned part[1024];
	int t = threadIdx.x;
	int chunk = (m + 1023) / 1024;
	int b = t * chunk, e = min(b + chunk, m);
	unsigned s = 0;
	for(int i = b; i < e; i++) s += data[i];
	part[t] = s;
	__syncthreads();
	for(int off = 1; off < 1024; off <<= 1) {
		unsigned v = t >= off ? part[t - off] : 0;
		__syncthreads();
		part[t] += v;
		__syncthreads();
	}
	unsigned run = part[t] - s;
	for(int i = b; i < e; i++) {
		unsigned v = data[i];
		data[i] = run;
		run += v;
	}
	if(t == 1023 && total) *total = part[1023];
}

/* photons in one or two runs of memory: those from n on are in b */
struct PhotonRuns {
	DevPhoton *a, *b;
	unsigned n;
	__device__ __forceinline__ DevPhoton &at(unsigned i) const { return i < n ? a[i] : b[i - n]; }
};

static PhotonRuns one_run(DevPhoton *p) { return PhotonRuns{p, nullptr, 0xffffffffu}; }

/* order-preserving compaction of one tile per block */
__global__ void k_compact(const int *valid, const DevPhoton *in, int n, const unsigned *boffs, PhotonRuns out)
{
	__shared__ int wsum[8];
	__shared__ int run;
	int base = blockIdx.x * TILE;
	int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	if(threadIdx.x == 0) run = (int)boffs[blockIdx.x];
	__syncthreads();
	for(int r = 0; r < TILE / 256; r++) {
		int i = base + r * 256 + threadIdx.x;
		int v = (i < n) ? valid[i] : 0;
		unsigned bal = __ballot_sync(0xffffffffu, v);
		int wpre = __popc(bal & ((1u << lane) - 1u));
		if(lane == 0) wsum[w] = __popc(bal);
		__syncthreads();
		int off = run;
		for(int k = 0; k < w; k++) off += wsum[k];
		if(v) out.at((unsigned)(off + wpre)) = in[i];
		__syncthreads();
		if(threadIdx.x == 0) {
			int t = 0;
			for(int k = 0; k < 8; k++) t += wsum[k];
			run += t;
		}
		__syncthreads();
	}
}

/* ---------------- grid keys and radix sort ---------------- */
__device__ __forceinline__ unsigned spread3(unsigned v)
{
	v &= 0x3ff;
	v = (v | (v << 16)) & 0x030000FF;
	v = (v | (v << 8)) & 0x0300F00F;
	v = (v | (v << 4)) & 0x030C30C3;
	v = (v | (v << 2)) & 0x09249249;
	return v;
}

__device__ __forceinline__ unsigned cell_key(const DevPhoton &p, const DPhotonMap &M, int morton)
{
	int c[3];
	for(int a = 0; a < 3; a++) {
		double v = floor(((double)p.p[a] - (double)M.org[a]) / (double)M.cell);
		c[a] = v < 0.0 ? 0 : (v > (double)(M.dims[a] - 1) ? M.dims[a] - 1 : (int)v);
	}
	return morton ? (spread3(c[0]) | (spread3(c[1]) << 1) | (spread3(c[2]) << 2))
		: (unsigned)(((size_t)c[2] * M.dims[1] + c[1]) * M.dims[0] + c[0]);
}

__global__ void k_keys(const DevPhoton *ph, int n, DPhotonMap M, int morton, unsigned *keys, unsigned *vals)
{
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
		keys[i] = cell_key(ph[i], M, morton);
		vals[i] = (unsigned)i;
	}
}

#define RS_THREADS 256

__global__ void k_rs_hist(const unsigned *keys, int n, int shift, unsigned *hist, int nblocks)
{
	__shared__ unsigned h[256];
	h[threadIdx.x] = 0;
	__syncthreads();
	int base = blockIdx.x * TILE;
	for(int i = base + threadIdx.x; i < base + TILE && i < n; i += RS_THREADS) atomicAdd(&h[(keys[i] >> shift) & 255u], 1u);
	__syncthreads();
	hist[(size_t)threadIdx.x * nblocks + blockIdx.x] = h[threadIdx.x];
}

/* stable scatter: tile items in order, ranks within a round from warp match masks */
__global__ void k_rs_scatter(const unsigned *keys, const unsigned *vals, int n, int shift, const unsigned *offs, int nblocks,
		unsigned *okeys, unsigned *ovals)
{
	__shared__ unsigned base[256];
	__shared__ unsigned wcnt[RS_THREADS / 32][257];
	int t = threadIdx.x, lane = t & 31, w = t >> 5;
	base[t] = offs[(size_t)t * nblocks + blockIdx.x];
	int tile = blockIdx.x * TILE;
	for(int r = 0; r < TILE / RS_THREADS; r++) {
		for(int k = 0; k < RS_THREADS / 32; k++) wcnt[k][t] = 0;
		if(t == 0) for(int k = 0; k < RS_THREADS / 32; k++) wcnt[k][256] = 0;
		__syncthreads();
		int i = tile + r * RS_THREADS + t;
		bool v = i < n;
		unsigned key = v ? keys[i] : 0u;
		unsigned d = v ? ((key >> shift) & 255u) : 256u;
		unsigned peers = __match_any_sync(0xffffffffu, d);
		int rank = __popc(peers & ((1u << lane) - 1u));
		if(lane == __ffs(peers) - 1) wcnt[w][d] = __popc(peers);
		__syncthreads();
		if(v) {
			unsigned pos = base[d] + rank;
			for(int k = 0; k < w; k++) pos += wcnt[k][d];
			okeys[pos] = key;
			ovals[pos] = vals[i];
		}
		__syncthreads();
		unsigned add = 0;
		for(int k = 0; k < RS_THREADS / 32; k++) add += wcnt[k][t];
		base[t] += add;
		__syncthreads();
	}
}

__global__ void k_permute(PhotonRuns in, const unsigned *vals, int n, PhotonRuns out)
{
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out.at((unsigned)i) = in.at(vals[i]);
}

/* the first of keys[lo, hi) (ascending) that is at least k */
__device__ __forceinline__ unsigned lower_key(const unsigned *keys, unsigned lo, unsigned hi, unsigned k)
{
	while(lo < hi) {
		unsigned mid = (lo + hi) >> 1;
		if(__ldg(keys + mid) < k) lo = mid + 1;
		else hi = mid;
	}
	return lo;
}

/* A map's cell table from the sorted cell keys (cell + k0) of its photons
 * [i0, i1): start[c] = its photons (counted from i0) in cells before c, for every cell
 * and one past the last.  A block takes START_CELLS cells: two searches find
 * its photons, counters in shared memory their cells, a scan the starts;
 * what bounds it is the table's own write (4 bytes a cell). */
#define START_CELLS 2048
__device__ __forceinline__ void cell_starts(const unsigned *keys, unsigned i0, unsigned i1, unsigned k0, size_t ncells, unsigned *start)
{
	__shared__ unsigned cnt[START_CELLS];
	__shared__ unsigned range[2];
	__shared__ unsigned wsum[8];
	const size_t c0 = (size_t)blockIdx.x * START_CELLS;
	const int t = threadIdx.x, lane = t & 31, w = t >> 5;
	if(t < 2) range[t] = lower_key(keys, i0, i1, (unsigned)min(k0 + c0 + (size_t)t * START_CELLS, (size_t)0xffffffffu));
	for(int i = t; i < START_CELLS; i += 256) cnt[i] = 0;
	__syncthreads();
	const unsigned b = range[0], e = range[1];
	for(unsigned i = b + t; i < e; i += 256) atomicAdd(&cnt[__ldg(keys + i) - (k0 + (unsigned)c0)], 1u);
	__syncthreads();
	/* eight cells per thread, scanned over the block */
	unsigned v[8], s = 0;
	#pragma unroll
	for(int k = 0; k < 8; k++) {
		v[k] = cnt[t * 8 + k];
		s += v[k];
	}
	unsigned incl = s;
	for(int o = 1; o < 32; o <<= 1) {
		unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
		if(lane >= o) incl += u;
	}
	if(lane == 31) wsum[w] = incl;
	__syncthreads();
	unsigned run = b - i0 + incl - s;
	for(int k = 0; k < w; k++) run += wsum[k];
	#pragma unroll
	for(int k = 0; k < 8; k++) {
		cnt[t * 8 + k] = run;
		run += v[k];
	}
	__syncthreads();
	for(int i = t; i < START_CELLS && c0 + i <= ncells; i += 256) start[c0 + i] = cnt[i];
}

__global__ void __launch_bounds__(256) k_starts(const unsigned *keys, int n, size_t ncells, unsigned *start)
{
	cell_starts(keys, 0, (unsigned)n, 0, ncells, start);
}

/* Photon launches run beside the frame's higher-priority stream: a block
 * per `block` items, so that blocks are short-lived and the frame's kernels
 * get SMs as they free, instead of a capped grid whose blocks stride over
 * the whole launch and hold their SMs until it ends. */
static int grid_n(int n, int block)
{
	int g = (n + block - 1) / block;
	return g < 1 ? 1 : g;
}

#define PCK(call, where) do { cudaError_t e_ = (call); if(e_ != cudaSuccess) return R.cuda_fail(e_, where); } while(0)

/* emission counts of one map of a frame: photons split by mean light
 * intensity (src/render.cc:87-110); appends the per-light prefix sums
 * (nl + 1) and power scales (nl), returns the map's total */
static int split_photons(const Renderer &R, int light0, int nl, int num, std::vector<int> &prefix, std::vector<float> &scale)
{
	size_t p0 = prefix.size();
	prefix.resize(p0 + nl + 1, 0);
	scale.resize(scale.size() + nl, 0.0f);
	size_t s0 = scale.size() - nl;
	if(num <= 0 || nl <= 0) return 0;
	std::vector<double> inten(nl);
	double accp = 0.0;
	for(int i = 0; i < nl; i++) {
		const double *c = R.sc.lights[light0 + i].col;
		inten[i] = (c[0] + c[1] + c[2]) / 3.0;
		accp += inten[i];
	}
	for(int i = 0; i < nl; i++) {
		int nphot = (int)ceil((double)num * (inten[i] / accp));
		prefix[p0 + i + 1] = prefix[p0 + i] + nphot;
		scale[s0 + i] = nphot ? (float)(1.0 / (double)nphot) : 0.0f;
	}
	return prefix[p0 + nl];
}

/* the projection maps' inputs on the host: kept until the stream that copies
 * them has been waited for */
struct ProjHost {
	std::vector<ProjSample> samples;
	std::vector<ProjBox> boxes;
};

/* What is made at a time, so that the workspace does not grow with lights,
 * objects and jobs: pairs of a light sample and a box (72 bytes each),
 * lights (33 kB each), boxes (56 bytes each).  What a frame or a batch of
 * some hundred objects needs is one group. */
#define PROJ_VIEWS (1 << 20)
#define PROJ_LIGHTS 1024
#define PROJ_BOXES (1 << 20)

/* every job's projection maps on stream s: bits (128 words per light of a
 * job: 2048 cells of the map, then of the caustic map) in R.pw_bits, the two
 * coverages in R.pw_cov; and the jobs' boxes, of the same bounds */
static int project_jobs(Renderer &R, std::vector<PhotonJobSpec> &spec, ProjHost &host, cudaStream_t s)
{
	double tp = Renderer::host_now_ms();
	const int small = g_faults.photon_group.load();
	const size_t max_views = small > 0 ? small : PROJ_VIEWS, max_boxes = small > 0 ? small : PROJ_BOXES;
	const int max_lights = small > 0 ? 2 : PROJ_LIGHTS;
	int slots = 0;
	for(const PhotonJobSpec &J : spec) slots += J.nlights;
	if(slots > 0) {
		if(!R.pj_tables_ready) {
			PCK(R.pj_tables.ensure(sizeof(ProjTables)), "projection tables");
			PCK(cudaMemcpyAsync(R.pj_tables.p, &proj_tables(), sizeof(ProjTables), cudaMemcpyHostToDevice, s), "projection tables");
			R.h2d += (int64_t)sizeof(ProjTables);
			R.pj_tables_ready = true;
		}
		PCK(R.pw_bits.ensure((size_t)slots * 128 * sizeof(uint32_t)), "projection maps");
		PCK(R.pw_cov.ensure((size_t)slots * 2 * sizeof(float)), "coverage");
	}
	int done = 0, lights = 0, most = 0;   /* lights of earlier groups and of this one; its samples' largest box count */
	auto send = [&]() -> int {
		if(lights == 0) return 0;
		const size_t bytes = (size_t)lights * 2 * PROJ_SLOT * sizeof(unsigned long long);
		PCK(R.pj_first.ensure(bytes), "projection cells");
		PCK(cudaMemsetAsync(R.pj_first.p, 0xff, bytes, s), "projection cells");
		const int ns = (int)host.samples.size();
		if(ns > 0) {
			PCK(R.pj_samples.upload(host.samples, s), "light samples");
			PCK(R.pj_boxes.upload(host.boxes, s), "object boxes");
			R.h2d += (int64_t)(ns * sizeof(ProjSample) + host.boxes.size() * sizeof(ProjBox));
			const int per = (int)std::max<size_t>(1, std::min<size_t>(max_views / most, ns));
			PCK(R.pj_views.ensure((size_t)per * most * sizeof(ProjView)), "projections");
			const ProjBox *boxes = R.pj_boxes.as<ProjBox>();
			ProjView *views = R.pj_views.as<ProjView>();
			const ProjTables *tables = R.pj_tables.as<ProjTables>();
			unsigned long long *first = R.pj_first.as<unsigned long long>();
			for(int q = 0; q < ns; q += per) {
				const ProjSample *smp = R.pj_samples.as<ProjSample>() + q;
				const int m = std::min(per, ns - q);
				LAUNCH(R, "projmaps", s, k_proj_view<<<(unsigned)std::min<size_t>(((size_t)m * most + 127) / 128, 1 << 20), 128, 0, s>>>(smp,
						m, most, boxes, views, tables, first));
				LAUNCH(R, "projmaps", s, k_proj_mark<<<dim3((unsigned)most, (unsigned)std::min(m, 65535)), 128, 0, s>>>(smp, m, most, boxes,
						views, tables, first));
			}
		}
		LAUNCH(R, "projmaps", s, k_proj_cover<<<lights * 2, 1024, 0, s>>>(R.pj_first.as<unsigned long long>(), R.pj_tables.as<ProjTables>(),
				small > 0 ? 1.0 : 1.0 / 1099511627776.0, R.pw_bits.as<uint32_t>() + (size_t)done * 128, R.pw_cov.as<float>() + (size_t)done * 2));
		PCK(cudaGetLastError(), "projection maps");
		return 0;
	};
	/* the next group, whose inputs take the place of the last one's */
	auto next = [&]() -> int {
		if(int r = send()) return r;
		PCK(cudaStreamSynchronize(s), "projection maps");
		done += lights;
		lights = most = 0;
		host.samples.clear();
		host.boxes.clear();
		return 0;
	};
	std::vector<ProjBox> ends[2];
	std::vector<Vec3> pts;
	std::vector<int> times;
	for(PhotonJobSpec &J : spec) {
		/* the job's object boxes at its interval's ends, and their union */
		const int at[2] = {J.t0, J.t1}, nend = J.t0 == J.t1 ? 1 : 2;
		for(int k = 0; k < 3; k++) { J.box.mn[k] = FLT_MAX; J.box.mx[k] = -FLT_MAX; }
		for(int e = 0; e < nend; e++) {
			ends[e].clear();
			for(int i = J.obj0; i < J.obj0 + J.nobj; i++) {
				const Box b = R.sc.object_bounds((size_t)i, at[e]);
				const Material &m = R.sc.objs[i].mat >= 0 ? R.sc.mats[R.sc.objs[i].mat] : R.sc.defmat;
				ProjBox d;
				for(int k = 0; k < 3; k++) {
					d.mn[k] = b.mn[k];
					d.mx[k] = b.mx[k];
					J.box.mn[k] = std::min(J.box.mn[k], b.mn[k]);
					J.box.mx[k] = std::max(J.box.mx[k], b.mx[k]);
				}
				d.caustic = m.refl > 0.0 || m.refr > 0.0 ? 1 : 0;
				d.pad = 0;
				ends[e].push_back(d);
			}
		}
		int box0[2] = {-1, -1};
		for(int k = 0; k < J.nlights; k++) {
			if(lights >= max_lights || (box0[0] < 0 && lights > 0 && host.boxes.size() + nend * ends[0].size() > max_boxes)) {
				if(int r = next()) return r;
				box0[0] = -1;
			}
			const int slot = lights++;
			if(J.nobj <= 0) continue;
			if(box0[0] < 0) {
				for(int e = 0; e < nend; e++) {
					box0[e] = (int)host.boxes.size();
					host.boxes.insert(host.boxes.end(), ends[e].begin(), ends[e].end());
				}
			}
			pts.clear();
			times.clear();
			R.sc.light_samples((size_t)(J.light0 + k), J.t0, J.t1, R.opt.seed, k, pts, times);
			for(size_t q = 0; q < pts.size(); q++) {
				ProjSample d;
				for(int c = 0; c < 3; c++) d.lp[c] = pts[q][c];
				d.box0 = box0[times[q] == J.t0 ? 0 : 1];
				d.nbox = J.nobj;
				d.slot = slot;
				d.order = (unsigned)q;
				host.samples.push_back(d);
				most = std::max(most, J.nobj);
			}
		}
	}
	if(int r = send()) return r;
	R.host_time("host.projmaps", tp);
	return 0;
}

/* Both photon maps of every job, traced as one wavefront on stream s: their
 * projection maps, the emission of all jobs' photons in one launch, then
 * passes of closest hits and interactions over one queue (each photon finds its job, and through
 * it its scene, lights, interval and projection maps), then the tail.  The
 * stored photons and their flags stay in R.pw_out / R.pw_valid by global
 * index; jobs[j].base and total[] locate each job's two segments. */
int photon_trace_jobs(Renderer &R, const DScene &base, std::vector<PhotonJobSpec> &spec, std::vector<PJobOut> &out, cudaStream_t s)
{
	ProjHost proj_host;
	int n = (int)spec.size();
	out.assign(n, PJobOut());
	std::vector<PJob> jobs(n);
	std::vector<int> prefix;
	std::vector<float> scale;
	std::vector<DevJob> pj(n);
	int proj = 0;
	int64_t all = 0;
	for(int j = 0; j < n; j++) {
		const PhotonJobSpec &J = spec[j];
		PJob &d = jobs[j];
		memset(&d, 0, sizeof d);
		d.base = (int)all;
		d.light0 = J.light0;
		d.nlights = J.nlights;
		d.prefix0 = (int)prefix.size();
		d.scale0 = (int)scale.size();
		d.proj0 = proj;
		proj += J.nlights;
		d.t0 = J.t0;
		d.t1 = J.t1;
		for(int m = 0; m < 2; m++) d.total[m] = split_photons(R, J.light0, J.nlights, J.num[m], prefix, scale);
		memset(&pj[j], 0, sizeof pj[j]);
		pj[j].pix0 = d.base;
		pj[j].scene = J.scene;
		out[j].base = d.base;
		out[j].total[0] = d.total[0];
		out[j].total[1] = d.total[1];
		all += (int64_t)d.total[0] + d.total[1];
		if(all > INT_MAX / 2) return R.fail(SRAY_EINVAL, "too many photons in one wavefront");
	}
	if(all == 0) return 0;
	if(int r = project_jobs(R, spec, proj_host, s)) return r;
	PCK(R.pw_jobs.upload(jobs, s), "photon jobs");
	PCK(R.pw_prefix.upload(prefix, s), "photon prefix");
	PCK(R.pw_scale.upload(scale, s), "photon scale");
	PCK(R.pw_pix.upload(pj, s), "photon job table");
	R.h2d += (int64_t)(jobs.size() * sizeof(PJob) + prefix.size() * 4 + scale.size() * 4 + pj.size() * sizeof(DevJob));
	PCK(R.pw_out.ensure((size_t)all * sizeof(DevPhoton)), "photon buffer");
	PCK(R.pw_valid.ensure((size_t)all * sizeof(int)), "photon flags");
	PhotonSet PSet;
	PSet.njobs = n;
	PSet.total = (int)all;
	PSet.jobs = R.pw_jobs.as<PJob>();
	PSet.prefix = R.pw_prefix.as<int>();
	PSet.scale = R.pw_scale.as<float>();
	PSet.projbits = R.pw_bits.as<uint32_t>();
	PSet.coverage = R.pw_cov.as<float>();
	PSet.out = R.pw_out.as<DevPhoton>();
	PSet.valid = R.pw_valid.as<int>();
	PCK(R.pctr.ensure(sizeof(DevCounters)), "counters");
	PCK(R.pcounts.ensure(64 * sizeof(int)), "counts");
	PCK(cudaMemsetAsync(R.pctr.p, 0, sizeof(DevCounters), s), "counters");
	PCK(cudaMemsetAsync(R.pcounts.p, 0, 4 * sizeof(int), s), "photon queue counts");
	int *cnt = R.pcounts.as<int>();
	R.pq[0].count = cnt + 0;
	R.pq[1].count = cnt + 1;
	R.pq[0].order = R.pq[1].order = nullptr;
	if(R.ensure_pqueue(0, (int)all) || R.ensure_pqueue(1, (int)all)) return SRAY_ECUDA;
	PCK(R.phits.ensure((size_t)all * 16), "photon hits");
	/* the scene as the photon kernels see it: in a scene set with the photon
	 * job table, through which a photon's global index finds its scene (the
	 * render's pixel table is not theirs) */
	DScene PS = base;
	PS.jobs = PS.nscenes > 1 ? R.pw_pix.as<DevJob>() : nullptr;
	PS.njobs = PS.nscenes > 1 ? n : 0;
	DevCounters *pctr = R.pctr.as<DevCounters>();
	/* photons per warp: a lane each once they fill the GPU's 2,048 lanes per
	 * SM, else as few as fill it with their tries */
	int per = 32;
	while(per > 2 && all * (32 / per) * 2 <= (int64_t)R.nsm * 2048) per >>= 1;
	LAUNCH(R, "photon_emit", s, k_photon_emit<<<grid_n((int)all, 4 * per), 128, 0, s>>>(PS, PSet, per, R.pq[0], pctr));
	/* the emitted count (a photon whose direction sampling fails is not queued) */
	PCK(cudaMemcpyAsync(R.pin + 8, R.pq[0].count, sizeof(int), cudaMemcpyDeviceToHost, s), "photon queue count");
	PCK(cudaStreamSynchronize(s), "photon emission");
	int cur = 0;
	int n_live = R.pin[8];
	R.d2h += sizeof(int);
	R.prof_collect();
	bool finished = false;
	for(int pass = 0; n_live > 0; pass++) {
		if(pass >= 2 * PHOTON_GUARD + 4) return R.fail(SRAY_EDEVICE, "photon paths did not terminate");
		PCK(cudaMemsetAsync(R.pq[cur ^ 1].count, 0, sizeof(int), s), "reset photon queue");
		if(!finished && pass > 0 && n_live <= R.tune.photon_tail) {
			/* the tail in one launch; what it hands back continues pass-wise */
			finished = true;
			PCK(cudaMemsetAsync(cnt + 2, 0, sizeof(int), s), "reset photon tail counter");
			LAUNCH(R, "photon_finish", s, k_photon_finish<<<grid_n(n_live, 128), 128, 0, s>>>(PS, PSet, R.pq[cur], cnt + 2,
					R.pq[cur ^ 1], pctr));
			PCK(cudaMemcpyAsync(R.pin + 8, R.pq[cur ^ 1].count, sizeof(int), cudaMemcpyDeviceToHost, s), "photon queue count");
			PCK(cudaStreamSynchronize(s), "photon tail");
			n_live = R.pin[8];
			R.d2h += sizeof(int);
			R.prof_collect();
			cur ^= 1;
			continue;
		}
		/* a large emission pass in the order of direction octant and origin
		 * cell: the photons of a warp then leave one light into one octant
		 * (the queue's order is arbitrary anyway: its slots come from
		 * atomics, and each entry carries its photon's identity); the
		 * bounced passes gain less than their sort costs */
		if(pass == 0 && n_live >= PHOTON_SORT_MIN)
			if(int r = R.sort_photon_pass(cur, n_live, s)) return r;
		if(launch_trace(R, PS, R.pq[cur], n_live, "photon_trace", s)) return SRAY_ECUDA;
		LAUNCH(R, "photon_bounce", s, k_photon_bounce<<<grid_n(n_live, 128), 128, 0, s>>>(PS, PSet, R.pq[cur], R.phits.as<int4>(),
				R.pq[cur ^ 1]));
		R.pq[cur].order = nullptr;
		PCK(cudaMemcpyAsync(R.pin + 8, R.pq[cur ^ 1].count, sizeof(int), cudaMemcpyDeviceToHost, s), "photon queue count");
		PCK(cudaStreamSynchronize(s), "photon pass");
		n_live = R.pin[8];
		R.d2h += sizeof(int);
		R.prof_collect();
		cur ^= 1;
	}
	DevCounters hc;
	PCK(cudaMemcpyAsync(&hc, pctr, sizeof hc, cudaMemcpyDeviceToHost, s), "counters");
	PCK(cudaStreamSynchronize(s), "photon trace");
	R.d2h += sizeof(DevCounters);
	if(hc.overflow) return R.fail(SRAY_EDEVICE, "traversal stack overflow while tracing photons");
	if(hc.gen_dir_fail) return R.fail(SRAY_EDEVICE, "projection-map sampling found no covered cell");
	return 0;
}

/* a map's stored photons from its segment of the wavefront's output
 * (flags `valid`, photons `in`, `total` of them): compacted in emission
 * order, sorted by grid cell, with the cell table */
int photon_finalize(Renderer &R, int global, const int *valid, const DevPhoton *in, int total, cudaStream_t s, int *stored)
{
	PhotonBufs &P = global ? R.gi : R.caust;
	*stored = 0;
	P.map.n = 0;
	if(total <= 0) return 0;
	/* compaction in emission order */
	int nb = (total + TILE - 1) / TILE;
	PCK(R.pw_tiles.ensure((size_t)(nb + 4) * sizeof(unsigned)), "scan");
	unsigned *bc = R.pw_tiles.as<unsigned>();
	LAUNCH(R, "photon_compact", s, k_count_valid<<<nb, 256, 0, s>>>(valid, total, bc));
	LAUNCH(R, "photon_compact", s, k_scan_excl<<<1, 1024, 0, s>>>(bc, nb, bc + nb));
	unsigned h_n = 0;
	PCK(cudaMemcpyAsync(&h_n, bc + nb, sizeof(unsigned), cudaMemcpyDeviceToHost, s), "stored count");
	PCK(cudaStreamSynchronize(s), "photon compaction");
	R.d2h += sizeof(unsigned);
	R.prof_collect();
	int n = (int)h_n;
	*stored = n;
	if(n == 0) return 0;
	PCK(P.ph.ensure((size_t)n * sizeof(DevPhoton)), "photon map");
	LAUNCH(R, "photon_compact", s, k_compact<<<nb, 256, 0, s>>>(valid, in, total, bc, one_run(P.ph.as<DevPhoton>())));
	return photon_map_build(R, global, n, s);
}

/* both photon maps of the frame (one job): the wavefront, then each map from
 * its segment */
int photon_shoot_maps(Renderer &R, const DScene &base, cudaStream_t s, int *nc, int *ng)
{
	*nc = *ng = 0;
	R.caust.map.n = 0;
	R.gi.map.n = 0;
	std::vector<PhotonJobSpec> spec(1);
	PhotonJobSpec &J = spec[0];
	J.num[0] = R.opt.caust_photons;
	J.num[1] = R.opt.gi_photons;
	J.light0 = 0;
	J.nlights = (int)R.sc.lights.size();
	J.t0 = base.t0;
	J.t1 = base.t1;
	J.scene = -1;
	J.nobj = (int)R.sc.objs.size();
	std::vector<PJobOut> out;
	int r = photon_trace_jobs(R, base, spec, out, s);
	if(r) return r;
	/* a map alone: its own build (320x240 frames with 20,000 photons in one
	 * map 582 us, 618 by the joint build, which uploads its tables) */
	if(out[0].total[0] == 0 || out[0].total[1] == 0 || R.sc.oct.nodes.empty()) {
		const DevPhoton *ph = R.pw_out.as<DevPhoton>();
		const int *valid = R.pw_valid.as<int>();
		if((r = photon_finalize(R, 0, valid, ph, out[0].total[0], s, nc))) return r;
		int o1 = out[0].total[0];
		return photon_finalize(R, 1, valid + o1, ph + o1, out[0].total[1], s, ng);
	}
	/* the boxes and radii of photon_map_build, the scene's extents; two
	 * tables are at most 2^27 cells */
	std::vector<DPhotonMap> maps;
	r = photon_finalize_jobs(R, out, std::vector<Box>(1, R.map_has_box ? R.map_box : R.sc.oct.nodes[0].box),
			std::vector<double>(1, R.map_gather_dist >= 0.0 ? R.map_gather_dist : R.sc.gather_dist), maps, s, true);
	if(r) return r;
	*nc = maps[0].n;
	*ng = maps[1].n;
	return 0;
}

/* A map's grid over box rb: cells of the given width, at most 2^26 of them;
 * returns their number */
static size_t map_cells(double width, const Box &rb, DPhotonMap &M)
{
	double cell = width;
	double ext[3];
	for(int a = 0; a < 3; a++) ext[a] = rb.mx[a] - rb.mn[a];
	int dims[3];
	for(;;) {
		double total_cells = 1.0;
		for(int a = 0; a < 3; a++) {
			double d = floor(ext[a] / cell) + 1.0;
			dims[a] = d < 67108864.0 ? (int)d : 67108864;
			total_cells *= d;
		}
		if(total_cells <= (double)(1 << 26)) break;
		cell *= 1.25;
	}
	M.cell = (float)cell;
	while((double)M.cell < cell) M.cell = nextafterf(M.cell, INFINITY);
	for(int a = 0; a < 3; a++) { M.dims[a] = dims[a]; M.org[a] = (float)rb.mn[a]; }
	for(int a = 0; a < 3; a++) while((double)M.org[a] > rb.mn[a]) M.org[a] = nextafterf(M.org[a], -INFINITY);
	return (size_t)dims[0] * dims[1] * dims[2];
}

/* The map of n photons over box rb for gathers of radius rad (k nearest, or
 * all within rad when k = 0): its range constants and the grid that queries
 * walk.  A query reads the photons of whole cells; on a surface, the cells
 * that the range reaches cover 1.7 times its disc when they are half the
 * radius wide, 2.6 times at the radius and 4.8 times at twice the radius.
 * Measured, 500,009 points of a map of 500k emitted photons: 1.17 ms at half
 * the radius, 1.25 at the radius, 1.43 at twice, and 1.28 at a third, where
 * the rows to look up outweigh the photons saved.  A finer grid costs its
 * table, 4 bytes a cell to write at every build: the finest of the three
 * widths whose table has at most 32 cells per photon (and 65,536) is taken,
 * so that the table stays small beside the photons (48 bytes each, moved
 * several times by the sort). */
static size_t map_grid(int k, double rad, const Box &rb, int n, DPhotonMap &M)
{
	const double most = 32.0 * n + 65536.0;
	size_t ncells = 0;
	const double f[3] = {0.5, 1.0, 2.0};
	for(int i = 0; i < 3; i++) {
		double w = rad > 0.0 ? f[i] * rad : 1.0;
		double cells = 1.0;
		for(int a = 0; a < 3; a++) cells *= floor((rb.mx[a] - rb.mn[a]) / w) + 1.0;
		if(cells > most && i < 2) continue;
		ncells = map_cells(w, rb, M);
		break;
	}
	M.n = n;
	M.k = k;
	M.range = (double)(float)rad;
	M.inv_area = (float)(1.0 / (M_PI * (rad * rad)));
	M.range_f = (float)rad;
	{
		double r2 = (double)M.range_f * (double)M.range_f;   /* exact: 48 significant bits */
		M.r2_hi = (float)r2;
		M.r2_lo = (float)(r2 - (double)M.r2_hi);
		M.screen = (float)(r2 * (1.0 + 1.0 / 1048576.0));
	}
	M.inv_cell = (float)(1.0 / (double)M.cell);
	M.reach = (float)((double)M.range_f / (double)M.cell * (1.0 + 1e-6));
	return ncells;
}

static int key_bits(unsigned maxkey)
{
	int bits = 0;
	while(bits < 32 && (maxkey >> bits)) bits++;
	return bits;
}

/* photons ph[0, n) in the order of their cells in M (of the cells' Morton
 * codes): the sorted keys and the photons' indices, in the wavefront's key
 * buffer until its next use */
static int sort_by_cell(Renderer &R, const DevPhoton *ph, int n, const DPhotonMap &M, int morton, cudaStream_t s, unsigned **keys_out,
		unsigned **vals_out)
{
	int bits = key_bits((unsigned)((size_t)M.dims[0] * M.dims[1] * M.dims[2] - 1));
	if(morton) {
		bits = 0;
		for(int a = 0; a < 3; a++) if(M.dims[a] > 1) bits = std::max(bits, 3 * key_bits((unsigned)M.dims[a] - 1) - 2 + a);
	}
	PCK(R.pw_keys.ensure((size_t)n * 16), "keys");
	unsigned *keys = R.pw_keys.as<unsigned>(), *vals = keys + n, *keys2 = keys + 2 * (size_t)n, *vals2 = keys + 3 * (size_t)n;
	LAUNCH(R, "photon_sort", s, k_keys<<<grid_n(n, 256), 256, 0, s>>>(ph, n, M, morton, keys, vals));
	return sort_pairs(R, keys, vals, keys2, vals2, n, bits, R.pw_hist, R.pw_part, "photon_sort", s, keys_out, vals_out);
}

/* the map over the n photons in P.ph: grid, sort by cell, cell table.  The
 * photons as given stay in P.tmp_ph (photon_map_read's order starts from
 * them). */
int photon_map_build(Renderer &R, int global, int n, cudaStream_t s)
{
	PhotonBufs &P = global ? R.gi : R.caust;
	const sray_opts &opt = R.opt;
	if(R.sc.oct.nodes.empty()) return R.fail(SRAY_ESTATE, "no scene bounds (build the frame first)");
	/* grid over the scene bounds (a batch job's: its scene over its own
	 * interval, the box its frame alone would have) */
	const Box &rb = R.map_has_box ? R.map_box : R.sc.oct.nodes[0].box;
	int k = global ? opt.gi_k : opt.caust_k;
	/* a job of a batch gathers with the radius of its own interval */
	double rad = k > 0 ? (double)opt.gather_rcap : (R.map_gather_dist >= 0.0 ? R.map_gather_dist : R.sc.gather_dist);
	DPhotonMap M = DPhotonMap();
	const size_t ncells = map_grid(k, rad, rb, n, M);
	map_cells(rad > 0.0 ? 2.0 * rad : 1.0, rb, P.order);
	PCK(P.starts.ensure((ncells + 1) * sizeof(unsigned)), "cell table");
	PCK(P.tmp_ph.ensure((size_t)n * sizeof(DevPhoton)), "photon buffer");
	unsigned *keys = nullptr, *vals = nullptr;
	if(int r = sort_by_cell(R, P.ph.as<DevPhoton>(), n, M, 0, s, &keys, &vals)) return r;
	LAUNCH(R, "photon_sort", s, k_permute<<<grid_n(n, 256), 256, 0, s>>>(one_run(P.ph.as<DevPhoton>()), vals, n, one_run(P.tmp_ph.as<DevPhoton>())));
	LAUNCH(R, "photon_sort", s, k_starts<<<(unsigned)((ncells + START_CELLS) / START_CELLS), 256, 0, s>>>(keys, n, ncells,
			P.starts.as<unsigned>()));
	std::swap(P.ph, P.tmp_ph);
	M.ph = P.ph.as<DevPhoton>();
	M.start = P.starts.as<unsigned>();
	P.map = M;
	PCK(cudaStreamSynchronize(s), "photon map build");
	R.prof_collect();
	return 0;
}

/* The first m photons of map `global` as programs see them
 * (sray_gpu_get_photons, dumps): in Morton order of cells twice the gather
 * radius (linear order where a dimension passes 10 bits), ties in emission
 * order, into h.  Sorted for each call, in the buffers that the map's own
 * making left: the wavefront's keys and photons, the latter only too small
 * for a restored map, whose photons are picked on the host where there is no
 * memory for them. */
int photon_map_read(Renderer &R, int global, int m, std::vector<DevPhoton> &h, cudaStream_t s)
{
	PhotonBufs &P = global ? R.gi : R.caust;
	const int n = P.map.n;
	h.clear();
	if(n <= 0 || m <= 0) return 0;
	const DPhotonMap &M = P.order;
	const int morton = M.dims[0] <= 1024 && M.dims[1] <= 1024 && M.dims[2] <= 1024;
	unsigned *keys = nullptr, *vals = nullptr;
	if(int r = sort_by_cell(R, P.tmp_ph.as<DevPhoton>(), n, M, morton, s, &keys, &vals)) return r;
	if(R.pw_out.ensure((size_t)m * sizeof(DevPhoton)) == cudaSuccess) {
		h.resize(m);
		LAUNCH(R, "photon_sort", s, k_permute<<<grid_n(m, 256), 256, 0, s>>>(one_run(P.tmp_ph.as<DevPhoton>()), vals, m, one_run(R.pw_out.as<DevPhoton>())));
		PCK(cudaMemcpyAsync(h.data(), R.pw_out.p, (size_t)m * sizeof(DevPhoton), cudaMemcpyDeviceToHost, s), "read photons");
		PCK(cudaStreamSynchronize(s), "read photons");
	} else {
		cudaGetLastError();
		std::vector<unsigned> order(m);
		std::vector<DevPhoton> all(n);
		PCK(cudaMemcpyAsync(order.data(), vals, (size_t)m * sizeof(unsigned), cudaMemcpyDeviceToHost, s), "read photons");
		PCK(cudaMemcpyAsync(all.data(), P.tmp_ph.p, (size_t)n * sizeof(DevPhoton), cudaMemcpyDeviceToHost, s), "read photons");
		PCK(cudaStreamSynchronize(s), "read photons");
		for(unsigned i : order) h.push_back(all[i]);
	}
	R.prof_collect();
	return 0;
}

/* ---------------- the maps of many jobs at once (a batch) ----------------
 * The wavefront's output holds every job's two maps as segments (job-major,
 * caustic then global).  One compaction keeps the stored photons of all
 * segments in emission order; each photon's key is its cell in its own
 * map's grid, counted on from the cells of the segments before it; a stable
 * LSD radix sort leaves the segments in order, each sorted by cell with ties
 * in emission order -- the order a map sorted alone gets -- and each
 * segment's cell table indexes its own photons.  (A sort by cell and another
 * by segment, as before, took 2.41 ms for six 480x270 frames, 2.35 now.) */

#define SCAN_PART 8192   /* entries per block of the long scan */

/* exclusive scan of each SCAN_PART-entry part in place (1024 threads, 8
 * entries each); the part's total into sums */
__global__ void k_scan_part(unsigned *data, int m, unsigned *sums)
{
	__shared__ unsigned part[1024];
	int t = threadIdx.x;
	int b = blockIdx.x * SCAN_PART + t * 8;
	unsigned v[8], sum = 0;
	#pragma unroll
	for(int k = 0; k < 8; k++) {
		v[k] = b + k < m ? data[b + k] : 0u;
		sum += v[k];
	}
	part[t] = sum;
	__syncthreads();
	for(int off = 1; off < 1024; off <<= 1) {
		unsigned u = t >= off ? part[t - off] : 0u;
		__syncthreads();
		part[t] += u;
		__syncthreads();
	}
	unsigned run = part[t] - sum;
	#pragma unroll
	for(int k = 0; k < 8; k++) {
		if(b + k < m) data[b + k] = run;
		run += v[k];
	}
	if(t == 1023) sums[blockIdx.x] = part[1023];
}

__global__ void k_scan_add(unsigned *data, int m, const unsigned *offs)
{
	unsigned o = offs[blockIdx.x];
	int b = blockIdx.x * SCAN_PART;
	for(int i = b + threadIdx.x; i < b + SCAN_PART && i < m; i += blockDim.x) data[i] += o;
}

/* the segment holding compacted index i: the last s with offs[s] <= i */
__device__ __forceinline__ int seg_of(const unsigned *offs, int nseg, unsigned i)
{
	int lo = 0, hi = nseg - 1;
	while(lo < hi) {
		int mid = (lo + hi + 1) >> 1;
		if(offs[mid] <= i) lo = mid;
		else hi = mid - 1;
	}
	return lo;
}

/* compacted index of each segment boundary: the tile's offset plus the
 * stored photons of the tile before it (one block per boundary) */
__global__ void k_seg_offsets(const int *valid, const unsigned *tile_offs, const int *bounds, unsigned *offs)
{
	__shared__ int red[256];
	int b = bounds[blockIdx.x], tile = b / TILE, c = 0;
	for(int i = tile * TILE + threadIdx.x; i < b; i += blockDim.x) c += valid[i];
	red[threadIdx.x] = c;
	__syncthreads();
	for(int off = 128; off > 0; off >>= 1) {
		if(threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
		__syncthreads();
	}
	if(threadIdx.x == 0) offs[blockIdx.x] = tile_offs[tile] + (unsigned)red[0];
}

/* keys of the compacted photons: their cells, each in its segment's grid,
 * the segments' cells one after the other */
__global__ void k_keys_seg(PhotonRuns ph, int n, const DPhotonMap *grids, const unsigned *offs, const unsigned long long *cell_base,
		int nseg, unsigned *keys, unsigned *vals)
{
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
		const int sg = seg_of(offs, nseg, (unsigned)i);
		keys[i] = (unsigned)cell_base[sg] + cell_key(ph.at((unsigned)i), grids[sg], 0);
		vals[i] = (unsigned)i;
	}
}

/* every segment's cell table (block row y: segment y), one after the other
 * in `starts`, or the second in a buffer of its own */
__global__ void __launch_bounds__(256) k_starts_seg(const unsigned *keys, const unsigned *offs, const unsigned long long *cell_base,
		unsigned *starts, unsigned *second)
{
	const int sg = blockIdx.y;
	const size_t ncells = (size_t)(cell_base[sg + 1] - cell_base[sg]) - 1;
	if((size_t)blockIdx.x * START_CELLS > ncells) return;
	cell_starts(keys, offs[sg], offs[sg + 1], (unsigned)cell_base[sg], ncells, second && sg == 1 ? second : starts + cell_base[sg]);
}

/* exclusive scan of m entries (scratch `part` for the parts' totals); the
 * total into *total when given */
static int scan_long(Renderer &R, unsigned *data, int m, unsigned *total, DevBuf &part, const char *name, cudaStream_t s)
{
	if(m <= 65536) {
		LAUNCH(R, name, s, k_scan_excl<<<1, 1024, 0, s>>>(data, m, total));
		return 0;
	}
	int parts = (m + SCAN_PART - 1) / SCAN_PART;
	PCK(part.ensure((size_t)(parts + 4) * sizeof(unsigned)), "scan parts");
	unsigned *sums = part.as<unsigned>();
	LAUNCH(R, name, s, k_scan_part<<<parts, 1024, 0, s>>>(data, m, sums));
	LAUNCH(R, name, s, k_scan_excl<<<1, 1024, 0, s>>>(sums, parts, total));
	LAUNCH(R, name, s, k_scan_add<<<parts, 256, 0, s>>>(data, m, sums));
	return 0;
}

/* stable LSD radix sort of n (key, value) pairs over the low `bits` bits of
 * the keys, ping-ponging with keys2 / vals2; *keys_out and *vals_out are the
 * buffers that hold the sorted pairs (scratch: hist, part) */
int sort_pairs(Renderer &R, unsigned *keys, unsigned *vals, unsigned *keys2, unsigned *vals2, int n, int bits, DevBuf &hist,
		DevBuf &part, const char *name, cudaStream_t s, unsigned **keys_out, unsigned **vals_out)
{
	int nbr = (n + TILE - 1) / TILE;
	PCK(hist.ensure((size_t)256 * nbr * sizeof(unsigned) + 16), "radix histogram");
	unsigned *h = hist.as<unsigned>();
	for(int shift = 0; shift < bits; shift += 8) {
		LAUNCH(R, name, s, k_rs_hist<<<nbr, RS_THREADS, 0, s>>>(keys, n, shift, h, nbr));
		if(scan_long(R, h, 256 * nbr, nullptr, part, name, s)) return SRAY_ECUDA;
		LAUNCH(R, name, s, k_rs_scatter<<<nbr, RS_THREADS, 0, s>>>(keys, vals, n, shift, h, nbr, keys2, vals2));
		std::swap(keys, keys2);
		std::swap(vals, vals2);
	}
	*keys_out = keys;
	*vals_out = vals;
	return 0;
}

/* every job's two maps from the wavefront's output: maps[2j] caustic,
 * maps[2j + 1] global, over the boxes and range radii of the jobs' own
 * frames.  All photons are sorted at once, by their cells with the maps'
 * cells one after the other.  Returns 1 (no map built) when the maps' cell
 * tables together would pass 2^28 cells, for the map-by-map build to take
 * over.  own (one job): into the renderer's own two maps, which outlive the
 * next wavefront, rather than the wavefront's buffers: a frame's two maps of
 * 100,000 emitted photons together, 321x181 frames 1310 us one map after the
 * other (230 us of it in 24 short launches and 3 waits), 1220 together. */
int photon_finalize_jobs(Renderer &R, const std::vector<PJobOut> &jobs, const std::vector<Box> &boxes,
		const std::vector<double> &gather_dist, std::vector<DPhotonMap> &maps, cudaStream_t s, bool own)
{
	const sray_opts &opt = R.opt;
	int nj = (int)jobs.size(), nseg = 2 * nj;
	maps.assign(nseg, DPhotonMap());
	const PJobOut &last = jobs[nj - 1];
	int total = last.base + last.total[0] + last.total[1];
	if(total == 0) return 0;
	const int *valid = R.pw_valid.as<int>();
	int nb = (total + TILE - 1) / TILE;
	PCK(R.pw_tiles.ensure((size_t)(nb + 4) * sizeof(unsigned)), "scan");
	unsigned *bc = R.pw_tiles.as<unsigned>();
	LAUNCH(R, "photon_compact", s, k_count_valid<<<nb, 256, 0, s>>>(valid, total, bc));
	if(scan_long(R, bc, nb, bc + nb, R.pw_part, "photon_compact", s)) return SRAY_ECUDA;
	std::vector<int> bounds(nseg + 1);
	for(int j = 0; j < nj; j++) {
		bounds[2 * j] = jobs[j].base;
		bounds[2 * j + 1] = jobs[j].base + jobs[j].total[0];
	}
	bounds[nseg] = total;
	PCK(R.pw_bounds.upload(bounds, s), "segment bounds");
	PCK(R.pw_offs.ensure((size_t)(nseg + 1) * sizeof(unsigned)), "segment offsets");
	unsigned *offs = R.pw_offs.as<unsigned>();
	LAUNCH(R, "photon_compact", s, k_seg_offsets<<<nseg + 1, 256, 0, s>>>(valid, bc, R.pw_bounds.as<int>(), offs));
	std::vector<unsigned> h_offs(nseg + 1);
	PCK(cudaMemcpyAsync(h_offs.data(), offs, (nseg + 1) * sizeof(unsigned), cudaMemcpyDeviceToHost, s), "segment offsets");
	PCK(cudaStreamSynchronize(s), "photon compaction");
	R.d2h += (int64_t)(nseg + 1) * sizeof(unsigned);
	R.h2d += (int64_t)bounds.size() * sizeof(int);
	R.prof_collect();
	int n = (int)h_offs[nseg];
	/* a table per map: its cells and one entry more */
	std::vector<unsigned long long> cell_base(nseg + 1, 0);
	unsigned long long most_cells = 0;
	for(int sg = 0; sg < nseg; sg++) {
		int k = (sg & 1) ? opt.gi_k : opt.caust_k;
		double rad = k > 0 ? (double)opt.gather_rcap : gather_dist[sg >> 1];
		unsigned long long nc = map_grid(k, rad, boxes[sg >> 1], (int)(h_offs[sg + 1] - h_offs[sg]), maps[sg]);
		cell_base[sg + 1] = cell_base[sg] + nc + 1;
		most_cells = std::max(most_cells, nc);
	}
	if(cell_base[nseg] > (1ull << 28)) return 1;
	if(n == 0) return 0;
	PhotonRuns given, sorted;
	unsigned *starts = nullptr, *second = nullptr;
	if(own) {
		PhotonBufs *P[2] = {&R.caust, &R.gi};
		for(int g = 0; g < 2; g++) {
			double rad = (g ? opt.gi_k : opt.caust_k) > 0 ? (double)opt.gather_rcap : gather_dist[0];
			map_cells(rad > 0.0 ? 2.0 * rad : 1.0, boxes[0], P[g]->order);
			PCK(P[g]->tmp_ph.ensure((size_t)maps[g].n * sizeof(DevPhoton)), "photon buffer");
			PCK(P[g]->ph.ensure((size_t)maps[g].n * sizeof(DevPhoton)), "photon map");
			PCK(P[g]->starts.ensure((size_t)(cell_base[g + 1] - cell_base[g]) * sizeof(unsigned)), "cell table");
		}
		given = PhotonRuns{P[0]->tmp_ph.as<DevPhoton>(), P[1]->tmp_ph.as<DevPhoton>(), h_offs[1]};
		sorted = PhotonRuns{P[0]->ph.as<DevPhoton>(), P[1]->ph.as<DevPhoton>(), h_offs[1]};
		starts = P[0]->starts.as<unsigned>();
		second = P[1]->starts.as<unsigned>();
	} else {
		PCK(R.pw_ph.ensure((size_t)n * sizeof(DevPhoton)), "photon maps");
		PCK(R.pw_sorted.ensure((size_t)n * sizeof(DevPhoton)), "photon maps");
		PCK(R.pw_starts.ensure((size_t)cell_base[nseg] * sizeof(unsigned)), "cell tables");
		given = one_run(R.pw_ph.as<DevPhoton>());
		sorted = one_run(R.pw_sorted.as<DevPhoton>());
		starts = R.pw_starts.as<unsigned>();
	}
	PCK(R.pw_keys.ensure((size_t)n * 16), "keys");
	LAUNCH(R, "photon_compact", s, k_compact<<<nb, 256, 0, s>>>(valid, R.pw_out.as<DevPhoton>(), total, bc, given));
	PCK(R.pw_grids.upload(maps, s), "map grids");
	PCK(R.pw_cellbase.upload(cell_base, s), "cell tables");
	R.h2d += (int64_t)(maps.size() * sizeof(DPhotonMap) + cell_base.size() * 8);
	unsigned *keys = R.pw_keys.as<unsigned>(), *vals = keys + n, *keys2 = keys + 2 * (size_t)n, *vals2 = keys + 3 * (size_t)n;
	const unsigned long long *base = R.pw_cellbase.as<unsigned long long>();
	LAUNCH(R, "photon_sort", s, k_keys_seg<<<grid_n(n, 256), 256, 0, s>>>(given, n, R.pw_grids.as<DPhotonMap>(), offs, base, nseg, keys,
			vals));
	if(int r = sort_pairs(R, keys, vals, keys2, vals2, n, key_bits((unsigned)(cell_base[nseg] - 1)), R.pw_hist, R.pw_part, "photon_sort", s,
			&keys, &vals))
		return r;
	LAUNCH(R, "photon_sort", s, k_permute<<<grid_n(n, 256), 256, 0, s>>>(given, vals, n, sorted));
	LAUNCH(R, "photon_sort", s, k_starts_seg<<<dim3((unsigned)((most_cells + START_CELLS) / START_CELLS), nseg), 256, 0, s>>>(keys, offs,
			base, starts, second));
	if(own) {
		PhotonBufs *P[2] = {&R.caust, &R.gi};
		for(int g = 0; g < 2; g++) {
			if(maps[g].n == 0) continue;
			maps[g].ph = P[g]->ph.as<DevPhoton>();
			maps[g].start = P[g]->starts.as<unsigned>();
			P[g]->map = maps[g];
		}
	} else {
		for(int sg = 0; sg < nseg; sg++) {
			maps[sg].ph = R.pw_sorted.as<DevPhoton>() + h_offs[sg];
			maps[sg].start = R.pw_starts.as<unsigned>() + cell_base[sg];
		}
	}
	PCK(cudaStreamSynchronize(s), "photon map build");
	R.prof_collect();
	return 0;
}

/* map `global` from host photons (a restored dump) */
int photon_map_restore(Renderer &R, int global, const std::vector<DevPhoton> &h, cudaStream_t s)
{
	PhotonBufs &P = global ? R.gi : R.caust;
	int n = (int)h.size();
	P.map.n = 0;
	if(n == 0) return 0;
	PCK(P.ph.ensure((size_t)n * sizeof(DevPhoton)), "photon map");
	PCK(P.tmp_ph.ensure((size_t)n * sizeof(DevPhoton)), "photon buffer");
	PCK(cudaMemcpyAsync(P.ph.p, h.data(), (size_t)n * sizeof(DevPhoton), cudaMemcpyHostToDevice, s), "upload photons");
	R.h2d += (int64_t)n * sizeof(DevPhoton);
	return photon_map_build(R, global, n, s);
}

}  // namespace sray
