/* An object's reach (HostScene::object_reach) on the host, built and run by
 * tests/test_reach_box.py: every point of a sphere or mesh at every time of
 * the frame's table lies in it, a still object's box is no larger than its
 * points (to 1e-3 of its size), and cylinders and objects whose extent over
 * time is not known have none.
 * Usage: reach_check <scene xml> <t0> <t1> <shutter> */
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <string>
#include <vector>
#include "scene_host.h"

using namespace sray;

int main(int argc, char **argv)
{
	if(argc < 5) return 2;
	FILE *f = fopen(argv[1], "rb");
	if(!f) return 2;
	std::string text;
	char buf[1 << 16];
	size_t n;
	while((n = fread(buf, 1, sizeof buf, f)) > 0) text.append(buf, n);
	fclose(f);
	sray_opts o;
	memset(&o, 0, sizeof o);
	o.meshoct_max_depth = 8; o.meshoct_max_items = 8; o.scnoct_max_depth = 8; o.scnoct_max_items = 8;
	HostScene sc;
	std::string err;
	if(!sc.load(text.c_str(), text.size(), o, err)) { printf("load: %s\n", err.c_str()); return 1; }
	const int t0 = atoi(argv[2]), t1 = atoi(argv[3]), sh = atoi(argv[4]), tlo = t0 - sh - 2, thi = t1 + sh + 2;
	sc.build_tree(t0, t1, o);
	int bad = 0, known = 0, still = 0;
	for(size_t i = 0; i < sc.objs.size(); i++) {
		const Object &ob = sc.objs[i];
		Box b;
		const bool have = sc.object_reach(i, tlo, thi, b);
		const bool turns = ob.xf.rot.time.size() > 1 || ob.xf.scale.time.size() > 1 || ob.xf.pos.interp == INTERP_CUBIC;
		if(have != (ob.type != OBJ_CYLINDER && !turns)) { printf("object %zu: reach %d\n", i, have); bad++; }
		if(!have) continue;
		known++;
		still += ob.is_static;
		for(int t = tlo; t <= thi; t++) {
			double m[4][4], mn[3] = {1e30, 1e30, 1e30}, mx[3] = {-1e30, -1e30, -1e30};
			ob.xf.matrix(t, m);
			std::vector<Vec3> pts;
			if(ob.type == OBJ_SPHERE) {
				for(int u = 0; u <= 60; u++) for(int v = 0; v < 120; v++)
					pts.push_back(Vec3(ob.rad * sin(u * M_PI / 60) * cos(v * M_PI / 60), ob.rad * cos(u * M_PI / 60), ob.rad * sin(u * M_PI / 60) * sin(v * M_PI / 60)));
			} else {
				const std::vector<double> &p = sc.meshes[ob.mesh].posd;
				for(size_t k = 0; k + 2 < p.size(); k += 3) pts.push_back(Vec3(p[k], p[k + 1], p[k + 2]));
			}
			for(const Vec3 &p : pts) {
				for(int a = 0; a < 3; a++) {
					double w = m[a][0] * p.x + m[a][1] * p.y + m[a][2] * p.z + m[a][3];
					mn[a] = std::min(mn[a], w);
					mx[a] = std::max(mx[a], w);
				}
			}
			for(int a = 0; a < 3; a++) {
				if(mn[a] < b.mn[a] || mx[a] > b.mx[a]) { printf("object %zu at %d: [%g, %g] outside [%g, %g]\n", i, t, mn[a], mx[a], b.mn[a], b.mx[a]); bad++; }
				const double slack = ob.is_static ? (mx[a] - mn[a]) * 2e-3 + 2.0 * std::max(fabs(b.mn[a]), fabs(b.mx[a])) * 2e-4 : 1e30;
				if(b.mn[a] < mn[a] - slack || b.mx[a] > mx[a] + slack) { printf("object %zu: [%g, %g] far beyond [%g, %g]\n", i, b.mn[a], b.mx[a], mn[a], mx[a]); bad++; }
			}
		}
	}
	printf("%d known, %d of them still, %d bad\n", known, still, bad);
	return bad || !known || !still || known == still ? 1 : 0;
}
