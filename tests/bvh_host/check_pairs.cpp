/*
 * check_pairs.cpp - host check of the pairs of triangles that join_pairs
 * (bvh.cpp) makes of a tree with leaves of one: read triangles from stdin ("n",
 * then 9 coordinates each) and rays ("m", then origin and direction each), cast
 * every ray and `extra` seeded ones, aimed from above random triangles at points
 * within 1e-5 of corners of others and at points of edges, with the traversal of
 * kernels_device.cuh in FP32, and compare triangle and distance of the closest
 * and of the first hit. Prints the rays, those that hit, and those whose hit
 * would differ if a triangle of a pair did not need its own box.
 */
#include "bvh.h"
#include "device_scene.h"

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <iostream>
#include <random>
#include <vector>

using namespace ssolb;

namespace {

struct Tri { float v[3][3]; };
struct Hit { float t; int tri; };

bool slab(const float* lo, const float* hi, const float* inv, const float* oinv, float tmax,
          float& t0)
{
  float t1 = tmax;
  t0 = 0.f;
  for(int c = 0; c < 3; ++c) {
    const float a = std::fma(lo[c], inv[c], -oinv[c]), b = std::fma(hi[c], inv[c], -oinv[c]);
    t0 = std::fmax(t0, std::fmin(a, b));
    t1 = std::fmin(t1, std::fmax(a, b));
  }
  return t0 <= t1;
}

void test(const std::vector<Tri>& tris, int i, const float* o, const float* d, const float* inv,
          const float* oinv, bool own, float tleaf, Hit& best)
{
  const Tri& T = tris[(size_t)i];
  double a[3][3];
  for(int k = 0; k < 3; ++k)
    for(int c = 0; c < 3; ++c) a[k][c] = (double)T.v[k][c] - o[c];
  /* sides of the ray's line: products of its direction with the edges */
  double s[3];
  for(int k = 0; k < 3; ++k) {
    const double *p = a[(k + 1) % 3], *q = a[(k + 2) % 3];
    s[k] = d[0] * (p[1] * q[2] - p[2] * q[1]) + d[1] * (p[2] * q[0] - p[0] * q[2])
         + d[2] * (p[0] * q[1] - p[1] * q[0]);
  }
  if((s[0] < 0 || s[1] < 0 || s[2] < 0) && (s[0] > 0 || s[1] > 0 || s[2] > 0)) return;
  double n[3], num = 0, den = 0;
  for(int c = 0; c < 3; ++c) {
    const int x = (c + 1) % 3, y = (c + 2) % 3;
    n[c] = (a[1][x] - a[0][x]) * (a[2][y] - a[0][y]) - (a[1][y] - a[0][y]) * (a[2][x] - a[0][x]);
    num += n[c] * a[0][c];
    den += n[c] * d[c];
  }
  const float t = (float)(num / den);
  if(!(t < best.t) || t <= 1e-4f) return;
  if(own) {
    float lo[3], hi[3], te;
    for(int c = 0; c < 3; ++c) {
      lo[c] = std::fmin(T.v[0][c], std::fmin(T.v[1][c], T.v[2][c]));
      hi[c] = std::fmax(T.v[0][c], std::fmax(T.v[1][c], T.v[2][c]));
    }
    if(!slab(lo, hi, inv, oinv, tleaf, te)) return;
  }
  best = {t, i};
}

Hit cast(const std::vector<DNode<float>>& nodes, const std::vector<uint32_t>& refs,
         const std::vector<Tri>& tris, const float* o, const float* d, bool any, bool own)
{
  float inv[3], oinv[3];
  for(int c = 0; c < 3; ++c) { inv[c] = 1.f / d[c]; oinv[c] = o[c] * inv[c]; }
  Hit best = {3.4e38f, -1};
  int stack[32], sp = 0, node = 0;
  while(node >= 0) {
    if(node & PAIR_LEAF) {
      const size_t first = (size_t)(node ^ PAIR_LEAF);
      const float tleaf = best.t;
      node = sp ? stack[--sp] : -1;
      for(size_t p = 0; p < 2; ++p) {
        test(tris, (int)primref_index(refs[first + p]), o, d, inv, oinv, own, tleaf, best);
        if(any && best.tri >= 0) return best;
      }
      continue;
    }
    const DNode<float>& N = nodes[(size_t)node];
    float te[2];
    bool h[2];
    for(int k = 0; k < 2; ++k)
      h[k] = slab(N.lo[k], N.hi[k], inv, oinv, best.t, te[k]) && N.count[k] >= 0;
    const bool in0 = h[0] && N.count[0] == 0, in1 = h[1] && N.count[1] == 0;
    if(in0 && in1) {
      const bool first0 = te[0] <= te[1];
      stack[sp++] = N.child[first0 ? 1 : 0];
      node = N.child[first0 ? 0 : 1];
    } else if(in0 || in1) {
      node = N.child[in0 ? 0 : 1];
    } else {
      node = sp ? stack[--sp] : -1;
    }
    for(int k = 0; k < 2; ++k)
      if(h[k] && N.count[k] > 0) {
        test(tris, (int)primref_index((uint32_t)N.child[k]), o, d, inv, oinv, false, 0.f, best);
        if(any && best.tri >= 0) return best;
      }
  }
  return best;
}

} /* namespace */

int main(int argc, char** argv)
{
  const long extra = argc > 1 ? std::atol(argv[1]) : 0;
  size_t n = 0, m = 0;
  std::cin >> n;
  std::vector<Tri> tris(n);
  std::vector<PrimBox> boxes(n);
  for(size_t i = 0; i < n; ++i) {
    double x;
    for(auto& v : tris[i].v)
      for(float& c : v) { std::cin >> x; c = (float)x; }
    for(int c = 0; c < 3; ++c) {
      boxes[i].lo[c] = std::fmin(tris[i].v[0][c], std::fmin(tris[i].v[1][c], tris[i].v[2][c]));
      boxes[i].hi[c] = std::fmax(tris[i].v[0][c], std::fmax(tris[i].v[1][c], tris[i].v[2][c]));
    }
    boxes[i].ref = primref_make(PRIM_TRIANGLE, (uint32_t)i);
  }
  std::cin >> m;
  std::vector<float> rays(6 * m);
  for(float& c : rays) { double x; std::cin >> x; c = (float)x; }

  BvhBuildParams prm;
  prm.max_leaf = 1;
  BvhResult r;
  build_bvh(boxes, prm, r);
  const std::vector<DNode<float>> one = bvh_nodes<float>(r);
  std::vector<DNode<float>> pairs = one;
  std::vector<uint32_t> refs = r.primrefs;
  join_pairs(pairs, refs);

  /* Every triangle once, and no node but the root that should be a pair */
  std::vector<int> seen(n, 0);
  for(size_t i = 0; i < pairs.size(); ++i) {
    const DNode<float>& N = pairs[i];
    if(i && N.count[0] == 1 && N.count[1] == 1) { std::printf("node of two left\n"); return 1; }
    for(int k = 0; k < 2; ++k) {
      if(N.count[k] == 1) ++seen.at(primref_index((uint32_t)N.child[k]));
      if(N.count[k] == 0 && (N.child[k] & PAIR_LEAF))
        for(int p = 0; p < 2; ++p)
          ++seen.at(primref_index(refs.at((size_t)(N.child[k] ^ PAIR_LEAF) + p)));
    }
  }
  for(size_t i = 0; i < n; ++i)
    if(seen[i] != 1) { std::printf("triangle %zu in %d leaves\n", i, seen[i]); return 1; }

  std::mt19937 gen(7);
  std::uniform_real_distribution<double> u(0.0, 1.0);
  long hits = 0, boxed = 0;
  for(long k = 0; k < (long)m + extra; ++k) {
    float o[3], d[3];
    if(k < (long)m) {
      for(int c = 0; c < 3; ++c) { o[c] = rays[6 * k + c]; d[c] = rays[6 * k + 3 + c]; }
    } else {
      const Tri &A = tris[gen() % n], &B = tris[gen() % n];
      const int v = (int)(gen() % 3);
      const double w = k & 1 ? u(gen) : 0.0, off = k & 1 ? 0.0 : 1e-5;
      double l = 0, e[3];
      for(int c = 0; c < 3; ++c) {
        o[c] = (float)((A.v[0][c] + A.v[1][c] + A.v[2][c]) / 3 + (c == 2 ? 1e-2 : 0));
        e[c] = B.v[v][c] + w * ((double)B.v[(v + 1) % 3][c] - B.v[v][c])
             + off * (2 * u(gen) - 1) - o[c];
        l += e[c] * e[c];
      }
      for(int c = 0; c < 3; ++c) d[c] = (float)(e[c] / std::sqrt(l));
    }
    for(int any = 0; any < 2; ++any) {
      const Hit a = cast(one, r.primrefs, tris, o, d, any, false);
      const Hit b = cast(pairs, refs, tris, o, d, any, true);
      if(a.tri != b.tri || a.t != b.t) {
        std::printf("ray %ld (any %d): triangle %d at %.9g, with pairs %d at %.9g\n", k, any, a.tri,
                    a.t, b.tri, b.t);
        return 1;
      }
      if(any) continue;
      hits += a.tri >= 0;
      const Hit f = cast(pairs, refs, tris, o, d, false, false);
      boxed += a.tri != f.tri || a.t != f.t;
    }
  }
  std::printf("ok %ld %ld %ld\n", (long)m + extra, hits, boxed);
  return 0;
}
