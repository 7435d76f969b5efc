// The FP32 triangle test of the contact search (csrc/xd_triangle.cuh) on the
// host: contacts that it would lose, over triangles of every length and width
// with the short edge at each vertex in turn, and of every kind of touch.
//   triangle_near <samples of each kind> <largest coordinate, m>
// prints "<contacts> <lost> <spheres clear of an ordinary triangle> <of those called near>".
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "xd_triangle.cuh"

struct V {
    double x, y, z;
};
static V operator-(V a, V b) { return { a.x - b.x, a.y - b.y, a.z - b.z }; }
static V operator+(V a, V b) { return { a.x + b.x, a.y + b.y, a.z + b.z }; }
static V operator*(double s, V a) { return { s * a.x, s * a.y, s * a.z }; }
static double dot(V a, V b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
static V cross(V a, V b) { return { a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x }; }
static double length(V a) { return std::sqrt(dot(a, a)); }

// FP64 rounded towards zero, as the search cuts its coordinates.
static float cut(double x)
{
    const float f = (float)x;
    return std::fabs((double)f) > std::fabs(x) ? std::nextafter(f, 0.f) : f;
}

// The distance in long double, from the face if the foot lies in it and the edges.
using LD = long double;
static double distance(V a, V b, V c, V p)
{
    const LD E[3][2][3] = { { { a.x, a.y, a.z }, { b.x, b.y, b.z } },
                            { { b.x, b.y, b.z }, { c.x, c.y, c.z } },
                            { { c.x, c.y, c.z }, { a.x, a.y, a.z } } };
    const LD q[3] = { p.x, p.y, p.z };
    LD best = INFINITY, n[3], u[3], v[3];
    for (auto& e : E) {
        LD ee = 0, ed = 0, d2 = 0;
        for (int k = 0; k < 3; ++k) ee += (e[1][k] - e[0][k]) * (e[1][k] - e[0][k]);
        for (int k = 0; k < 3; ++k) ed += (e[1][k] - e[0][k]) * (q[k] - e[0][k]);
        const LD t = ee > 0 ? std::min((LD)1, std::max((LD)0, ed / ee)) : 0;
        for (int k = 0; k < 3; ++k) {
            const LD d = q[k] - e[0][k] - t * (e[1][k] - e[0][k]);
            d2 += d * d;
        }
        best = std::min(best, std::sqrt(d2));
    }
    for (int k = 0; k < 3; ++k) u[k] = E[0][1][k] - E[0][0][k], v[k] = E[2][0][k] - E[0][0][k];
    for (int k = 0; k < 3; ++k) n[k] = u[(k + 1) % 3] * v[(k + 2) % 3] - u[(k + 2) % 3] * v[(k + 1) % 3];
    const LD nn = n[0] * n[0] + n[1] * n[1] + n[2] * n[2];
    bool inside = nn > 0;
    for (auto& e : E) {   // on the inner side of every edge
        LD s = 0;
        for (int k = 0; k < 3; ++k) {
            const int a1 = (k + 1) % 3, a2 = (k + 2) % 3;
            s += n[k] * ((e[1][a1] - e[0][a1]) * (q[a2] - e[0][a2]) - (e[1][a2] - e[0][a2]) * (q[a1] - e[0][a1]));
        }
        inside &= s >= 0;
    }
    if (inside) {
        LD h = 0;
        for (int k = 0; k < 3; ++k) h += n[k] * (q[k] - E[0][0][k]);
        best = std::min(best, std::fabs(h) / std::sqrt(nn));
    }
    return (double)best;
}

int main(int argc, char** argv)
{
    const long each = argc > 1 ? std::atol(argv[1]) : 2000;
    const double off = argc > 2 ? std::atof(argv[2]) : 0.3;
    std::mt19937_64 g(7);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    std::normal_distribution<double> G;
    auto dir = [&] {
        const V a{ G(g), G(g), G(g) };
        return (1 / length(a)) * a;
    };
    long contacts = 0, lost = 0, clear = 0, called = 0;
    for (double r : { 3e-5, 3e-3, 0.1 })
        for (double L : { 1e-5, 1e-3, 1e-2, 0.1, 0.3, 1.0, 3.0 })
            for (double w : { 1e-10, 1e-8, 1e-7, 1e-6, 3e-6, 1e-5, 3e-5, 1e-4, 3e-4, 1e-3, 1e-2, 0.1, 1.0 }) {
                if (w > L) continue;
                for (int kind = 0; kind < 4; ++kind)   // the short edge's place, or none (the third vertex over the edge)
                    for (long i = 0; i < each; ++i) {
                        const V e = dir();
                        V f = dir();
                        f = f - dot(f, e) * e;
                        f = (1 / length(f)) * f;
                        const V o = off * U(g) * dir();
                        const double a = kind == 3 ? (0.05 + 0.9 * U(g)) * L : (U(g) - 0.5) * 2 * w;
                        const V T[3] = { o, o + a * e + w * f, o + L * e };
                        V P = T[kind % 3], Q = T[(kind + 1) % 3], R = T[(kind + 2) % 3];
                        if (U(g) < 0.5) std::swap(Q, R);
                        double b1 = U(g), b2 = U(g);   // a point of the face or of an edge
                        if (b1 + b2 > 1) b1 = 1 - b1, b2 = 1 - b2;
                        if (i % 4 == 1) b1 = 0;
                        if (i % 4 == 2) b2 = 0;
                        if (i % 4 == 3) b2 = 1 - b1;
                        const V q = P + b1 * (Q - P) + b2 * (R - P), n = cross(Q - P, R - P);
                        const V d = i % 3 || !(length(n) > 0) ? dir() : (U(g) < 0.5 ? 1.0 : -1.0) / length(n) * n;
                        const V s = q + r * (i % 8 == 7 ? 1.3 + U(g) : 1.0 - 0.01 * U(g) * U(g)) * d;
                        const double dist = distance(P, Q, R, s);
                        const float px = cut(s.x), py = cut(s.y), pz = cut(s.z);
                        const bool near = xd::tri_near(px, py, pz, cut(r), std::fabs(px) + std::fabs(py) + std::fabs(pz),
                                                       cut(P.x), cut(P.y), cut(P.z), cut(Q.x), cut(Q.y), cut(Q.z),
                                                       cut(R.x), cut(R.y), cut(R.z));
                        if (dist < r) {
                            ++contacts;
                            lost += !near;
                        } else if (dist > 1.3 * r && w > 0.2 * L && L < 30 * r && L > r && off <= 1.0 && r > 1e-3) {
                            ++clear;
                            called += near;
                        }
                    }
            }
    std::printf("%ld %ld %ld %ld\n", contacts, lost, clear, called);
}
