// cell_box.cuh - which edges may cross an arc inside a lattice cell.
//
// A leaf answers a query by the edges that cross arc(R, q), R the cell's
// center and q a point of the cell, so an edge belongs in a cell's list when
// it may meet the geodesic convex hull of the cell (with the locate margin).
// The gnomonic projection at a cell's center maps great-circle arcs to
// straight segments, so the hull's bounding rectangle in that plane is convex
// on the sphere too, and "does the edge meet it" is a segment-rectangle test
// in the plane: two projections, a bounding-interval test and one cross
// product.  The rectangle hugs the cell, where the cap around it (the test
// used before, and still for cells too wide for the plane) has five times
// the cell's area: on a 1.1M-edge polygon the leaves hold fewer edges and the
// index fewer leaves (the figures are beside the build's pair kernels).
//
// Why lists need no nesting of the rectangles: a child's cell lies in its
// parent's cell, so the child's hull lies in the parent's hull, and an edge
// that meets the child's hull meets the parent's and passes the parent's
// (conservative) test.  By induction a child's list, filtered from its
// parent's, holds every edge that meets the child's hull.
//
// Host and device; no fused multiply-add (the sources build without
// contraction), so the host tests run the device's arithmetic.
#pragma once

#include <math.h>

#include "gahhg_canon.h"
#include "geom.cuh"

namespace gahhg {
namespace cellbox {

// Added to every side of a rectangle (radians): the margin between where the
// index arithmetic places a query and where its canonical XYZ lies (2e-8,
// LOC_MARGIN), times the plane's stretch inside a cell (1 / cos^2(MAX_REACH) <
// 1.07), and the rounding of the projections.
constexpr double MARGIN = 3.0e-8;
// Cells whose corners are at most this far from the center (radians) and at
// most MAX_HALF_WIDE wide in longitude on each side use the rectangle: then
// every point of the cell projects with R.q > 0.96 and the coordinates are
// monotone along the cell's sides (see corner()).
constexpr double MAX_REACH = 0.25;
constexpr double MAX_HALF_WIDE = 0.2;
// An edge end with X.R below this (more than 60 degrees from the center) is
// not projected; the caller falls back to the cap test.
constexpr double MIN_DOT = 0.5;
// Bound on a projected coordinate's absolute error, per unit of the
// magnitudes beside it: the dot products of unit vectors carry about 3e-16,
// the division by X.R >= 0.5 doubles it, the frame's canonical sine and
// cosine (1 ulp) and the canonical R's rounding add as much again, about
// 2e-15 for coordinates up to 1.8; five times that.
constexpr double ERR = 1.0e-14;

// The tangent frame of a center: canonical sine and cosine of its latitude
// and longitude; R = (ca so, sa, ca co) is the canonical XYZ bit for bit,
// e1 = (co, 0, -so) points east, e2 = (-sa so, ca, -sa co) north.
struct Frame {
    double sa, ca, so, co;
};

GHD Frame frame_at(double lonc, double latc)
{
    Frame f;
    gahhg_canon_sincos(gahhg_canon_rad(latc), &f.sa, &f.ca);
    gahhg_canon_sincos(gahhg_canon_rad(lonc), &f.so, &f.co);
    return f;
}

GHD D3 center_of(const Frame& f) { return d3(f.ca * f.so, f.sa, f.ca * f.co); }

// Gnomonic coordinates of A; false when A is too far from the center.
GHD bool project(const Frame& f, const D3& A, double& x, double& y)
{
    const double t = A.x * f.so + A.z * f.co;
    const double w = f.ca * t + f.sa * A.y;
    if (!(w >= MIN_DOT)) return false;
    const double i = 1.0 / w;
    x = (A.x * f.co - A.z * f.so) * i;
    y = (f.ca * A.y - f.sa * t) * i;
    return true;
}

// Gnomonic coordinates of the point at angle differences (dl, dp) from the
// center (bounds only: sin and cos of the platform).  For |dl| up to
// MAX_HALF_WIDE and points within MAX_REACH, x grows with dl along a
// parallel, y moves one way with |dl| there (dy/dl has the sign of
// dl sin(phi)), and along a meridian both are monotone (it is a straight
// line), so a rectangle over corners and, where dl = 0 lies between them, the
// middles of the parallels, covers the cell; a rectangle covers the hull of
// what it covers.
GHD void corner_at(double sa, double ca, double sl, double h, double sp, double cp, double& x, double& y)
{
    const double cphi = ca * cp - sa * sp;
    const double v = 2.0 * h * h;  // 1 - cos dl
    const double i = 1.0 / (cp - ca * cphi * v);
    x = cphi * sl * i;
    y = (sp + sa * cphi * v) * i;
}

GHD void corner(double sa, double ca, double dl, double dp, double& x, double& y)
{
    corner_at(sa, ca, sin(dl), sin(0.5 * dl), sin(dp), cos(dp), x, y);
}

// A rectangle [x0, x1] x [y0, y1] in the plane.
struct Box {
    double x0, x1, y0, y1;
};

// Whether cells of half sizes hl x hp (radians of longitude, latitude; cosine
// of latitude at most cmax) use rectangles.
GHD bool use_box(double hl, double hp, double cmax)
{
    return hl <= MAX_HALF_WIDE && hp + hl * cmax <= MAX_REACH;
}

// The cell around its own center.
GHD Box own_box(double sa, double ca, double hl, double hp)
{
    double xa, ya, xb, yb, xm, ym, xn, yn;
    corner(sa, ca, hl, hp, xa, ya);
    corner(sa, ca, hl, -hp, xb, yb);
    corner(sa, ca, 0.0, hp, xm, ym);
    corner(sa, ca, 0.0, -hp, xn, yn);
    Box b;
    b.x1 = fmax(fabs(xa), fabs(xb)) + MARGIN;
    b.x0 = -b.x1;
    b.y1 = fmax(fmax(ya, ym), fmax(yb, yn)) + MARGIN;
    b.y0 = fmin(fmin(ya, ym), fmin(yb, yn)) - MARGIN;
    return b;
}

// The rectangle over four corners of a cell on one side of the center in
// longitude (a child of the 4 x 4 split never straddles its parent's center).
GHD Box corners_box(double xa, double ya, double xb, double yb, double xc, double yc, double xd, double yd)
{
    Box b;
    b.x0 = fmin(fmin(xa, xb), fmin(xc, xd)) - MARGIN;
    b.x1 = fmax(fmax(xa, xb), fmax(xc, xd)) + MARGIN;
    b.y0 = fmin(fmin(ya, yb), fmin(yc, yd)) - MARGIN;
    b.y1 = fmax(fmax(ya, yb), fmax(yc, yd)) + MARGIN;
    return b;
}

// A projected edge, with what its tests share.
struct alignas(16) Segment {
    double ax, ay, bx, by;  // the ends
    double x0, x1, y0, y1;  // around them
    double dx, dy;          // b - a
    double c1;              // side of the center
    double n;               // magnitudes |a| + |b| + |d|
};

GHD Segment segment(double ax, double ay, double bx, double by)
{
    Segment s;
    s.ax = ax;
    s.ay = ay;
    s.bx = bx;
    s.by = by;
    s.x0 = fmin(ax, bx);
    s.x1 = fmax(ax, bx);
    s.y0 = fmin(ay, by);
    s.y1 = fmax(ay, by);
    s.dx = bx - ax;
    s.dy = by - ay;
    s.c1 = ax * s.dy - ay * s.dx;
    s.n = fabs(ax) + fabs(ay) + fabs(bx) + fabs(by) + fabs(s.dx) + fabs(s.dy);
    return s;
}

// May the segment meet the rectangle?  Never false for one that does.
GHD bool meets(const Segment& s, const Box& b)
{
    if (s.x1 < b.x0 || s.x0 > b.x1 || s.y1 < b.y0 || s.y0 > b.y1) return false;
    const double cx = 0.5 * (b.x0 + b.x1), cy = 0.5 * (b.y0 + b.y1);
    const double ux = s.ax - cx, uy = s.ay - cy;
    const double side = fabs(ux * s.dy - uy * s.dx);
    const double reach = (b.x1 - cx) * fabs(s.dy) + (b.y1 - cy) * fabs(s.dx);
    return side <= reach + ERR * (s.n + fabs(ux) + fabs(uy));
}

GHD bool meets(double ax, double ay, double bx, double by, const Box& b) { return meets(segment(ax, ay, bx, by), b); }

// Does the segment cross the one from the origin (the center) to q?  1 or 0
// when the signs of the four orientations are certain, -1 otherwise.  One
// bound serves all four (the largest of theirs).
GHD int crosses_from_center(const Segment& s, double qx, double qy)
{
    const double e = ERR * (s.n + (fabs(qx) + fabs(qy)));
    const double c2 = s.c1 + (s.dx * qy - s.dy * qx);  // side of q
    const double c3 = qx * s.ay - qy * s.ax, c4 = qx * s.by - qy * s.bx;
    const bool p1 = s.c1 > e, n1 = s.c1 < -e, p2 = c2 > e, n2 = c2 < -e;
    const bool p3 = c3 > e, n3 = c3 < -e, p4 = c4 > e, n4 = c4 < -e;
    if ((p1 & p2) | (n1 & n2) | (p3 & p4) | (n3 & n4)) return 0;
    return (p1 | n1) & (p2 | n2) & (p3 | n3) & (p4 | n4) ? 1 : -1;
}

GHD int crosses_from_center(double ax, double ay, double bx, double by, double qx, double qy)
{
    return crosses_from_center(segment(ax, ay, bx, by), qx, qy);
}

}  // namespace cellbox
}  // namespace gahhg
