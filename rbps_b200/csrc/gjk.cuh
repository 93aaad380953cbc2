// gjk.cuh - GJK, EPA and the convex contact manifold on the device: the
// narrowphase of every convex pair without an analytic routine (a convex
// hull against a sphere, box, capsule or hull), as rbc::gjk_epa_manifold
// runs it (ContactManifoldGenerator.cpp:415-440).
//
// Same operation order as the reference, so the FP64 instantiation gives the
// same bits:
//   * GJK (GJK.cpp:18-97) over the simplex of Simplex.hpp, its vertices newest
//     first as the reference's order array lists them (DoSimplex.cpp:6-16),
//     and the line / triangle / tetrahedron cases of Line.cpp, Triangle.cpp,
//     Tetrahedron.cpp;
//   * EPA (EPA.cpp:141-378): at most 256 faces and 128 vertices, faces never
//     freed, the seed-coplanar shortcut, horizon edges cancelled in both
//     directions with order-preserving erase, the barycentric witness on A;
//   * the manifold (ContactManifoldGenerator.cpp:176-413): for two hulls
//     with polygon tables the reference / incident polygon clip
//     (Clipping.cpp:37-101) or the edge-edge closest points
//     (Clipping.cpp:103-128); one EPA point otherwise; reduce_to_4
//     (ContactManifoldGenerator.hpp:88-154).
// One warp runs one pair: the two shapes' supports on its halves, the scans
// over hull vertices, EPA faces and horizon edges split across its lanes; the
// polytope, edge list and clipping buffers live in the warp's shared-memory
// workspace (two views of one region: the polytope while EPA runs, the
// clipping buffers after).
//
// What bounds it is the latency of a pair's own chain, one iteration after
// another, and the fetch of its instructions: most queued pairs separate in
// one or two iterations, and a few of thousands run long.  So the code is
// kept small (one out-of-line support for every call), the simplex in
// registers, and a pair that goes round in circles is stopped at once.
#pragma once
#include <cfloat>
#include <cstdint>

#include "narrow.cuh"

namespace rbps_gpu
{
    // A workspace limit of the GJK path was hit: the device error word gets
    // RBPS_ERR_INTERNAL with site 20 + k (the pair reports no contact).
    __device__ __forceinline__ void set_gjk_error(int *err, int k)
    {
        if (err && atomicCAS(err, 0, -6) == 0)
        {
            err[1] = 20 + k;
            err[2] = 0;
        }
    }

    template <class T> __device__ __forceinline__ T big_value();
    template <> __device__ __forceinline__ double big_value<double>() { return DBL_MAX; }
    template <> __device__ __forceinline__ float big_value<float>() { return FLT_MAX; }

    constexpr int kEpaMaxFaces = 256;
    constexpr int kEpaMaxVerts = 128;
    constexpr int kEpaMaxIter = 128;
    constexpr int kGjkMaxIter = 128;
    constexpr int kEpaMaxEdges = 3 * kEpaMaxFaces;
    constexpr int kClipMaxPoly = 64;                     // polygon vertices / neighbour planes handled
    constexpr int kClipCap = (kClipMaxPoly * 2) * 2 + 8; // (inc_n + planes) * 2 + 8 at the limits

    template <class T>
    struct SVert
    {
        vec3<T> w0, w1, w;
    };

    template <class T>
    struct EpaFace
    {
        vec3<T> n, centroid;
        T d;
        uint8_t v[3];
        uint8_t obsolete;
    };

    // The clipping buffers of the hull-hull manifold alone: the second view
    // of a warp's shared workspace, over the EPA polytope it no longer needs.
    template <class T>
    struct GjkClipWork
    {
        vec3<T> inc[kClipMaxPoly], ref[kClipMaxPoly];
        vec3<T> pl_n[kClipMaxPoly], pl_p[kClipMaxPoly];
        vec3<T> buf_a[kClipCap + 4], buf_b[kClipCap + 4];
        T keep_d[kClipCap + 4];
    };

    // The EPA polytope of one warp's evaluation (first view of its workspace).
    template <class T>
    struct GjkEpaWork
    {
        SVert<T> verts[kEpaMaxVerts];
        EpaFace<T> faces[kEpaMaxFaces];
        uint16_t edges[kEpaMaxEdges]; // a | b << 8
        uint8_t seen[kEpaMaxFaces];   // the faces that see the new vertex, in order
    };

    // Bytes of one warp's shared workspace: the two views overlap.
    template <class T>
    constexpr size_t gjk_warp_bytes()
    {
        return ((sizeof(GjkEpaWork<T>) > sizeof(GjkClipWork<T>) ? sizeof(GjkEpaWork<T>) : sizeof(GjkClipWork<T>)) +
                15) / 16 * 16;
    }

    // shape_support (ShapeTypes.hpp:130-133) of every kind but the hull, whose
    // scan is the warp's (pair_support).
    template <class T>
    __device__ __forceinline__ vec3<T> local_support(int kind, const double *p, const vec3<T> &d)
    {
        switch (kind)
        {
        case kSphere: // Sphere.hpp:48-51
            return normalize(d) * T(p[0]);
        case kBox: // Box.hpp:49-55
            return vec3<T>(d.x > T(0) ? T(p[0]) : -T(p[0]), d.y > T(0) ? T(p[1]) : -T(p[1]),
                           d.z > T(0) ? T(p[2]) : -T(p[2]));
        case kCapsule: // Capsule.hpp:72-79
        {
            const vec3<T> endpoint(T(0.0), d.y >= T(0.0) ? T(p[0]) : -T(p[0]), T(0.0));
            const T len = length(d);
            if (len < T(kEpsilon))
                return endpoint;
            return endpoint + (d / len) * T(p[1]);
        }
        case kEllipsoid:
        case kCylinder:
        case kCone:
            return support_round<T>(kind, p, d);
        default:
            return vec3<T>();
        }
    }

    // ------------------------------------------------------------ one warp per pair
    // In the warp forms below every lane of the warp runs the same control
    // flow on the same values (scalar state is computed redundantly, so it
    // is bit-identical on every lane); the loops over hull vertices, EPA
    // faces, vertices and horizon edges are split across the lanes and
    // joined by warp reductions that keep the serial scans' tie rules.
    // Shared memory is written by one lane (or each lane its own entries)
    // between __syncwarp()s.
    constexpr unsigned kWarpAll = 0xffffffffu;

    // One shape of the pair as a half-warp holds it: lanes 0-15 shape A, lanes
    // 16-31 shape B, so both supports of an iteration run as one.  A hull of
    // up to 32 vertices is kept in registers, two a lane.
    template <class T>
    struct HalfShape
    {
        int kind;
        double p[3];
        tf<T> t;
        const double *V; // the hull's vertices, or null
        uint32_t nv;
        vec3<T> p0, p1;  // vertices sub and sub + 16 (sub: the lane in its half)
        bool any_hull;   // either shape of the pair is a hull
    };

    template <class T>
    __device__ __forceinline__ HalfShape<T> half_shape(const ShapeDev &sa, const tf<T> &ta, const ShapeDev &sb,
                                                       const tf<T> &tb, const HullSetDev &hs)
    {
        const bool b = threadIdx.x & 16u;
        const uint32_t sub = threadIdx.x & 15u;
        HalfShape<T> h;
        const ShapeDev &s = b ? sb : sa;
        h.kind = s.kind;
        for (int k = 0; k < 3; ++k)
            h.p[k] = s.p[k];
        h.t = b ? tb : ta;
        h.any_hull = sa.kind == kHull || sb.kind == kHull;
        h.V = nullptr;
        h.nv = 0;
        if (h.kind == kHull)
        {
            const uint32_t v0 = hs.v_off[s.hull];
            h.nv = hs.v_off[s.hull + 1] - v0;
            h.V = hs.verts + 3 * (size_t)v0;
            if (sub < h.nv)
                h.p0 = vec3<T>(T(h.V[3 * sub]), T(h.V[3 * sub + 1]), T(h.V[3 * sub + 2]));
            if (sub + 16u < h.nv)
                h.p1 = vec3<T>(T(h.V[3 * sub + 48]), T(h.V[3 * sub + 49]), T(h.V[3 * sub + 50]));
        }
        return h;
    }

    // The Minkowski support along dir (MinkowskiDiff.hpp support_a / _b): A's
    // along dir on lanes 0-15 and B's along -dir on lanes 16-31, in `own`;
    // returns their difference.  A hull's is the first vertex (lowest index)
    // of maximal dot product, as the serial scan's strict `>` keeps
    // (ConvexHull.hpp:457-472); a NaN first dot keeps vertex 0 as that scan
    // does.  Inline, at three calls in all: out of line the shapes and the
    // simplex went through the stack, whose 200 KB an SM the L1 left beside
    // the workspaces cannot hold.
    template <class T>
    __device__ __forceinline__ vec3<T> pair_support(const HalfShape<T> &h, const vec3<T> &dir, vec3<T> &own)
    {
        const bool b = threadIdx.x & 16u;
        const vec3<T> d = h.t.inverse_rotate_vector(b ? -dir : dir);
        vec3<T> l;
        if (h.any_hull)
        {
            const uint32_t sub = threadIdx.x & 15u;
            T best_d = T(0);
            uint32_t best_i = ~0u;
            bool nan0 = false;
            for (uint32_t i = sub; i < h.nv; i += 16)
            {
                const vec3<T> p = i < 16u && h.nv <= 32u ? h.p0
                                  : h.nv <= 32u          ? h.p1
                                                : vec3<T>(T(h.V[3 * i]), T(h.V[3 * i + 1]), T(h.V[3 * i + 2]));
                const T dd = dot(p, d);
                nan0 = nan0 || (i == 0 && dd != dd);
                if (dd == dd && (best_i == ~0u || dd > best_d))
                {
                    best_d = dd;
                    best_i = i;
                }
            }
            for (int o = 8; o > 0; o >>= 1)
            {
                const T od = __shfl_xor_sync(kWarpAll, best_d, o);
                const uint32_t oi = __shfl_xor_sync(kWarpAll, best_i, o);
                if (oi != ~0u && (best_i == ~0u || od > best_d || (od == best_d && oi < best_i)))
                {
                    best_d = od;
                    best_i = oi;
                }
            }
            const unsigned nan = __ballot_sync(kWarpAll, nan0) & (b ? 0xffff0000u : 0xffffu);
            const uint32_t i = nan || best_i == ~0u ? 0u : best_i;
            if (h.nv)
                l = vec3<T>(T(h.V[3 * i]), T(h.V[3 * i + 1]), T(h.V[3 * i + 2]));
        }
        if (h.kind != kHull)
            l = local_support(h.kind, h.p, d);
        own = h.t.transform_point(l);
        const vec3<T> other(__shfl_xor_sync(kWarpAll, own.x, 16), __shfl_xor_sync(kWarpAll, own.y, 16),
                            __shfl_xor_sync(kWarpAll, own.z, 16));
        return b ? other - own : own - other;
    }

    // Both supports of vertex `at` of a warp's shared list: lane 0 holds A's,
    // lane 16 B's (pair_support); w is the same on every lane.
    template <class T>
    __device__ __forceinline__ void store_vertex(SVert<T> &at, const vec3<T> &own, const vec3<T> &w)
    {
        const uint32_t lane = threadIdx.x & 31u;
        if (lane == 0)
        {
            at.w0 = own;
            at.w = w;
        }
        if (lane == 16)
            at.w1 = own;
        __syncwarp();
    }

    // ------------------------------------------------------------ GJK
    // The live vertices, newest first: their differences in registers (every
    // index is a constant), and the slot of a warp's shared list that holds
    // each one's supports.
    template <class T>
    struct Simplex
    {
        vec3<T> w[4];
        int slot[4];
        int rank;
    };

    template <class T>
    __device__ __forceinline__ vec3<T> triple_cross(const vec3<T> &a, const vec3<T> &b, const vec3<T> &c)
    {
        return cross(cross(a, b), c);
    }

    // Adds w as the newest; returns its slot, one that no live vertex holds.
    template <class T>
    __device__ __forceinline__ int simplex_add(Simplex<T> &s, const vec3<T> &w)
    {
        int free = 15;
        for (int i = 0; i < 3; ++i) // at most three are live
            if (i < s.rank)
                free &= ~(1 << s.slot[i]);
        const int slot = __ffs(free) - 1;
        for (int i = 3; i > 0; --i)
        {
            s.w[i] = s.w[i - 1];
            s.slot[i] = s.slot[i - 1];
        }
        s.w[0] = w;
        s.slot[0] = slot;
        if (s.rank < 4)
            ++s.rank;
        return slot;
    }

    template <class T>
    __device__ __forceinline__ void do_simplex_2(Simplex<T> &s, vec3<T> &dir)
    {
        const vec3<T> a = s.w[0], b = s.w[1];
        const vec3<T> ao = -a, ab = b - a;
        if (dot(ab, ao) >= T(0.0))
        {
            s.rank = 2;
            dir = triple_cross(ab, ao, ab);
            if (length_sq(dir) < T(1e-6))
            {
                const T ax = rabs(ab.x), ay = rabs(ab.y), az = rabs(ab.z);
                const vec3<T> axis = (ax <= ay && ax <= az) ? vec3<T>(T(1), T(0), T(0))
                                     : (ay <= az ? vec3<T>(T(0), T(1), T(0)) : vec3<T>(T(0), T(0), T(1)));
                dir = cross(ab, axis);
                if (length_sq(dir) < T(1e-6))
                    dir = cross(ab, vec3<T>(T(0), T(0), T(1)));
            }
        }
        else
        {
            s.rank = 1;
            dir = ao;
        }
    }

    template <class T>
    __device__ __forceinline__ void do_simplex_3(Simplex<T> &s, vec3<T> &dir)
    {
        const vec3<T> a = s.w[0], b = s.w[1], c = s.w[2];
        const vec3<T> ao = -a, ab = b - a, ac = c - a;
        const vec3<T> abc = cross(ab, ac);
        if (dot(cross(abc, ac), ao) >= T(0.0))
        {
            if (dot(ac, ao) >= T(0.0))
            {
                s.w[1] = c;
                s.slot[1] = s.slot[2];
                s.rank = 2;
                dir = triple_cross(ac, ao, ac);
            }
            else if (dot(ab, ao) >= T(0.0))
            {
                s.rank = 2;
                dir = triple_cross(ab, ao, ab);
            }
            else
            {
                s.rank = 1;
                dir = ao;
            }
        }
        else if (dot(cross(ab, abc), ao) >= T(0.0))
        {
            if (dot(ab, ao) >= T(0.0))
            {
                s.rank = 2;
                dir = triple_cross(ab, ao, ab);
            }
            else
            {
                s.rank = 1;
                dir = ao;
            }
        }
        else if (dot(abc, ao) >= T(0.0))
        {
            s.rank = 3;
            dir = abc;
        }
        else
        {
            s.w[1] = c;
            s.w[2] = b;
            const int tmp = s.slot[1];
            s.slot[1] = s.slot[2];
            s.slot[2] = tmp;
            s.rank = 3;
            dir = -abc;
        }
    }

    // Keeps the listed vertices (their constant places) in order.
    template <class T>
    __device__ __forceinline__ void keep(Simplex<T> &s, int r, int x0, int x1 = 0, int x2 = 0)
    {
        const vec3<T> a = s.w[x0], b = s.w[x1], c = s.w[x2];
        const int i = s.slot[x0], j = s.slot[x1], k = s.slot[x2];
        s.w[0] = a;
        s.slot[0] = i;
        if (r > 1)
        {
            s.w[1] = b;
            s.slot[1] = j;
        }
        if (r > 2)
        {
            s.w[2] = c;
            s.slot[2] = k;
        }
        s.rank = r;
    }

    // Returns true when the origin is inside the tetrahedron.
    template <class T>
    __device__ __forceinline__ bool do_simplex_4(Simplex<T> &s, vec3<T> &dir)
    {
        constexpr int va = 0, vb = 1, vc = 2, vd = 3;
        const vec3<T> a = s.w[va], b = s.w[vb], c = s.w[vc], d = s.w[vd];
        const vec3<T> ao = -a, ab = b - a, ac = c - a, ad = d - a;
        const vec3<T> abc = cross(ab, ac), acd = cross(ac, ad), adb = cross(ad, ab);
        const T kInside = T(1e-10);
        unsigned info = 0;
        if (dot(abc, ao) > kInside)
            info |= 1u;
        if (dot(acd, ao) > kInside)
            info |= 2u;
        if (dot(adb, ao) > kInside)
            info |= 4u;
        switch (info)
        {
        case 0:
            return true;
        case 1:
            if (dot(cross(abc, ac), ao) >= T(0.0))
            {
                if (dot(ac, ao) >= T(0.0)) { keep(s, 2, va, vc); dir = triple_cross(ac, ao, ac); }
                else if (dot(ab, ao) >= T(0.0)) { keep(s, 2, va, vb); dir = triple_cross(ab, ao, ab); }
                else { keep(s, 1, va); dir = ao; }
            }
            else if (dot(cross(ab, abc), ao) >= T(0.0))
            {
                if (dot(ab, ao) >= T(0.0)) { keep(s, 2, va, vb); dir = triple_cross(ab, ao, ab); }
                else { keep(s, 1, va); dir = ao; }
            }
            else { keep(s, 3, va, vb, vc); dir = abc; }
            break;
        case 2:
            if (dot(cross(acd, ad), ao) >= T(0.0))
            {
                if (dot(ad, ao) >= T(0.0)) { keep(s, 2, va, vd); dir = triple_cross(ad, ao, ad); }
                else if (dot(ac, ao) >= T(0.0)) { keep(s, 2, va, vc); dir = triple_cross(ac, ao, ac); }
                else { keep(s, 1, va); dir = ao; }
            }
            else if (dot(cross(ac, acd), ao) >= T(0.0))
            {
                if (dot(ac, ao) >= T(0.0)) { keep(s, 2, va, vc); dir = triple_cross(ac, ao, ac); }
                else { keep(s, 1, va); dir = ao; }
            }
            else { keep(s, 3, va, vc, vd); dir = acd; }
            break;
        case 3:
            if (dot(ac, ao) >= T(0.0)) { keep(s, 2, va, vc); dir = triple_cross(ac, ao, ac); }
            else { keep(s, 1, va); dir = ao; }
            break;
        case 4:
            if (dot(cross(adb, ab), ao) >= T(0.0))
            {
                if (dot(ab, ao) >= T(0.0)) { keep(s, 2, va, vb); dir = triple_cross(ab, ao, ab); }
                else if (dot(ad, ao) >= T(0.0)) { keep(s, 2, va, vd); dir = triple_cross(ad, ao, ad); }
                else { keep(s, 1, va); dir = ao; }
            }
            else if (dot(cross(ad, adb), ao) >= T(0.0))
            {
                if (dot(ad, ao) >= T(0.0)) { keep(s, 2, va, vd); dir = triple_cross(ad, ao, ad); }
                else { keep(s, 1, va); dir = ao; }
            }
            else { keep(s, 3, va, vd, vb); dir = adb; }
            break;
        case 5:
            if (dot(ab, ao) >= T(0.0)) { keep(s, 2, va, vb); dir = triple_cross(ab, ao, ab); }
            else { keep(s, 1, va); dir = ao; }
            break;
        case 6:
            if (dot(ad, ao) >= T(0.0)) { keep(s, 2, va, vd); dir = triple_cross(ad, ao, ad); }
            else { keep(s, 1, va); dir = ao; }
            break;
        default:
            keep(s, 1, va);
            dir = ao;
            break;
        }
        return false;
    }

    enum
    {
        kGjkValid = 0,
        kGjkInside = 1,
        kGjkFailed = 2
    };

    template <class T>
    __device__ __forceinline__ bool same_bits(const vec3<T> &a, const vec3<T> &b)
    {
        auto bits = [](T x) { return __double_as_longlong(double(x)); };
        return bits(a.x) == bits(b.x) && bits(a.y) == bits(b.y) && bits(a.z) == bits(b.z);
    }

    // Every lane of a warp runs it.  `sv` holds the simplex's supports and
    // `mark` is scratch, four and one entries of the warp's shared memory.
    // An iteration is a function of the simplex and the direction alone, so
    // one that comes back to an earlier state goes round for good and ends
    // in kGjkFailed at iteration 128: it is returned as soon as the state is
    // met again (bit for bit; Brent's marks at iterations 1, 2, 4, 8, ...).
    // Two hulls that almost touch do this: 34 of the 19,362 queued pairs of
    // a 65,536-body world's step, and each took 0.25 ms of a 0.29 ms pass.
    template <class T>
    __device__ __forceinline__ int gjk_evaluate(const HalfShape<T> &h, const vec3<T> &guess, Simplex<T> &s, SVert<T> *sv,
                                                SVert<T> &mark)
    {
        s.rank = 0;
        vec3<T> dir = length_sq(guess) > T(kEpsilon) ? guess : vec3<T>(T(1.0), T(0.0), T(0.0));
        vec3<T> mark_dir;
        int mark_rank = 0, mark_it = 1;
        for (int it = -1; it < kGjkMaxIter; ++it)
        {
            vec3<T> own;
            const vec3<T> w = pair_support(h, dir, own);
            if (it >= 0 && dot(w, dir) < T(0.0))
                return kGjkValid;
            store_vertex(sv[simplex_add(s, w)], own, w);
            if (s.rank == 2)
                do_simplex_2(s, dir);
            else if (s.rank == 3)
                do_simplex_3(s, dir);
            else if (s.rank == 4)
            {
                if (do_simplex_4(s, dir))
                    return kGjkInside;
            }
            else if (it < 0)
                dir = -w;
            if (s.rank == mark_rank && same_bits(dir, mark_dir) && same_bits(s.w[0], mark.w0) &&
                (s.rank < 2 || same_bits(s.w[1], mark.w1)) && (s.rank < 3 || same_bits(s.w[2], mark.w)))
                return kGjkFailed;
            if (it == mark_it)
            {
                mark_it = 2 * it;
                mark_dir = dir;
                mark_rank = s.rank;
                __syncwarp();
                if ((threadIdx.x & 31u) == 0)
                {
                    mark = SVert<T>{s.w[0], s.w[1], s.w[2]};
                }
                __syncwarp();
            }
        }
        return kGjkFailed;
    }

    // ------------------------------------------------------------ EPA
    enum
    {
        kEpaValid = 0,
        kEpaFailed = 1,
        kEpaOutOfFaces = 2,
        kEpaOutOfVertices = 3,
        kEpaNonLinear = 4
    };

    // compute_face_normal (EPA.cpp:19-67)
    template <class T>
    __device__ bool epa_face_normal(EpaFace<T> &f, const SVert<T> *V, int n_all)
    {
        const vec3<T> a = V[f.v[0]].w, b = V[f.v[1]].w, c = V[f.v[2]].w;
        vec3<T> n = cross(b - a, c - a);
        const T n_len = length(n);
        if (n_len < T(kEpsilon))
            return false;
        n = n / n_len;
        T d = dot(n, a);
        const T kCop = T(1e-12);
        if (d < -kCop)
        {
            n = -n;
            d = -d;
        }
        else if (d <= kCop)
        {
            bool fixed = false;
            for (int i = 0; i < n_all; ++i)
            {
                const T t = dot(n, V[i].w);
                if (t > kCop)
                {
                    n = -n;
                    d = T(0.0);
                    fixed = true;
                    break;
                }
                if (t < -kCop)
                {
                    d = T(0.0);
                    fixed = true;
                    break;
                }
            }
            if (!fixed)
                return false;
        }
        f.n = n;
        f.centroid = (a + b + c) * (T(1.0) / T(3.0));
        f.d = d;
        f.obsolete = 0;
        return true;
    }

    template <class T>
    struct EpaResult
    {
        vec3<T> normal;
        T depth;
        vec3<T> contact;
    };

    // ------------------------------------------------------------ manifold
    template <class T>
    __device__ __forceinline__ vec3<T> hull_vertex(const HullSetDev &hs, uint32_t hull, uint32_t i)
    {
        const double *p = hs.verts + 3 * (size_t)(hs.v_off[hull] + i);
        return vec3<T>(T(p[0]), T(p[1]), T(p[2]));
    }

    template <class T>
    __device__ __forceinline__ vec3<T> hull_poly_normal(const HullSetDev &hs, const HullDesc &h, uint32_t p)
    {
        const double *n = hs.poly_n + 3 * (size_t)(h.pn + p);
        return vec3<T>(T(n[0]), T(n[1]), T(n[2]));
    }

    // support_vertex_index (ContactManifoldGenerator.cpp:25-38)
    template <class T>
    __device__ uint32_t support_vertex_index(const HullSetDev &hs, uint32_t hull, const tf<T> &t, const vec3<T> &wd)
    {
        const vec3<T> ld = t.inverse_rotate_vector(wd);
        const uint32_t nv = hs.v_off[hull + 1] - hs.v_off[hull];
        uint32_t best = 0;
        T best_d = dot(hull_vertex<T>(hs, hull, 0), ld);
        for (uint32_t i = 1; i < nv; ++i)
        {
            const T d = dot(hull_vertex<T>(hs, hull, i), ld);
            if (d > best_d)
            {
                best_d = d;
                best = i;
            }
        }
        return best;
    }

    // pick_best_polygon (ContactManifoldGenerator.cpp:40-60)
    template <class T>
    __device__ uint32_t pick_best_polygon(const HullSetDev &hs, const HullDesc &h, const tf<T> &t, uint32_t sv,
                                          const vec3<T> &wd, T &align)
    {
        const uint32_t *off = hs.u32 + h.v2p_o, *idx = hs.u32 + h.v2p_i;
        const uint32_t s = off[sv], e = off[sv + 1];
        uint32_t best = (s < e) ? idx[s] : 0u;
        T best_d = -big_value<T>();
        for (uint32_t i = s; i < e; ++i)
        {
            const uint32_t p = idx[i];
            const T d = dot(t.rotate_vector(hull_poly_normal<T>(hs, h, p)), wd);
            if (d > best_d)
            {
                best_d = d;
                best = p;
            }
        }
        align = best_d;
        return best;
    }

    // pick_best_edge_pair (ContactManifoldGenerator.cpp:68-126)
    template <class T>
    __device__ bool pick_best_edge_pair(const HullSetDev &hs, uint32_t ha, const HullDesc &da, const tf<T> &ta,
                                        uint32_t sa, uint32_t hb, const HullDesc &db, const tf<T> &tb, uint32_t sb,
                                        const vec3<T> &wn, uint32_t e[4], vec3<T> &out_n, T &align)
    {
        const vec3<T> wsa = ta.transform_point(hull_vertex<T>(hs, ha, sa));
        const vec3<T> wsb = tb.transform_point(hull_vertex<T>(hs, hb, sb));
        const uint32_t *ao = hs.u32 + da.v2n_o, *ai = hs.u32 + da.v2n_i;
        const uint32_t *bo = hs.u32 + db.v2n_o, *bi = hs.u32 + db.v2n_i;
        const uint32_t na_s = ao[sa], na_e = ao[sa + 1], nb_s = bo[sb], nb_e = bo[sb + 1];
        if (na_s >= na_e || nb_s >= nb_e)
            return false;
        T best_d = -big_value<T>();
        bool found = false;
        for (uint32_t i = na_s; i < na_e; ++i)
        {
            const uint32_t na = ai[i];
            const vec3<T> ea = wsa - ta.transform_point(hull_vertex<T>(hs, ha, na));
            for (uint32_t j = nb_s; j < nb_e; ++j)
            {
                const uint32_t nb = bi[j];
                const vec3<T> eb = wsb - tb.transform_point(hull_vertex<T>(hs, hb, nb));
                const vec3<T> c = cross(ea, eb);
                const T c_len = length(c);
                if (c_len < T(kEpsilon))
                    continue;
                const vec3<T> cn = c / c_len;
                const T d_pos = dot(cn, wn);
                if (d_pos > best_d)
                {
                    best_d = d_pos;
                    e[0] = sa; e[1] = na; e[2] = sb; e[3] = nb;
                    out_n = cn;
                    found = true;
                }
                const T d_neg = -d_pos;
                if (d_neg > best_d)
                {
                    best_d = d_neg;
                    e[0] = sa; e[1] = na; e[2] = sb; e[3] = nb;
                    out_n = -cn;
                    found = true;
                }
            }
        }
        align = best_d;
        return found;
    }

    // skew_line_closest_points (Clipping.cpp:103-128)
    template <class T>
    __device__ bool skew_closest(const vec3<T> &p1, const vec3<T> &d1, const vec3<T> &p2, const vec3<T> &d2,
                                 vec3<T> &l1, vec3<T> &l2)
    {
        const T n1 = d1.x * d2.x + d1.y * d2.y + d1.z * d2.z;
        const T n2 = d2.x * d2.x + d2.y * d2.y + d2.z * d2.z;
        const T m1 = -d1.x * d1.x - d1.y * d1.y - d1.z * d1.z;
        const T m2 = -d2.x * d1.x - d2.y * d1.y - d2.z * d1.z;
        const T r1 = -d1.x * p2.x + d1.x * p1.x - d1.y * p2.y + d1.y * p1.y - d1.z * p2.z + d1.z * p1.z;
        const T r2 = -d2.x * p2.x + d2.x * p1.x - d2.y * p2.y + d2.y * p1.y - d2.z * p2.z + d2.z * p1.z;
        const T denom = (n1 * m2) - (n2 * m1);
        if (rabs(denom) < T(kEpsilon))
            return false;
        const T n = ((r1 * m2) - (r2 * m1)) / denom;
        const T m = ((n1 * r2) - (n2 * r1)) / denom;
        l1 = p1 + d1 * m;
        l2 = p2 + d2 * n;
        return true;
    }

    // sutherland_hodgman (Clipping.cpp:37-101) from `in` through the planes,
    // ping-ponging between a and b; returns min(count, cap) points in *res.
    template <class T>
    __device__ int sutherland_hodgman(const vec3<T> *in, int n_in, const vec3<T> *pn, const vec3<T> *pp, int n_planes,
                                      bool remove_only, vec3<T> *a, vec3<T> *b, int cap, const vec3<T> **res,
                                      int *err)
    {
        *res = a;
        if (n_in <= 0 || n_planes <= 0 || cap <= 0)
            return 0;
        int na = n_in;
        for (int i = 0; i < n_in; ++i)
            a[i] = in[i];
        for (int p = 0; p < n_planes; ++p)
        {
            if (na == 0)
                break;
            const vec3<T> N = pn[p], P = pp[p];
            const T dplane = -dot(N, P);
            int nb = 0;
            vec3<T> start = a[na - 1];
            for (int j = 0; j < na; ++j)
            {
                const vec3<T> end = a[j];
                const bool start_in = dot(start, N) + dplane >= T(0.0);
                const bool end_in = dot(end, N) + dplane >= T(0.0);
                if (nb + 2 > kClipCap + 4)
                {
                    set_gjk_error(err, 2);
                    return 0;
                }
                if (remove_only)
                {
                    if (end_in)
                        b[nb++] = end;
                }
                else
                {
                    // plane_edge_intersection (Clipping.cpp:15-33)
                    bool cut_ok = false;
                    vec3<T> cut;
                    if (start_in != end_in)
                    {
                        const vec3<T> ab = end - start;
                        const T ab_p = dot(N, ab);
                        if (!(rabs(ab_p) <= T(1e-6)))
                        {
                            const vec3<T> p_co = N * (-dplane);
                            T fac = -dot(N, start - p_co) / ab_p;
                            if (fac < T(0.0))
                                fac = T(0.0);
                            if (fac > T(1.0))
                                fac = T(1.0);
                            cut = start + ab * fac;
                            cut_ok = true;
                        }
                    }
                    if (start_in && end_in)
                        b[nb++] = end;
                    else if (start_in && !end_in)
                    {
                        if (cut_ok)
                            b[nb++] = cut;
                    }
                    else if (!start_in && end_in)
                    {
                        if (cut_ok)
                            b[nb++] = cut;
                        b[nb++] = end;
                    }
                }
                start = end;
            }
            vec3<T> *t = a;
            a = b;
            b = t;
            na = nb;
        }
        *res = a;
        return na < cap ? na : cap;
    }

    // reduce_to_4 (ContactManifoldGenerator.hpp:88-154)
    template <class T>
    __device__ int reduce_to_4(const vec3<T> *pts, const T *dep, int n, Manifold<T> &m)
    {
        if (n <= 4)
        {
            for (int i = 0; i < n; ++i)
            {
                m.pos[i] = pts[i];
                m.depth[i] = dep[i];
            }
            return n;
        }
        int i0 = 0;
        for (int i = 1; i < n; ++i)
            if (dep[i] > dep[i0])
                i0 = i;
        int i1 = (i0 == 0) ? 1 : 0;
        T best = length_sq(pts[i1] - pts[i0]);
        for (int i = 0; i < n; ++i)
        {
            if (i == i0)
                continue;
            const T d = length_sq(pts[i] - pts[i0]);
            if (d > best)
            {
                best = d;
                i1 = i;
            }
        }
        int i2 = -1;
        best = T(0.0);
        const vec3<T> seg = pts[i1] - pts[i0];
        for (int i = 0; i < n; ++i)
        {
            if (i == i0 || i == i1)
                continue;
            const T d = length_sq(cross(pts[i] - pts[i0], seg));
            if (d > best)
            {
                best = d;
                i2 = i;
            }
        }
        if (i2 < 0)
            for (int i = 0; i < n; ++i)
                if (i != i0 && i != i1)
                {
                    i2 = i;
                    break;
                }
        int i3 = -1;
        best = T(0.0);
        if (i2 >= 0)
        {
            const vec3<T> tri_n = cross(pts[i1] - pts[i0], pts[i2] - pts[i0]);
            for (int i = 0; i < n; ++i)
            {
                if (i == i0 || i == i1 || i == i2)
                    continue;
                const T d = rabs(dot(pts[i] - pts[i0], tri_n));
                if (d > best)
                {
                    best = d;
                    i3 = i;
                }
            }
            if (i3 < 0)
                for (int i = 0; i < n; ++i)
                    if (i != i0 && i != i1 && i != i2)
                    {
                        i3 = i;
                        break;
                    }
        }
        m.pos[0] = pts[i0];
        m.depth[0] = dep[i0];
        m.pos[1] = pts[i1];
        m.depth[1] = dep[i1];
        if (i2 >= 0)
        {
            m.pos[2] = pts[i2];
            m.depth[2] = dep[i2];
        }
        if (i3 >= 0)
        {
            m.pos[3] = pts[i3];
            m.depth[3] = dep[i3];
            return 4;
        }
        return (i2 >= 0) ? 3 : 2;
    }

    template <class T>
    __device__ __forceinline__ void single_point(Manifold<T> &m, const vec3<T> &n, const vec3<T> &p, T d)
    {
        m.normal = n;
        m.n = 1;
        m.pos[0] = p;
        m.depth[0] = d;
    }

    // manifold_convex_convex (ContactManifoldGenerator.cpp:176-379) for two
    // hulls with polygon tables.
    // WS: the clipping buffers (GjkClipWork, the second view of a warp's
    // shared workspace).
    template <class T, class WS>
    __device__ void manifold_hull_hull(const EpaResult<T> &r, const HullSetDev &hs, uint32_t ha, const tf<T> &ta,
                                       uint32_t hb, const tf<T> &tb, WS &ws, Manifold<T> &m, int *err)
    {
        m.normal = r.normal;
        m.n = 0;
        const HullDesc da = hs.desc[ha], db = hs.desc[hb];
        const vec3<T> inv_normal = -r.normal;
        const uint32_t sa = support_vertex_index(hs, ha, ta, r.normal);
        const uint32_t sb = support_vertex_index(hs, hb, tb, inv_normal);
        T align_a, align_b;
        const uint32_t poly_a = pick_best_polygon(hs, da, ta, sa, r.normal, align_a);
        const uint32_t poly_b = pick_best_polygon(hs, db, tb, sb, inv_normal, align_b);
        uint32_t e[4] = {0, 0, 0, 0};
        vec3<T> edge_n(T(0), T(0), T(0));
        T align_e = -big_value<T>();
        const bool has_edge = pick_best_edge_pair(hs, ha, da, ta, sa, hb, db, tb, sb, r.normal, e, edge_n, align_e);
        const T EPS = T(1e-4);
        if (has_edge && align_e > align_a + EPS && align_e > align_b + EPS)
        {
            const vec3<T> p1 = ta.transform_point(hull_vertex<T>(hs, ha, e[0]));
            const vec3<T> d1 = ta.transform_point(hull_vertex<T>(hs, ha, e[1])) - p1;
            const vec3<T> p2 = tb.transform_point(hull_vertex<T>(hs, hb, e[2]));
            const vec3<T> d2 = tb.transform_point(hull_vertex<T>(hs, hb, e[3])) - p2;
            vec3<T> l1, l2;
            if (skew_closest(p1, d1, p2, d2, l1, l2))
                single_point(m, r.normal, (l1 + l2) * T(0.5), r.depth);
            else
                single_point(m, r.normal, r.contact, r.depth);
            return;
        }
        const bool ref_is_a = align_a > align_b;
        const HullDesc &dref = ref_is_a ? da : db;
        const HullDesc &dinc = ref_is_a ? db : da;
        const uint32_t href = ref_is_a ? ha : hb, hinc = ref_is_a ? hb : ha;
        const tf<T> &tref = ref_is_a ? ta : tb;
        const tf<T> &tinc = ref_is_a ? tb : ta;
        const uint32_t ref_poly = ref_is_a ? poly_a : poly_b;
        const uint32_t inc_poly = ref_is_a ? poly_b : poly_a;
        const vec3<T> ref_n = tref.rotate_vector(hull_poly_normal<T>(hs, dref, ref_poly));
        const uint32_t *inc_off = hs.u32 + dinc.po, *inc_idx = hs.u32 + dinc.pi;
        const uint32_t inc_s = inc_off[inc_poly], inc_e = inc_off[inc_poly + 1];
        const int inc_n = (int)(inc_e - inc_s);
        if (inc_n < 3)
        {
            single_point(m, r.normal, r.contact, r.depth);
            return;
        }
        const uint32_t *ref_off = hs.u32 + dref.po, *ref_idx = hs.u32 + dref.pi;
        const uint32_t ref_s = ref_off[ref_poly], ref_e = ref_off[ref_poly + 1];
        const uint32_t *p2o = hs.u32 + dref.p2p_o, *p2i = hs.u32 + dref.p2p_i;
        const uint32_t n_s = p2o[ref_poly], n_e = p2o[ref_poly + 1];
        if (inc_n > kClipMaxPoly || (int)(ref_e - ref_s) > kClipMaxPoly || (int)(n_e - n_s) > kClipMaxPoly)
        {
            set_gjk_error(err, 3); // polygon beyond the workspace: no contact
            return;
        }
        for (int i = 0; i < inc_n; ++i)
            ws.inc[i] = tinc.transform_point(hull_vertex<T>(hs, hinc, inc_idx[inc_s + i]));
        for (uint32_t i = 0; i < ref_e - ref_s; ++i)
            ws.ref[i] = tref.transform_point(hull_vertex<T>(hs, href, ref_idx[ref_s + i]));
        const vec3<T> ref_pt = ws.ref[0];
        const int n_planes = (int)(n_e - n_s);
        for (int i = 0; i < n_planes; ++i)
        {
            const uint32_t nbp = p2i[n_s + i];
            const uint32_t first_v = ref_idx[ref_off[nbp]];
            ws.pl_p[i] = tref.transform_point(hull_vertex<T>(hs, href, first_v));
            ws.pl_n[i] = -tref.rotate_vector(hull_poly_normal<T>(hs, dref, nbp));
        }
        const int clip_cap = (inc_n + n_planes) * 2 + 8;
        const vec3<T> *clipped = ws.inc;
        int n_clipped = inc_n;
        if (n_planes > 0)
            n_clipped = sutherland_hodgman(ws.inc, inc_n, ws.pl_n, ws.pl_p, n_planes, false, ws.buf_a, ws.buf_b,
                                           clip_cap, &clipped, err);
        // the ref-plane pass starts in the buffer that holds the clipped
        // polygon (a copy onto itself), and the kept points stay in the one
        // it ends in
        const vec3<T> rpn = -ref_n;
        const vec3<T> *fin = ws.buf_a;
        vec3<T> *from = clipped == ws.buf_b ? ws.buf_b : ws.buf_a;
        const int n_final = sutherland_hodgman(clipped, n_clipped, &rpn, &ref_pt, 1, true, from,
                                               from == ws.buf_a ? ws.buf_b : ws.buf_a, clip_cap + 4, &fin, err);
        vec3<T> *kept = fin == ws.buf_a ? ws.buf_a : ws.buf_b;
        int n_keep = 0;
        for (int i = 0; i < n_final; ++i)
        {
            const vec3<T> p = fin[i];
            const T d_to_plane = dot(p - ref_pt, ref_n);
            const vec3<T> diff = ref_n * d_to_plane;
            const T pen = ref_is_a ? dot(diff, r.normal) : -dot(diff, r.normal);
            if (pen <= T(0.0))
            {
                kept[n_keep] = p;
                ws.keep_d[n_keep] = -pen;
                ++n_keep;
            }
        }
        if (n_keep == 0)
        {
            single_point(m, r.normal, r.contact, r.depth);
            return;
        }
        m.n = reduce_to_4(kept, ws.keep_d, n_keep, m);
    }

    // ------------------------------------------------------------ EPA on a warp
    // add_edge (EPA.cpp:71-84) over n edges in order, on a warp.  The reference
    // erases a stored edge equal to the new one in either direction and
    // otherwise appends the new one, so an edge met an even number of times
    // is gone and one met an odd number stands where it was met last.
    // Compacts E in place, in order; returns the count.
    __device__ __forceinline__ int warp_horizon(uint16_t *E, int n)
    {
        const int lane = (int)(threadIdx.x & 31u);
        auto key = [](uint32_t e) { return min(e & 255u, e >> 8) | (max(e & 255u, e >> 8) << 8); };
        int kept = 0;
        // an entry is read by every later round's scan: results are written
        // behind the scan only, at or below the place they came from
        uint32_t keep_bits[(kEpaMaxEdges + 31) / 32 / 8 + 1]; // 8 rounds of flags a word
        for (uint32_t &k : keep_bits)
            k = 0;
        for (int base = 0, r = 0; base < n; base += 32, ++r)
        {
            const int i = base + lane;
            const uint32_t mine = i < n ? key(E[i]) : ~0u;
            int met = 0, last = -1;
            for (int j = 0; j < n; ++j)
                if (key(E[j]) == mine)
                {
                    ++met;
                    last = j;
                }
            if (i < n && (met & 1) && last == i)
                keep_bits[r >> 3] |= 1u << (r & 7);
        }
        __syncwarp();
        for (int base = 0, r = 0; base < n; base += 32, ++r)
        {
            const int i = base + lane;
            const bool k = (keep_bits[r >> 3] >> (r & 7)) & 1u;
            const uint16_t e = i < n ? E[i] : 0;
            const unsigned m = __ballot_sync(kWarpAll, k);
            if (k)
                E[kept + __popc(m & ((1u << lane) - 1u))] = e;
            kept += __popc(m);
            __syncwarp();
        }
        return kept;
    }

    // epa_evaluate on one warp, the polytope in the warp's shared workspace.
    // The same steps in the same order as the serial form (EPA.cpp:141-378):
    // the nearest live face is a warp argmin keeping the lowest index on
    // ties (the serial scan's strict `<`); the faces that see the new vertex
    // are tested 32 at a time and their edges added in face order; the new
    // faces are built 32 at a time and packed in edge order, a degenerate
    // one leaving no slot, with OutOfFaces where the serial loop would meet
    // 256 faces.  Every lane returns the same result.
    template <class T>
    __device__ int epa_evaluate_warp(const Simplex<T> &seed, const HalfShape<T> &h, GjkEpaWork<T> &ws, EpaResult<T> &out)
    {
        const uint32_t lane = threadIdx.x & 31u;
        out.normal = vec3<T>(T(0), T(0), T(0));
        out.depth = T(0.0);
        out.contact = vec3<T>(T(0), T(0), T(0));
        if (seed.rank != 4)
            return kEpaNonLinear;
        SVert<T> *V = ws.verts;
        EpaFace<T> *F = ws.faces;
        {
            // the simplex's supports lie in its slots: into its order
            SVert<T> mine;
            for (int i = 0; i < 4; ++i)
                if (lane == (uint32_t)i)
                    mine = V[seed.slot[i]];
            __syncwarp();
            if (lane < 4)
                V[lane] = mine;
            __syncwarp();
        }
        int nv = 4, nf = 0;
        {
            const vec3<T> va = V[0].w, vb = V[1].w, vc = V[2].w, vd = V[3].w;
            const T e2 = T(kEpsilon) * T(kEpsilon);
            vec3<T> pn = cross(vb - va, vc - va);
            if (length_sq(pn) < e2)
                pn = cross(vb - va, vd - va);
            if (length_sq(pn) < e2)
                pn = cross(vc - va, vd - va);
            if (length_sq(pn) > e2)
            {
                pn = normalize(pn);
                const T dist_d = rabs(dot(vd - va, pn));
                if (dist_d < T(1e-5))
                {
                    T dist[2]; // along pn, along -pn
#pragma unroll 1
                    for (int k = 0; k < 2; ++k)
                    {
                        const vec3<T> dn = k ? -pn : pn;
                        vec3<T> own;
                        dist[1] = dot(pair_support(h, dn, own) - va, dn);
                        if (k == 0)
                            dist[0] = dist[1];
                    }
                    const T dist_pos = dist[0], dist_neg = dist[1];
                    if (dist_pos < T(1e-4) || dist_neg < T(1e-4))
                    {
                        out.normal = (dist_pos <= dist_neg) ? pn : -pn;
                        out.depth = T(0.0);
                        out.contact = (V[0].w0 + V[1].w0 + V[2].w0 + V[3].w0) * T(0.25);
                        return kEpaValid;
                    }
                }
            }
        }
        {
            // initial tetrahedron faces (A,B,C), (A,C,D), (A,D,B), (B,C,D): lane k builds face k
            const uint8_t init[4][3] = {{0, 1, 2}, {0, 2, 3}, {0, 3, 1}, {1, 2, 3}};
            EpaFace<T> f;
            bool ok = true;
            if (lane < 4)
            {
                f.v[0] = init[lane][0];
                f.v[1] = init[lane][1];
                f.v[2] = init[lane][2];
                f.obsolete = 0;
                ok = epa_face_normal(f, V, nv);
            }
            if (__ballot_sync(kWarpAll, !ok))
                return kEpaNonLinear;
            if (lane < 4)
                F[lane] = f;
            nf = 4;
            __syncwarp();
        }
        for (int it = 0; it < kEpaMaxIter; ++it)
        {
            T min_d = big_value<T>();
            int ci = -1;
            for (int i = (int)lane; i < nf; i += 32)
                if (!F[i].obsolete && F[i].d < min_d)
                {
                    min_d = F[i].d;
                    ci = i;
                }
            for (int o = 16; o > 0; o >>= 1)
            {
                const T od = __shfl_xor_sync(kWarpAll, min_d, o);
                const int oi = __shfl_xor_sync(kWarpAll, ci, o);
                if (oi >= 0 && (ci < 0 || od < min_d || (od == min_d && oi < ci)))
                {
                    min_d = od;
                    ci = oi;
                }
            }
            if (ci < 0)
                return kEpaFailed;
            const EpaFace<T> cf = F[ci];
            const vec3<T> dir = cf.n;
            vec3<T> own;
            const vec3<T> w = pair_support(h, dir, own);
            const T d_proj = dot(w, dir);
            if (d_proj - min_d < T(1e-6))
            {
                out.normal = cf.n;
                out.depth = min_d;
                const vec3<T> q = cf.n * min_d;
                const vec3<T> p0 = V[cf.v[0]].w, p1 = V[cf.v[1]].w, p2 = V[cf.v[2]].w;
                const vec3<T> e0 = p1 - p0, e1 = p2 - p0, r = q - p0;
                const T d00 = dot(e0, e0), d01 = dot(e0, e1), d11 = dot(e1, e1);
                const T d20 = dot(r, e0), d21 = dot(r, e1);
                const T denom = d00 * d11 - d01 * d01;
                if (rabs(denom) < T(kEpsilon))
                    out.contact = V[cf.v[0]].w0;
                else
                {
                    const T v_w = (d11 * d20 - d01 * d21) / denom;
                    const T w_w = (d00 * d21 - d01 * d20) / denom;
                    const T u_w = T(1.0) - v_w - w_w;
                    out.contact = V[cf.v[0]].w0 * u_w + V[cf.v[1]].w0 * v_w + V[cf.v[2]].w0 * w_w;
                }
                return kEpaValid;
            }
            bool dup = false;
            for (int i = (int)lane; i < nv; i += 32)
                dup = dup || length_sq(V[i].w - w) < T(kEpsilon) * T(kEpsilon);
            if (__any_sync(kWarpAll, dup))
            {
                out.normal = cf.n;
                out.depth = min_d;
                out.contact = V[cf.v[0]].w0;
                return kEpaValid;
            }
            if (nv >= kEpaMaxVerts)
                return kEpaOutOfVertices;
            const uint8_t wi = (uint8_t)nv;
            store_vertex(V[nv], own, w);
            ++nv;
            // the horizon: the faces that see w, their edges in face order
            int n_seen = 0;
            for (int base = 0; base < nf; base += 32)
            {
                const int i = base + (int)lane;
                bool vis = false;
                if (i < nf && !F[i].obsolete)
                {
                    vis = dot(F[i].n, w - F[i].centroid) > T(0.0);
                }
                const unsigned m = __ballot_sync(kWarpAll, vis);
                if (vis)
                {
                    F[i].obsolete = 1;
                    ws.seen[n_seen + __popc(m & ((1u << lane) - 1u))] = (uint8_t)i;
                }
                n_seen += __popc(m);
            }
            __syncwarp();
            for (int k = (int)lane; k < 3 * n_seen; k += 32)
            {
                const uint8_t *fv = F[ws.seen[k / 3]].v;
                const int c = k % 3;
                ws.edges[k] = (uint16_t)(fv[c] | (fv[c == 2 ? 0 : c + 1] << 8));
            }
            __syncwarp();
            const int ne = warp_horizon(ws.edges, 3 * n_seen);
            // new faces on the horizon edges, packed in edge order
            for (int base = 0; base < ne; base += 32)
            {
                const int e = base + (int)lane;
                EpaFace<T> f;
                bool ok = false;
                if (e < ne)
                {
                    f.v[0] = (uint8_t)ws.edges[e];
                    f.v[1] = (uint8_t)(ws.edges[e] >> 8);
                    f.v[2] = wi;
                    f.obsolete = 0;
                    ok = epa_face_normal(f, V, nv);
                }
                const unsigned okm = __ballot_sync(kWarpAll, ok);
                const int before = nf + __popc(okm & ((1u << lane) - 1u));
                if (__any_sync(kWarpAll, e < ne && before >= kEpaMaxFaces))
                    return kEpaOutOfFaces;
                if (ok)
                    F[before] = f;
                nf += __popc(okm);
            }
            __syncwarp();
        }
        return kEpaFailed;
    }

    // gjk_epa_manifold on one warp: every lane calls it with the same pair
    // and `ws` the warp's shared workspace (gjk_warp_bytes<T>()).  The
    // return value is the same on every lane; the manifold is complete on
    // lane 0 (a hull-hull manifold is clipped by lane 0 alone, in the
    // workspace's second view).
    template <class T>
    __device__ bool gjk_epa_manifold_warp(const ShapeDev &sa, const tf<T> &ta, const ShapeDev &sb, const tf<T> &tb,
                                          const HullSetDev &hs, unsigned char *ws, Manifold<T> &m, int *err)
    {
        GjkEpaWork<T> &work = *reinterpret_cast<GjkEpaWork<T> *>(ws);
        const HalfShape<T> h = half_shape(sa, ta, sb, tb, hs);
        vec3<T> guess = tb.pos - ta.pos;
        if (length_sq(guess) < T(kEpsilon))
            guess = vec3<T>(T(1.0), T(0.0), T(0.0));
        Simplex<T> s;
        if (gjk_evaluate(h, guess, s, work.verts, work.verts[4]) != kGjkInside)
            return false;
        EpaResult<T> r;
        if (epa_evaluate_warp(s, h, work, r) != kEpaValid)
            return false;
        m.normal = r.normal;
        m.n = 0;
        const bool adj_a = sa.kind == kHull && hs.desc[sa.hull].np > 0;
        const bool adj_b = sb.kind == kHull && hs.desc[sb.hull].np > 0;
        __syncwarp(); // the polytope is dead: the clipping view may overwrite it
        if (adj_a && adj_b)
        {
            if ((threadIdx.x & 31u) == 0)
                manifold_hull_hull(r, hs, (uint32_t)sa.hull, ta, (uint32_t)sb.hull, tb,
                                   *reinterpret_cast<GjkClipWork<T> *>(ws), m, err);
        }
        else
            single_point(m, r.normal, r.contact, r.depth);
        __syncwarp();
        return true;
    }
} // namespace rbps_gpu
