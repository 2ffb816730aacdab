// gb_step.cuh -- candidate pairs, narrow phase + contact law, and the fused
// per-particle reduction / walls / gravity / integration kernel.
#pragma once

#include "gb_broadphase.cuh"
#include "gb_dem.cuh"

namespace gb
{

// Particle state on the device, structure of arrays.  Positions are FP64 in
// every mode.  Orientation: in the FP64 modes the 3x3 basis of Grains'
// Transform3 (9 arrays, row-major), updated exactly as
// Transform3::composeLeftByRotation; in the mixed mode a unit quaternion
// (w, x, y, z) as a compensated FP32 pair: rot[0..3] hold the FP32 value,
// read by the FP32 bounding tests, and rot[4..7] the FP32 remainder, so that
// hi + lo (read by the FP64 contact geometry) keeps the orientation to FP64
// accuracy (an FP32 quaternion alone rounds a pose by ~6e-8 rad, which moves
// GJK's stopping point on resting contacts).
template <typename St>
struct State
{
    double*   pos[3];
    St*       rot[9]; // basis (FP64 modes) or quaternion hi in rot[0..3], lo in rot[4..7] (mixed)
    St*       vel[3];
    St*       omg[3];
    St*       frc[3];
    St*       trq[3];
    uint32_t* rb_id;
};

template <typename S>
struct Tables
{
    const RBShape<store_t<S>>*   shape;
    const RBInertia<store_t<S>>* inertia;
    const Vert<store_t<S>>*      verts;
    const Law<store_t<S>>*       law; // material-pair table
    const RBShape<store_t<S>>*   obs_shape;
    const double*                obs_tr; // 12 per obstacle (basis, origin)
    const double*                obs_mass;
    const double4*               obs_plane; // Rectangle planes: normal, normal . origin
    const double*                obs_vel;   // 6 per obstacle: velocity, angular velocity
    uint32_t                     obs_rect;  // bit o: obstacle o (< 32) is a Rectangle
    int                          n_obs;
    // FP64 copies of the shape tables (read by the mixed mode's FP64 GJK)
    const RBShape<double>* shape64;
    const Vert<double>*    verts64;
    const RBShape<double>* obs_shape64;
    // FP32 ones, read by the certified FP32 passes of every mode (the mixed
    // mode's own tables; rounded copies in the FP64 modes)
    const RBShape<float>* shape32;
    const Vert<float>*    verts32;
};

// ---- records of the particles that have candidates ------------------------------
// The narrow phase gathers its particles at random ids.  From the
// structure-of-arrays state a particle's pose is seven to twelve 4- and 8-byte
// loads in as many sectors, beside a dozen of its body record; the fill pass,
// which runs over the particles that have candidates anyway, packs what the
// culls read into one aligned record.  Pose: the centre, the body, and what
// the oriented-box test reads in FP32 (the mixed mode's quaternion, the FP64
// modes' basis).  `r` is the bounding radius: negative for a sphere, infinite
// for a pose that the FP32 certificates do not cover (a basis off orthonormal
// by more than 2e-5: its pairs all go to the FP64 solve).
template <typename St>
struct alignas(32) PoseRec // FP64 modes: 96 bytes, three sectors
{
    double   x, y, z;
    uint32_t rb;
    float    r;
    float    R[9];
    float    bb[3];
    float    pad[4];
};
template <>
struct alignas(32) PoseRec<float> // mixed: 64 bytes, two sectors
{
    double   x, y, z;
    uint32_t rb;
    float    r;
    float    q[4];
    float    bb[3];
    float    pad;
};

// Spheres, where every body is one: all that a contact reads of a particle.
template <typename St>
struct alignas(32) SphereRec // 64 bytes mixed, 96 FP64
{
    double   x, y, z, r;
    St       v[3], w[3], mass;
    uint32_t material;
};

// a record in 32-byte loads and stores, a sector each (sm_100's widest)
template <typename T>
GB_D T load_rec(const T* p)
{
    constexpr int kWords = sizeof(T) / 32;
    uint64_t      w[4 * kWords];
#pragma unroll
    for(int k = 0; k < kWords; ++k)
        asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];"
            : "=l"(w[4 * k]), "=l"(w[4 * k + 1]), "=l"(w[4 * k + 2]), "=l"(w[4 * k + 3])
            : "l"(reinterpret_cast<const char*>(p) + 32 * k));
    T t;
    memcpy(&t, w, sizeof(t));
    return t;
}

template <typename T>
GB_D void store_rec(T* p, const T& t)
{
    constexpr int kWords = sizeof(T) / 32;
    uint64_t      w[4 * kWords];
    memcpy(w, &t, sizeof(t));
#pragma unroll
    for(int k = 0; k < kWords; ++k)
        asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(
                         reinterpret_cast<char*>(p) + 32 * k),
                     "l"(w[4 * k]), "l"(w[4 * k + 1]), "l"(w[4 * k + 2]), "l"(w[4 * k + 3])
                     : "memory");
}

// the records' arrays, by particle id; null where the step does not read them
template <typename St>
struct Records
{
    PoseRec<St>*   pose;
    SphereRec<St>* sphere;
};

// ---- mixed precision narrow phase --------------------------------------------
// The bounding-sphere and OBB tests run in FP32 on FP32 poses (their margins
// are absolute: LOWEPS on the OBB axes, the crust-free bounding box), and every
// pair that survives them and that the FP32 stages (GJK's first iteration, the
// FP32 GJK) do not certify as separated is solved by the FP64 GJK of the FP64
// mode, with FP64 shape tables and the compensated quaternion: FP32 support
// points on mm-size grains carry ~1e-10 m of rounding, the order of a resting
// contact's overlap (m g / kn ~ 1e-8 m), so contact points and overlaps come
// from FP64.

GB_D Quat<double> load_quat64(const State<float>& st, uint32_t i)
{
    Quat<double> q;
    q.w = (double)st.rot[0][i] + (double)st.rot[4][i];
    q.v = mk<double>((double)st.rot[1][i] + (double)st.rot[5][i],
                     (double)st.rot[2][i] + (double)st.rot[6][i],
                     (double)st.rot[3][i] + (double)st.rot[7][i]);
    return q;
}

GB_D M3<double> load_rot64(const State<float>& st, uint32_t i)
{
    const Quat<double> q = load_quat64(st, i);
    return quat_to_matrix<double>(q.w, q.v.x, q.v.y, q.v.z);
}

GB_D Contact<float> to_f(const Contact<double>& c)
{
    Contact<float> r;
    r.pt      = cvt3<float>(c.pt);
    r.vec     = cvt3<float>(c.vec);
    r.overlap = (float)c.overlap;
    return r;
}

// closestPointsSpheres (CollisionDetection.cpp:26-48) for the mixed mode:
// the closed form directly in FP64, the point relative to A's centre.
GB_D Contact<float> closest_spheres_mixed(double rA, double rB, const double xa[3],
                                          const double xb[3])
{
    const V3<double> d64 = mk<double>(xb[0] - xa[0], xb[1] - xa[1], xb[2] - xa[2]);
    const double     nd = norm(d64), overlap = nd - rA - rB;
    if(!(overlap < 0.0))
        return no_contact<float>();
    // one FP64 division (the result is rounded to FP32)
    const V3<double> u = (1.0 / nd) * d64;
    Contact<double>  c;
    c.pt      = (rA + 0.5 * overlap) * u;
    c.vec     = overlap * u;
    c.overlap = overlap;
    return to_f(c);
}

// closestPointsRigidBodies for the mixed mode on a lane pair (kGjkPaired; not
// two spheres); points relative to A's centre.  VAR: the GJK variant of the
// FP64 solve; active: the lane has a pair.
template <int VAR>
GB_D Contact<float> closest_mixed(const Tables<float>& tb, const State<float>& st, uint32_t a,
                                  uint32_t b, uint32_t ra, uint32_t rb, const Body<float>& A,
                                  const Body<float>& B, const M3<float>& RA, const M3<float>& RB,
                                  const double xa[3], const double xb[3], int* iters, bool active)
{
    const V3<double> d64 = mk<double>(xb[0] - xa[0], xb[1] - xa[1], xb[2] - xa[2]);
    const V3<float>  d   = cvt3<float>(d64);
    active = active && norm(d) - (A.rcirc + B.rcirc) < 0.0f && obb_overlap(A.bb, B.bb, RA, RB, d);
    // every pair that passes the bounding tests is solved on the FP64 path of
    // the FP64 mode
    const Body<double> A64 = load_body<double>(tb.shape64, ra, tb.verts64);
    const Body<double> B64 = load_body<double>(tb.shape64, rb, tb.verts64);
    const M3<double>   RA64 = load_rot64(st, a), RB64 = load_rot64(st, b);
    Tr<double>         b2a64;
    const M3<double>   RAt64 = transpose(RA64);
    b2a64.R                  = mul(RAt64, RB64);
    b2a64.o                  = mul(RAt64, d64);
    const GjkResult<double> g = gjk<VAR>(A64, B64, b2a64, active);
    *iters += g.iters;
    const double distance = g.dist - (A64.crust + B64.crust);
    if(!active || distance > 0.0)
        return no_contact<float>();
    const V3<double> ptA = mul(RA64, g.pa);
    const V3<double> ptB = mul(RB64, g.pb) + d64;
    Contact<double>  c;
    c.pt      = (ptA + ptB) / 2.0;
    V3<double> vec = ptA - ptB;
    vec            = round3(vec / norm(vec), 1e-10);
    c.vec          = (-distance) * vec;
    c.overlap      = distance;
    return to_f(c);
}

template <typename S>
GB_D constexpr bool is_mixed()
{
    return sizeof(store_t<S>) == 4;
}

template <typename S>
GB_D M3<S> load_rot(const State<store_t<S>>& st, uint32_t i)
{
    if constexpr(is_mixed<S>())
        return quat_to_matrix<S>(S(st.rot[0][i]), S(st.rot[1][i]), S(st.rot[2][i]),
                                 S(st.rot[3][i]));
    else
    {
        M3<S> R;
#pragma unroll
        for(int k = 0; k < 9; ++k)
            R.m[k] = S(st.rot[k][i]);
        return R;
    }
}

template <typename S>
GB_D V3<S> load3(store_t<S>* const a[3], uint32_t i)
{
    return mk<S>(S(a[0][i]), S(a[1][i]), S(a[2][i]));
}

template <typename S>
GB_D Law<S> load_law(const Law<store_t<S>>* t, int ma, int mb)
{
    // ContactForceModelBuilderFactory::computeHash (ContactForceModelBuilderFactory.cpp:77-83)
    const unsigned s = ma < mb ? ma : mb, l = ma < mb ? mb : ma;
    const Law<store_t<S>> L = t[l * (l + 1) / 2 + s];
    Law<S>                r;
    r.kn   = S(L.kn);
    r.muen = S(L.muen);
    r.etat = S(L.etat);
    r.muc  = S(L.muc);
    r.kr   = S(L.kr);
    r.kt   = S(L.kt);
    return r;
}

// ---- candidate pairs ----------------------------------------------------------
// One thread per particle in cell-sorted order.  Enumerates the 27 neighbour
// cells in the reference's order (k = z outer, j = y, i = x inner; the
// neighbour table of LinkedCell.cpp:41-70) and the particles of each cell in
// ascending id, keeping ordered pairs (A, B != A) whose bounding spheres
// overlap: norm(xB - xA) - (rA + rB) < 0 (CollisionDetection.cpp:209-211).
// The three cells x-1, x, x+1 of one (y, z) row have consecutive keys, so
// their particles are one contiguous range of the sorted order: the walk is
// nine ranges, visiting the candidates in the same order as the 27 cells.
// A conservative FP32 test on spos32 (put_sorted inflates its radii by a bound
// on the FP32 rounding, so an FP32 rejection implies an FP64 rejection) skips
// most non-candidates before the FP64 test, in every mode: the candidate set
// is the FP64 test's.
// Candidates kept per particle by the count pass: 32 covers all but ~1e-4 of
// the particles of a dense polydisperse bed (mean ~7, 99.9th percentile ~25);
// the fill pass enumerates the rest again.
constexpr int kPairSlots = 32;

// Particle-obstacle pairs (ComponentManagerCPU.cpp:301-351) share the pair
// list: after the particle pairs of A come A's obstacle candidates in obstacle
// order, as b = kObstacleBit | o, so that the segmented sum adds the obstacle
// forces after the particle forces, in the reference's order.
constexpr uint32_t kObstacleBit     = 0x80000000u;
constexpr uint8_t  kContactParticle = 1; // contact flags of a pair record
constexpr uint8_t  kContactObstacle = 2;
constexpr int      kMaskObstacles   = 32; // obstacles beyond these are always candidates

// Frame of obstacle o for particle A at xa: A's centre oA and the obstacle's
// origin oO (relative to xa in the mixed mode, absolute in the FP64 modes).
template <typename S>
GB_D void obstacle_frame(const Tables<S>& tb, int o, const double xa[3], V3<S>& oA, V3<S>& oO,
                         M3<S>& RO)
{
    const double* ot = tb.obs_tr + 12 * o;
    if constexpr(is_mixed<S>())
    {
        oA = zero3<S>();
        oO = mk<S>(S(ot[9] - xa[0]), S(ot[10] - xa[1]), S(ot[11] - xa[2]));
    }
    else
    {
        oA = mk<S>(S(xa[0]), S(xa[1]), S(xa[2]));
        oO = mk<S>(S(ot[9]), S(ot[10]), S(ot[11]));
    }
#pragma unroll
    for(int k = 0; k < 9; ++k)
        RO.m[k] = S(ot[k]);
}

// Obstacles that particle a may touch, bit o for obstacle o < kMaskObstacles.
// A lies in its bounding box (half extents bb), so its support point towards
// a Rectangle's plane is at most bb . |RA^T n| from its centre: a centre
// farther than that from the plane (plus a bound on the rounding of both
// sides) cannot touch it, and the full test of closest_rectangle would reject
// it too.  Other obstacle types are always candidates.
// The box's extent along any unit normal is at most |bb| (Cauchy-Schwarz), so
// a centre farther than |bb| from every plane is decided without the
// rotation: `rot` (a callable returning RA) runs only for the planes within
// that reach.
template <typename S, typename Rot>
GB_D uint32_t obstacle_mask_at(const Tables<S>& tb, uint32_t r, Rot&& rot, const double xa[3])
{
    const int nm = tb.n_obs < kMaskObstacles ? tb.n_obs : kMaskObstacles;
    if(nm == 0)
        return 0u;
    // in FP64 throughout: the plane distance from the exact centre, the box
    // extent along the normal from this mode's rotation; the slack covers the
    // rounding of both and the 1e-7 difference between the mixed mode's FP32
    // rotation and the FP64 one its contact recomputation uses
    const double bb[3] = {(double)tb.inertia[r].bb[0], (double)tb.inertia[r].bb[1],
                          (double)tb.inertia[r].bb[2]};
    const double ax    = fabs(xa[0]) + fabs(xa[1]) + fabs(xa[2]);
    uint32_t     mask  = ~tb.obs_rect & ((nm == 32) ? ~0u : ((1u << nm) - 1u));
    const double reach = sqrt(bb[0] * bb[0] + bb[1] * bb[1] + bb[2] * bb[2]);
    bool         have  = false;
    M3<S>        RA;
    for(int o = 0; o < nm; ++o)
    {
        if(!((tb.obs_rect >> o) & 1u))
            continue;
        const double4 pl = tb.obs_plane[o];
        const double  dc = fabs(pl.x * xa[0] + pl.y * xa[1] + pl.z * xa[2] - pl.w);
        if(dc - reach > 1e-6 * reach + 1e-12 * (1.0 + ax + fabs(pl.w)))
            continue; // beyond the box's reach whatever its orientation
        if(!have)
        {
            RA   = rot();
            have = true;
        }
        double hb, slack;
        if constexpr(is_mixed<S>())
        {
            // the extent from the FP32 rotation in FP32: each |(RA^T n)_k|
            // is off by a few 1e-7 (its rounding, and the FP32 rotation's
            // distance from the FP64 one), so the slack takes 1e-6 of the
            // box's half-extents' sum
            const float n32[3] = {(float)pl.x, (float)pl.y, (float)pl.z};
            float       h32    = 0.0f;
#pragma unroll
            for(int k = 0; k < 3; ++k)
                h32 += (float)bb[k]
                       * fabsf(RA.m[k] * n32[0] + RA.m[3 + k] * n32[1] + RA.m[6 + k] * n32[2]);
            hb    = (double)h32;
            slack = 1e-6 * (bb[0] + bb[1] + bb[2]) + 1e-12 * (1.0 + ax + fabs(pl.w));
        }
        else
        {
            hb = 0.0;
#pragma unroll
            for(int k = 0; k < 3; ++k)
            {
                // (RA^T n)_k = sum_j RA[j][k] n_j
                const double nk = to_d(RA.m[k]) * pl.x + to_d(RA.m[3 + k]) * pl.y
                                  + to_d(RA.m[6 + k]) * pl.z;
                hb += bb[k] * fabs(nk);
            }
            slack = 1e-6 * hb + 1e-12 * (1.0 + ax + fabs(pl.w));
        }
        if(!(dc - hb > slack))
            mask |= 1u << o;
    }
    return mask;
}

// The mask is computed where the pose is at hand: by k_particles right after
// each move, and by k_obstacle_mask after the state was set from the host.
template <typename S>
__global__ void __launch_bounds__(kBlock)
    k_obstacle_mask(int n, State<store_t<S>> st, Tables<S> tb, uint32_t* __restrict__ mask)
{
    grid_dep_sync();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n)
        return;
    const double xa[3] = {st.pos[0][i], st.pos[1][i], st.pos[2][i]};
    mask[i] = obstacle_mask_at<S>(tb, st.rb_id[i], [&] { return load_rot<S>(st, i); }, xa);
}

// A particle's obstacle candidates, in ascending obstacle order (the order of
// the reference's obstacle loop, ComponentManagerCPU.cpp:301-351).  The
// Rectangles among the first kMaskObstacles are decided by the particle's
// mask (walls within reach after the last move); every other obstacle comes
// from its linked cell's list -- the obstacles whose surface a particle of
// that cell may reach, binned on the host when the obstacles are set.
// Without lists (every obstacle a Rectangle among the first 32, or none) the
// mask decides alone; its bits of the other first-32 obstacles are set.
struct ObsCand
{
    const uint32_t* mask;       // by particle id
    int             n;          // obstacles
    uint32_t        rect;       // bit o: obstacle o (< 32) is a Rectangle
    const uint32_t* cell_start; // C + 1 offsets into cell_ids, by linked cell (or null)
    const uint32_t* cell_ids;   // the listed obstacles, ascending per cell
    const uint32_t* skeys;      // linked-cell key by sorted position
};

GB_D int obstacle_candidates(const ObsCand& oc, uint32_t a, uint32_t s)
{
    if(!oc.n)
        return 0;
    if(oc.cell_start)
    {
        const uint32_t key = oc.skeys[s];
        return __popc(oc.mask[a] & oc.rect) + (int)(oc.cell_start[key + 1] - oc.cell_start[key]);
    }
    return __popc(oc.mask[a]) + (oc.n > kMaskObstacles ? oc.n - kMaskObstacles : 0);
}

template <typename Visit>
GB_D void for_each_obstacle_candidate(const ObsCand& oc, uint32_t a, uint32_t s, Visit&& visit)
{
    if(!oc.n)
        return;
    uint32_t mask = oc.mask[a];
    if(oc.cell_start)
    {
        // the mask's Rectangles merged into the cell's list, both ascending
        mask &= oc.rect;
        const uint32_t key = oc.skeys[s];
        for(uint32_t k = oc.cell_start[key]; k < oc.cell_start[key + 1]; ++k)
        {
            const uint32_t o = oc.cell_ids[k];
            while(mask && (uint32_t)(__ffs(mask) - 1) < o)
            {
                visit((uint32_t)(__ffs(mask) - 1));
                mask &= mask - 1u;
            }
            visit(o);
        }
        for(; mask; mask &= mask - 1u)
            visit((uint32_t)(__ffs(mask) - 1));
        return;
    }
    const int nm = oc.n < kMaskObstacles ? oc.n : kMaskObstacles;
    for(int o = 0; o < nm; ++o)
        if((mask >> o) & 1u)
            visit((uint32_t)o);
    for(int o = kMaskObstacles; o < oc.n; ++o)
        visit((uint32_t)o);
}

template <typename S>
GB_D constexpr bool is_strict()
{
    return std::is_same<S, dstrict>::value;
}

// The candidate test of sorted particles a and b: |d| - (rA + rB) < 0 in
// FP64 (ComponentManagerCPU.cpp:372-380; the strict mode in the reference's
// operation order), behind the FP32 pre-test, whose rejection is certified
// (put_sorted inflates the FP32 radii).  The
// products and sums are written as explicit round-to-nearest operations, so
// that every kernel that enumerates candidates -- the count pass and the
// re-enumeration of the fill pass -- takes the same decisions.
GB_D bool pretest_rejects(const float4& a32, const float4& q)
{
    const float fx = __fsub_rn(q.x, a32.x), fy = __fsub_rn(q.y, a32.y);
    const float fz = __fsub_rn(q.z, a32.z), fr = __fadd_rn(a32.w, q.w);
    return __fmaf_rn(fz, fz, __fmaf_rn(fy, fy, __fmul_rn(fx, fx))) >= __fmul_rn(fr, fr);
}

template <bool STRICT>
GB_D bool exact_hit(const double4& pa, const double4& pb)
{
    if constexpr(STRICT)
    {
        const dstrict dx = dstrict(pb.x) - dstrict(pa.x);
        const dstrict dy = dstrict(pb.y) - dstrict(pa.y);
        const dstrict dz = dstrict(pb.z) - dstrict(pa.z);
        return s_sqrt(dx * dx + dy * dy + dz * dz) - (dstrict(pa.w) + dstrict(pb.w))
               < dstrict(0.0);
    }
    else
    {
        const double dx = __dsub_rn(pb.x, pa.x), dy = __dsub_rn(pb.y, pa.y);
        const double dz = __dsub_rn(pb.z, pa.z), r = __dadd_rn(pa.w, pb.w);
        return __fma_rn(dz, dz, __fma_rn(dy, dy, __dmul_rn(dx, dx))) < __dmul_rn(r, r);
    }
}

// The 27 neighbour cells of cell (cx, cy, cz) in the reference's enumeration
// order (LinkedCell.cpp:66-112, k then j then i) are 9 rows of up to 3 cells;
// the cells of a row are consecutive keys, so each row is one contiguous
// range [begin, end) of sorted positions.
GB_D void neighbour_row(const uint32_t* __restrict__ cstart, uint32_t nx, uint32_t ny, uint32_t nz,
                        int cx, int cy, int cz, int r, uint32_t& begin, uint32_t& end)
{
    const int z = cz + r / 3 - 1, y = cy + r % 3 - 1;
    begin = end = 0;
    if(z < 0 || z >= (int)nz || y < 0 || y >= (int)ny)
        return;
    const int      x0  = cx > 0 ? cx - 1 : 0, x1 = cx + 1 < (int)nx ? cx + 1 : cx;
    const uint32_t row = ((uint32_t)z * ny + (uint32_t)y) * nx;
    begin              = cstart[row + (uint32_t)x0];
    end                = cstart[row + (uint32_t)x1 + 1];
}

// Count pass over half of the stencil, five threads per sorted particle s,
// one per row.  The candidate test is symmetric bit for bit (b - a is
// -(a - b) exactly, and the radius sum commutes), so each unordered pair is
// tested once: by s for the partners t after it in the stencil's enumeration
// order -- the rest of its own row (the cells x, x + 1 of row (dz, dy) =
// (0, 0) from s + 1 on, one contiguous range) and the 4 rows (0, +1),
// (+1, -1), (+1, 0), (+1, +1).  A hit is recorded for both particles
// (record_candidate): pcount[id] (zeroed) counts by one atomic, whose result
// is the partner's slot, and the first kPairSlots partners go to the id's
// slots in arrival order.  The enumeration order of a particle's candidates
// is ascending sorted position (rows ascend in (z, y), cells in x, ids within
// a cell), so the fill pass restores it by sorting the slots.  Obstacle
// candidates are counted in obs_count[id] by the particle's own-row thread;
// the scan adds the two.
//
// The rows are walked by threads of their own because the walk is a chain of
// dependent loads (row bounds, then candidates): one thread per particle
// waited through five chains in turn, and a small packing left the chip idle
// (12k spheres 32 -> 14 us a launch).
//
// The FP32 test passes one candidate in some 5 to 15, so in nearly every round
// a few lanes of a warp have a hit; tested and recorded where they are found,
// the FP64 test and the two atomics ran in nearly every round for those few
// lanes and were most of the instructions.  The hits of a warp are queued in
// shared memory instead and taken 32 at a time (1M bed: fine-grid count 252 ->
// 164 us, large grains 162 -> 67 us; 1M spheres' count 112 -> 90 us).

// Candidate v (a sorted position) of particle id u: its slot and the count.
GB_D void record_candidate(uint32_t id_u, uint32_t v, uint32_t* __restrict__ pcount,
                           uint32_t* __restrict__ slot)
{
    const uint32_t k = atomicAdd(pcount + id_u, 1u);
    if(k < kPairSlots)
        slot[(size_t)id_u * kPairSlots + k] = v;
}

// A warp's FP32 hits (s, t): at most 31 left over and two rounds of 32.
struct HitQueue
{
    uint32_t s[96], t[96];
};

GB_D void push_hit(HitQueue& q, unsigned& n, bool hit, uint32_t s, uint32_t t)
{
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    if(hit)
    {
        const unsigned k = n + __popc(m & ((1u << (threadIdx.x & 31u)) - 1u));
        q.s[k]           = s;
        q.t[k]           = t;
    }
    n += __popc(m);
}

// record(s, t) for the queued hits that the FP64 test keeps, while a whole
// round of them is queued, or all of them (`flush`)
template <bool STRICT, typename Record>
GB_D void take_hits(HitQueue& q, unsigned& n, bool flush, const double4* __restrict__ pos,
                    Record&& record)
{
    while(n >= 32u || (flush && n))
    {
        const unsigned lane = threadIdx.x & 31u, k = n < 32u ? n : 32u;
        n -= k;
        __syncwarp();
        if(lane < k)
        {
            const uint32_t s = q.s[n + lane], t = q.t[n + lane];
            if(exact_hit<STRICT>(pos[s], pos[t]))
                record(s, t);
        }
        __syncwarp();
    }
}

// A warp walks its lanes' candidate ranges [t0, t1) of the lanes' particles s
// (an empty range on the lanes without one).
template <bool STRICT, typename Record>
GB_D void walk_rows(uint32_t s, uint32_t t0, uint32_t t1, const double4* __restrict__ pos,
                    const float4* __restrict__ pos32, HitQueue& q, Record&& record)
{
    const uint32_t len    = t1 > t0 ? t1 - t0 : 0u;
    const uint32_t rounds = __reduce_max_sync(0xffffffffu, len);
    if(!rounds)
        return;
    const float4 a32 = len ? pos32[s] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    unsigned     n   = 0; // queued hits, warp-uniform
    for(uint32_t k = 0; k < rounds; k += 2)
    {
        const bool h0 = k < len && !pretest_rejects(a32, pos32[t0 + k]);
        const bool h1 = k + 1 < len && !pretest_rejects(a32, pos32[t0 + k + 1]);
        if(__any_sync(0xffffffffu, h0 || h1))
        {
            push_hit(q, n, h0, s, t0 + k);
            push_hit(q, n, h1, s, t0 + k + 1);
        }
        take_hits<STRICT>(q, n, k + 2 >= rounds, pos, record);
    }
}

constexpr int kHalfRows = 5; // the rows of the half stencil, one thread each

template <bool STRICT>
__global__ void __launch_bounds__(kBlock, 8)
    k_pair_count(int n, const uint32_t* __restrict__ skeys, const uint32_t* __restrict__ sids,
                 const double4* __restrict__ spos, const float4* __restrict__ spos32,
                 const uint32_t* __restrict__ cstart, uint32_t nx, uint32_t ny, uint32_t nz,
                 uint32_t* __restrict__ obs_count, uint32_t* __restrict__ pcount,
                 uint32_t* __restrict__ slot, ObsCand oc, const int* abort_flags)
{
    grid_dep_sync();
    __shared__ HitQueue s_hits[kWarps];
    const int           r = 4 + (int)(blockIdx.x % kHalfRows); // row r of the 3 x 3 (dz, dy)
    const int           s = (int)(blockIdx.x / kHalfRows * blockDim.x + threadIdx.x);
    if(step_aborted(abort_flags))
        return;
    uint32_t t0 = 0, t1 = 0;
    if(s < n)
    {
        if(oc.n && r == 4)
        {
            const uint32_t a   = sids[s];
            const int      obs = obstacle_candidates(oc, a, (uint32_t)s);
            if(obs)
                obs_count[a] = (uint32_t)obs;
        }
        const uint32_t key = skeys[s];
        const int      cx = key % nx, cy = (key / nx) % ny, cz = key / (nx * ny);
        neighbour_row(cstart, nx, ny, nz, cx, cy, cz, r, t0, t1);
        if(r == 4)
            t0 = (uint32_t)s + 1;
    }
    walk_rows<STRICT>((uint32_t)s, t0, t1, spos, spos32, s_hits[threadIdx.x >> 5],
                      [&](uint32_t u, uint32_t v) {
                          record_candidate(sids[u], v, pcount, slot);
                          record_candidate(sids[v], u, pcount, slot);
                      });
}

// A warp walks the concatenation of up to 32 ranges [t0, t1) of sorted
// positions, lane r holding range r (lanes past the last range hold empty
// ones), ROUNDS x 32 entries at a time in range order: visit(t, valid) with
// the lane's ROUNDS entries (entry k of a lane is the k-th group of 32's) runs
// on every lane (warp-uniform).  All ranges' bounds are loaded at once, by
// their lanes, and short ranges share rounds, where a range-at-a-time walk
// pays a dependent load pair and a mostly idle round per range.  More rounds
// at a time put more loads in flight where a warp works alone.
template <int ROUNDS, typename Visit>
GB_D void warp_ranges(uint32_t t0, uint32_t t1, Visit&& visit)
{
    const unsigned lane = threadIdx.x & 31u;
    const uint32_t len  = t1 > t0 ? t1 - t0 : 0u;
    uint32_t       inc  = len; // inclusive prefix of the lengths
#pragma unroll
    for(int o = 1; o < 32; o <<= 1)
    {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if(lane >= (unsigned)o)
            inc += y;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, inc, 31);
    const uint32_t exc   = inc - len;
    for(uint32_t base = 0; base < total; base += 32 * ROUNDS)
    {
        uint32_t t[ROUNDS];
        bool     valid[ROUNDS];
#pragma unroll
        for(int k = 0; k < ROUNDS; ++k)
        {
            const uint32_t idx = base + 32u * k + lane;
            // the last range that starts at or before idx (exclusive prefixes
            // do not decrease; an empty range shares its start with the next)
            unsigned r = 0;
#pragma unroll
            for(unsigned step = 16; step >= 1; step >>= 1)
                if(__shfl_sync(0xffffffffu, exc, r + step) <= idx)
                    r += step;
            t[k] = __shfl_sync(0xffffffffu, t0, r) + (idx - __shfl_sync(0xffffffffu, exc, r));
            valid[k] = idx < total;
        }
        visit(t, valid);
    }
}

// ---- candidate search on a finer grid (polydisperse packings) -----------------
// The reference's cell is twice the LARGEST bounding radius, so in a
// polydisperse packing a particle's 27 cells hold hundreds of others (~960 in
// the 2.2 mm bed of 0.5-2 mm grains, 7.2 mm cells).  The same candidate set
// is found with far fewer tests on a second grid of cell h >= 2 r_s, r_s a
// bounding radius that most particles do not exceed ("small"; the others are
// "large"):
//   small-small pairs: |d| < rA + rB <= 2 r_s <= h, adjacent fine cells --
//     the half stencil of k_pair_count on the fine grid (k_pair_count_fine);
//   small-large pairs: the large particle scans the fine cells within its
//     reach rL + r_s (k_pair_count_large, one warp per large particle);
//   large-large pairs: the large particle scans the fine cells within its
//     reach rL + r_max for large partners after it in the fine order.
// Each unordered pair is tested once, with the same symmetric test
// (pretest_rejects + exact_hit), and recorded for both particles into the
// same slots and counts as k_pair_count (the partner by its reference sorted
// position): the fill pass's sort restores the reference's order, so the
// pair list is the same, bit for bit.  A large particle's key is its
// fine cell plus nf (the fine cell count): the fine order holds the small
// particles by cell, then the large ones by cell.
struct FineGrid
{
    double   mn[3];
    double   h;    // fine cell edge
    double   rs;   // the small particles' bounding-radius limit
    double   rmax; // the largest bounding radius
    uint32_t nx, ny, nz;
};

GB_D uint32_t fine_axis(double x, double mn, double h, uint32_t n)
{
    const double f = (x - mn) / h; // NaN falls to cell 0
    return f >= 0.0 ? (f < (double)n ? (uint32_t)f : n - 1u) : 0u;
}

__global__ void __launch_bounds__(kBlock)
    k_fine_hash(int n, const double* __restrict__ px, const double* __restrict__ py,
                const double* __restrict__ pz, const uint32_t* __restrict__ rb_id,
                const double* __restrict__ rcirc, FineGrid g, uint32_t* __restrict__ fkey,
                uint32_t* __restrict__ fcount, const int* abort_flags)
{
    grid_dep_sync();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n || step_aborted(abort_flags))
        return;
    uint32_t key = (fine_axis(pz[i], g.mn[2], g.h, g.nz) * g.ny + fine_axis(py[i], g.mn[1], g.h, g.ny))
                       * g.nx
                   + fine_axis(px[i], g.mn[0], g.h, g.nx);
    if(rcirc[rb_id[i]] > g.rs)
        key += g.nx * g.ny * g.nz; // the large particles' cells
    fkey[i] = key;
    atomicAdd(&fcount[key], 1u);
}

// each particle into a free slot of its fine cell (any order within a cell:
// the fill pass sorts), with its key, id, reference sorted position and
// positions (put_sorted); leaves the counts at zero
__global__ void __launch_bounds__(kBlock)
    k_fine_scatter(int n, const uint32_t* __restrict__ fkey, const uint32_t* __restrict__ fstart,
                   uint32_t* __restrict__ fcount, const double* __restrict__ px,
                   const double* __restrict__ py, const double* __restrict__ pz,
                   const uint32_t* __restrict__ rb_id, const double* __restrict__ rcirc,
                   const uint32_t* __restrict__ sorted_of, uint32_t* __restrict__ fskey,
                   uint32_t* __restrict__ fids, uint32_t* __restrict__ fref,
                   double4* __restrict__ fpos, float4* __restrict__ fpos32, const int* abort_flags)
{
    grid_dep_sync();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n || step_aborted(abort_flags))
        return;
    const uint32_t key  = fkey[i];
    const uint32_t slot = fstart[key] + atomicSub(&fcount[key], 1u) - 1u;
    fskey[slot]         = key;
    fids[slot]          = (uint32_t)i;
    fref[slot]          = sorted_of[i];
    put_sorted(slot, (uint32_t)i, px, py, pz, rb_id, rcirc, fpos, fpos32);
}

// small particles: k_pair_count's half stencil on the fine grid (whose cells
// hold small particles only); a thread per row of a fine sorted position
template <bool STRICT>
__global__ void __launch_bounds__(kBlock, 8)
    k_pair_count_fine(int n, const uint32_t* __restrict__ fstart, FineGrid g,
                      const uint32_t* __restrict__ fskey, const uint32_t* __restrict__ fids,
                      const uint32_t* __restrict__ fref, const double4* __restrict__ fpos,
                      const float4* __restrict__ fpos32, uint32_t* __restrict__ obs_count,
                      uint32_t* __restrict__ pcount, uint32_t* __restrict__ slot,
                      ObsCand oc, const int* abort_flags)
{
    grid_dep_sync();
    __shared__ HitQueue s_hits[kWarps];
    const int           r = 4 + (int)(blockIdx.x % kHalfRows);
    const int           f = (int)(blockIdx.x / kHalfRows * blockDim.x + threadIdx.x);
    if(step_aborted(abort_flags))
        return;
    uint32_t t0 = 0, t1 = 0;
    if(f < n && (uint32_t)f < fstart[g.nx * g.ny * g.nz])
    {
        if(oc.n && r == 4)
        {
            const int obs = obstacle_candidates(oc, fids[f], fref[f]);
            if(obs)
                obs_count[fids[f]] = (uint32_t)obs;
        }
        const uint32_t key = fskey[f];
        const int cx = key % g.nx, cy = (key / g.nx) % g.ny, cz = key / (g.nx * g.ny);
        neighbour_row(fstart, g.nx, g.ny, g.nz, cx, cy, cz, r, t0, t1);
        if(r == 4)
            t0 = (uint32_t)f + 1;
    }
    walk_rows<STRICT>((uint32_t)f, t0, t1, fpos, fpos32, s_hits[threadIdx.x >> 5],
                      [&](uint32_t u, uint32_t v) {
                          record_candidate(fids[u], fref[v], pcount, slot);
                          record_candidate(fids[v], fref[u], pcount, slot);
                      });
}

// large particles (keys past the small ones'), one warp each: small partners
// from the fine cells within reach rL + r_s, then large partners after it in
// the fine order from the large particles' cells within reach rL + r_max
template <bool STRICT>
__global__ void __launch_bounds__(kBlock)
    k_pair_count_large(int n, const uint32_t* __restrict__ fstart, FineGrid g,
                       const uint32_t* __restrict__ fids, const uint32_t* __restrict__ fref,
                       const double4* __restrict__ fpos, const float4* __restrict__ fpos32,
                       uint32_t* __restrict__ obs_count, uint32_t* __restrict__ pcount,
                       uint32_t* __restrict__ slot, ObsCand oc, const int* abort_flags)
{
    grid_dep_sync();
    __shared__ HitQueue s_hits[kWarps];
    HitQueue&           hits  = s_hits[threadIdx.x >> 5];
    unsigned            nhits = 0;
    const unsigned lane = threadIdx.x & 31u;
    const uint32_t nf   = g.nx * g.ny * g.nz;
    const int64_t  f    = (int64_t)fstart[nf] + ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    if(f >= n || step_aborted(abort_flags)) // warp-uniform
        return;
    const uint32_t a = fids[f], sa = fref[f];
    if(oc.n && lane == 0)
    {
        const int obs = obstacle_candidates(oc, a, sa);
        if(obs)
            obs_count[a] = (uint32_t)obs;
    }
    const double4 pa = fpos[f];
    const float4  pa32 = fpos32[f];
    auto          record = [&](uint32_t u, uint32_t v) {
        record_candidate(fids[u], fref[v], pcount, slot);
        record_candidate(fids[v], fref[u], pcount, slot);
    };
    for(int large = 0; large < 2; ++large)
    {
        // the fine cells of the box [x - reach, x + reach]
        const double   reach = (pa.w + (large ? g.rmax : g.rs)) * (1.0 + 1e-6) + 1e-6 * g.h;
        const uint32_t base  = large ? nf : 0u;
        const uint32_t x0    = fine_axis(pa.x - reach, g.mn[0], g.h, g.nx);
        const uint32_t x1    = fine_axis(pa.x + reach, g.mn[0], g.h, g.nx);
        const uint32_t y0    = fine_axis(pa.y - reach, g.mn[1], g.h, g.ny);
        const uint32_t y1    = fine_axis(pa.y + reach, g.mn[1], g.h, g.ny);
        const uint32_t z0    = fine_axis(pa.z - reach, g.mn[2], g.h, g.nz);
        const uint32_t z1    = fine_axis(pa.z + reach, g.mn[2], g.h, g.nz);
        // the rows (z, y) of the box, 32 at a time, lane i holding row i of
        // the chunk, walked as one sequence
        const uint32_t wy = y1 - y0 + 1, rows = (z1 - z0 + 1) * wy;
        for(uint32_t c0 = 0; c0 < rows; c0 += 32)
        {
            uint32_t t0 = 0, t1 = 0;
            if(c0 + lane < rows)
            {
                const uint32_t z   = z0 + (c0 + lane) / wy, y = y0 + (c0 + lane) % wy;
                const uint32_t row = base + (z * g.ny + y) * g.nx;
                t0                 = fstart[row + x0];
                t1                 = fstart[row + x1 + 1];
                if(large && t0 < (uint32_t)f + 1)
                    t0 = (uint32_t)f + 1; // each large pair once
            }
            warp_ranges<2>(t0, t1, [&](const uint32_t(&t)[2], const bool(&valid)[2]) {
                const bool h0 = valid[0] && !pretest_rejects(pa32, fpos32[t[0]]);
                const bool h1 = valid[1] && !pretest_rejects(pa32, fpos32[t[1]]);
                push_hit(hits, nhits, h0, (uint32_t)f, t[0]);
                push_hit(hits, nhits, h1, (uint32_t)f, t[1]);
                take_hits<STRICT>(hits, nhits, false, fpos, record);
            });
        }
    }
    take_hits<STRICT>(hits, nhits, true, fpos, record);
}

// Ascending sort of t[0, N) in registers by a bitonic network (Batcher, 1968):
// every index is a compile-time constant once unrolled.
template <int N, int M>
GB_D void bitonic_sort(uint32_t (&t)[M])
{
    static_assert(N <= M && (N & (N - 1)) == 0, "a power of two within the array");
#pragma unroll
    for(int k = 2; k <= N; k <<= 1)
#pragma unroll
        for(int j = k >> 1; j > 0; j >>= 1)
#pragma unroll
            for(int i = 0; i < N; ++i)
            {
                const int l = i ^ j;
                if(l > i)
                {
                    const uint32_t x = t[i], y = t[l];
                    const uint32_t lo = min(x, y), hi = max(x, y);
                    const bool     up = (i & k) == 0;
                    t[i]              = up ? lo : hi;
                    t[l]              = up ? hi : lo;
                }
            }
}

// Particle a's pose or sphere record (Records).
template <typename S>
GB_D void write_records(uint32_t a, const State<store_t<S>>& st, const Tables<S>& tb,
                        const Records<store_t<S>>& rec)
{
    using St          = store_t<S>;
    const uint32_t rb = st.rb_id[a];
    if(rec.sphere)
    {
        SphereRec<St> o;
        o.x = st.pos[0][a];
        o.y = st.pos[1][a];
        o.z = st.pos[2][a];
        o.r = tb.shape64[rb].p[0];
#pragma unroll
        for(int k = 0; k < 3; ++k)
        {
            o.v[k] = st.vel[k][a];
            o.w[k] = st.omg[k][a];
        }
        o.mass     = tb.inertia[rb].mass;
        o.material = (uint32_t)tb.shape[rb].material;
        store_rec(rec.sphere + a, o);
    }
    if(rec.pose)
    {
        const RBShape<float>& sh = tb.shape32[rb];
        PoseRec<St>           o;
        o.x  = st.pos[0][a];
        o.y  = st.pos[1][a];
        o.z  = st.pos[2][a];
        o.rb = rb;
        o.r  = sh.type == GB_SPHERE ? -sh.rcirc : sh.rcirc;
        if constexpr(is_mixed<S>())
        {
#pragma unroll
            for(int k = 0; k < 4; ++k)
                o.q[k] = st.rot[k][a];
        }
        else
        {
#pragma unroll
            for(int k = 0; k < 9; ++k)
                o.R[k] = (float)st.rot[k][a];
            // the certificates hold for both orders of a pair, whose frames
            // agree only as far as the bases are rotations
            bool ok = true;
#pragma unroll
            for(int i = 0; i < 3; ++i)
#pragma unroll
                for(int j = i; j < 3; ++j)
                {
                    const float g = o.R[3 * i] * o.R[3 * j] + o.R[3 * i + 1] * o.R[3 * j + 1]
                                    + o.R[3 * i + 2] * o.R[3 * j + 2];
                    ok = ok && fabsf(g - (i == j ? 1.0f : 0.0f)) < 2e-5f;
                }
            if(!ok && sh.type != GB_SPHERE)
                o.r = INFINITY;
        }
#pragma unroll
        for(int k = 0; k < 3; ++k)
            o.bb[k] = sh.bb[k];
        store_rec(rec.pose + a, o);
    }
}

// Fill pass, one thread per particle id a (most have no candidate and read
// only its two counts): the pair records of a at offset[a] -- its particle
// candidates from its slots, sorted ascending (the enumeration order), or
// enumerated again in order when there were more than kPairSlots -- then its
// obstacle candidates.  Every record's
// contact flag starts at 0, so that the narrow phase writes the records of
// contacts only (outputs are read where the flag is set).  A warp's particles
// have consecutive ids and so nearly consecutive records: their sorted slots
// are staged in shared memory and written out together, consecutive records
// by consecutive lanes, where each lane writing its own few records cost a
// partial sector per lane and array (1M bed 114 -> 74 us a launch).
template <typename S>
__global__ void __launch_bounds__(kBlock)
    k_pair_fill(int n, const uint32_t* __restrict__ sids, const uint32_t* __restrict__ sorted_of,
                uint32_t* __restrict__ obs_count, uint32_t* __restrict__ pcount,
                const uint32_t* __restrict__ slot, ObsCand oc,
                const uint32_t* __restrict__ offset, uint32_t* __restrict__ pair_a,
                uint32_t* __restrict__ pair_b, int64_t cap, int* __restrict__ flags,
                uint32_t* __restrict__ gjk_count, uint32_t* __restrict__ ovf_list, int ovf_phase,
                uint32_t* __restrict__ obs_queue, uint8_t* __restrict__ contact,
                State<store_t<S>> st, Tables<S> tb, Records<store_t<S>> rec)
{
    grid_dep_sync();
    __shared__ uint32_t s_partner[kWarps][32 * kPairSlots]; // sorted positions ...
    __shared__ uint8_t  s_owner[kWarps][32 * kPairSlots];   // ... and the lane they belong to
    const int           a = blockIdx.x * blockDim.x + threadIdx.x;
    if(a == 0)
    {
        // the narrow phase's GJK queues of this step start empty: [0] the
        // cull pass's, [1] the FP32 stage's; [2 + phase] counts
        // this step's overflowing particles and [4 + phase] its obstacle
        // records, [3 - phase] and [5 - phase] (last step's, read by its
        // overflow and obstacle passes) start the next step at zero
        gjk_count[0]             = 0;
        gjk_count[1]             = 0;
        gjk_count[3 - ovf_phase] = 0;
        gjk_count[5 - ovf_phase] = 0;
    }
    // (this pass sets the capacity flag itself, so the lanes of a warp may read
    // it apart: one answer for all of them, who go on together from here)
    if(__any_sync(0xffffffffu, step_aborted(flags)))
        return;
    const unsigned lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    uint32_t       cp = a < n ? pcount[a] : 0u, k_obs = a < n && oc.n ? obs_count[a] : 0u;
    if(!__any_sync(0xffffffffu, cp + k_obs))
        return;
    int64_t out = cp + k_obs ? offset[a] : 0;
    if(out + cp + k_obs > cap)
    {
        atomicOr(flags, kFlagCapacity);
        cp = k_obs = 0u;
    }
    // the count pass's counters start the next step at zero (an aborted step
    // leaves them for the host's memset before its replay)
    if(cp)
        pcount[a] = 0u;
    if(k_obs)
        obs_count[a] = 0u;
    const uint32_t m    = cp <= kPairSlots ? cp : 0u;
    const uint32_t wmax = __reduce_max_sync(0xffffffffu, m);
    if(wmax)
    {
        // the slots in registers (unused ones as 0xffffffff, above every
        // sorted position), sorted with static indices only, so nothing goes
        // to local memory
        const uint4* mine = reinterpret_cast<const uint4*>(slot + (size_t)a * kPairSlots);
        uint32_t     t[kPairSlots];
#pragma unroll
        for(int q = 0; q < kPairSlots / 4; ++q)
        {
            uint4 x = make_uint4(~0u, ~0u, ~0u, ~0u);
            if((uint32_t)(4 * q) < m)
                x = mine[q];
            t[4 * q]     = (uint32_t)(4 * q) < m ? x.x : ~0u;
            t[4 * q + 1] = (uint32_t)(4 * q + 1) < m ? x.y : ~0u;
            t[4 * q + 2] = (uint32_t)(4 * q + 2) < m ? x.z : ~0u;
            t[4 * q + 3] = (uint32_t)(4 * q + 3) < m ? x.w : ~0u;
        }
        // a bitonic network over the warp's largest count (rounded up to 8,
        // 16 or 32 slots): one code path per warp, ~80 compare-exchanges for
        // the common 16 instead of 32 x 32 rank comparisons
        if(wmax <= 8)
            bitonic_sort<8>(t);
        else if(wmax <= 16)
            bitonic_sort<16>(t);
        else
            bitonic_sort<kPairSlots>(t);
        const uint32_t incl  = warp_incl_scan(m);
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
#pragma unroll
        for(int k = 0; k < kPairSlots; ++k)
            if((uint32_t)k < m)
            {
                s_partner[w][incl - m + k] = t[k];
                s_owner[w][incl - m + k]   = (uint8_t)lane;
            }
        __syncwarp();
        const uint32_t shift = (uint32_t)out - (incl - m); // record minus staged index
        for(uint32_t i0 = 0; i0 < total; i0 += 32)
        {
            const uint32_t i     = i0 + lane;
            const unsigned owner = i < total ? s_owner[w][i] : 0u;
            const uint32_t p     = __shfl_sync(0xffffffffu, shift, owner) + i;
            if(i < total)
            {
                pair_a[p]  = (uint32_t)a - lane + owner;
                pair_b[p]  = sids[s_partner[w][i]];
                contact[p] = 0;
            }
        }
    }
    out += cp;
    if(cp > kPairSlots)
    {
        // more partners than slots (the largest grains of a polydisperse
        // packing): k_pair_fill_overflow writes them, a warp per particle
        ovf_list[atomicAdd(gjk_count + 2 + ovf_phase, 1u)] = (uint32_t)a;
    }
    // the particle's obstacle records, contiguous after its particle pairs,
    // into the obstacle pass's queue
    if(k_obs)
    {
        const uint32_t q = atomicAdd(gjk_count + 4 + ovf_phase, k_obs);
        for(uint32_t j = 0; j < k_obs; ++j)
            obs_queue[q + j] = (uint32_t)out + j;
        for_each_obstacle_candidate(oc, a, sorted_of[a], [&](uint32_t o) {
            pair_a[out]  = a;
            pair_b[out]  = kObstacleBit | o;
            contact[out] = 0;
            ++out;
        });
    }
    if(cp)
        write_records<S>((uint32_t)a, st, tb, rec);
}

// The particle pairs of the particles whose partners overflowed their slots,
// one warp per particle: the 27 cells in the reference's order,
// four rounds of 32 candidates at a time (a particle is one chain of dependent
// rounds), the hits of a round written in lane order (ballot + prefix count).
template <bool STRICT>
__global__ void __launch_bounds__(128)
    k_pair_fill_overflow(const uint32_t* __restrict__ ovf_count,
                         const uint32_t* __restrict__ ovf_list, const uint32_t* __restrict__ skeys,
                         const uint32_t* __restrict__ sids, const uint32_t* __restrict__ sorted_of,
                         const double4* __restrict__ spos, const float4* __restrict__ spos32,
                         const uint32_t* __restrict__ cstart, uint32_t nx, uint32_t ny, uint32_t nz,
                         const uint32_t* __restrict__ offset, uint32_t* __restrict__ pair_a,
                         uint32_t* __restrict__ pair_b, uint8_t* __restrict__ contact,
                         const int* __restrict__ flags)
{
    grid_dep_sync();
    if(step_aborted(flags))
        return;
    const unsigned lane  = threadIdx.x & 31u;
    const uint32_t total = *ovf_count;
    const uint32_t warps = gridDim.x * (blockDim.x / 32);
    for(uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) / 32; w < total; w += warps)
    {
        const uint32_t a   = ovf_list[w];
        const uint32_t s   = sorted_of[a];
        uint32_t       out = offset[a];
        const uint32_t key = skeys[s];
        const double4  pa  = spos[s];
        const float4   pa32 = spos32[s];
        const int cx = key % nx, cy = (key / nx) % ny, cz = key / (nx * ny);
        // the 9 rows of 3 cells, lane r holding row r, walked as one sequence
        uint32_t t0 = 0, t1 = 0;
        if(lane < 9)
            neighbour_row(cstart, nx, ny, nz, cx, cy, cz, (int)lane, t0, t1);
        warp_ranges<4>(t0, t1, [&](const uint32_t(&t)[4], const bool(&valid)[4]) {
            bool hit[4];
#pragma unroll
            for(int k = 0; k < 4; ++k)
                hit[k] = valid[k] && t[k] != s && !pretest_rejects(pa32, spos32[t[k]]);
#pragma unroll
            for(int k = 0; k < 4; ++k)
            {
                const bool     h    = hit[k] && exact_hit<STRICT>(pa, spos[t[k]]);
                const unsigned bits = __ballot_sync(0xffffffffu, h);
                if(h)
                {
                    const uint32_t q = out + __popc(bits & ((1u << lane) - 1u));
                    pair_a[q]        = a;
                    pair_b[q]        = sids[t[k]];
                    contact[q]       = 0;
                }
                out += __popc(bits);
            }
        });
    }
}

// ---- narrow phase + contact law, one thread per candidate pair ---------------
template <typename St>
struct PairOut
{
    St*      f[3];
    St*      t[3];
    St*      m[3];     // rolling moment (only when some kr != 0)
    uint8_t* contact;  // kContactParticle / kContactObstacle when overlap < 0, else 0 (set
                       // to 0 by the fill pass; the other outputs are written, and
                       // read, for contacts only)
    uint32_t* pcount;  // 1 where particle id has a contact (zero before the narrow phase;
                       // the per-particle kernel reads and clears it)
    double*  info;     // optional: 7 per pair (point, vector, overlap) in world frame
    // tangential history (history law): current step out, previous step in
    St*             xi[3];
    const uint32_t* prev_off;
    const uint32_t* prev_b;
    const uint8_t*  prev_contact;
    const St*       prev_xi[3];
};

// the tangential spring of the pair (a, b) at the end of the last step (zero
// where it was no contact)
template <typename S>
GB_D V3<S> previous_spring(const PairOut<store_t<S>>& po, uint32_t a, uint32_t b)
{
    for(uint32_t k = po.prev_off[a]; k < po.prev_off[a + 1]; ++k)
        if(po.prev_b[k] == b)
            return po.prev_contact[k]
                       ? mk<S>(S(po.prev_xi[0][k]), S(po.prev_xi[1][k]), S(po.prev_xi[2][k]))
                       : zero3<S>();
    return zero3<S>();
}

// the outputs of contact p of particle a: force, torque, rolling moment,
// spring, contact flag, and (when recorded) the contact point in world frame,
// vector and overlap
template <typename S>
GB_D void store_pair(const PairOut<store_t<S>>& po, int64_t p, uint32_t a, const Force<S>& F,
                     const V3<S>& xi_new, uint8_t flag, int law_kind, int has_kr,
                     const Contact<S>& ci, const double xa[3])
{
    po.pcount[a] = 1u;
#pragma unroll
    for(int k = 0; k < 3; ++k)
    {
        const S fk[3] = {F.f.x, F.f.y, F.f.z}, tk[3] = {F.t.x, F.t.y, F.t.z};
        po.f[k][p] = (store_t<S>)to_d(fk[k]);
        po.t[k][p] = (store_t<S>)to_d(tk[k]);
    }
    if(has_kr)
    {
        po.m[0][p] = (store_t<S>)to_d(F.m.x);
        po.m[1][p] = (store_t<S>)to_d(F.m.y);
        po.m[2][p] = (store_t<S>)to_d(F.m.z);
    }
    if(law_kind != GB_LAW_HOOKE)
    {
        po.xi[0][p] = (store_t<S>)to_d(xi_new.x);
        po.xi[1][p] = (store_t<S>)to_d(xi_new.y);
        po.xi[2][p] = (store_t<S>)to_d(xi_new.z);
    }
    po.contact[p] = flag;
    if(po.info)
    {
        double* o = po.info + 7 * p;
        if constexpr(is_mixed<S>())
        {
            o[0] = xa[0] + to_d(ci.pt.x);
            o[1] = xa[1] + to_d(ci.pt.y);
            o[2] = xa[2] + to_d(ci.pt.z);
        }
        else
        {
            o[0] = to_d(ci.pt.x);
            o[1] = to_d(ci.pt.y);
            o[2] = to_d(ci.pt.z);
        }
        o[3] = to_d(ci.vec.x);
        o[4] = to_d(ci.vec.y);
        o[5] = to_d(ci.vec.z);
        o[6] = to_d(ci.overlap);
    }
}

// Pair p of particle a with obstacle o: closestPointsRigidBodies against the
// obstacle and the contact law with the obstacle at rest
// (ComponentManagerCPU.cpp:301-351).  The history law starts a fresh spring
// for obstacle contacts every step.  GEN: some obstacle is not a Rectangle
// and needs the general GJK (of variant VAR).
template <typename S, bool GEN, int VAR>
GB_D void narrow_obstacle(int64_t p, uint32_t a, int o, const State<store_t<S>>& st,
                          const Tables<S>& tb, const PairOut<store_t<S>>& po, int law_kind,
                          int has_kr, S dt, unsigned long long* counters)
{
    const uint32_t ra    = st.rb_id[a];
    const Body<S>  A     = load_body<S>(tb.shape, ra, tb.verts);
    const M3<S>    RA    = load_rot<S>(st, a);
    const double   xa[3] = {st.pos[0][a], st.pos[1][a], st.pos[2][a]};
    const double*  ot    = tb.obs_tr + 12 * o;
    const Body<S>  O     = load_body<S>(tb.obs_shape, o, tb.verts);
    V3<S>          oA, oO;
    M3<S>          RO;
    obstacle_frame(tb, o, xa, oA, oO, RO);
    int        iters = 0;
    Contact<S> ci    = no_contact<S>();
    if constexpr(is_mixed<S>())
    {
        if(O.type == GB_DRUM)
        {
            // the wall point nearest A's centre and its tangent plane, in FP64
            // relative to the centre; the FP32 pre-test, then the FP64 plane
            // contact as for Rectangles
            const V3<double> ax = mk<double>(ot[2], ot[5], ot[8]);
            const V3<double> d  = mk<double>(xa[0] - ot[9], xa[1] - ot[10], xa[2] - ot[11]);
            const V3<double> r  = d - dot(ax, d) * ax;
            const double     nr = norm(r), R = tb.obs_shape64[o].p[0];
            if(nr > 1e-12 * R)
            {
                const V3<double> e  = (1.0 / nr) * r;
                const V3<double> w  = (R - nr) * e; // the wall point, from A's centre
                const V3<S>      e32 = cvt3<S>(e);
                const V3<S>      pA  = mul(RA, support(A, mul_t(RA, e32)));
                if(S(R - nr) - dot(e32, pA) < S(1e-6))
                {
                    const Body<double> A64  = load_body<double>(tb.shape64, ra, tb.verts64);
                    const M3<double>   RA64 = load_rot64(st, a);
                    ci = to_f(closest_rectangle(A64, RA64, zero3<double>(), w, -e));
                }
            }
        }
        else if(O.type == GB_RECTANGLE)
        {
            // FP32 first; a contact (or a near miss within the rounding
            // margin) is recomputed in FP64 relative to the particle centre
            const V3<S> rn  = mk<S>(RO.m[2], RO.m[5], RO.m[8]);
            const V3<S> rnA = s_copysign(S(1.0), dot(rn, oA - oO)) * rn;
            const V3<S> pA  = mul(RA, support(A, mul_t(RA, -rnA)));
            const S     sep = dot(rnA, pA - oO);
            if(sep < S(1e-6))
            {
                const Body<double> A64  = load_body<double>(tb.shape64, ra, tb.verts64);
                const M3<double>   RA64 = load_rot64(st, a);
                const V3<double>   oO64 = mk<double>(ot[9] - xa[0], ot[10] - xa[1], ot[11] - xa[2]);
                ci = to_f(closest_rectangle(A64, RA64, zero3<double>(), oO64,
                                            mk<double>(ot[2], ot[5], ot[8])));
            }
        }
        else if constexpr(GEN)
            ci = closest_points<VAR>(A, O, RA, RO, oA, oO, oO - oA, &iters);
    }
    else if(O.type == GB_RECTANGLE)
        ci = closest_rectangle(A, RA, oA, oO, mk<S>(RO.m[2], RO.m[5], RO.m[8]));
    else if(O.type == GB_DRUM)
        ci = closest_drum(A, RA, oA, oO, mk<S>(RO.m[2], RO.m[5], RO.m[8]), O.p[0]);
    else if constexpr(GEN)
        ci = closest_points<VAR>(A, O, RA, RO, oA, oO, oO - oA, &iters);
    if(ci.overlap < S(0.0))
    {
        Force<S>     F;
        const Law<S> L  = load_law<S>(tb.law, tb.shape[ra].material, tb.obs_shape[o].material);
        const S      m1 = S(tb.inertia[ra].mass);
        const S      m2 = S(tb.obs_mass[o]);
        const V3<S>  vA = load3<S>(st.vel, a), wA = load3<S>(st.omg, a);
        V3<S>        arm, ptw, armO;
        if constexpr(is_mixed<S>())
        {
            arm  = ci.pt;
            ptw  = mk<S>(S(xa[0] + to_d(ci.pt.x)), S(xa[1] + to_d(ci.pt.y)), S(xa[2] + to_d(ci.pt.z)));
            armO = mk<S>(S(xa[0] - ot[9]), S(xa[1] - ot[10]), S(xa[2] - ot[11])) + ci.pt;
        }
        else
        {
            arm  = ci.pt - oA;
            ptw  = ci.pt;
            armO = ci.pt - oO;
        }
        // the wall's velocity at the contact point, v + w x (p - origin): zero
        // for the reference's walls at rest (ComponentManagerCPU.cpp:330-340)
        const double* ov  = tb.obs_vel + 6 * o;
        const V3<S>   wO  = mk<S>(S(ov[3]), S(ov[4]), S(ov[5]));
        const V3<S>   vOp = mk<S>(S(ov[0]), S(ov[1]), S(ov[2])) + cross(wO, armO);
        if(law_kind == GB_LAW_HOOKE)
        {
            const V3<S> rel = (vA + cross(wA, ptw)) - vOp;
            F               = hooke(L, ci, rel, wA - wO, m1, m2, arm);
        }
        else
        {
            V3<S> xi;
            F = hooke_history(L, ci, (vA + cross(wA, arm)) - vOp, m1, m2, dt, zero3<S>(), xi,
                              arm);
        }
        atomicAdd(&counters[0], 1ull);
        store_pair<S>(po, p, a, F, zero3<S>(), kContactObstacle, law_kind, has_kr, ci, xa);
    }
    if(iters)
        atomicAdd(&counters[1], (unsigned long long)iters);
}

// The first iteration of GJK-JH (gjk_jh, GJK_JH.cpp:332-371), where it
// decides the pair on its own.  From v = sA(0) - b2a(sB(0)) and the first
// Minkowski support w = sA(-v) - b2a(sB(R^T v)), g = v.w / |v| is a lower
// bound on the distance of the cores, and GJK returns a distance of at
// least g wherever it stops (|v| of a point of the Minkowski difference).
// So:
//   g > crustA + crustB + margin: GJK's distance exceeds the crusts: no
//     contact;
//   g < -margin: mu stays 0 < the absolute tolerance, GJK stops at this
//     iteration and returns |v|; if that exceeds the crusts: no contact.
// Every other pair (in particular every contact) takes the full GJK.  It is
// evaluated in FP32 in every mode (supports, frames and dot products), with a
// margin of 1e-4 of the bounding radii, some eleven times a bound on the FP32
// error of g: a support value is short by up to 7.8e-6 of its radius
// (support_sq_log32), and the direction's error of ~3e-7 (support values are
// Lipschitz in the direction with constant |x| <= R_circ) and the frames' add
// 1e-6.  A pair decided here is one that the FP64 GJK also finds out of
// contact, so long as it converges (a signed-volume iteration that breaks down
// on a separated pair ends at distance 0, a contact with a 0/0 normal; such a
// pair is none here), so the contact set and the
// contact geometry stay those of the FP64 GJK.  Both rules are the same for
// (A, B) and (B, A): the pair of the other order has v and w mirrored, so
// each unordered pair is decided once, for both its records.
// The first rule holds for every GJK variant (each returns the norm of a
// point of the Minkowski difference, at least the true distance, which g
// bounds from below); the second is GJK-JH's own stopping rule (JH_RULE).
// `s` is the sum of the bounding radii (infinite: nothing is decided).
template <bool JH_RULE>
GB_D bool gjk_first_iteration_separates(const Body<float>& A, const Body<float>& B,
                                        const M3<float>& RA, const M3<float>& RB,
                                        const V3<float>& d, float s)
{
    Tr<float>       b2a;
    const M3<float> RAt = transpose(RA);
    b2a.R               = mul(RAt, RB);
    b2a.o               = mul(RAt, d);
    const V3<float> v    = support_zero(A) - apply(b2a, support_zero(B));
    const float     dist = norm(v);
    const V3<float> pa = support_first(A, -v), qb = support_first(B, mul_t(b2a.R, v));
    const V3<float> w  = pa - apply(b2a, qb);
    const float     g  = dot(v, w) / dist;
    const float     ct = A.crust + B.crust;
    const float     margin = 1e-4f * s + 1e-9f;
    if(g > ct + margin)
        return true;
    return JH_RULE && g < -margin && dist - ct > margin;
}

// ---- the FP32 GJK stage ------------------------------------------
// Closest point to the origin of the segment (a, b) or the triangle (a, b, c)
// (Ericson, Real-Time Collision Detection, 5.1.2 and 5.1.5, by Voronoi
// regions), with the vertices of the feature it lies on put in y0..y(n-1).
// The vertices come by value: the callers pass the simplex they overwrite
// (with references, an edge (b, c) result read b after y1 = c had replaced
// it and returned c instead of the edge's closest point).
GB_D V3<float> closest_on_segment(const V3<float> a, const V3<float> b, V3<float>& y0,
                                  V3<float>& y1, int& n)
{
    const V3<float> ab = b - a;
    const float     t  = -dot(a, ab);
    if(t <= 0.0f)
    {
        y0 = a;
        n  = 1;
        return a;
    }
    const float den = dot(ab, ab);
    if(t >= den)
    {
        y0 = b;
        n  = 1;
        return b;
    }
    y0 = a;
    y1 = b;
    n  = 2;
    return a + (t / den) * ab;
}

GB_D V3<float> closest_on_triangle(const V3<float> a, const V3<float> b, const V3<float> c,
                                   V3<float>& y0, V3<float>& y1, V3<float>& y2, int& n)
{
    const V3<float> ab = b - a, ac = c - a;
    const float     d1 = -dot(ab, a), d2 = -dot(ac, a);
    if(d1 <= 0.0f && d2 <= 0.0f)
    {
        y0 = a;
        n  = 1;
        return a;
    }
    const float d3 = -dot(ab, b), d4 = -dot(ac, b);
    if(d3 >= 0.0f && d4 <= d3)
    {
        y0 = b;
        n  = 1;
        return b;
    }
    const float vc = d1 * d4 - d3 * d2;
    if(vc <= 0.0f && d1 >= 0.0f && d3 <= 0.0f)
    {
        y0 = a;
        y1 = b;
        n  = 2;
        return a + (d1 / (d1 - d3)) * ab;
    }
    const float d5 = -dot(ab, c), d6 = -dot(ac, c);
    if(d6 >= 0.0f && d5 <= d6)
    {
        y0 = c;
        n  = 1;
        return c;
    }
    const float vb = d5 * d2 - d1 * d6;
    if(vb <= 0.0f && d2 >= 0.0f && d6 <= 0.0f)
    {
        y0 = a;
        y1 = c;
        n  = 2;
        return a + (d2 / (d2 - d6)) * ac;
    }
    const float va = d3 * d6 - d5 * d4;
    if(va <= 0.0f && d4 - d3 >= 0.0f && d5 - d6 >= 0.0f)
    {
        y0 = b;
        y1 = c;
        n  = 2;
        return b + ((d4 - d3) / ((d4 - d3) + (d5 - d6))) * (c - b);
    }
    const float den = 1.0f / (va + vb + vc);
    y0              = a;
    y1              = b;
    y2              = c;
    n               = 3;
    return a + (vb * den) * ab + (vc * den) * ac;
}

constexpr int kGjk32MaxIter = 24;

// For a pair that GJK's first iteration leaves open: GJK iterations in
// FP32 on at most a triangle (a new point added to a triangle keeps the
// nearest of the three faces through it), kept only for their support
// planes.  Any direction v and the Minkowski support w along -v give the
// lower bound v.w/|v| on the distance of the cores, whatever the simplex
// arithmetic did, with the FP32 error bound of gjk_first_iteration_separates.
// True: the largest bound exceeds the crusts by that margin, so the FP64 GJK
// finds no contact either.  False (the FP64 GJK decides): an iterate came
// within the crusts and the margin (a contact or a near miss), reached the
// origin, left the finite range, or they ran out of iterations.
// Called by whole warps (gjk_goes_on), lanes without a pair with run = false.
GB_D bool gjk_fp32_separates(const Body<float>& A, const Body<float>& B, const M3<float>& RA,
                             const M3<float>& RB, const V3<float>& d, float s, bool run)
{
    Tr<float>       b2a;
    const M3<float> RAt = transpose(RA);
    b2a.R               = mul(RAt, RB);
    b2a.o               = mul(RAt, d);
    const float ct      = A.crust + B.crust;
    const float margin  = 1e-4f * s + 1e-9f;
    V3<float>   y0 = support_zero(A) - apply(b2a, support_zero(B));
    V3<float>   y1 = y0, y2 = y0;
    int         n  = 1;
    V3<float>   v  = y0;
    float       mu = -INFINITY;
    bool        separates = false;
    for(int k = 0; k < kGjk32MaxIter && gjk_goes_on<true>(run); ++k)
    {
        const float vv = dot(v, v);
        run            = run && vv > 1e-30f;
        if(!run)
            continue;
        const V3<float> w = support_first(A, -v)
                            - apply(b2a, support_first(B, mul_t(b2a.R, v)));
        const float vw = dot(v, w);
        const float nv = sqrtf(vv);
        const float g  = vw / nv;
        mu             = fmaxf(mu, g); // (a NaN g ends it below)
        separates      = mu > ct + margin;
        // nv bounds the distance from above: within the crusts and the margin
        // no lower bound can pass them
        if(separates || !(g == g) || nv <= ct + margin || vv - vw <= 1e-6f * vv)
        {
            run = false;
            continue;
        }
        if(n == 1)
            v = closest_on_segment(y0, w, y0, y1, n);
        else if(n == 2)
            v = closest_on_triangle(y0, y1, w, y0, y1, y2, n);
        else
        {
            // the faces of the tetrahedron through w: the nearest one
            V3<float>       a0, a1, a2, b0, b1, b2, c0, c1, c2;
            int             na, nb, nc;
            const V3<float> pa = closest_on_triangle(w, y0, y1, a0, a1, a2, na);
            const V3<float> pb = closest_on_triangle(w, y1, y2, b0, b1, b2, nb);
            const V3<float> pc = closest_on_triangle(w, y0, y2, c0, c1, c2, nc);
            const float     da = dot(pa, pa), db = dot(pb, pb), dc = dot(pc, pc);
            if(da <= db && da <= dc)
            {
                v  = pa;
                y0 = a0;
                y1 = a1;
                y2 = a2;
                n  = na;
            }
            else if(db <= dc)
            {
                v  = pb;
                y0 = b0;
                y1 = b1;
                y2 = b2;
                n  = nb;
            }
            else
            {
                v  = pc;
                y0 = c0;
                y1 = c1;
                y2 = c2;
                n  = nc;
            }
        }
    }
    return separates;
}

// The contact law for contact `ci` of the particle pair record p = (a, b) and
// its outputs.  B's centre is at oB in the working coordinates.
template <typename S>
GB_D void pair_contact(int64_t p, uint32_t a, uint32_t b, const Law<S>& L, S m1, S m2,
                       const V3<S>& vA, const V3<S>& vB, const V3<S>& wA, const V3<S>& wB,
                       const V3<S>& oA, const V3<S>& oB, const Contact<S>& ci, const double xa[3],
                       const PairOut<store_t<S>>& po, int law_kind, int has_kr, S dt)
{
    Force<S> F;
    V3<S>    xi_new = zero3<S>();
    // arm = contact point - A's centre
    V3<S> arm, ptw;
    if constexpr(is_mixed<S>())
    {
        arm = ci.pt;
        ptw = mk<S>(S(xa[0] + to_d(ci.pt.x)), S(xa[1] + to_d(ci.pt.y)), S(xa[2] + to_d(ci.pt.z)));
    }
    else
    {
        arm = ci.pt - oA;
        ptw = ci.pt;
    }
    if(law_kind == GB_LAW_HOOKE)
    {
        // Kinematics::kinematicsAtPoint with the absolute contact point
        const V3<S> rel = (vA + cross(wA, ptw)) - (vB + cross(wB, ptw));
        F               = hooke(L, ci, rel, wA - wB, m1, m2, arm);
    }
    else
    {
        const V3<S> armB = ci.pt - oB;
        const V3<S> rel  = (vA + cross(wA, arm)) - (vB + cross(wB, armB));
        F = hooke_history(L, ci, rel, m1, m2, dt, previous_spring<S>(po, a, b), xi_new, arm);
    }
    store_pair<S>(po, p, a, F, xi_new, kContactParticle, law_kind, has_kr, ci, xa);
}

// Pair record p: closestPointsRigidBodies, contact law, outputs.  SPHERES: a
// pair of spheres, whose closed form needs no rotation and no body record.
template <typename S, int VAR, bool SPHERES = false>
GB_D void narrow_pair(int64_t p, uint32_t a, uint32_t b, const State<store_t<S>>& st,
                      const Tables<S>& tb, const PairOut<store_t<S>>& po, int law_kind, int has_kr,
                      S dt, unsigned long long* __restrict__ counters, bool active = true)
{
    const uint32_t ra = st.rb_id[a], rb = st.rb_id[b];
    const double   xa[3] = {st.pos[0][a], st.pos[1][a], st.pos[2][a]};
    const double   xb[3] = {st.pos[0][b], st.pos[1][b], st.pos[2][b]};
    V3<S>          oA, oB, d;
    if constexpr(is_mixed<S>())
    {
        d  = mk<S>(S(xb[0] - xa[0]), S(xb[1] - xa[1]), S(xb[2] - xa[2]));
        oA = zero3<S>();
        oB = d;
    }
    else
    {
        oA = mk<S>(S(xa[0]), S(xa[1]), S(xa[2]));
        oB = mk<S>(S(xb[0]), S(xb[1]), S(xb[2]));
        d  = oB - oA;
    }
    int        iters = 0;
    Contact<S> ci;
    if constexpr(SPHERES)
    {
        const double rA = tb.shape64[ra].p[0], rB = tb.shape64[rb].p[0];
        if constexpr(is_mixed<S>())
            ci = closest_spheres_mixed(rA, rB, xa, xb);
        else
            ci = closest_spheres(S(rA), S(rB), oA, oB);
    }
    else
    {
        const Body<S> A  = load_body<S>(tb.shape, ra, tb.verts);
        const Body<S> B  = load_body<S>(tb.shape, rb, tb.verts);
        const M3<S>   RA = load_rot<S>(st, a), RB = load_rot<S>(st, b);
        if constexpr(is_mixed<S>())
            ci = closest_mixed<VAR>(tb, st, a, b, ra, rb, A, B, RA, RB, xa, xb, &iters, active);
        else
            ci = closest_points<VAR>(A, B, RA, RB, oA, oB, d, &iters, active);
    }
    // the lanes of a pair hold the same results: the first one stores them
    if((VAR & kGjkPaired) && (!active || (threadIdx.x & (gjk_lanes(VAR) - 1))))
        return;
    if(ci.overlap < S(0.0))
        pair_contact<S>(p, a, b, load_law<S>(tb.law, tb.shape[ra].material, tb.shape[rb].material),
                        S(tb.inertia[ra].mass), S(tb.inertia[rb].mass), load3<S>(st.vel, a),
                        load3<S>(st.vel, b), load3<S>(st.omg, a), load3<S>(st.omg, b), oA, oB, ci,
                        xa, po, law_kind, has_kr, dt);
    if(iters)
        atomicAdd(&counters[1], (unsigned long long)iters);
}

// The pair records of a narrow-phase launch, p in [0, npairs).  A list longer
// than the grid is walked with a grid stride (consecutive records in
// consecutive lanes).  A shorter one -- the common case of a loose packing,
// a few thousand candidates -- is spread over all warps, ceil(npairs / warps)
// consecutive records per warp: one thread's GJK is a long dependent chain,
// and the divergent chains of a warp run one after the other, so the step
// waits for the warp with the most records, not for the longest chain alone.
template <typename F>
GB_D void for_each_pair(int64_t npairs, F&& f)
{
    const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
    const int64_t tid      = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t nwarps   = nthreads >> 5, lane = threadIdx.x & 31;
    // records per warp and round: a short list's share, or one per lane
    const int64_t k = npairs < nthreads ? (npairs + nwarps - 1) / nwarps : 32;
    if(lane < k)
        for(int64_t p = (tid >> 5) * k + lane; p < npairs; p += nwarps * k)
            f(p);
}

// The same for passes that whole warps run together: f(p, valid) on every lane
// of the warp, STEP (1, 2 or 4) lanes per pair, lanes without a pair with
// valid = false and a p that may be read (npairs > 0).
template <int STEP, typename F>
GB_D void for_each_pair_converged(int64_t npairs, F&& f)
{
    constexpr int kPairs = 32 / STEP; // pairs a warp holds at a time
    const int64_t nwarps = (int64_t)gridDim.x * blockDim.x / 32;
    const int64_t warp   = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const int     slot   = (int)(threadIdx.x & 31u) / STEP;
    // pairs per warp and round: a short list's share, or all a warp holds
    const int64_t k = npairs < nwarps * kPairs ? (npairs + nwarps - 1) / nwarps : kPairs;
    for(int64_t base = warp * k; base < npairs; base += nwarps * k)
    {
        const bool valid = slot < k && base + slot < npairs;
        f(valid ? base + slot : npairs - 1, valid);
    }
}

// The narrow phase of a run whose bodies are all spheres: every record's
// closed form and law in one pass, one thread per record, from the sphere
// records of the fill pass (two to three sectors a particle, where the
// structure-of-arrays state costs a sector per component).  Issue-bound on the
// FP64 closed form (48% of issue slots); a launch, against the general kernel
// on the state arrays: 1M spheres mixed 254 -> 160 us, 400k FP64 246 -> 91 us.
template <typename S>
__global__ void __launch_bounds__(kBlock)
    k_narrow_spheres(const uint32_t* __restrict__ total, const int* __restrict__ flags,
                     const uint32_t* __restrict__ pair_a, const uint32_t* __restrict__ pair_b,
                     const SphereRec<store_t<S>>* __restrict__ rec, Tables<S> tb,
                     PairOut<store_t<S>> po, int law_kind, int has_kr, S dt)
{
    grid_dep_sync();
    if(step_aborted(flags))
        return;
    const int64_t np = *total, stride = (int64_t)gridDim.x * blockDim.x;
    for(int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < np; p += stride)
    {
        const uint32_t a = pair_a[p], b = pair_b[p];
        if(b & kObstacleBit) // k_narrow_obstacles
            continue;
        const SphereRec<store_t<S>> A = load_rec(rec + a), B = load_rec(rec + b);
        const double                xa[3] = {A.x, A.y, A.z}, xb[3] = {B.x, B.y, B.z};
        V3<S>                       oA, oB;
        Contact<S>                  ci;
        if constexpr(is_mixed<S>())
        {
            oA = zero3<S>();
            oB = mk<S>(S(xb[0] - xa[0]), S(xb[1] - xa[1]), S(xb[2] - xa[2]));
            ci = closest_spheres_mixed(A.r, B.r, xa, xb);
        }
        else
        {
            oA = mk<S>(S(A.x), S(A.y), S(A.z));
            oB = mk<S>(S(B.x), S(B.y), S(B.z));
            ci = closest_spheres(S(A.r), S(B.r), oA, oB);
        }
        if(!(ci.overlap < S(0.0)))
            continue;
        pair_contact<S>(p, a, b, load_law<S>(tb.law, (int)A.material, (int)B.material), S(A.mass),
                        S(B.mass), mk<S>(S(A.v[0]), S(A.v[1]), S(A.v[2])),
                        mk<S>(S(B.v[0]), S(B.v[1]), S(B.v[2])),
                        mk<S>(S(A.w[0]), S(A.w[1]), S(A.w[2])),
                        mk<S>(S(B.w[0]), S(B.w[1]), S(B.w[2])), oA, oB, ci, xa, po, law_kind,
                        has_kr, dt);
    }
}

// the pose record of a particle for the FP32 passes
struct Pose32
{
    double    x, y, z;
    uint32_t  rb;
    float     r;
    M3<float> R;
    V3<float> bb;
};

template <typename St>
GB_D Pose32 load_pose(const PoseRec<St>* __restrict__ rec, uint32_t i)
{
    const PoseRec<St> o = load_rec(rec + i);
    Pose32            p;
    p.x  = o.x;
    p.y  = o.y;
    p.z  = o.z;
    p.rb = o.rb;
    p.r  = o.r;
    p.bb = mk<float>(o.bb[0], o.bb[1], o.bb[2]);
    if constexpr(sizeof(St) == 4)
        p.R = quat_to_matrix<float>(o.q[0], o.q[1], o.q[2], o.q[3]);
    else
    {
#pragma unroll
        for(int k = 0; k < 9; ++k)
            p.R.m[k] = o.R[k];
    }
    return p;
}

GB_D V3<float> centre_difference(const Pose32& A, const Pose32& B)
{
    return mk<float>(float(B.x - A.x), float(B.y - A.y), float(B.z - A.z));
}

// the record (b, a) of record (a, b): b's records hold the mirror of each of
// a's (the candidate test is symmetric); kNoRecord, never expected, if not.
// They ascend in the partner's sorted position, obstacles after them (the fill
// pass), so a long list is halved first: a large grain among small ones has
// thousands of records, and each of its pairs looks through them (a detect of
// 60,000 grains around one, mixed 25.2 -> 15.3 ms, of 1,350 0.48 -> 0.40 ms).
// Where halving stops matters little (8, 32 and 128 records: the same within
// 1%); lists of up to 32, all but a few in other packings, read no positions.
constexpr uint32_t kNoRecord     = 0xffffffffu;
constexpr uint32_t kMirrorLinear = 32; // records looked through one by one

GB_D uint32_t mirror_record(const uint32_t* __restrict__ off, const uint32_t* __restrict__ pair_b,
                            const uint32_t* __restrict__ sorted_of, uint32_t a, uint32_t b)
{
    uint32_t k = off[b], e = off[b + 1];
    if(e - k > kMirrorLinear)
    {
        const uint32_t s = sorted_of[a];
        while(e - k > kMirrorLinear)
        {
            const uint32_t m = k + (e - k) / 2, q = pair_b[m];
            if(!(q & kObstacleBit) && sorted_of[q] <= s)
                k = m;
            else
                e = m;
        }
    }
    for(; k < e; ++k)
        if(pair_b[k] == a)
            return k;
    return kNoRecord;
}

// A warp's queue of pairs in shared memory: lanes push what they keep, packed
// by a ballot, and the warp pops 32 at a time, so that each stage of the cull
// runs with all lanes busy whatever the stage before it left.
struct WarpQueue
{
    uint32_t p[64], a[64], b[64];
};

GB_D void warp_push(WarpQueue& q, unsigned& n, bool take, uint32_t p, uint32_t a, uint32_t b)
{
    const unsigned m = __ballot_sync(0xffffffffu, take);
    if(take)
    {
        const unsigned k = n + __popc(m & ((1u << (threadIdx.x & 31u)) - 1u));
        q.p[k]           = p;
        q.a[k]           = a;
        q.b[k]           = b;
    }
    n += __popc(m);
    __syncwarp();
}

// The last min(n, 32) entries of the queue, one per lane; false on the lanes
// past them.
GB_D bool warp_pop(const WarpQueue& q, unsigned& n, uint32_t& p, uint32_t& a, uint32_t& b)
{
    const unsigned lane = threadIdx.x & 31u;
    const unsigned k    = n < 32u ? n : 32u;
    const bool     mine = lane < k;
    n -= k;
    if(mine)
    {
        p = q.p[n + lane];
        a = q.a[n + lane];
        b = q.b[n + lane];
    }
    __syncwarp();
    return mine;
}

// The cull, k_narrow: every unordered candidate pair once, in FP32, in stages
// that a warp runs on packed lanes (WarpQueue): its record (a, b) with a < b
// is taken from the list; two spheres are solved for both records (closed
// form); a sphere against another shape is no contact (the reference's GJK
// starts from Sphere::support(0), whose 0/0 makes every distance NaN:
// Sphere.cpp:111); the oriented boxes, then GJK's first iteration, drop the
// pairs that both records' FP64 tests drop; what is left goes to gjk_queue as
// record p (k_narrow_gjk32).  Decisions are certified (obb_apart,
// gjk_first_iteration_separates), so every mode, the bit-exact one included,
// keeps the contacts of its own FP64 tests, which the last pass repeats for
// each record it solves.  Bound by FP32 issue and the latency of the records
// (44% of issue slots at five blocks per SM; six gave the 1M bed 1% and cost
// the 100k polyhedra 2%).  A launch, against a thread per ordered record in
// the mode's own precision: 1M bed mixed 398 -> 176 us, 130k bed FP64 242 ->
// 30 us, 400k drum 334 -> 107 us, 100k polyhedra 149 -> 94 us (and less since
// support(0) is not evaluated).
template <typename S, bool JH_RULE, bool SPHERES>
__global__ void __launch_bounds__(128, 5)
    k_narrow(const uint32_t* __restrict__ total, const int* __restrict__ flags,
             const uint32_t* __restrict__ pair_a, const uint32_t* __restrict__ pair_b,
             const uint32_t* __restrict__ off, const uint32_t* __restrict__ sorted_of,
             const PoseRec<store_t<S>>* __restrict__ pose, State<store_t<S>> st, Tables<S> tb,
             PairOut<store_t<S>> po, int law_kind, int has_kr, S dt,
             unsigned long long* __restrict__ counters, uint32_t* __restrict__ gjk_queue,
             uint32_t* __restrict__ gjk_count)
{
    grid_dep_sync();
    __shared__ WarpQueue s_boxes[4], s_first[4], s_sphere[SPHERES ? 4 : 1];
    if(step_aborted(flags))
        return;
    const unsigned lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    WarpQueue &    boxes = s_boxes[w], &first = s_first[w], &sphere = s_sphere[SPHERES ? w : 0];
    unsigned       nboxes = 0, nfirst = 0, nsphere = 0; // warp-uniform
    const int64_t  np     = *total;
    const int64_t  stride = (int64_t)gridDim.x * blockDim.x;
    int64_t        base   = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~int64_t(31);
    while(true)
    {
        const bool more = base < np;
        if(more)
        {
            const int64_t p    = base + lane;
            uint32_t      a    = 0, b = 0;
            bool          take = false;
            if(p < np)
            {
                a    = pair_a[p];
                b    = pair_b[p];
                take = a < b && !(b & kObstacleBit);
            }
            warp_push(boxes, nboxes, take, (uint32_t)p, a, b);
            base += stride;
        }
        if(nboxes >= 32 || (!more && nboxes))
        {
            uint32_t   p = 0, a = 0, b = 0;
            const bool mine = warp_pop(boxes, nboxes, p, a, b);
            bool       keep = false, both = false;
            if(mine)
            {
                const Pose32 A = load_pose(pose, a), B = load_pose(pose, b);
                const bool   sa = SPHERES && A.r < 0.0f, sb = SPHERES && B.r < 0.0f;
                both            = sa && sb;
                if(!sa && !sb)
                    keep = !obb_apart(A.bb, B.bb, A.R, B.R, centre_difference(A, B),
                                      1e-4f * (A.r + B.r));
            }
            warp_push(first, nfirst, keep, p, a, b);
            if constexpr(SPHERES)
                warp_push(sphere, nsphere, both, p, a, b);
        }
        const bool flush = !more && !nboxes;
        if(nfirst >= 32 || (flush && nfirst))
        {
            uint32_t   p = 0, a = 0, b = 0;
            const bool mine = warp_pop(first, nfirst, p, a, b);
            bool       keep = false;
            if(mine)
            {
                const Pose32      A  = load_pose(pose, a), B = load_pose(pose, b);
                const Body<float> bA = load_body<float>(tb.shape32, A.rb, tb.verts32);
                const Body<float> bB = load_body<float>(tb.shape32, B.rb, tb.verts32);
                keep = !gjk_first_iteration_separates<JH_RULE>(bA, bB, A.R, B.R,
                                                               centre_difference(A, B), A.r + B.r);
            }
            const unsigned m = __ballot_sync(0xffffffffu, keep);
            uint32_t       k = 0;
            if(lane == 0 && m)
                k = atomicAdd(gjk_count, (uint32_t)__popc(m));
            k = __shfl_sync(0xffffffffu, k, 0);
            if(keep)
                gjk_queue[k + __popc(m & ((1u << lane) - 1u))] = p;
        }
        if constexpr(SPHERES)
            if(nsphere >= 32 || (flush && nsphere))
            {
                uint32_t p = 0, a = 0, b = 0;
                if(warp_pop(sphere, nsphere, p, a, b))
                {
                    const uint32_t pm = mirror_record(off, pair_b, sorted_of, a, b);
                    for(int k = 0; k < (pm == kNoRecord ? 1 : 2); ++k)
                        narrow_pair<S, GB_GJK_JH, true>(k ? pm : p, k ? b : a, k ? a : b, st, tb,
                                                        po, law_kind, has_kr, dt, counters);
                }
                __syncwarp();
            }
        if(flush && !nfirst && !nsphere)
            break;
    }
}

// The FP32 GJK stage over the cull's queue: a pair that gjk_fp32_separates
// decides has no contact (its certificate, a lower bound on the distance,
// holds for every GJK variant and for both records); of every other pair both
// records go to the FP64 GJK's queue.  Bound by issue with 5 to 12 of 32 lanes
// active (lanes of a warp need different numbers of iterations); a launch on
// the 1M bed 210 us for each record on its own, 112 us now.  Four blocks per
// SM: two cost the bed 4% and the polyhedra 15% of a step, five the 10k column
// 3% (spills).
template <typename St>
__global__ void __launch_bounds__(128)
    k_narrow_gjk32(const uint32_t* __restrict__ gjk_count, const int* __restrict__ flags,
                   const uint32_t* __restrict__ gjk_queue, const uint32_t* __restrict__ pair_a,
                   const uint32_t* __restrict__ pair_b, const uint32_t* __restrict__ off,
                   const uint32_t* __restrict__ sorted_of, const PoseRec<St>* __restrict__ pose,
                   const RBShape<float>* __restrict__ shape, const Vert<float>* __restrict__ verts,
                   uint32_t* __restrict__ queue64, uint32_t* __restrict__ count64)
{
    grid_dep_sync();
    if(step_aborted(flags))
        return;
    for_each_pair_converged<1>(*gjk_count, [&](int64_t q, bool valid) {
        const uint32_t    p = gjk_queue[q];
        const uint32_t    a = pair_a[p], b = pair_b[p];
        const Pose32      A = load_pose(pose, a), B = load_pose(pose, b);
        const Body<float> bA = load_body<float>(shape, A.rb, verts);
        const Body<float> bB = load_body<float>(shape, B.rb, verts);
        const bool        open = !gjk_fp32_separates(bA, bB, A.R, B.R, centre_difference(A, B),
                                                     A.r + B.r, valid);
        if(valid && open)
        {
            const uint32_t pm = mirror_record(off, pair_b, sorted_of, a, b);
            const uint32_t k  = atomicAdd(count64, pm == kNoRecord ? 1u : 2u);
            queue64[k]        = p;
            if(pm != kNoRecord)
                queue64[k + 1] = pm;
        }
    });
}

// One queued pair per lane pair (kGjkPaired: the two supports of a GJK
// iteration in parallel), the warp's pairs going through the iterations
// together; a short queue is spread over all warps, a long one walked with a
// stride.  Both lanes of a pair take the same path throughout, so their
// shuffles always meet.  MIN_BLOCKS > 1
// caps its registers for more resident warps (Johnson's tables and some
// values spill to local memory): faster where the supports are closed forms
// (superquadrics) and the queue outnumbers the default's lane pairs, slower
// where they loop over polyhedron vertices or one round takes the queue.
// The launch does its work only for a queue length in [min_queue,
// max_queue), read on the device, so that the host can launch both forms
// and let the queue pick one.
template <typename S, int VAR, int MIN_BLOCKS = 1>
__global__ void __launch_bounds__(128, MIN_BLOCKS)
    k_narrow_gjk(const uint32_t* __restrict__ gjk_count, const int* __restrict__ flags,
                 const uint32_t* __restrict__ gjk_queue, const uint32_t* __restrict__ pair_a,
                 const uint32_t* __restrict__ pair_b, State<store_t<S>> st, Tables<S> tb,
                 PairOut<store_t<S>> po, int law_kind, int has_kr, S dt,
                 unsigned long long* __restrict__ counters, uint32_t min_queue,
                 uint32_t max_queue)
{
    grid_dep_sync();
    if(step_aborted(flags))
        return;
    const int64_t nq     = *gjk_count;
    if(nq < (int64_t)min_queue || nq >= (int64_t)max_queue)
        return;
    for_each_pair_converged<gjk_lanes(VAR | kGjkPaired)>(nq, [&](int64_t q, bool valid) {
        const uint32_t p = gjk_queue[q];
        narrow_pair<S, VAR | kGjkPaired>(p, pair_a[p], pair_b[p], st, tb, po, law_kind, has_kr,
                                         dt, counters, valid);
    });
}

// ---- per-particle kernel -------------------------------------------------------
// PHASE_DETECT:  torce = sum of the particle's pair forces in enumeration
//                order, then obstacle contacts in obstacle order
//                (ComponentManagerCPU.cpp:356-423 then :301-351).
// PHASE_GRAVITY: torce.force += m g (ComponentManagerCPU.cpp:448-460).
// PHASE_MOVE:    integrate from the stored torce, then reset it
//                (ComponentManagerCPU.cpp:465-500).
// PHASE_STEP:    all three fused, no torce round trip.
enum Phase
{
    PHASE_DETECT  = 1,
    PHASE_GRAVITY = 2,
    PHASE_MOVE    = 4,
    PHASE_STEP    = 7
};

template <typename S>
struct StepParams
{
    S        dt;      // time step
    S        h;       // velocity kick of this move (dt; dt/2 on the first Verlet move)
    V3<S>    g;       // gravity
    int      integrator;
    int      law_kind;
    int      has_kr;
    int      phases;
    int      accumulate; // PHASE_DETECT adds to the stored torce instead of to zero
    int      rb_identity; // particle i's rigid body is body i
};

// The particle-obstacle records of the pair list, one thread per record, in a
// kernel of their own: the two kinds interleave in the list, and one kernel
// for both would run both code paths in every warp.
template <typename S, bool GEN, int VAR>
__global__ void __launch_bounds__(128)
    k_narrow_obstacles(const uint32_t* __restrict__ n_obs_records,
                       const uint32_t* __restrict__ obs_queue, const int* __restrict__ flags,
                       const uint32_t* __restrict__ pair_a, const uint32_t* __restrict__ pair_b,
                       State<store_t<S>> st, Tables<S> tb, PairOut<store_t<S>> po, int law_kind,
                       int has_kr, S dt, unsigned long long* __restrict__ counters)
{
    if(step_aborted(flags))
        return;
    // the step's obstacle records, queued by the fill pass
    for_each_pair(*n_obs_records, [&](int64_t q) {
        const uint32_t p = obs_queue[q];
        narrow_obstacle<S, GEN, VAR>(p, pair_a[p], (int)(pair_b[p] & ~kObstacleBit), st, tb, po,
                                     law_kind, has_kr, dt, counters);
    });
}

// ---- per-particle kernel: segmented sum, gravity, integration -----------------
// A latency-bound streaming kernel.  Its loads are all issued before the pair
// loop; the mixed instantiation runs four 256-thread blocks per SM at 64
// registers with a few spilled (measured 3% faster than three blocks at 79
// registers without, and than five at 48); the FP64 ones need about 125
// registers and get two blocks.
// LOADED (mixed mode): the plain loop over a grain's records, for packings
// whose grains have many contacts (many_contacts).
template <typename S, bool LOADED>
__global__ void __launch_bounds__(kBlock, sizeof(store_t<S>) == 4 ? 4 : 2)
    k_particles(int n, State<store_t<S>> st, Tables<S> tb, const uint32_t* __restrict__ off,
                PairOut<store_t<S>> po, StepParams<S> sp, int* __restrict__ contacts_out,
                uint32_t* __restrict__ mask_out, int* __restrict__ flags,
                unsigned int* __restrict__ done)
{
    grid_dep_sync();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n || step_aborted(flags))
        return;
    const uint32_t            r   = sp.rb_identity ? (uint32_t)i : st.rb_id[i];
    const RBInertia<store_t<S>>* in = tb.inertia + r;
    // the body record (mass, inertia, inverse inertia, box) in 16-byte loads
    store_t<S> rec[16];
    {
        constexpr int per = 16 / sizeof(store_t<S>);
        using Vec         = typename std::conditional<per == 4, float4, double2>::type;
        const Vec* v4     = reinterpret_cast<const Vec*>(in);
#pragma unroll
        for(int k = 0; k < 16 / per; ++k)
        {
            const Vec x = __ldg(v4 + k);
            if constexpr(per == 4)
            {
                rec[4 * k]     = x.x;
                rec[4 * k + 1] = x.y;
                rec[4 * k + 2] = x.z;
                rec[4 * k + 3] = x.w;
            }
            else
            {
                rec[2 * k]     = x.x;
                rec[2 * k + 1] = x.y;
            }
        }
    }
    const S                   m   = S(rec[0]);
    V3<S>                     F, T;
    V3<S>                     v = load3<S>(st.vel, i), w = load3<S>(st.omg, i);
    int                       nc = 0;
    // The pose and the body record do not depend on the pair loop: they are
    // loaded before it, and every store comes after all loads, so that these
    // loads and the loop's gathers are in flight together.
    const bool move = (sp.phases & PHASE_MOVE) != 0;
    S            I[6], I1[6];
    Quat<S>      q;
    float        qlo[4]; // mixed: the orientation's FP32 remainder (q + qlo is the orientation)
    M3<S>        R;
    double       x0[3];
    if(move)
    {
#pragma unroll
        for(int k = 0; k < 6; ++k)
        {
            I[k]  = S(rec[1 + k]);
            I1[k] = S(rec[7 + k]);
        }
        if constexpr(is_mixed<S>())
        {
            q.w = S(st.rot[0][i]);
            q.v = mk<S>(S(st.rot[1][i]), S(st.rot[2][i]), S(st.rot[3][i]));
#pragma unroll
            for(int k = 0; k < 4; ++k)
                qlo[k] = st.rot[4 + k][i];
        }
        else
            R = load_rot<S>(st, i);
#pragma unroll
        for(int k = 0; k < 3; ++k)
            x0[k] = st.pos[k][i];
    }
    if(sp.phases & PHASE_DETECT)
    {
        // Torce::addForce onto the torce accumulated since the last move
        // (zero unless set_torces, add_external_forces or a detect came first)
        if(sp.accumulate)
        {
            F = load3<S>(st.frc, i);
            T = load3<S>(st.trq, i);
        }
        else
        {
            F = zero3<S>();
            T = zero3<S>();
        }
        // the particle's pairs, then its obstacle pairs, in list order; most
        // particles have no contact (the narrow phase marks those that have)
        // and skip their list
        const uint32_t ncon = po.pcount[i];
        if(ncon)
        {
            po.pcount[i] = 0u;
            const uint32_t pe = off[i + 1];
            if constexpr(LOADED)
                for(uint32_t p = off[i]; p < pe; ++p)
                {
                    const uint8_t hit = po.contact[p];
                    if(!hit)
                        continue;
                    nc += hit == kContactParticle;
                    F = F + mk<S>(S(po.f[0][p]), S(po.f[1][p]), S(po.f[2][p]));
                    T = T + mk<S>(S(po.t[0][p]), S(po.t[1][p]), S(po.t[2][p]));
                    if(sp.has_kr)
                        T = T + mk<S>(S(po.m[0][p]), S(po.m[1][p]), S(po.m[2][p]));
                }
            else
            {
                // The FP64 modes take two records at a time, their loads in
                // flight together (a record out of contact is loaded and
                // dropped): two resident blocks per SM do not hide a chain of
                // dependent loads per partner (400k spheres 2790 -> 2746 us
                // per ten steps).
                constexpr uint32_t kBatch = is_mixed<S>() ? 1 : 2;
                for(uint32_t p = off[i]; p < pe; p += kBatch)
                {
                    uint8_t hit[kBatch];
                    V3<S>   f[kBatch], t[kBatch];
#pragma unroll
                    for(uint32_t k = 0; k < kBatch; ++k)
                    {
                        const uint32_t q = p + k < pe ? p + k : pe - 1;
                        hit[k]           = p + k < pe ? po.contact[q] : uint8_t(0);
                        if(kBatch == 1 && !hit[k])
                            break;
                        f[k] = mk<S>(S(po.f[0][q]), S(po.f[1][q]), S(po.f[2][q]));
                        t[k] = mk<S>(S(po.t[0][q]), S(po.t[1][q]), S(po.t[2][q]));
                    }
#pragma unroll
                    for(uint32_t k = 0; k < kBatch; ++k)
                        if(hit[k])
                        {
                            nc += hit[k] == kContactParticle;
                            F = F + f[k];
                            T = T + t[k];
                            if(sp.has_kr)
                                T = T
                                    + mk<S>(S(po.m[0][p + k]), S(po.m[1][p + k]),
                                            S(po.m[2][p + k]));
                        }
                }
            }
        }
    }
    else
    {
        F = load3<S>(st.frc, i);
        T = load3<S>(st.trq, i);
    }
    if(sp.phases & PHASE_GRAVITY)
        F = F + m * sp.g; // Torce::addForce(mass * g)
    if(move)
    {
        // RigidBody::computeMomentum + FirstOrderExplicit::Move
        // (RigidBody.cpp:267-307, FirstOrderExplicit.cpp:46-60) or the Verlet kick-drift
        if constexpr(!is_mixed<S>())
            q = quat_from_basis(R);
        const V3<S> acc   = mk<S>(F.x / m, F.y / m, F.z / m);
        const V3<S> alpha = angular_acceleration(I, I1, w, T, q);
        V3<S>       trans;
        Quat<S>     dq;
        if(sp.integrator == GB_FIRST_ORDER_EXPLICIT)
        {
            trans = sp.dt * v;
            v     = v + sp.dt * acc;
            dq    = quaternion_change(w, sp.dt);
            w     = w + sp.dt * alpha;
        }
        else
        {
            v     = v + sp.h * acc;
            w     = w + sp.h * alpha;
            trans = sp.dt * v;
            dq    = quaternion_change(w, sp.dt);
        }
        // Transform3::updateTransform (Transform3.cpp:324-329)
        double xn[3];
#pragma unroll
        for(int k = 0; k < 3; ++k)
        {
            const S tk[3] = {trans.x, trans.y, trans.z};
            if constexpr(is_mixed<S>())
                xn[k] = x0[k] + (double)tk[k];
            else
                xn[k] = to_d(S(x0[k]) + tk[k]);
            st.pos[k][i] = xn[k];
        }
        float hi[4]; // mixed: the new orientation's FP32 part
        if constexpr(is_mixed<S>())
        {
            // the increment from the FP32 angular velocity, composed with the
            // compensated orientation and renormalised in FP64
            Quat<double> dq64, q64;
            dq64.w          = (double)dq.w;
            dq64.v          = cvt3<double>(dq.v);
            q64.w           = (double)q.w + (double)qlo[0];
            q64.v           = mk<double>((double)q.v.x + (double)qlo[1], (double)q.v.y + (double)qlo[2],
                                         (double)q.v.z + (double)qlo[3]);
            Quat<double> qn = qmul(dq64, q64);
            const double rn = 1.0 / sqrt(qn.w * qn.w + norm2(qn.v));
            const double c[4] = {qn.w * rn, qn.v.x * rn, qn.v.y * rn, qn.v.z * rn};
#pragma unroll
            for(int k = 0; k < 4; ++k)
            {
                hi[k]            = (float)c[k];
                st.rot[k][i]     = hi[k];
                st.rot[4 + k][i] = (float)(c[k] - (double)hi[k]);
            }
        }
        else
        {
            compose_left_by_rotation(R, dq);
#pragma unroll
            for(int k = 0; k < 9; ++k)
                st.rot[k][i] = to_d(R.m[k]);
        }
        // the obstacle candidates of the next detect, from the new pose
        if(mask_out)
            mask_out[i] = obstacle_mask_at<S>(
                tb, r,
                [&] {
                    if constexpr(is_mixed<S>())
                        return quat_to_matrix<S>(hi[0], hi[1], hi[2], hi[3]);
                    else
                        return R;
                },
                xn);
        st.vel[0][i] = (store_t<S>)to_d(v.x);
        st.vel[1][i] = (store_t<S>)to_d(v.y);
        st.vel[2][i] = (store_t<S>)to_d(v.z);
        st.omg[0][i] = (store_t<S>)to_d(w.x);
        st.omg[1][i] = (store_t<S>)to_d(w.y);
        st.omg[2][i] = (store_t<S>)to_d(w.z);
        // a move that leaves a non-finite state is reported by its own step
        // (the next step's hash would report it one step late)
        if(!(isfinite(xn[0]) && isfinite(xn[1]) && isfinite(xn[2]) && isfinite(to_d(v.x))
             && isfinite(to_d(v.y)) && isfinite(to_d(v.z)) && isfinite(to_d(w.x))
             && isfinite(to_d(w.y)) && isfinite(to_d(w.z))))
            atomicOr(flags, kFlagNonFinite);
        if(sp.phases != PHASE_STEP || sp.accumulate)
        {
            // Torce::reset
#pragma unroll
            for(int k = 0; k < 3; ++k)
            {
                st.frc[k][i] = store_t<S>(0);
                st.trq[k][i] = store_t<S>(0);
            }
        }
    }
    else
    {
        st.frc[0][i] = (store_t<S>)to_d(F.x);
        st.frc[1][i] = (store_t<S>)to_d(F.y);
        st.frc[2][i] = (store_t<S>)to_d(F.z);
        st.trq[0][i] = (store_t<S>)to_d(T.x);
        st.trq[1][i] = (store_t<S>)to_d(T.y);
        st.trq[2][i] = (store_t<S>)to_d(T.z);
    }
    if(contacts_out && (sp.phases & PHASE_DETECT))
        contacts_out[i] = nc;
    if(i == 0)
        atomicAdd(done, 1u); // the host counts the launches that completed
}

} // namespace gb
