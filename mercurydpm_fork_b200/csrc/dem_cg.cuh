// dem_cg.cuh -- Gaussian coarse-graining, CG<Coordinates, Gauss, StandardFields>.
//
// Restates CG::evaluateParticle and CG::evaluateContact (Kernel/CG/CG.hcc:333-528)
// with the Gauss function (Kernel/CG/Functions/Gauss.hcc:61-270), the
// coordinate systems O, XZ and XYZ (Kernel/CG/Coordinates/{O,XZ,XYZ}.cc,
// Base_XY_XZ_YZ.cc:32-53) and StandardFields (Kernel/CG/Fields/StandardFields.cc:184-250):
//   particles: phi = prefactor exp(-|r - x|^2 / 2w^2) within the cutoff;
//   contacts:  psi = line integral of the Gauss function between the two
//              ends the reference's IntegralType selects (I to P, contact to P,
//              I to contact), contact stress += F (x) branch psi, and
//              interaction force density += (+-F) phi(contact point) for
//              contacts with a fixed partner or a wall.
// Every point gathers its sums in a fixed order, so an evaluation is
// bit-for-bit reproducible: each particle and contact gets its point range per
// dimension (CG.hcc:340-395 and 478-495) and the bin of the range's first
// point; stable radix sorts order them by (bin, particle slot) and (bin,
// contact pair) (contact records arrive in launch order; the pair key makes
// their order canonical), and their values are written in that order, one array
// per value. A block then takes a tile of up to 8 points, one per warp, and
// brings the entries of the bins that can reach the tile through shared memory
// a chunk at a time; each lane takes a fixed stride of every chunk, and a
// fixed butterfly sums the lanes. Few tiles are split over several blocks by
// chunk, whose sums are added in block order.
// The contact records are those of the last force evaluation, i.e. the
// interactions the reference holds when writeOutputFiles evaluates CG at the
// start of the next step. Positions are the particles' own (for a pair that
// meets across a periodic boundary the reference's kept interaction joins the
// two real particles, InteractionHandler.cc:316-368, and CG uses those).
#pragma once
#include "dem_records.cuh"

namespace dem {

constexpr double CG_PI = 3.1415926535897932384626433832795;
constexpr double CG_SQRT_PI = 1.7724538509055160272981674833411;
constexpr double CG_SQRT_2 = 1.4142135623730950488016887242097;

struct CGDev {
    int coord;           // DEM_CG_*
    int instance;
    int n[3];            // points per dimension (1 for unresolved dimensions)
    int resolved[3];
    double min[3], max[3];
    double start[3], delta[3];
    double width, cutoff;
    double prefactor;    // Coordinates::getGaussPrefactor
    int direct[3];       // points a direct contact's range can cover, per dimension
};

__device__ __forceinline__ int cg_dims(const CGDev& g) { return g.coord == DEM_CG_XYZ ? 3 : (g.coord == DEM_CG_XZ ? 2 : 0); }

// squared distance in the resolved dimensions (XZ::getDistanceSquared, XYZ::getDistanceSquared)
__device__ __forceinline__ double cg_dist2(const CGDev& g, V3 p, V3 r)
{
    if (g.coord == DEM_CG_XYZ) return len2(r - p);
    if (g.coord == DEM_CG_XZ) return (p.x - r.x) * (p.x - r.x) + (p.z - r.z) * (p.z - r.z);
    return 0.0;
}

// Gauss::evaluateCGFunction
__device__ __forceinline__ double cg_phi(const CGDev& g, V3 p, V3 r)
{
    if (g.coord == DEM_CG_O) return 1.0;
    const double d2 = cg_dist2(g, p, r);
    return (d2 > g.cutoff * g.cutoff) ? 0.0 : g.prefactor * exp(-d2 / (2.0 * g.width * g.width));
}

// Coordinates::getGaussIntegralPrefactor (Base_XY_XZ_YZ.cc:40-53, XYZ.cc:157-171)
__device__ __forceinline__ double cg_integral_prefactor(const CGDev& g, double distance)
{
    const double widthSqrt2 = g.width * CG_SQRT_2;
    const double a = -g.cutoff;
    const double b = g.cutoff + distance;
    double prefactor;
    if (g.coord == DEM_CG_XZ) {
        prefactor = 1.0 / (widthSqrt2 * CG_SQRT_PI);
        prefactor /= erf(g.cutoff / (widthSqrt2));
    } else {
        prefactor = 1.0 / (CG_SQRT_2 * CG_SQRT_PI * g.width);
        prefactor = prefactor * prefactor / (1.0 - exp(-0.5 * ((g.cutoff / g.width) * (g.cutoff / g.width))));
    }
    return prefactor * 0.5 /
           (+erf(b / widthSqrt2) * b + widthSqrt2 / CG_SQRT_PI * exp(-((b / widthSqrt2) * (b / widthSqrt2))) -
            erf(a / widthSqrt2) * a - widthSqrt2 / CG_SQRT_PI * exp(-((a / widthSqrt2) * (a / widthSqrt2))));
}

__device__ __forceinline__ V3 cg_point(const CGDev& g, int i, int j, int k)
{
    return v3(g.start[0] + g.delta[0] * i, g.start[1] + g.delta[1] * j, g.start[2] + g.delta[2] * k);
}

// index range of the points a support [lo, hi] (in index units) touches: CG.hcc:340-395, 478-495
__device__ __forceinline__ void cg_range(const CGDev& g, int d, double lo_idx, double hi_idx, int& lo, int& hi)
{
    if (!g.resolved[d]) {
        lo = 0;
        hi = 1;
        return;
    }
    const double a = lo_idx + 1.0;
    const double b = hi_idx + 1.0;
    lo = a > 0.0 ? (a < (double)g.n[d] ? (int)a : g.n[d]) : 0;
    hi = b > 0.0 ? (b < (double)g.n[d] ? (int)b : g.n[d]) : 0;
}

// Words (8 bytes) of a particle as the gather reads it, one array each: position,
// mass, velocity, radius, and the first and last point of its range per
// dimension as int2. StandardFields::setFields(const BaseParticle&) is evaluated
// from them per point (fields 0-10 and 23-28).
enum CGParticleWord { CGP_X = 0, CGP_M = 3, CGP_V = 4, CGP_R = 7, CGP_RANGE = 8, CGP_WORDS = 11 };

// IntegralType of CG::getIntegralType (CG.hcc:451-466)
enum CGIntegral { CG_NONE = 0, CG_I_TO_P, CG_CONTACT_TO_P, CG_I_TO_CONTACT };

// Words of a contact: the ends of its line integral I and P, the particle P and
// the contact point, the direction of the line, force, the branch and
// interaction force density vectors of StandardFields::setFields(const
// BaseInteraction&), the integral prefactor, (IntegralType, whether the line has
// a length in the resolved dimensions) as int2, and the ranges.
enum CGContactWord {
    CGC_IE = 0, CGC_PE = 3, CGC_P = 6, CGC_C = 9, CGC_DIR = 12, CGC_F = 15, CGC_BRANCH = 18, CGC_IFD = 21,
    CGC_PREFACTOR = 24, CGC_TYPE = 25, CGC_RANGE = 26, CGC_WORDS = 29
};

__device__ __forceinline__ double cg_word(int a, int b)
{
    return __longlong_as_double(((long long)b << 32) | (long long)(unsigned)a);
}
__device__ __forceinline__ int2 cg_ints(double w)
{
    const long long v = __double_as_longlong(w);
    return make_int2((int)(unsigned)(v & 0xffffffffll), (int)(v >> 32));
}

// bins: one per point; a particle or contact goes to the point its range starts
// at. A contact whose range is wider than a direct one's can be (the ends of one
// across a periodic boundary lie a period apart) would widen every point's search
// to the whole period: it goes to a list of its own, bin npts; what adds to no
// point, to npts + 1.
__device__ __forceinline__ int cg_bin(const CGDev& g, const int lo[3]) { return (lo[0] * g.n[1] + lo[1]) * g.n[2] + lo[2]; }

__device__ __forceinline__ void cg_width_max(int* wmax, const int lo[3], const int hi[3])
{
    for (int k = 0; k < 3; ++k) atomicMax(wmax + k, hi[k] - lo[k]);
}

// range of a particle; false when it adds to no point
__device__ __forceinline__ bool cg_particle_range(const CGDev& g, V3 x, int lo[3], int hi[3])
{
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double pos = (&x.x)[k] - g.min[k];
        const double invDelta = g.n[k] / (g.max[k] - g.min[k]);
        const double idPos = pos * invDelta - 0.5;
        const double idCutoff = g.cutoff * invDelta;
        cg_range(g, k, idPos - idCutoff, idPos + idCutoff, lo[k], hi[k]);
        if (lo[k] >= hi[k]) return false;
    }
    return true;
}

// Particle s: its bin.
__global__ void __launch_bounds__(128) k_cg_particle_bins(DevPtrs d, CGDev g, unsigned* bin, int* slot, int* wmax)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= d.n) return;
    slot[s] = s;
    const int c = d.ctl->cur;
    const int4 is = d.info[c][s];
    int lo[3], hi[3];
    unsigned b = (unsigned)(g.n[0] * g.n[1] * g.n[2]) + 1u;
    // StandardFields::evaluateFixedParticles() is false
    if (is.z == g.instance && !(is.w & FLAG_FIXED) && cg_particle_range(g, xyz(d.pr[c][s]), lo, hi)) {
        b = (unsigned)cg_bin(g, lo);
        cg_width_max(wmax, lo, hi);
    }
    bin[s] = b;
}

// The particle at sorted position e: its words.
__global__ void __launch_bounds__(128) k_cg_particle_words(DevPtrs d, CGDev g, const int* order, const unsigned* bin,
                                                            double* out, int stride)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= d.n || bin[e] >= (unsigned)(g.n[0] * g.n[1] * g.n[2])) return;
    const int s = order[e], c = d.ctl->cur;
    const double4 p4 = d.pr[c][s];
    const double4 v4 = d.vm[c][s];
    int lo[3], hi[3];
    cg_particle_range(g, xyz(p4), lo, hi);
    const double w[CGP_WORDS] = {p4.x, p4.y, p4.z, 1.0 / v4.w, v4.x, v4.y, v4.z, p4.w,
                                 cg_word(lo[0], hi[0]), cg_word(lo[1], hi[1]), cg_word(lo[2], hi[2])};
#pragma unroll
    for (int k = 0; k < CGP_WORDS; ++k) out[(size_t)k * stride + e] = w[k];
}

// Contact record rix: its canonical key (P's slot, wall flag, I's slot or wall;
// bits: of a slot or wall index).
__global__ void __launch_bounds__(128) k_cg_contact_keys(DevPtrs d, unsigned nrec, int bits, unsigned long long* key,
                                                         int* idx)
{
    const unsigned rix = blockIdx.x * blockDim.x + threadIdx.x;
    if (rix >= nrec) return;
    const ContactRecord& r = d.records[rix];
    key[rix] = ((unsigned long long)(unsigned)r.slot_p << (bits + 1)) | ((unsigned long long)(r.is_wall ? 1u : 0u) << bits) |
               (unsigned long long)(unsigned)r.slot_i;
    idx[rix] = (int)rix;
}

// IntegralType and ends of a contact record; false when it adds to no point
__device__ __forceinline__ bool cg_contact_ends(const DevPtrs& d, const CGDev& g, const ContactRecord& rec, int c, int& type,
                                                V3& P, V3& C, V3& Ipos, int lo[3], int hi[3])
{
    const int4 ip = d.info[c][rec.slot_p];
    if (ip.z != g.instance) return false;
    const bool p_fixed = (ip.w & FLAG_FIXED) != 0;
    const bool i_fixed = rec.is_wall ? true : ((d.info[c][rec.slot_i].w & FLAG_FIXED) != 0);
    if (p_fixed)
        type = i_fixed ? CG_NONE : CG_I_TO_CONTACT;
    else
        type = i_fixed ? CG_CONTACT_TO_P : CG_I_TO_P;
    if (type == CG_NONE) return false;
    P = xyz(d.pr[c][rec.slot_p]);
    C = v3(rec.contact_point[0], rec.contact_point[1], rec.contact_point[2]);
    if (rec.is_wall) {
        const dem_wall& w = d.walls[rec.slot_i];
        Ipos = v3(w.position[0], w.position[1], w.position[2]);
    } else {
        Ipos = xyz(d.pr[c][rec.slot_i]);
    }
    // point range between P and I (the contact point when I is fixed): CG.hcc:478-495
    const V3 Iend = i_fixed ? C : Ipos;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (g.n[k] == 1) {
            lo[k] = 0;
            hi[k] = 1;
            continue;
        }
        const double invDelta = g.n[k] / (g.max[k] - g.min[k]);
        const double pk = ((&P.x)[k] - g.min[k]) * invDelta - 0.5;
        const double ik = ((&Iend.x)[k] - g.min[k]) * invDelta - 0.5;
        const double ck = g.cutoff * invDelta;
        cg_range(g, k, fmin(pk, ik) - ck, fmax(pk, ik) + ck, lo[k], hi[k]);
        if (lo[k] >= hi[k]) return false;
    }
    return true;
}

// The contact at canonical position j (record order[j]): its bin.
__global__ void __launch_bounds__(128) k_cg_contact_bins(DevPtrs d, CGDev g, unsigned nrec, const int* order, unsigned* bin,
                                                          int* rix, int* wmax)
{
    const unsigned j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= nrec) return;
    rix[j] = order[j];
    int type, lo[3], hi[3];
    V3 P, C, I;
    unsigned b = (unsigned)(g.n[0] * g.n[1] * g.n[2]);
    if (cg_contact_ends(d, g, d.records[order[j]], d.ctl->cur, type, P, C, I, lo, hi)) {
        if (hi[0] - lo[0] <= g.direct[0] && hi[1] - lo[1] <= g.direct[1] && hi[2] - lo[2] <= g.direct[2]) {
            b = (unsigned)cg_bin(g, lo);
            cg_width_max(wmax + 3, lo, hi);
        }
    } else {
        ++b;
    }
    bin[j] = b;
}

// The contact at sorted position e (record order[e]): its words.
__global__ void __launch_bounds__(128) k_cg_contact_words(DevPtrs d, CGDev g, unsigned nrec, const int* order,
                                                           const unsigned* bin, double* out, int stride)
{
    const unsigned e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nrec || bin[e] > (unsigned)(g.n[0] * g.n[1] * g.n[2])) return;
    const ContactRecord& rec = d.records[order[e]];
    int type, lo[3], hi[3];
    V3 P, C, Ipos;
    cg_contact_ends(d, g, rec, d.ctl->cur, type, P, C, Ipos, lo, hi);
    const V3 F = v3(rec.force[0], rec.force[1], rec.force[2]);
    const V3 n = v3(rec.normal[0], rec.normal[1], rec.normal[2]);
    // StandardFields::setFields(const BaseInteraction&, IntegralType); the
    // vectors of BaseInteraction.cc:459-476 (normal x distance, so a periodic
    // pair gets its image branch)
    V3 branch, ifd = zero3();
    const double dist = rec.is_wall ? 0.0 : sqrt(len2(v3(rec.branch[0], rec.branch[1], rec.branch[2])));
    if (type == CG_I_TO_P) {
        branch = n * dist;                  // getIP
    } else if (type == CG_I_TO_CONTACT) {
        ifd = -F;
        branch = n * dist + C - P;          // getIC
    } else {
        ifd = F;
        branch = P - C;                     // getCP
    }
    // Gauss::evaluateCGIntegral (Gauss.hcc:207-270)
    double nlen = 0.0;
    V3 dir = n;
    if (g.coord == DEM_CG_XZ) {
        nlen = sqrt(n.x * n.x + n.z * n.z);
        dir = n / nlen;
    } else if (g.coord == DEM_CG_XYZ) {
        nlen = sqrt(n.x * n.x + n.y * n.y + n.z * n.z);
    }
    const V3 ie = (type != CG_CONTACT_TO_P) ? Ipos : C;
    const V3 pe = (type != CG_I_TO_CONTACT) ? P : C;
    const bool line = g.coord != DEM_CG_O && !(fabs(nlen) < 1e-10);
    // the integral prefactor, from the length of the line: the reference takes it
    // at the first point of the range that passes the support test, where pN - iN
    // is the same length
    double prefactor = 0.0;
    if (line) {
        const V3 r = cg_point(g, lo[0], lo[1], lo[2]);
        double iN, pN;
        if (g.coord == DEM_CG_XZ) {
            iN = (ie.x - r.x) * dir.x + (ie.z - r.z) * dir.z;
            pN = (pe.x - r.x) * dir.x + (pe.z - r.z) * dir.z;
        } else {
            iN = dot(ie - r, dir);
            pN = dot(pe - r, dir);
        }
        prefactor = cg_integral_prefactor(g, pN - iN);
    }
    const double w[CGC_WORDS] = {ie.x, ie.y, ie.z, pe.x, pe.y, pe.z, P.x, P.y, P.z, C.x, C.y, C.z, dir.x, dir.y, dir.z,
                                 F.x, F.y, F.z, branch.x, branch.y, branch.z, ifd.x, ifd.y, ifd.z, prefactor,
                                 cg_word(type, line ? 1 : 0), cg_word(lo[0], hi[0]), cg_word(lo[1], hi[1]),
                                 cg_word(lo[2], hi[2])};
#pragma unroll
    for (int k = 0; k < CGC_WORDS; ++k) out[(size_t)k * stride + e] = w[k];
}

// First position of every bin in a list sorted by bin, start[0 .. npts + 1]:
// the entries of bin b are start[b] .. start[b + 1] - 1.
__global__ void k_cg_bin_starts(const unsigned* sorted_bin, int m, int npts, int* start)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > npts + 1) return;
    int lo = 0, hi = m;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (sorted_bin[mid] < (unsigned)b) lo = mid + 1;
        else hi = mid;
    }
    start[b] = lo;
}

constexpr int CG_ACC = 29;
constexpr int CG_TILE = 8;                    // points of a block, one per warp
constexpr int CG_THREADS = 32 * CG_TILE;
constexpr int CG_CHUNK = 128;                 // entries in shared memory at a time

struct CGTiles {
    int t[3];      // points of a tile per dimension (their product is at most CG_TILE)
    int n[3];      // tiles per dimension
    int split;     // blocks of a tile
};

// What one particle (column e of the words in shared memory) adds at point r.
__device__ __forceinline__ void cg_add_particle(const CGDev& g, const double* w, int e, V3 r, double (&acc)[CG_ACC])
{
    const double phi = cg_phi(g, v3(w[CGP_X * CG_CHUNK + e], w[(CGP_X + 1) * CG_CHUNK + e], w[(CGP_X + 2) * CG_CHUNK + e]), r);
    if (phi == 0.0) return;
    const double m = w[CGP_M * CG_CHUNK + e], rad = w[CGP_R * CG_CHUNK + e];
    const V3 v = v3(w[CGP_V * CG_CHUNK + e], w[(CGP_V + 1) * CG_CHUNK + e], w[(CGP_V + 2) * CG_CHUNK + e]);
    acc[0] += 4.0 / 3.0 * CG_PI * rad * rad * rad * phi; // BaseParticle::getVolume (3D)
    acc[1] += m * phi;
    acc[2] += v.x * m * phi; acc[3] += v.y * m * phi; acc[4] += v.z * m * phi;
    acc[5] += v.x * v.x * m * phi; acc[6] += v.x * v.y * m * phi; acc[7] += v.x * v.z * m * phi;
    acc[8] += v.y * v.y * m * phi; acc[9] += v.y * v.z * m * phi; acc[10] += v.z * v.z * m * phi;
    double ps = 1.0;
#pragma unroll
    for (int f = 0; f < 6; ++f) {
        acc[23 + f] += ps * phi;
        ps *= rad;
    }
}

// What one contact adds at point r.
__device__ __forceinline__ void cg_add_contact(const CGDev& g, const double* w, int e, V3 r, double (&acc)[CG_ACC])
{
    auto vec = [&](int k) { return v3(w[k * CG_CHUNK + e], w[(k + 1) * CG_CHUNK + e], w[(k + 2) * CG_CHUNK + e]); };
    const int2 type = cg_ints(w[CGC_TYPE * CG_CHUNK + e]); // (IntegralType, has a line)
    double psi;
    if (g.coord == DEM_CG_O) {
        psi = 1.0;
    } else if (!type.y) {
        psi = cg_phi(g, vec(CGC_C), r);
    } else {
        double iN, pN, t2;
        const V3 ie = vec(CGC_IE), pe = vec(CGC_PE), P = vec(CGC_P), n = vec(CGC_DIR);
        if (g.coord == DEM_CG_XZ) {
            iN = (ie.x - r.x) * n.x + (ie.z - r.z) * n.z;
            pN = (pe.x - r.x) * n.x + (pe.z - r.z) * n.z;
            t2 = (P.x - r.x) * (P.x - r.x) + (P.z - r.z) * (P.z - r.z) - pN * pN;
        } else {
            iN = dot(ie - r, n);
            pN = dot(pe - r, n);
            t2 = len2(P - r) - pN * pN;
        }
        const double w_sqrt_2 = CG_SQRT_2 * g.width;
        if (iN > g.cutoff || pN < -g.cutoff || t2 > g.cutoff * g.cutoff)
            psi = 0.0;
        else
            psi = w[CGC_PREFACTOR * CG_CHUNK + e] * (erf(pN / w_sqrt_2) - erf(iN / w_sqrt_2)) *
                  exp(-0.5 * t2 / (g.width * g.width));
    }
    if (psi != 0.0) {
        const V3 F = vec(CGC_F), b = vec(CGC_BRANCH);
        acc[11] += F.x * b.x * psi; acc[12] += F.x * b.y * psi; acc[13] += F.x * b.z * psi;
        acc[14] += F.y * b.x * psi; acc[15] += F.y * b.y * psi; acc[16] += F.y * b.z * psi;
        acc[17] += F.z * b.x * psi; acc[18] += F.z * b.y * psi; acc[19] += F.z * b.z * psi;
    }
    if (type.x != CG_I_TO_P) {
        const double phi = cg_phi(g, vec(CGC_C), r);
        if (phi != 0.0) {
            const V3 ifd = vec(CGC_IFD);
            acc[20] += ifd.x * phi;
            acc[21] += ifd.y * phi;
            acc[22] += ifd.z * phi;
        }
    }
}

// One chunk: its m entries (src) through shared memory, then every warp's point.
template <int WORDS, int RANGE, typename Add>
__device__ __forceinline__ void cg_chunk(const double* words, int stride, int m, bool active, const int (&pidx)[3],
                                         double* sh, const int* src, Add add)
{
    __syncthreads(); // src is there
    for (int k = threadIdx.x; k < WORDS * CG_CHUNK; k += CG_THREADS) {
        const int e = k & (CG_CHUNK - 1);
        if (e < m) sh[k] = words[(size_t)(k / CG_CHUNK) * stride + src[e]];
    }
    __syncthreads();
    if (active)
        for (int e = threadIdx.x & 31; e < m; e += 32) {
            bool in = true;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int2 range = cg_ints(sh[(RANGE + k) * CG_CHUNK + e]);
                in = in && range.x <= pidx[k] && pidx[k] < range.y;
            }
            if (in) add(sh, e);
        }
    __syncthreads();
}

// The entries of one kind that can reach the tile, a chunk at a time: the bins
// from w - 1 points before the tile's first point to its last, rows of bins
// along the last dimension (contiguous entries), CG_THREADS rows at a time.
// `part` of `split` blocks takes every split-th chunk.
template <int WORDS, int RANGE, typename Add>
__device__ __forceinline__ void cg_walk(const CGDev& g, const int (&p0)[3], const int (&p1)[3], const int* width,
                                        const int* start, const double* words, int stride, int split, int part,
                                        bool active, const int (&pidx)[3], double* sh, int* src, int* row_at, int* row_off,
                                        int* warp_sums, Add add)
{
    int lo[3], n[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        lo[k] = max(0, p0[k] - width[k] + 1);
        n[k] = p1[k] - lo[k] + 1;
    }
    const int nrows = n[0] * n[1];
    int chunk = 0;
    for (int r0 = 0; r0 < nrows; r0 += CG_THREADS) {
        const int row = r0 + (int)threadIdx.x;
        int len = 0;
        if (row < nrows) {
            const int b = ((lo[0] + row / n[1]) * g.n[1] + lo[1] + row % n[1]) * g.n[2] + lo[2];
            const int a = start[b];
            len = start[b + n[2]] - a;
            row_at[threadIdx.x] = a;
        }
        int total;
        const int off = block_exclusive_scan(len, warp_sums, total);
        row_off[threadIdx.x] = off; // the rows of this batch, ascending
        __syncthreads();
        for (int c0 = 0; c0 < total; c0 += CG_CHUNK, ++chunk) {
            if (chunk % split != part) continue;
            const int m = min(CG_CHUNK, total - c0);
            if ((int)threadIdx.x < m) { // the entry's place: the last row that starts at or before it
                const int e = c0 + threadIdx.x;
                int a = 0, b = CG_THREADS;
                while (b - a > 1) {
                    const int mid = (a + b) >> 1;
                    if (row_off[mid] <= e) a = mid;
                    else b = mid;
                }
                src[threadIdx.x] = row_at[a] + e - row_off[a];
            }
            cg_chunk<WORDS, RANGE>(words, stride, m, active, pidx, sh, src, add);
        }
        __syncthreads();
    }
}

// The entries begin .. end - 1, whatever their ranges: those whose range meets
// the tile, in order.
template <int WORDS, int RANGE, typename Add>
__device__ __forceinline__ void cg_walk_wide(const int (&p0)[3], const int (&p1)[3], int begin, int end, const double* words,
                                             int stride, int split, int part, bool active, const int (&pidx)[3], double* sh,
                                             int* src, int* warp_sums, Add add)
{
    for (int b = begin + part * CG_THREADS; b < end; b += split * CG_THREADS) {
        const int e = b + (int)threadIdx.x;
        bool meets = e < end;
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (meets) {
                const int2 range = cg_ints(words[(size_t)(RANGE + k) * stride + e]);
                meets = range.x <= p1[k] && p0[k] < range.y;
            }
        int total;
        const int at = block_exclusive_scan(meets ? 1 : 0, warp_sums, total);
        for (int c0 = 0; c0 < total; c0 += CG_CHUNK) {
            if (meets && at >= c0 && at < c0 + CG_CHUNK) src[at - c0] = e;
            cg_chunk<WORDS, RANGE>(words, stride, min(CG_CHUNK, total - c0), active, pidx, sh, src, add);
        }
        __syncthreads();
    }
}

// Bound by the latency of its FP64 chains (two error functions and an exponential
// per contact and point in reach) in warps that are partly idle: of a box of
// 20,000 on 20 x 20 x 24 points, 18.8 of 32 lanes active (the others' entries
// failed the range or cutoff test), 16 warps per SM, 44 % of the issue slots, 27 %
// of the FP64 pipe, DRAM idle. One warp per point read every candidate's record from L2
// again for each point, some 6.8 GB per evaluation of the 200,000 chute on 100 x
// 50 points, and searched the whole period once a contact crossed it. Tiles of
// 8 points with a list of their own for those contacts: 1.25 -> 0.75 ms there,
// 1.23 -> 0.40 ms for a box of 20,000 on 20 x 20 x 24 points (without that list
// the chute took 2.3 ms).
__global__ void __launch_bounds__(CG_THREADS, 2) k_cg_gather(CGDev g, CGTiles tiles, const double* pwords, int pstride,
                                                             const int* pstart, const double* cwords, int cstride,
                                                             const int* cstart, const int* wmax, double volume, double* out)
{
    __shared__ double sh[CGC_WORDS * CG_CHUNK];
    __shared__ int src[CG_CHUNK], row_at[CG_THREADS], row_off[CG_THREADS], warp_sums[CG_TILE];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int part = blockIdx.x % tiles.split, tile = blockIdx.x / tiles.split;
    const int tidx[3] = {tile / (tiles.n[2] * tiles.n[1]), (tile / tiles.n[2]) % tiles.n[1], tile % tiles.n[2]};
    int p0[3], p1[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        p0[k] = tidx[k] * tiles.t[k];
        p1[k] = min(g.n[k], p0[k] + tiles.t[k]) - 1;
    }
    const int pidx[3] = {p0[0] + wid / (tiles.t[2] * tiles.t[1]), p0[1] + (wid / tiles.t[2]) % tiles.t[1],
                         p0[2] + wid % tiles.t[2]};
    const bool active = pidx[0] <= p1[0] && pidx[1] <= p1[1] && pidx[2] <= p1[2];
    const V3 r = cg_point(g, pidx[0], pidx[1], pidx[2]);
    double acc[CG_ACC];
#pragma unroll
    for (int f = 0; f < CG_ACC; ++f) acc[f] = 0.0;
    cg_walk<CGP_WORDS, CGP_RANGE>(g, p0, p1, wmax, pstart, pwords, pstride, tiles.split, part, active, pidx, sh, src, row_at,
                                  row_off, warp_sums, [&](const double* w, int e) { cg_add_particle(g, w, e, r, acc); });
    // the direct contacts, then those across a periodic boundary
    auto add = [&](const double* w, int e) { cg_add_contact(g, w, e, r, acc); };
    const int npts_ = g.n[0] * g.n[1] * g.n[2];
    for (int wide = 0; wide < 2; ++wide) {
        if (wide)
            cg_walk_wide<CGC_WORDS, CGC_RANGE>(p0, p1, cstart[npts_], cstart[npts_ + 1], cwords, cstride, tiles.split, part,
                                               active, pidx, sh, src, warp_sums, add);
        else
            cg_walk<CGC_WORDS, CGC_RANGE>(g, p0, p1, wmax + 3, cstart, cwords, cstride, tiles.split, part, active, pidx, sh,
                                          src, row_at, row_off, warp_sums, add);
    }
    if (!active) return;
    // fixed butterfly over the lanes; lane f writes field f
    double mine = 0.0;
#pragma unroll
    for (int f = 0; f < CG_ACC; ++f) {
        double v = acc[f];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == f) mine = v;
    }
    const size_t pt = (size_t)(pidx[0] * g.n[1] + pidx[1]) * g.n[2] + pidx[2];
    const size_t npts = (size_t)g.n[0] * g.n[1] * g.n[2];
    if (lane < CG_ACC) out[(part * npts + pt) * DEM_CG_NFIELDS + lane] = tiles.split == 1 ? mine / volume : mine;
}

// the parts of split tiles, in block order
__global__ void __launch_bounds__(256) k_cg_join(const double* parts, int split, size_t nvals, double volume, double* out)
{
    const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nvals) return;
    double v = 0.0;
    for (int s = 0; s < split; ++s) v += parts[s * nvals + k];
    out[k] = v / volume;
}

} // namespace dem

extern "C" int dem_cg_eval(dem_handle* hh, const dem_cg_grid* grid, double* fields_out)
{
    Handle* h = reinterpret_cast<Handle*>(hh);
    if (!h || !grid || !fields_out) return fail(h, DEM_ERR_BAD_INPUT, "dem_cg_eval: bad arguments");
    if (!h->uploaded || h->initial_pending) return fail(h, DEM_ERR_STATE, "no force evaluation yet (call dem_step)");
    if (!h->records_valid)
        return fail(h, DEM_ERR_CAPACITY, "contact records of the last evaluation overflowed; step again");
    if (grid->coordinates != DEM_CG_O && grid->coordinates != DEM_CG_XZ && grid->coordinates != DEM_CG_XYZ)
        return fail(h, DEM_ERR_BAD_INPUT, "dem_cg_eval: coordinates must be DEM_CG_O, DEM_CG_XZ or DEM_CG_XYZ");
    if (grid->instance < 0 || grid->instance >= (int)h->inst.size())
        return fail(h, DEM_ERR_BAD_INPUT, "dem_cg_eval: instance out of range");
    if (!(grid->width > 0.0)) return fail(h, DEM_ERR_BAD_INPUT, "dem_cg_eval: width must be positive");
    CGDev g{};
    g.coord = grid->coordinates;
    g.instance = grid->instance;
    const bool res[3] = {g.coord != DEM_CG_O, g.coord == DEM_CG_XYZ, g.coord != DEM_CG_O};
    long long npts = 1;
    for (int k = 0; k < 3; ++k) {
        g.resolved[k] = res[k];
        g.n[k] = res[k] ? grid->n[k] : 1;
        if (g.n[k] < 1) return fail(h, DEM_ERR_BAD_INPUT, "dem_cg_eval: point counts must be >= 1");
        g.min[k] = grid->min[k];
        g.max[k] = grid->max[k];
        // spaceEvenly (Kernel/CG/Coordinates/XZ.h:136-152, XYZ.h:189-210)
        g.delta[k] = (g.max[k] - g.min[k]) / g.n[k];
        g.start[k] = g.min[k] + 0.5 * g.delta[k];
        npts *= g.n[k];
    }
    g.width = grid->width;
    double rmax = 0.0;
    const dem::InstanceDev& I = h->inst[grid->instance];
    for (int l = 0; l < I.n_levels; ++l) rmax = std::max(rmax, I.level_rmax[l]);
    g.cutoff = (grid->cutoff_factor > 0.0 ? grid->cutoff_factor : 3.0) * grid->width; // Gauss::setWidth
    for (int k = 0; k < 3; ++k) // centres at most two radii and the interaction distance apart, two cutoffs beyond them
        g.direct[k] = (int)std::min(1e9, std::ceil((2.0 * rmax + I.max_interaction_distance + 2.0 * g.cutoff) / g.delta[k]) + 2.0);
    // Coordinates::getGaussPrefactor
    const double pf = 1.0 / (CG_SQRT_2 * CG_SQRT_PI * g.width);
    if (g.coord == DEM_CG_XZ) {
        g.prefactor = pf * pf / (1.0 - exp(-0.5 * ((g.cutoff / g.width) * (g.cutoff / g.width))));
    } else if (g.coord == DEM_CG_XYZ) {
        const double cw = g.cutoff / g.width;
        g.prefactor = pf * pf * pf / (erf(cw / CG_SQRT_2) - CG_SQRT_2 / CG_SQRT_PI * cw * exp(-0.5 * (cw * cw)));
    } else {
        g.prefactor = 1.0;
    }
    // CG::volumeAverageVariables: volume of the averaged dimensions
    double volume = 1.0;
    if (g.coord == DEM_CG_XZ) volume = g.max[1] - g.min[1];
    if (g.coord == DEM_CG_O) volume = (g.max[0] - g.min[0]) * (g.max[1] - g.min[1]) * (g.max[2] - g.min[2]);
    CU(cudaSetDevice(h->device));
    using namespace dem;
    const int n = h->d.n;
    const int nrec = (int)h->n_records;
    const size_t nvals = (size_t)npts * DEM_CG_NFIELDS;
    if (npts > (1ll << 30)) return fail(h, DEM_ERR_BAD_INPUT, "dem_cg_eval: too many points");
    auto bits_for = [](unsigned long long v) { // of values 0 .. v
        int b = 1;
        while ((v >> b) != 0) ++b;
        return b;
    };
    const int bits = bits_for((unsigned long long)npts + 1); // bin keys 0 .. npts + 1
    const int index_bits = bits_for((unsigned long long)std::max(n, h->d.n_walls));
    const int key_bits = std::min(64, 2 * index_bits + 1);
    size_t t1 = 0, t2 = 0, t3 = 0;
    CU(cub::DeviceRadixSort::SortPairs(nullptr, t1, (const unsigned*)nullptr, (unsigned*)nullptr, (const int*)nullptr,
                                       (int*)nullptr, std::max(n, 1), 0, bits, h->stream));
    CU(cub::DeviceRadixSort::SortPairs(nullptr, t2, (const unsigned long long*)nullptr, (unsigned long long*)nullptr,
                                       (const int*)nullptr, (int*)nullptr, std::max(nrec, 1), 0, key_bits, h->stream));
    CU(cub::DeviceRadixSort::SortPairs(nullptr, t3, (const unsigned*)nullptr, (unsigned*)nullptr, (const int*)nullptr,
                                       (int*)nullptr, std::max(nrec, 1), 0, bits, h->stream));
    const size_t tmp_bytes = std::max(t1, std::max(t2, t3));
    // tiles of up to 8 neighbouring points; too few of them for two blocks on
    // every SM are split by chunk
    CGTiles tiles{};
    const int shape[3][3] = {{1, 1, 1}, {2, 1, 4}, {2, 2, 2}}; // O, XZ, XYZ
    const int* t = shape[g.coord == DEM_CG_O ? 0 : (g.coord == DEM_CG_XZ ? 1 : 2)];
    long long n_tiles = 1;
    for (int k = 0; k < 3; ++k) {
        tiles.t[k] = t[k];
        tiles.n[k] = (g.n[k] + t[k] - 1) / t[k];
        n_tiles *= tiles.n[k];
    }
    tiles.split = (int)std::max<long long>(1, std::min<long long>(64, 8ll * h->sm_count / n_tiles));
    // one scratch arena for the evaluation
    Arena arena;
    auto take = [&arena](size_t bytes) { return arena.take(bytes); };
    const size_t nn = std::max(n, 1), nr = std::max(nrec, 1);
    const size_t o_out = take(nvals * sizeof(double));
    const size_t o_parts = tiles.split > 1 ? take(tiles.split * nvals * sizeof(double)) : o_out;
    const size_t o_pwords = take(nn * CGP_WORDS * 8), o_cwords = take(nr * CGC_WORDS * 8);
    const size_t o_pbin0 = take(nn * 4), o_pbin1 = take(nn * 4), o_pslot0 = take(nn * 4), o_pslot1 = take(nn * 4);
    const size_t o_ckey0 = take(nr * 8), o_ckey1 = take(nr * 8), o_cidx0 = take(nr * 4), o_cidx1 = take(nr * 4);
    const size_t o_cbin0 = take(nr * 4), o_cbin1 = take(nr * 4);
    const size_t o_pstart = take(((size_t)npts + 2) * 4), o_cstart = take(((size_t)npts + 2) * 4);
    const size_t o_wmax = take(6 * sizeof(int));
    const size_t o_tmp = take(tmp_bytes);
    Scratch scratch(h);
    CU(scratch.take(arena.total));
    auto at = [&scratch](size_t off) { return (void*)(scratch.p + off); };
    double *dout = (double*)at(o_out), *parts = (double*)at(o_parts);
    double *pwords = (double*)at(o_pwords), *cwords = (double*)at(o_cwords);
    unsigned *pbin0 = (unsigned*)at(o_pbin0), *pbin1 = (unsigned*)at(o_pbin1);
    int *pslot0 = (int*)at(o_pslot0), *pslot1 = (int*)at(o_pslot1);
    unsigned long long *ckey0 = (unsigned long long*)at(o_ckey0), *ckey1 = (unsigned long long*)at(o_ckey1);
    int *cidx0 = (int*)at(o_cidx0), *cidx1 = (int*)at(o_cidx1);
    unsigned *cbin0 = (unsigned*)at(o_cbin0), *cbin1 = (unsigned*)at(o_cbin1);
    int *pstart = (int*)at(o_pstart), *cstart = (int*)at(o_cstart);
    int* wmax = (int*)at(o_wmax);
    void* tmp = at(o_tmp);
    CU(cudaMemsetAsync(wmax, 0, 6 * sizeof(int), h->stream));
    size_t tb;
    if (n > 0) {
        k_cg_particle_bins<<<grid_for(n, 128), 128, 0, h->stream>>>(h->d, g, pbin0, pslot0, wmax);
        tb = tmp_bytes;
        CU(cub::DeviceRadixSort::SortPairs(tmp, tb, pbin0, pbin1, pslot0, pslot1, n, 0, bits, h->stream));
        k_cg_particle_words<<<grid_for(n, 128), 128, 0, h->stream>>>(h->d, g, pslot1, pbin1, pwords, (int)nn);
    }
    k_cg_bin_starts<<<grid_for(npts + 2, 256), 256, 0, h->stream>>>(pbin1, n, (int)npts, pstart);
    if (nrec > 0) {
        k_cg_contact_keys<<<grid_for(nrec, 128), 128, 0, h->stream>>>(h->d, (unsigned)nrec, index_bits, ckey0, cidx0);
        tb = tmp_bytes;
        CU(cub::DeviceRadixSort::SortPairs(tmp, tb, ckey0, ckey1, cidx0, cidx1, nrec, 0, key_bits, h->stream));
        k_cg_contact_bins<<<grid_for(nrec, 128), 128, 0, h->stream>>>(h->d, g, (unsigned)nrec, cidx1, cbin0, cidx0, wmax);
        tb = tmp_bytes;
        CU(cub::DeviceRadixSort::SortPairs(tmp, tb, cbin0, cbin1, cidx0, cidx1, nrec, 0, bits, h->stream));
        k_cg_contact_words<<<grid_for(nrec, 128), 128, 0, h->stream>>>(h->d, g, (unsigned)nrec, cidx1, cbin1, cwords, (int)nr);
    }
    k_cg_bin_starts<<<grid_for(npts + 2, 256), 256, 0, h->stream>>>(cbin1, nrec, (int)npts, cstart);
    k_cg_gather<<<(unsigned)(n_tiles * tiles.split), CG_THREADS, 0, h->stream>>>(g, tiles, pwords, (int)nn, pstart, cwords,
                                                                                (int)nr, cstart, wmax, volume, parts);
    if (tiles.split > 1)
        k_cg_join<<<grid_for((long long)nvals, 256), 256, 0, h->stream>>>(parts, tiles.split, nvals, volume, dout);
    CU(cudaGetLastError());
    CU(cudaMemcpyAsync(fields_out, dout, nvals * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CU(cudaStreamSynchronize(h->stream));
    return DEM_OK;
}
