// cm_scene.h -- flattened scene description shared by host and device.
//
// The host facade records the reference's object graph (Region tree,
// NormalShapes, MONSEL_MaterialScatterModel with its ScatterMechanisms) and
// flattens it into these plain arrays.  Device units: energy in eV, length in
// nm, rates in 1/nm.  Geometry is double precision in every mode.
#pragma once
#include <stdint.h>

namespace cm {

constexpr int kMaxMech = 8;
constexpr int kMaxElem = 8;
constexpr int kMaxCore = 16;
constexpr int kMaxShapeDepth = 4;
constexpr int kGridMinChildren = 24;  // regions with at least this many bounded children get a ChildGrid

// NISTMonte/MonteCarloSS.cu:32-33 in nm
constexpr double kChamberRadiusNm = 0.1e9;
constexpr double kSmallDispNm = 1.0e-6;
constexpr double kPi = 3.14159265358979323846;

enum ShapeKind : int { SHAPE_SPHERE = 1, SHAPE_PLANES = 2, SHAPE_INTERSECTION = 3, SHAPE_CYLINDER = 4, SHAPE_UNION = 5 };
enum MechKind : int { MECH_NISTMOTT = 1, MECH_TABULATED = 2, MECH_FITTED = 3, MECH_PHONON = 4, MECH_POLARON = 5 };

struct Shape {
  int kind;
  int anyunion;      // a union below (or at) this node
  int a, b;          // intersection / union children
  int plane0, np;    // planes [plane0, plane0+np)
  double c[3], r;    // sphere (nm)
  // NormalCylindricalShape (nm): end0, axis = end1 - end0, axis / |axis| as the
  // reference computed it, radius^2, |axis|^2, |axis|
  double e0[3], ax[3], nax[3], rad2, len2, len;
};

struct Plane {
  double n[3];
  double p[3];       // nm
};

struct Region {
  int parent, msm, shape;
  int child0, nchild;  // children indices in Scene::children
  int cls;             // wave segment of electrons in this region (by material model)
  double bb[6];        // axis-aligned box holding the region's shape (nm): min xyz, max xyz
  int grid;            // index of the grid over this region's children, -1: scan them in order
};

// A uniform x-y grid over the children of a region with many of them.  Each cell lists, ascending,
// the positions (in the region's child list) of the children whose box overlaps it; children whose
// box is unbounded in x or y are listed once apart.  Searches visit only the listed children and
// resolve ties by position, so they find what the in-order scan finds.
struct ChildGrid {
  double x0, y0, dx, dy;  // nm
  double z0, z1;          // the listed children's boxes lie between
  int nx, ny;
  int cell0;              // cell (ix, iy) lists grid_items[cell_start[cell0 + iy * nx + ix] .. next)
  int unb0, nunb;         // the unbounded children: grid_items[unb0 .. unb0 + nunb)
};

// The part of a region that lies strictly inside its shape, for the childless regions of models with
// mechanisms, as half-spaces (FastPlane) and at most one cylinder wall.  A step whose two ends are both in
// there meets no boundary, and the region test and the boundary search need not run: kFastMarginNm is far
// above the rounding of either evaluation (at most ~1e-6 nm for coordinates below 1e9 nm; shapes given by
// larger ones keep a wider margin, see inside_of), so both decide alike.
struct alignas(16) FastRegion {
  int msm, cls;          // as the Region's
  int plane0, np;        // half-spaces fast_planes[plane0, plane0 + np); np < 0: no such description
  int cyl;               // fast_cyls index, -1: none
  int pad[3];
};
struct alignas(16) FastPlane {
  double n[3], d;        // inside: n . p < d
};
struct FastCyl {
  double e0[3], ax[3];   // a point of the axis and its unit vector
  double rad2;           // inside: squared distance from the axis < rad2
};
constexpr double kFastMarginNm = 1e-4;

// electrons are kept in one wave segment per material class, so that the
// threads of a warp mostly run the same material's code
// (of the models with mechanisms: vacuum has none and takes no fast flight)
constexpr int kClasses = 3;
// a wave has two segments per class: electrons at or above kSegmentSplitEv and below it (the low band
// takes the Browning branch of the elastic cross sections and the low-energy secondary paths), so that
// a warp's threads mostly run the same branches
constexpr int kSegments = 2 * kClasses;
constexpr double kSegmentSplitEv = 50.0;
// and two more for the full flight: kSlowSegment for electrons that may meet a boundary of their region (at
// one just met, or handed back by the fast flight), kOpenSegment for those in a region without a FastRegion
// description (vacuum, a region with children), whose steps run through other code
constexpr int kSlowSegment = kSegments, kOpenSegment = kSegments + 1, kWaveSegments = kSegments + 2;
constexpr int kMaxWave = 1 << 27;  // electrons per wave segment: kWaveSegments x and 8 x (the pool) stay within int

// The structs the transport kernels read are in the compute precision R, rounded once when the scene is
// built: a value the physics casts to float would otherwise cost a double load and a conversion at a
// sixteenth of the arithmetic rate in every step.

// JoyLuoNieminenCSD (JMONSEL/JoyLuoNieminenCSD.cu:42-121) in eV/nm units
template <typename R>
struct Jln {
  int nce;
  R minE, breakE;            // eV
  R gamma15;                 // R(1.5) * R(gamma), gamma in eV^-1.5 nm^-1
  R coef[kMaxElem];          // eV^2 / nm
  R recipJ[kMaxElem];        // 1/eV
  R beta[kMaxElem];
};

// One element of a NISTMott mechanism: what its cross section (times the rate factor, 1/nm) takes.  kel is
// a0^2 * scalefactor * density * N_A per table unit, kbrown the same factor for a cross section in nm^2.
template <typename R>
struct alignas(16) ElemRate {
  R below;                   // extrapolation energy of the mechanism's method, eV
  R sf, kbrown;              // Browning's scale factor and rate factor
  R b0, b1, b2;              // Browning: b0 / (e + b1 sqrt(e) + b2 / sqrt(e)), e in keV
  R kel, lin;                // table rate factor; method 3: kel * table value at `below`
  R ra, rb;                  // screened Rutherford: ra / (E + rb)
  int off_spwem;             // the element's cross sections in the blob
  int mott;                  // index into Scene::mott
};

// A search guide of one axis of an NU table: the argument's bucket, found by arithmetic, holds at most one
// node, so one comparison with that node finds the interval the reference's bisection finds.  The bucket
// is (x - x0) * scale rounded down, or for kind 2 the leading bits of x (an axis spaced by a factor).
struct AxisGuide {
  int kind;                  // 0: none (bisection), 1: linear, 2: leading bits
  int off, n;                // entries guides[off, off + n)
  int shift, base;           // kind 2
  double x0, scale;          // kind 1
};
// bucket entry: nodes below the bucket, and the first index of the order-3 window of an argument that is
// not above (first0) or above (first1) the bucket's node
struct alignas(8) GuideEntry {
  unsigned short below, first0, first1, pad;
};

// NUTableInterpolation (dims 1..3) in the precision blob, with double copies in SceneView::dbl of every
// axis (window selection compares the argument with the reference's abscissae in double in both
// precisions) and of a 3-D table's values (its reference d3 step extrapolates from the first energy
// window, which amplifies rounding by orders of magnitude, so FP32 evaluates it in double too)
struct Table {
  int dim;
  int n[3];
  int off_x[3];
  int off_v;
  int off_x64[3];            // axes in dbl
  int off_v64;               // values in dbl (3-D tables), else -1
  AxisGuide guide[3];
  double domain[3][2];
  double range[2];
};

template <typename R>
struct Mech {
  int kind;
  // NISTMott via SelectableElasticSM
  int nel;
  int mottMethod;            // NISTMottRS method 1..3
  R belowMin, belowMax;      // smallest and largest extrapolation energy of its elements
  // TabulatedInelasticSM (JMONSEL/TabulatedInelasticSM.cu:461-498), energies in eV
  int methodSE;
  R energyOffset, minEgenSE, rateMult, energyCBbottom, bandgap, energyGap, offsetFermiEnergy, bEref;
  R eiDomain0, iimfpDomain0, rangeSE0lo, rangeSE0hi;
  // FittedInelSM: SE energy (and lowest energy with a rate), energy per SE
  R fittedSE, energySEgen;
  // phonon / polaron
  R prefactor, extinction, cutoff;
  double phononE, prefactor64;
  ElemRate<R> el[kMaxElem];
  int ncore;
  R core[kMaxCore];
  Jln<R> csd;
  Table iimfp, red, theta, se0;  // copies of the tables it uses
};

template <typename R>
struct alignas(16) Msm {
  int nmech, mech0;          // mechanisms [mech0, mech0+nmech)
  unsigned kinds;            // their kinds, 4 bits each, the first lowest
  int csd;                   // 0 = ZeroCSD, 1 = JoyLuoNieminenCSD
  R minE;                    // eV (may be -inf)
  R ecb;                     // E_CB bottom of this material, eV
  R u0;                      // barrier's u0 (= E_CB of the material it was built for), eV
  int classical;
  double lambda;
  R lambdaFactor;            // 1/sqrt(eV)
  int material;
  int vacuum;
  Jln<R> jln;
};

// NISTMottRS per element; the tables live in the precision blob, the extrapolation constants are
// indexed by method (1: Factory, 2: Factory100, 3: Factory100Lin; entry 0 copies method 1)
struct Mott {
  int Z;
  int off_spwem, off_x1;     // offsets of the cross sections in the table blob (off_x1 unused: -1)
  int off_x1d;               // offset of the 61 x 201 quantile table in the double copies (dbl)
  double extrapolateBelowEnergy[4];  // eV
  double sfBrowning[4];
  double mottXSatMin[4];             // table value (units of a0^2) at extrapolateBelowEnergy
  double zp17, zp2, zp3;
  double rutherfordA, rutherfordB;  // sigma = A / (E + B) in nm^2 with E in eV
  double rutherfordAlpha;           // alpha = rutherfordAlpha / E
};

// The whole scene as device pointers (one struct passed by value to kernels)
template <typename R>
struct SceneView {
  const Shape* shapes;
  const Plane* planes;
  const Region* regions;
  const int* children;
  const Msm<R>* msms;
  const Mech<R>* mechs;
  const Mott* mott;
  const Table* tables;
  const GuideEntry* guides;
  const ChildGrid* grids;
  const int* cell_start;
  const int* grid_items;
  const FastRegion* fast;    // per region
  const FastPlane* fast_planes;
  const FastCyl* fast_cyls;
  const R* blob;             // table data in compute precision
  const double* dbl;         // double copies: NISTMott quantile tables (sampled angles within 1e-6 in FP32
                             // too), NU-table axes and 3-D table values
  int chamber;
  int options;               // bit 0: JMONSEL fixes, bit 1: exact CSG in FP32
  int depth;                 // deepest intersection nesting; 0 = every shape is a leaf (plane set or sphere)
  double dl50, param;        // NISTMott log-energy grid (eV)
  R maxMott;                 // NISTMottRS MAX_NISTMOTT in eV
  int nstaged;               // elements of blob's prefix this kernel holds in shared memory (0: none)
  int nstage;                // elements of the prefix the scene places for staging (a multiple of 16 bytes)
};

}  // namespace cm
