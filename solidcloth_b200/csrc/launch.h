// launch.h — host-callable launchers for the cloth-step kernels (step_kernels.cu).
#pragma once
#include "sc_internal.cuh"

namespace sc {

constexpr int KVT = 48;        // self vertex-triangle contact slots per vertex
constexpr int KCAND = 256;     // BVH candidates kept per proximity query
constexpr int KRES = 96;       // distinct features tracked per vertex for the dedup
constexpr int BROAD_WALKS = 2; // broad-phase modes callers may name (one kernel serves both)
constexpr int CCD_VT_PAIRS = 128, CCD_EE_PAIRS = 96; // pair store per vertex / edge
constexpr int CCD_VT_HITS = 32, CCD_EE_HITS = 16;   // continuous contacts per vertex / edge
constexpr int MAX_COLOURS = 128; // independent-set colouring rounds per contact class
constexpr int WALL_SLOTS = 5;

// Vertex contact slot (walls, sphere, SDF, mesh vertex contacts).
struct VC { float4 point; float4 normal; float2 lam; int feature; int mesh; };
// Triangle contact (cloth triangle vs collider vertex / sphere / SDF).
struct TC { uint4 idx; float4 point; float4 normal; float4 w; float2 lam; int feature; int mesh; };
// Edge contact (cloth edge vs collider edge / sphere).
struct EC { uint4 idx; float4 point; float4 normal; float4 w; float2 lam; int feature; int mesh; };
// Self contact (vertex-triangle: i1..i3 triangle, i4 vertex; edge-edge: (i1,i2) x (i3,i4)).
struct SCt { uint4 idx; float4 normal; float4 w; float2 lam; float side; float error; };

// Vertex collider descriptor (world order).
struct VColl
{
    int type;        // 1 walls, 3 sphere, 7 sdf, 4 mesh
    int slotBase;    // first slot of this collider in the vertex-contact slot array
    int kmax;        // slots per vertex
    int vBegin, vCount; // particles it acts on (a batch instance's range; else all)
    int countBase;   // first of its vCount per-particle slot counts
    int mesh;        // mesh collider index for type 4
    float4 a, b;     // walls: lo, hi; sphere: centre (a.xyz), radius (a.w)
    cudaTextureObject_t val, grad; // sdf
    float4 sdfLo, sdfSteps;        // sdf box min, steps
    int4 sdfCells;
};

// scratch of one class's contact colouring: per particle its number of contacts (zero
// between substeps) and its list's end; per list entry the key and, sorted, the
// contact; per contact its successors' entries and how many particles hold it back
struct ColourScratch
{
    int* deg; int* cur;
    unsigned long long* key; int* sorted;
    int4* next; int* rem;
};

struct Buffers
{
    // vertex contacts: counts[coll][N] (uint8), slots[slotBase + i*kmax + k]
    uint8_t* vcCount;
    VC* vc;
    int numVColl;
    const VColl* vcoll;       // device copy
    const int2* instColl;     // batch: (first collider, count) per instance; null: all colliders act on all
    // triangle / edge contacts: per-collider slot arrays, flags, dense lists
    TC* tcSlot; int* tcFlag; TC* tcList; int* tcCount; int tcCap;
    EC* ecSlot; int* ecFlag; EC* ecList; int* ecCount; int ecCap;
    // self contacts
    int* stCnt; SCt* stSlot; SCt* stList; int* stCount; int stCap;
    int* seFlag; SCt* seSlot; SCt* seList; int* seCount; int seCap;
    // continuous collision: candidate pairs (query, candidate), those left to the full
    // test, and the hits among them with each query's number of hits
    int2* ccdVtPairs; int2* ccdEePairs; int* ccdVtPairCount; int* ccdEePairCount; int ccdVtCap, ccdEeCap;
    int2* ccdVtTest; int2* ccdEeTest; int* ccdVtTestCount; int* ccdEeTestCount;
    int2* ccdVtHits; int2* ccdEeHits; int* ccdVtHitTotal; int* ccdEeHitTotal;
    int* ccdVtHitCnt; int* ccdEeHitCnt;
    int2* ccdVtSorted; int2* ccdEeSorted;
    // colouring scratch
    ColourScratch colouring[2];  // self vertex-triangle, self edge-edge
    int* selfColours;            // colours of the two classes in this substep
    int* colour; int* order; int* colourStart; int colourCap;
    // scan scratch: block sums, per-item offsets, totals
    int* scanBlock; int* scanOff; int* scanTot;
    int* scanBlock2;           // second block-sum scratch for scans on the side stream
    int* scanOff2;             // second per-item offsets (side stream)
    const DevMesh* meshes;     // device array
    int numMeshes;
    // this substep's queries that reach a mesh collider, by kind (vertices, triangles,
    // edges): item, collider (index in vcoll), contact slot of the collider
    int4* meshQuery; int meshQueryBase[3]; int* meshQueryCount;
};

struct TileView;
// tv: the tile solver's view when it runs this substep; first: of its frame
void launch_predict(cudaStream_t s, const DevCloth& c, const SolverParams& P, const TileView* tv, bool first);
// state <-> 10 N floats: positions, velocities, previous positions (xyz), inverse masses
void launch_pack_state(cudaStream_t s, const DevCloth& c, float* out);
void launch_unpack_state(cudaStream_t s, const DevCloth& c, const float* in);
void launch_velocity(cudaStream_t s, const DevCloth& c, const SolverParams& P);
void launch_fem(cudaStream_t s, const DevCloth& c, const SolverParams& P, int first, int count);
void launch_links(cudaStream_t s, const DevCloth& c, const SolverParams& P, int first, int count);
void launch_reset_link_error(cudaStream_t s, const DevCloth& c);
void launch_bends(cudaStream_t s, const DevCloth& c, const SolverParams& P, int first, int count, int resetErr);
void launch_normals(cudaStream_t s, const DevCloth& c, bool prevMesh, const float4* verts);
// vertex contacts of every collider, triangle and edge contacts with their dense lists
void launch_colliders(cudaStream_t s, const DevCloth& c, const SolverParams& P, const Buffers& b, const VColl* hostColl,
                      int numColl, int flags);
void launch_solve_vertex_contacts(cudaStream_t s, const DevCloth& c, const SolverParams& P, const Buffers& b);
void launch_solve_multi_contacts(cudaStream_t s, const DevCloth& c, const SolverParams& P, const Buffers& b, int iter);
void launch_colour_contacts(cudaStream_t s, const DevCloth& c, const Buffers& b);
void launch_bvh_refit(cudaStream_t s, const DevBVH& bvh, const DevCloth& c, int kind, float tol);
// microseconds a phase of the cluster solver's barrier structure costs (kind 0:
// barrier only; 1: plus one distributed-shared-memory read and write), -1 if no
// cluster of the solver's size fits
float probe_cluster_phase(int kind, int phases);
void launch_self_proximity(cudaStream_t s, const DevCloth& c, const SolverParams& P, const Buffers& b,
                           const DevBVH& triBvh, const DevBVH& edgeBvh);
// swept boxes + continuous-collision broad and narrow phases; the vertex-triangle
// half runs on `side` (forked from / joined to s by the events); marks (optional,
// entries may be null): records around the edge-edge and the vertex-triangle
// halves {ee start, ee end, vt start, vt end}
void launch_ccd(cudaStream_t s, cudaStream_t side, cudaEvent_t fork, cudaEvent_t join, const DevCloth& c,
                const SolverParams& P, const Buffers& b, const BoxSet& tris, const BoxSet& edges, const VertexBlocks& verts,
                const cudaEvent_t* marks = nullptr);
// self-contact lists: proximity contacts (self) compacted, then the continuous
// hits appended (ccd)
void launch_compact_self(cudaStream_t s, const DevCloth& c, const SolverParams& P, const Buffers& b, bool self, bool ccd);
// clears the solver's error and exit words; with a tile plan also its exchange tags
void launch_reset_gs(cudaStream_t s, const DevCloth& c, const TileView* tv = nullptr);

// The reference's other link solvers (ClothModel::SetSolver, Physics/ClothPBD.cpp:293-298):
// links in index order, per-link displacements, and each particle's incident links
// in increasing link index ((link << 1) | 1 where the particle is the link's i2)
struct LinkSolve
{
    int L;
    const float4* link;     // L: i1, i2 (bits), rest length, stiffness; link index order
    float4* disp;           // L: this iteration's displacement of each link
    float* d;               // L: conjugate-residual search direction
    const int* incStart;    // N + 1
    const int* inc;         // 2 L
};
// SolveJacobi: `iterations` rounds of SolveLinksJacobi (omega 0.5)
void launch_solve_jacobi(cudaStream_t s, const DevCloth& c, const SolverParams& P, const LinkSolve& ls);
// SolveCR (alpha0 0.1): beta[k] of iteration k, (k / (iterations - 1))^0.6, computed by the caller
void launch_solve_cr(cudaStream_t s, const DevCloth& c, const SolverParams& P, const LinkSolve& ls, const float* beta);
// max |C| over warp / weft / shear constraints, as float bits into *out
void launch_residual(cudaStream_t s, const DevCloth& c, unsigned* out);
// residual-target mode for the per-colour path: residual + exit flag after an iteration
void launch_residual_exit(cudaStream_t s, const DevCloth& c, const SolverParams& P, int iter);
void launch_iteration_total(cudaStream_t s, const DevCloth& c);
void launch_gs_exit_test(cudaStream_t s, const DevCloth& c, const SolverParams& P, int iter);

// cluster-resident Gauss-Seidel solver (one cluster per cloth, one launch per substep)
constexpr int GS_THREADS = 512;
constexpr int GS_SMEM_MAX = 200 * 1024; // dynamic shared memory per CTA: particles + staged records
// A tile launch cannot solve self contacts that reach across its tiles: it works
// only while there are none, and a launch after it only when there are some (the
// counts are known on the device alone); of two launches after it, one with fewer
// contact colours than `colours` and the other with as many or more.
enum { GUARD_NONE = 0, GUARD_IF_SELF = 1, GUARD_IF_NO_SELF = 2, GUARD_IF_FEW = 3, GUARD_IF_MANY = 4 };
struct SolveGuard { int kind, colours; };
struct GsPlan
{
    int iterations, vpc, nFemCol, nBendCol;   // vpc: particles per CTA (cluster solver)
    int stage;               // 1: each CTA copies its constraint records to shared memory first
    int femStage, bendStage; // records per CTA when staged (max over the cluster's CTAs)
    int femStart[65];
    int bendStart[65];
    int nLinkCol;            // mass-spring path (FEM off): link colours
    int linkStart[65];
    SolveGuard guard;        // whether the launch does its work
};
// cluster size usable for N particles (0: too large or unsupported); sets the
// particles per CTA and the dynamic shared memory per CTA
int gs_cluster_size(int N, int& vpc, size_t& smem);
// variant 0: one constraint per thread; 1: two (their loads overlap)
int gs_cluster_variants();
bool launch_gs_cluster(cudaStream_t s, const DevCloth& c, const SolverParams& P, const Buffers& b, GsPlan plan,
                       int clusterSize, size_t smem, int variant);

// grid-resident solver (cooperative launch, any cloth or batch size); variants
// differ in threads per CTA and in constraints per thread (tiles)
int gs_grid_variants();
void gs_grid_variant_info(int variant, int& threads, int& femTile, int& bendTile);
int gs_grid_max_blocks_per_sm(int variant);
bool launch_gs_grid(cudaStream_t s, const DevCloth& c, const SolverParams& P, const Buffers& b, GsPlan plan,
                    int variant, int blocksPerSm);

// band-parallel solver (one cluster per cloth, one launch per substep): the
// particles in contiguous bands of 2^shift, one per CTA, resident in shared
// memory; each class's records split per band into interior records (every
// particle in the band) and boundary records (lowest particle in the band, the
// others in it or among the first `halo` particles of the next band)
struct BandView
{
    int shift, halo;
    int nFemCol, nBendCol, nLinkCol;
    // record offsets per (band, part, colour): [(band * 2 + part) * nCol + colour], nBands * 2 * nCol + 1 entries
    const int* femOff;
    const int* bendOff;
    const int* linkOff;
    // records in (band, part, colour, colour order) order: FEM 3 float4, bends uint4, links float4
    const float4* fem;
    const uint4* bend;
    const float4* link;
    // records staged in shared memory (1) or read through the non-coherent path (0),
    // and the most records one band holds (the staging layout)
    int stageFem, stageBend, stageLink;
    int femMax, bendMax, linkMax;
};
constexpr int BAND_SMEM_MAX = 220 * 1024;  // dynamic shared memory per CTA of the band solver
// threads-per-CTA variants of the band solver (same order, bit-identical results)
int gs_band_variants();
int gs_band_threads(int variant);
// resident CTAs of the tile solver per SM with smem bytes each (0: none)
int gs_tile_max_blocks_per_sm(int threads, bool whole, size_t smem);
// true if a cluster of clusterSize CTAs with smem bytes each can run the band solver
bool gs_band_fits(int clusterSize, size_t smem);

// tile solver (k_gs_tile): each CTA keeps a tile of the cloth in shared memory,
// its own particles and a halo around them, and runs several colours between two
// exchanges, with the halo's constraints computed redundantly
constexpr int TILE_SMEM_MAX = 200 * 1024;    // dynamic shared memory per CTA: local particles
constexpr int TILE_MAX_GROUPS = 4;           // exchanges of one class sweep
struct TileDesc
{
    int idBase, nOwn, nLoc;      // its particles in ids[]: nOwn own, then the halo
    int peers, peerFirst;        // tiles of its cloth and the first of them (1: closed, no exchange)
};
struct TileClass
{
    int nCol;
    unsigned long long cutMask;  // an exchange follows colour c inside the sweep (bit c)
    const int* off;                 // (tile * (nCol + 1) + colour): first record
};
// edge or triangle collider contacts: the cloth's edges / triangles a tile may have
// to solve contacts of, by static colour, and its contact records of the substep
constexpr int TILE_CT_WORDS = 6;
struct TileContacts
{
    int nSlot;                   // colliders that make such contacts (0: none)
    int nEntry;                  // entries of all tiles
    TileClass cls;
    const int4* entry;           // edge / triangle, its local particles (two or three)
    float4* rec;                 // nSlot x nEntry x TILE_CT_WORDS
};
struct TileView
{
    int nTiles, N;
    int threads;                 // per CTA: 128, 256 or 512
    int identity;                // one closed tile whose local indices are the particle indices
    const int* ctaStart;         // tiles of CTA b: ctaTile[ctaStart[b] .. ctaStart[b + 1])
    const int* ctaTile;
    const TileDesc* tile;
    const int* ids;              // global particle of each local one
    TileClass fem, bend, link;
    TileContacts edgeCt, triCt;
    const float4* femRec;        // records as in DevCloth, with local particle indices
    const uint4* bendRec;
    const float4* linkRec;
    float4* xch;                 // 2 N: exchanged positions, w = exchange number (as bits)
    unsigned long long* xred;    // 2 nTiles: exchanged iteration-end words (number << 32 | value)
    float4* selfRec;             // identity: 2 words per self contact (stCap, then seCap of them), in colour order
};

// The solver's entry points as one table per build of solver.cuh: IEEE division
// and square root without FMA contraction (bit-exact with the reference's
// operation order, the check-mode build) or the fast build (FMA contraction,
// approximate division and square root). Same kernels, same order, same
// launch shapes; detection is shared and always exact.
struct SolverOps
{
    void (*fem)(cudaStream_t, const DevCloth&, const SolverParams&, int, int);
    void (*links)(cudaStream_t, const DevCloth&, const SolverParams&, int, int);
    void (*reset_link_error)(cudaStream_t, const DevCloth&);
    void (*bends)(cudaStream_t, const DevCloth&, const SolverParams&, int, int, int);
    void (*vertex_contacts)(cudaStream_t, const DevCloth&, const SolverParams&, const Buffers&);
    void (*multi_contacts)(cudaStream_t, const DevCloth&, const SolverParams&, const Buffers&, int);
    int (*cluster_size)(int, int&, size_t&);
    bool (*cluster)(cudaStream_t, const DevCloth&, const SolverParams&, const Buffers&, GsPlan, int, size_t, int);
    int (*grid_max_blocks_per_sm)(int);
    bool (*grid)(cudaStream_t, const DevCloth&, const SolverParams&, const Buffers&, GsPlan, int, int);
    bool (*band)(cudaStream_t, const DevCloth&, const SolverParams&, const Buffers&, GsPlan, const BandView&, int, size_t,
                 int);
    bool (*tile)(cudaStream_t, const DevCloth&, const SolverParams&, const Buffers&, const TileView&, int, size_t, int, SolveGuard);
};
const SolverOps& solver_ops(bool fast);

// learned warm start (mlp_kernels.cuh): 9347 FP32 parameters, 27 normalisation values
constexpr int MLP_NPARAM = 9347, MLP_NNORM = 27, MLP_IN = 12, MLP_OUT = 3;
void launch_mlp_warm(cudaStream_t s, const DevCloth& c, const Buffers& b, const float* prm, const float* norm);
void launch_mlp_features(cudaStream_t s, const DevCloth& c, const Buffers& b, float* feat);
void launch_mlp_targets(cudaStream_t s, const DevCloth& c, float* target);
void launch_mlp_forward(cudaStream_t s, const float* X, int S, const float* prm, const float* norm, float* Y);
bool launch_mlp_grad(cudaStream_t s, const float* X, const float* T, int S, const float* prm, const float* norm,
                     float* grad, float* loss);
void launch_adam(cudaStream_t s, float* prm, const float* grad, float* m, float* v, int step, float lr);

// SDF::CreateFromMesh on the device: (nx+1)(ny+1)(nz+1) values, x fastest
bool launch_sdf_from_mesh(const DevMesh& m, int nx, int ny, int nz, float4 lo, float4 steps, float* out, int* status);

// exclusive scan of n ints (out may alias nothing); total written to *total if not null
void scan_ints(cudaStream_t s, const int* in, int* out, int n, int* total, int* tmp);

} // namespace sc
