// Internal definitions shared by the conehead_gb300 CUDA sources.
#pragma once

#include <cstdint>
#include <vector>
#include <cuda.h>
#include <cuda_runtime.h>

#include "../../include/conehead_gb300.h"

namespace ch {

// ------------------------------------------------------------------ sizes --
// Cone gather tile: 16 (x) x 16 (y) x 16 (z) outputs.  The 16 outputs of a
// tile line along the "run axis" of the walks being summed (x or y, chosen
// per walk on the host) are split between OUT_SPLIT consumer warps, each
// thread holding 16 / OUT_SPLIT of them in registers:
//   run axis x: half a warp covers 16 consecutive z of one y row, the other
//     half the same z two rows further (y + 2); 8 warps cover the 16 rows;
//   run axis y: half a warp covers 16 consecutive z of one x slice, the other
//     half the next slice (x + 1); 8 warps cover the 16 slices.
// More warps hide more shared-memory latency; every warp reads the run
// records and its own line ends.
constexpr int TZ = 16, TY = 16, TX = 16;
constexpr int TILE_VOX = TZ * TY * TX;
#ifndef CH_OUT_SPLIT
#define CH_OUT_SPLIT 2
#endif
constexpr int OUT_SPLIT = CH_OUT_SPLIT;
constexpr int OUT_PER_THREAD = 16 / OUT_SPLIT;
// A run is up to RUN_MAX consecutive taps of one walk whose steps all lie
// along the walk's run axis: its n taps read one line of 15 + n window values
// along that axis, so a thread loads each value once for up to n taps.
constexpr int RUN_MAX = 4;
// Shared-memory window of a chunk: [x][row][z] with z pitch P and `rows` y
// rows per x slice.  Three shapes ("variants") trade z reach for x and y reach
// in one fixed slot; the chunker picks the cheapest that holds the chunk.
// Every P is 8 mod 16, so 2P = 16 mod 32: the half-warps of the x layout
// (rows y and y + 2) hit disjoint banks.  Every `rows` is 2 mod 4, so the
// slice pitch rows * P is 16 mod 32: the half-warps of the y layout (slices x
// and x + 1) hit disjoint banks too.
constexpr int N_VARIANTS = 3;
__host__ __device__ constexpr int var_p(int v) { return v == 0 ? 24 : (v == 1 ? 40 : 56); }
__host__ __device__ constexpr int var_rows(int v) { return v == 0 ? 34 : (v == 1 ? 26 : 22); }
static_assert((2 * var_p(0)) % 32 == 16 && (2 * var_p(1)) % 32 == 16 && (2 * var_p(2)) % 32 == 16,
              "x layout: rows y and y + 2 must fall in disjoint banks");
static_assert((var_rows(0) * var_p(0)) % 32 == 16 && (var_rows(1) * var_p(1)) % 32 == 16 &&
                  (var_rows(2) * var_p(2)) % 32 == 16,
              "y layout: slices x and x + 1 must fall in disjoint banks");
constexpr int WIN_FLOATS = 27648;     // one pipeline slot (108 KiB)
__host__ __device__ constexpr int var_max_ex(int v) { return WIN_FLOATS / (var_p(v) * var_rows(v)); }
// largest tap-offset spread a chunk may have along each axis in variant v
// (z also absorbs the 4-float TMA alignment of the window origin)
__host__ __device__ constexpr int var_span_z(int v) { return var_p(v) - TZ - 3; }
__host__ __device__ constexpr int var_span_y(int v) { return var_rows(v) - TY; }
__host__ __device__ constexpr int var_span_x(int v) { return var_max_ex(v) - TX; }
// One TMA box loads a chunk's whole window: P x rows x ex floats, so every
// (variant, x extent) pair has its own tensor map.
__host__ __device__ constexpr int n_maps_before(int v) {
  return v == 0 ? 0 : (v == 1 ? var_max_ex(0) - TX + 1 : (var_max_ex(0) - TX + 1) + (var_max_ex(1) - TX + 1));
}
constexpr int N_TMAPS = n_maps_before(2) + (var_max_ex(2) - TX + 1);
__host__ __device__ constexpr int tmap_index(int v, int ex) { return n_maps_before(v) + (ex - TX); }
// Run record, two int4: {window offset of the run's base in its chunk's
// variant, n, w0, w1} and {w2, w3, 0, 0} (float bits).  The base is the tap
// furthest along the run axis; weight slot c belongs to the tap c steps
// behind it, which reads line value i + c for output i.
constexpr int RUN_REC_INT4 = 2;
constexpr int MAX_CHUNK_RUNS = 64;    // runs per chunk (their records are staged with the window)
constexpr int N_SLOTS = 2;
constexpr int CONE_CONSUMER_WARPS = (TY / 2) * OUT_SPLIT;
constexpr int CONE_THREADS = (CONE_CONSUMER_WARPS + 1) * 32;
constexpr int DIR_GROUP = 16;         // unique directions per work unit (default; ch_tuning.dir_group)
constexpr int MAX_DIR_GROUP = 1024;   // the producer walks a unit's directions 32 at a time

// Bounded device-side waits: try_wait iterations of an mbarrier wait before
// the gather gives up (its pipeline waits may be given a smaller bound per
// plan, ch_plan_set_wait_limit; the wait for its own copies in flight always
// has this one).
constexpr long long MBAR_LIMIT = 1ll << 22;

// device error flags (bit mask in Plan::d_flags[0])
constexpr int FLAG_TIMEOUT = 1;
constexpr int FLAG_PARALLEL_RAY = 2;
constexpr int FLAG_BAD_INDEX = 4;

// ---------------------------------------------------------- beam constants --
// Everything the per-voxel prologue needs about one beam, prepared on the
// host (float64 values mirrored from the reference's arrays, float32
// approximations for the fast blocking test).
struct BeamDev {
  // exact mirror inputs
  double src[3], vy[3], m0[3], m2[3];   // m0/m2: transform rows 0 and 2
  double vyw;                           // v_y . float32(src), reference order
  double srcd[3];                       // float32(src)
  float srcf[3], vyf[3], m0f[3], m2f[3], vywf;  // float32 copies (geom_f32 path)
  int geom_f32;
  // low parts of the float64 values beside vyf, m0f, m2f and vywh (project_pairs)
  float vyl[3], m0l[3], m2l[3], vywh, vywl;
  int pairs;                            // no product of them overflows (make_beam)
  // fast approximate projection: xb ~ c0 + si * (m0.S - m0.p), si = K / (n.S - n.p)
  float a_c0, a_c2, a_m0S, a_m2S, a_nS, a_K;
  // cull box in beam coordinates (cm) for voxel centres (inclusive)
  float cx_lo, cx_hi, cz_lo, cz_hi;
  float cull_margin_k;   // margin = k * SAD/depth
  int cull_enable;
  // block crop
  const float* block;
  int brows, bcols, br0, bc0, full_rows, full_cols;
  int uniform;          // every crop value is 1.0
  // sub-sample lattice (blocked_fraction)
  int lat;              // float64 source arrays on a sane grid: samples may be classified in float32
  int wraps;            // the crop holds the map's last row or column, which index -2000 reads
  float lat_n, lat_0, lat_2;   // largest |d nd|, |d x0|, |d x2| of a sub-sample from its voxel centre (cm)
  float err_x, err_n;   // float32 error bounds of x0 and nd against the reference's ray (cm)
  float uc, uh, wc, wh; // the crop's cells, centre and half width along u (rows) and w (columns)
  int rlim, clim;       // crop rows and columns a lookup can reach without the wrap
  // fluence / TERMA
  double sad;
  int sad_f32;
};

struct SettingsDev {
  float sPri, sAnn, zAnn, rInner, rOuter, zExp, sExp, kExp;
  float softRatio, softLimit, hornRatio;
  int samples;
  int n_energy;
  float E[CH_MAX_ENERGY], w[CH_MAX_ENERGY], mu[CH_MAX_ENERGY];
};

struct GridDev {
  int n[3];
  float origin[3];
  float spacing[3];
  int zp;             // padded z pitch of the internal TERMA volume
  int swap_xy;
};

// ------------------------------------------------------------ exact math --
// Reference arithmetic without FMA contraction (round after every op).
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fdiv(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double ddiv(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ float d2f(double a) { return __double2float_rn(a); }

// voxel centre: float32 store of f64(origin) + f64(spacing) * i.  The float64
// value is exact for any realistic grid, so one fused rounding equals it.
__device__ __forceinline__ float voxel_centre(float origin, float spacing, int i) {
  return __fmaf_rn(spacing, (float)i, origin);
}

// DDA initial t and increment for one axis (reference cuda_dda_3d):
// t0 = f32(f64(s/2) / f64(|d|)) == fdiv(s/2, |d|) (double rounding through
// float64 is innocuous for float32 operands), dt = s / |d| in float32.
__device__ __forceinline__ void dda_axis(float d, float s, int& step, float& t, float& dt) {
  step = d < 0.0f ? -1 : 1;
  float a = d < 0.0f ? -d : d;
  if (a == 0.0f) {
    t = 1000000000.0f;
    dt = 1000000000.0f;
  } else {
    t = fdiv(s * 0.5f, a);
    dt = fdiv(s, a);
  }
}

__device__ __forceinline__ int dda_pick(const float* t) {
  return (t[0] < t[1]) ? ((t[0] < t[2]) ? 0 : 2) : ((t[1] < t[2]) ? 1 : 2);
}

// ----------------------------------------------------- cone stage structs --
constexpr uint32_t RANGE_EMPTY = 0xffffffffu;

struct __align__(128) ConeBeam {
  CUtensorMap tmap[N_TMAPS];  // TERMA volume (dims nz, ny, nx; pitch zp), box P x rows x ex per map
  float* dose;
  const uint32_t* ranges; // [n_tiles][n_dirs]
  const uint32_t* cranges;
  int n[3];
  int ntile[3];
  int n_tiles;
  int unit_begin;
  int n_units;
  int pad[1];
};
static_assert(sizeof(ConeBeam) % 128 == 0, "ConeBeam must keep tensor maps aligned");

struct ConeDirs {
  int n_dirs;
  const int* tap_base;
  const int* tap_len;
  const int4* taps;        // window offset of O[m] in variants 0..2, float bits of w[m] (scatter path)
  const short4* offs;      // O[m] (x, y, z, step axis)
  const float* tvals;      // exit t of tap m
  const int4* runs;        // RUN_REC_INT4 per run, the runs of all walks back to back
  const int* run_base;     // first run of each walk
  const int* tap_run;      // per tap: its global run index * 8 + 2 + its weight slot (the word of its weight)
  const int* run_tap;      // per run: global index of its first tap (one trailing entry)
  const int* axis;         // per walk: run axis, 0 = x, 1 = y
  const int* chunk_base;
  const int* n_chunks;
  const int* chunk_start;  // first run of each chunk (walk-local)
  const int4* chunk_rec;   // 2 per chunk: {first run, last run, variant, span_x | span_y << 16},
                           //              {max O_x, max O_y, max O_z, 0} over the chunk's taps
  const float* dirs;       // unit direction (x, y, z)
  int group;               // unique directions per work unit (1..MAX_DIR_GROUP)
  int order;               // units: 0 = tile outer, group inner; 1 = group outer, tile inner
  long long wait_limit;    // try_wait iterations of a pipeline wait before the gather gives up
  int withhold;            // test hook: 0 = off; CH_WITHHOLD_WINDOWS / CH_WITHHOLD_SLOTS (the
                           // producer issues no window / the consumers free no slot)
};

struct RangeBeam {
  int n[3], ntile[3], n_tiles;
  float origin[3], spacing[3];
  int n_planes;
  float pa[4][3];
  float pk0[4];
  const int* aabb;          // box of the nonzero input (lo/hi pairs per axis)
  const int* out_aabb;      // if set, output tiles outside this box get no taps
  int n_out_planes;         // output tiles wholly outside one of these planes
  float opa[4][3];          // (the beam frustum, for the transposed cone of
  float opk0[4];            // the adjoint) get no taps either
  uint32_t* ranges;        // [n_tiles][n_dirs]: first | last run << 16 (walk-local), or RANGE_EMPTY
  uint32_t* cranges;       // [n_tiles][n_dirs]: first | last chunk << 16 (walk-local)
};

// Regular beamlet grid on the block map: beamlet (i, j) covers map rows
// r0 + i*cell_rows .. + cell_rows and columns c0 + j*cell_cols .. + cell_cols.
struct BeamletDev {
  int rows, cols, cell_rows, cell_cols, r0, c0;
};

// Chunks of 32 entries (one per lane) of a list.  Lists hold up to 2^31 - 1
// voxels, so entry numbers rounded up to a launch's stride pass 2^31: they are
// unsigned and compared as such.
__host__ __device__ __forceinline__ int list_chunks(int count) { return (int)(((unsigned)count + 31u) >> 5); }

struct Inter {
  double* blocked;
  float *d_eff, *oad, *fluence, *f_soften, *f_horn, *terma;
};

// ---------------------------------------------------- spectral cone stage --
// The cone stage as one convolution per grid shape (spectral.cu): periods
// M_k = the smallest allowed length >= 2 n_k - 1 along x and y, M_z = the
// smallest >= nz along z (spec_lengths), one transform per beam.
constexpr int SPEC_THREADS = 256;         // general kernels
constexpr int SPEC_CTAS_PER_SM = 3;       // their register budget (85 per thread)
constexpr int SPEC_ELEMS = 4096;          // complex values per CTA: 4096 / M lines of period M
constexpr int SPEC_MIN_GENERAL = 768, SPEC_MAX_PERIOD = 4096;
constexpr int SPEC_MAX_BEAMS = 32;        // beams per launch (their work buffers coexist)
constexpr int SPEC_SMEM = 2 * SPEC_ELEMS * 8;   // two ping-pong buffers of float2 per CTA
struct SpecBeam {
  const float* t;          // TERMA [nx][ny][zp]
  const unsigned char* l;  // lines of t that may be nonzero (NULL: every line is read)
  float2* a;               // [nx][ny][Mz]
  float2* b;               // [nx][My][Mz]
  float* d;                // dose [nx][ny][nz]
};
struct SpecGrid {
  int n[3], M[3];
  int logL[3];             // log2 of the lines per CTA of the general pass along x, y, z
  int zp;                  // z pitch of the TERMA volumes
  int conj;                // multiply by conj(S^): the transposed cone
  const float2* tw[3];     // twiddles exp(-2 pi i k / M_axis)
  const float2* tq;        // quarter steps exp(-2 pi i k / (4 Mz)): the twist along z
  const float2* shat;      // S^ [Mx][My][Mz], 1/(Mx My Mz) folded in; [Mz][My][Mx] on the plane path
  int plane;               // the plane path (spec_plane_path): A = [Mz][lp] plane-major, no B
  int lp;                  // plane pitch of A on the plane path (nx ny rounded up to 32)
  int skip;                // rows of A without TERMA are not written: their reader goes by the line flags
  int ahead;               // the y and x passes ask L2 for the lines of a later CTA
  int after;               // the passes start while their predecessors end (launch_after)
};
struct SpecLaunch {
  SpecGrid g;
  int n_beams;
  SpecBeam p[SPEC_MAX_BEAMS];
};
// forward transform of full lines in place: element i of line (o, c), c < 16,
// at data + (o / nb) os1 + (o mod nb) os2 + c cs + i is
struct SpecFull {
  float2* data;
  const float2* tw;
  const float2* tq;        // multiplied in first (NULL: not)
  int nb;
  size_t os1, os2, cs, is;
};
int spec_period(int n);                  // 0 when no length up to SPEC_MAX_PERIOD holds 2n - 1
int spec_length_z(int nz);               // 0 when none holds nz
int spec_lines_log2(int M);
int spec_pass_lines_log2(int M, int Mz);
std::vector<float2> spec_twiddles();      // every length (ascending), back to back
size_t spec_twiddle_offset(int M);       // of exp(-2 pi i k / M); the quarter steps follow
cudaError_t setup_spec_kernels();        // allow the kernels their dynamic shared memory
void launch_spec_beams(SpecLaunch& L, cudaStream_t st);   // sets L.g.after
// The plane path: periods of 256 along x and y (97 to 128 voxels).  z forward
// into plane-major A[kz][x y], one cluster of two CTAs per (beam, kz) plane for
// the y and x transforms, the S^ product and their inverses (the plane's
// spectrum held in the pair's shared memory), z inverse from A.  S^ is then
// kept as [Mz][My][Mx].
constexpr int SPEC_PLANE_M = 256;
// half the plane spectrum, an exchange buffer per warp, the twiddle table
constexpr int SPEC_PLANE_SMEM = (128 * 128 + 16 * 2 * 256 + 16 * 18) * 8;
inline bool spec_plane_path(const int* M) { return M[0] == SPEC_PLANE_M && M[1] == SPEC_PLANE_M; }
inline int spec_plane_pitch(const int* n) { return (n[0] * n[1] + 31) / 32 * 32; }
// S^ [Mx][My][Mz] -> [Mz][My][Mx]
void launch_spec_transpose(const float2* in, float2* out, int Mx, int My, int Mz, cudaStream_t st);
// S^ of one grid shape, in place: scatter the folded stencil's values (float
// indexes into s, zeroed, [Mx][My][Mz]), then three forward passes
void launch_spec_build(const SpecGrid& g, const long long* idx, const float* val, int n_val, float2* s,
                       cudaStream_t st);

// One beam of a batched prologue (device record).
struct PrologueBeam {
  GridDev g;
  BeamDev b;
  SettingsDev s;
  const float* rho;
  float* T;          // [nx][ny][zp]
  int* aabb;         // 8 ints: TERMA box, list count at [6]
  int* list_v;       // this beam's voxel list (nx ny nz entries)
  unsigned char* line_any;  // per (x, y) line: 1 when the line holds a listed voxel
  int zero_all;      // 1: zero TERMA on every line (the gather reads it anywhere);
                     // 0: only on lines with listed voxels (the spectral path reads line_any)
  int box;           // 1: the gather needs the TERMA box
};

// Records of the one-launch prologue, passed as a kernel parameter.
constexpr int FUSED_MAX_BEAMS = 4;
struct FusedRecords {
  PrologueBeam r[FUSED_MAX_BEAMS];
};
static_assert(sizeof(FusedRecords) <= 3968, "the records fit the smallest kernel parameter space");

// ---------------------------------------------- programmatic launches --
// A kernel launched with launch_after may start while its predecessor on the
// stream finishes: it sets up what no earlier kernel writes, then waits for the
// predecessor's memory (after_wait) before it reads or writes anything else.
// Each such kernel lets its own successor start (after_trigger) when its CTAs
// have started; the successor waits for its end all the same, so waits chain
// through the stream.  The short kernels of a single beam's call spend a good
// part of their time between launches.
__device__ __forceinline__ void after_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void after_trigger() { asm volatile("griddepcontrol.launch_dependents;"); }

// A load of what an earlier kernel wrote, zero unless ok: an ordinary one (the
// read-only path promises data that does not change while the kernel runs, and
// the compiler may move it above the wait), predicated so that a thread's loads
// stay one batch.  The compiler keeps them in place: issue them before the
// barrier that publishes a table, not after.
// KEEP: leave the line in L1 (the wider y and x passes, 1% at 160^3 and 192^3;
// the others are 5% faster without, 96^3).
template <bool KEEP = false>
__device__ __forceinline__ float2 load_after(const float2* p, bool ok) {
  float2 v;
  if (KEEP)
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %3, 0;\n mov.f32 %0, 0f00000000;\n mov.f32 %1, 0f00000000;\n"
        " @p ld.global.v2.f32 {%0, %1}, [%2];\n}"
        : "=f"(v.x), "=f"(v.y)
        : "l"(p), "r"((int)ok));
  else
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %3, 0;\n mov.f32 %0, 0f00000000;\n mov.f32 %1, 0f00000000;\n"
        " @p ld.global.L1::no_allocate.v2.f32 {%0, %1}, [%2];\n}"
        : "=f"(v.x), "=f"(v.y)
        : "l"(p), "r"((int)ok));
  return v;
}
__device__ __forceinline__ float load_after(const float* p, bool ok) {
  float v;
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %2, 0;\n mov.f32 %0, 0f00000000;\n"
               " @p ld.global.L1::no_allocate.f32 %0, [%1];\n}"
               : "=f"(v)
               : "l"(p), "r"((int)ok));
  return v;
}

// early = false: an ordinary launch.
template <typename... P, typename... A>
void launch_after(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = early ? 1 : 0;
  cudaLaunchKernelEx(&c, kernel, P(args)...);   // a failure is the caller's cudaGetLastError
}

// ------------------------------------------------------------ launchers --
void launch_prologue_fused(const FusedRecords& recs, int n_beams, long long max_lines, int* flag_word, int epoch,
                           cudaStream_t st);
void upload_unit_partials();
// work: a zeroed int, the TERMA launch's chunk counter
void launch_prologue_batch(const PrologueBeam* recs, int n_beams, long long max_voxels, long long max_lines,
                           int n_sm, int* flags, int* work, cudaStream_t st, int ctas_per_sm);
void launch_prologue(const float* rho, const GridDev& g, const BeamDev& b, const SettingsDev& s, float* T,
                     const Inter& inter, int all_voxels, int* aabb, bool box, int* list_v, int n_sm, int* flags,
                     cudaStream_t st, int ctas_per_sm = 8);   // box: the gather needs the TERMA box
// Frame of the cone directions: off = the room frame (the reference), on =
// rotated by a beam's world->beam matrix m (row major, xform of ch_beam).
struct ConeFrame {
  int on;
  double m[9];
};
void launch_stencil(const float* theta, int n_theta, const float* phi, int n_phi, const double* K, int n_r,
                    const float* spacing, const int* cap, int max_len, short4* off, float* t, float* dk,
                    int* len, float* dirs, const ConeFrame& frame, cudaStream_t st);
void launch_scatter_radiological(const float* T, const float* rho, const int* n, int zp, int swap_xy, int n_dirs,
                                 const int* tap_base, const int* tap_len, const short4* offs, const float* tvals,
                                 const int* walk_row, const int* walk_mult, const float2* K2, int n_r,
                                 const int* list_count, const int* list_v, int n_sm, float* dose, cudaStream_t st);
// K as float32 pairs (hi + lo), read by the radiological scatter
void launch_split_table(const double* K, int n, float2* out, cudaStream_t st);
void launch_reweight(const double* K, int n_r, int n_walks, const int* tap_base, const int* tap_len,
                     const float* tvals, const int* walk_row, const int* walk_mult, int4* taps, const int* tap_run,
                     int4* runs, cudaStream_t st);
void launch_dda_trace(const int* n, const float* sp, int n_rays, const int* starts, const float* dirs, int cap,
                      int* vox, float* t, int* len, cudaStream_t st);
void launch_scatter(const float* T, const int* n, int zp, int n_dirs, const int* tap_base, const int* tap_len,
                    const short4* offs, const int4* taps, float* dose, cudaStream_t st);
size_t cone_smem_bytes();
cudaError_t setup_cone_kernel();
void launch_range(const RangeBeam* rbs_dev, int n_beams, int max_tiles, const ConeDirs& D, cudaStream_t st);
void launch_gather(const ConeBeam* beams_dev, int n_beams, const ConeDirs& D, int total_units, int n_ctas,
                   int* unit_counter, unsigned long long* updates, int* flags, cudaStream_t st);
// keep: a bit per counter that is not reset
void launch_init_scratch(int* aabb, int n_beams, int* counters, cudaStream_t st, unsigned keep = 0);
void launch_mlc_raster(const ch_mlc& m, float* out, int rows, int cols, int r0, int c0, cudaStream_t st);
void launch_nonzero_box(const float* x, int n0, int n1, int n2, int* box, cudaStream_t st);
void launch_beamlet_fill(const float* w, const BeamletDev& bl, float* crop, cudaStream_t st);
void launch_to_float(const double* in, float* out, int n, cudaStream_t st);
cudaError_t launch_blocked_adjoint(const GridDev& g, const BeamDev& b, const BeamletDev& bl, int S, const float* T,
                                   const float* tbar, const int* list_count, const int* list_v, double* wbar,
                                   int n_sm, int* flags, cudaStream_t st);

}  // namespace ch
