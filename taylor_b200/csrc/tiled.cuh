// tiled.cuh -- tiles of consecutive rows (or columns) with their neighbour
// sets, for the shared-memory staged gathers of tiled.cu.
#pragma once
#include "mega_internal.cuh"

namespace mega {

// How a tile set's packed records are laid out (build_slices in tiled.cu):
// slices of 8 rows, 32 records per step, 4 consecutive entries of each row
struct SliceView {
  const uint8_t* ord = nullptr;    // per slot (tile, position): the row within the tile; rows past n come last
  const int64_t* sstep = nullptr;  // per slice of 8 slots: its first step (record 32 sstep), and the end
  int64_t nrec = 0;                // records, pads among them
  bool ahead = false;              // fetch a slice's records to L2 as its rows begin (records_ahead)
};

struct TileSet {
  int32_t R = 0;           // rows (columns) per tile; the kernels run 4, 8 or 16 threads per row
  int64_t ntiles = 0;
  int32_t jmax = 0;        // stride of jset per tile
  int32_t maxcnt = 0;      // largest neighbour set of any tile
  int32_t recmax = 0;      // most packed records of any tile (build_slices)
  int32_t* jset = nullptr; // [ntiles][jmax] sorted node ids
  int32_t* jcnt = nullptr; // [ntiles]
  uint16_t* lidx = nullptr;  // per entry: rank of its neighbour in the tile's set
  // the slices of its records (build_slices)
  uint8_t* ord = nullptr;
  int64_t* sstep = nullptr;
  int64_t* rbase = nullptr;  // per row: the record of its entry 0; entry k is 32 (k / 4) + k % 4 further
  int64_t nrec = 0;
  bool banked32 = false;     // the mixed records are in bank order
  SliceView view(bool ahead = false) const { return SliceView{ord, sstep, nrec, ahead}; }
};

// NSNI terms carried by the tiled gathers: the smoothed second derivatives
// S_q (XX, YY, ZZ, XY, YZ, XZ) of every list entry in the layout of the row
// records (srow) and of the column records, as planes of nrec values: float4
// (q 0-3) and float2 (q 4, 5), or three planes of double2; their row sums
// (mixed), and the per-node H output (row gather) and force weights (column
// gather)
struct NsniTiles {
  const void* srow = nullptr;
  const double* ssum = nullptr;  // mixed: 6 per node, sum_J S_q(i, J) of the float values in double
  double* hq = nullptr;          // out: sum_J S_q(i, J) du_J,k at [(6 k + q) fg_ld(n) + i]
};

struct TiledForceArgs {
  int32_t n;
  int32_t R;
  int64_t ntiles;
  int32_t jmax;
  int32_t maxcnt;
  int32_t recmax;
  const int32_t* jset;
  const int32_t* jcnt;
  const int64_t* colptr;
  SliceView sv;           // the layout of pk
  const void* pk;         // packed transposed entries (gradient + local index)
  const double* tshp;     // transposed shape values (body force) or null
  const void* tmat;       // 12 values per node
  int has_body;
  int predict;
  const int8_t* ebc;
  const double* mass;
  const uint16_t* matidx;
  const MatEntry* mats;
  const int8_t* body_id;
  double* fint;
  double* fext;
  double* vel;
  double* acl;
  double* dsp;
  double* dsp_tot;
  double* prforce;
  const void* ns_scol;    // NSNI: the S planes of the column records, or null
  const void* ns_w;       // NSNI: force weights, 20 values per node (18 used; floats when mixed)
  const double* vel2;     // prescribed velocities of fixity code 2 for this step (3), or null
  const double* ndt;      // per-node step of independent instances, or null (dt for all)
  double dt;
  StepAccum* acc;
  unsigned* status;
};

// Tiles of R consecutive rows of (ptr, idx), R halved from `rows` down to 8
// until every tile's neighbour set fits jmax = 1024.
int build_tiles(cudaStream_t s, int32_t n, const int64_t* ptr, const int32_t* idx, int64_t nnz, int32_t gmaxn,
                TileSet& ts, DevPool& pool, int32_t* maxcnt_out, int32_t rows = 64);
// The record layout of ts (row order, slices, record bases) into pool.
int build_slices(cudaStream_t s, int32_t n, const int64_t* ptr, TileSet& ts, DevPool& pool);
// records of ts.nrec entries in the slice layout: (gradient of entry pos[e],
// rank of e) as float4, or FP64 as planes of double2 (x, y), double (z) and
// uint16_t (rank): 16 or 26 bytes a record
int pack_entries(cudaStream_t s, int32_t n, const TileSet& ts, const int64_t* ptr, const double* gx,
                 const double* gy, const double* gz, const int64_t* pos, bool f64, void* out);
// mixed records of the transposed view from those of the rows
int pack_transposed32(cudaStream_t s, int32_t n, const TileSet& ct, const int64_t* colptr, const float4* in,
                      const int32_t* trow, const int64_t* pos, const int64_t* rowptr, const TileSet& rt,
                      float4* out);
// the pads of float records whose entries are written elsewhere
int pad_records32(cudaStream_t s, int32_t n, const TileSet& ts, const int64_t* ptr, float4* out);
// Reorder the entries within each row (column) of the tiles ts so that the
// lanes of a warp of a gather with `lanes` (4 or 8) lanes per row read
// distinct shared-memory banks of the staged neighbour data (16-byte vectors
// by rank) where possible.  lidx is reordered in place;
// pos, the identity on entry, receives each entry's position before.
int bank_order(cudaStream_t s, int32_t n, const TileSet& ts, const int64_t* ptr, uint16_t* lidx,
               int64_t* pos, int lanes);
// out[e] = e;  entry e takes the record of entry pos[e] of its row
int iota64(cudaStream_t s, int64_t m, int64_t* out);
int gather_records(cudaStream_t s, int32_t n, const TileSet& ts, const int64_t* ptr, const int64_t* pos, bool f64,
                   const void* in, void* out);
// NSNI's S (list order, at pos[e] when given) as planes in the records' layout,
// and those planes with the entries of each row reordered by pos
int pack_second(cudaStream_t s, int32_t n, const TileSet& ts, const int64_t* ptr, const int64_t* pos, const NsniS& src,
                bool f64, void* out);
int gather_second(cudaStream_t s, int32_t n, const TileSet& ts, const int64_t* ptr, const int64_t* pos, bool f64,
                  const void* in, void* out);
// launch variants of the two gathers: lanes per row x records in flight
// (register streams, variants 0-3 and 6, 7), and lanes per row with the
// tile's records streamed into shared memory by the copy engine (variants
// 4, 5)
constexpr int kTiledVariants = 8;
int tiled_variants();
// whether a variant's shared memory fits the row (defgrad) or column (force) tiles
bool tiled_variant_fits(const TileSet& ts, bool mixed, int variant, bool force, bool has_body);
// MEGA_ERR_UNSUPPORTED when the variant's shared memory does not fit the tiles
// ns: the NSNI H gather rides along (register variants; FP64 takes those of
// the same lanes per row for 4 and 5, mixed refuses them).
// full: F - I as well as G0 (else the stress update adds G0 to F - I)
// load_only: nothing is launched; the kernel the call would launch is loaded,
// so that a stream capture finds it ready
int launch_defgrad_tiled(cudaStream_t s, bool mixed, bool interp, int32_t n, const TileSet& ts,
                         const NsniTiles* ns, const int64_t* rowptr, const void* pk, const double* dsp,
                         const double* dsp_tot,
                         const double* sdphi, const double* shp, double* dsp_tot_phy, double* fg, StepAccum* acc,
                         unsigned* status, int variant, bool full, bool load_only = false);
// whether the gathers of these tiles fetch their records ahead
bool records_ahead(const TileSet& ts, bool mixed);
// The row gather of the increments that goes on to the stress update of its
// rows (finite strain, undamaged models, no NSNI, another step follows), and
// whether it is the faster way: all of its blocks resident at once.
bool defgrad_stress_fits(const TileSet& ts, int variant);
int launch_defgrad_stress(cudaStream_t s, bool mixed, int32_t n, const TileSet& ts, const int64_t* rowptr,
                          const void* pk, const double* dsp, const double* dsp_tot, const double* sdphi, double* fg,
                          const StressArgs& a, int variant, bool load_only = false);
int launch_force_tiled(cudaStream_t s, bool mixed, const TiledForceArgs& a, int variant = 0, bool load_only = false);

}  // namespace mega
