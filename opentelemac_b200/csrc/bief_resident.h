// bief_resident.h -- the solvers that keep their search direction in shared
// memory (bief_resident.cu), as bief_api.cu launches them.
#pragma once

#include "bief_device.cuh"

namespace bief {

constexpr int RES_T = 1024;      // threads of a virtual block (the tree's)
// Blocks of a cluster.  Measured with at most 8 against at most 16 (us per
// iteration, binary64 / mixed): 1 tree block as 8 or 16 blocks 3.51 / 3.21
// against 3.89 / 3.61; 6 tree blocks as 6 or 12, binary64, 7.31 against 5.39;
// 11 tree blocks in the grid form or as 11, 9.05 / 7.47 against 8.67 / 6.73;
// 15 tree blocks likewise 8.89 / 6.90 against 10.0 / 8.34.
constexpr int RES_MAXCL = 12;
constexpr int RES_TAG = 24;  // grid blocks up to which partial sums are tagged words

// Partition of the nodes over physical blocks, and the local index lists.
struct ResPart {
  int n, G, S, V, R, TP, NP;  // nodes; virtual blocks; splits; virtual blocks per block;
                              // rows per thread; threads per block; physical blocks
  int own;                    // V * R * TP: local indices of the block's own rows
  const int *halo_off;        // [NP+1]
  const int *halo;            // node numbers, ascending per block
  const unsigned *halo_loc;   // CL: owner block << 16 | owner's local index
};

constexpr int PLAN_W = 20480;

struct PlanP {
  ResPart Q;
  // neighbours that make the halo: the segments' when there are segments (each
  // element face is one, and a segment need not be a face), else the mesh's
  const int *nb_meta, *nb_off, *nb_col;
  const int *meta, *seg_off, *seg_col;   // binary32 slots: distinct neighbours
  const int *rec_off;                    // records: meta's low half entries
  const int2 *rec_idx;
  const int *sg_meta, *sg_off, *sg_col;  // segment slots
  int *halo_n;
  int *halo;           // null: there already
  unsigned *halo_loc;  // cluster form only
  // one of these: pairs, single, pairs, records
  unsigned short *seg_li, *sg_li, *sg_li2;
  ushort2 *rec_li;
  int shift;  // pairs: 2 = indices as byte offsets into a binary32 window
};

struct RedShared {
  unsigned long long mbar[2];
  double ws[2][32];
  double cold[3];   // scalars of the mixed solve
  double us[2][16];  // alternate: a warp may still read the previous reduction's
};

struct ResP {
  ResPart Q;
  Sell S;                     // operator of the storage (old-form lists for A x)
  const unsigned short *li;   // binary32 slots / segment slots: local neighbour
  const ushort2 *rli;         // records: local vertices
  int td;                     // working TYPDIA
  const double *da, *dsc;
  double *x;
  const double *b;
  Ctl *ctl;
  double *part;
  unsigned long long *box;    // tagged partial sums (grid form)
  long long timeout_ns;
  int cache;                  // operator slots (multiple of 32) kept in shared memory
  int halo_max;
  int nvec;                   // own-row vectors in shared memory
  // k_cg_res
  int nitmax;
  int keep;                   // steps whose slots are loaded to stay in L2
  double eps;
  double *r, *ad;
  // k_cgstab_res (r, ad: R and V published)
  double *tv, *p0;
  // k_mixed_res
  int max_outer, max_inner;
  double outer_tol, inner_tol;
  float *z, *ri, *q;
  int smem_limit;             // (host) most dynamic shared memory a launch may have
};

// Shared-memory layout, computed alike by host and kernel.
struct ResLayout {
  size_t win, vec, red, box, off, deg, cidx, ccoef, total;
};
// elt: bytes of a vector value (8 binary64, 4 binary32); nvec: own-row
// vectors kept beside the window; cb: operator bytes per slot without index,
// ib: index bytes per slot.
__host__ __device__ inline ResLayout res_layout(int own, int halo, int G, bool cl, int elt,
                                                int nvec, int cb, int ib, int cache) {
  ResLayout L;
  size_t o = 0;
  auto take = [&](size_t bytes) {
    const size_t at = o;
    o = (o + bytes + 15) & ~(size_t)15;
    return at;
  };
  L.win = take((size_t)elt * (size_t)(own + halo));
  L.vec = take((size_t)elt * own * nvec);
  L.red = take(sizeof(RedShared));
  L.box = take(cl ? (size_t)2 * 32 * G * 8 : 0);
  L.off = take(sizeof(int2) * (size_t)(own / 32));
  L.deg = take((size_t)own);
  L.ccoef = take((size_t)cb * cache);
  L.cidx = take((size_t)ib * cache);
  L.total = o;
  return L;
}

// Launchers (bief_resident.cu); they return cudaGetLastError()'s value.
cudaError_t res_launch_plan(bool fill, const PlanP &A, cudaStream_t st);
cudaError_t res_launch_cg(int sto, bool cl, const ResP &P, size_t smem, cudaStream_t st);
cudaError_t res_launch_cgstab(int sto, bool comp, const ResP &P, size_t smem, cudaStream_t st);
// shift: 0 when the local indices are byte offsets, else 2.
cudaError_t res_launch_mixed(int sto, bool cl, bool vs, int shift, const ResP &P, size_t smem,
                             cudaStream_t st);
// Whether a cluster of np blocks of tp threads with that much shared memory
// can be resident (one probe for all cluster kernels).
bool res_cluster_fits(int np, int tp, size_t smem);

// One block in a reduction that never completes: form 0 cluster, 1 tagged
// sums, 2 counter; part: 4 values, box: 8 words, cleared.
cudaError_t res_wait_test(int form, Ctl *ctl, double *part, unsigned long long *box,
                          long long timeout_ns);
// The limit of dynamic shared memory that the cluster form's GRACJG (blocks
// of at most 512 threads) has now.
cudaError_t res_smem_limit(int *bytes);

}  // namespace bief
