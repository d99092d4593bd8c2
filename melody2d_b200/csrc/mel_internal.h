// Internal definitions of the B200 solver: device-resident model and kernel entry points.
// Layout (HBM): body-sorted structure-of-arrays; node pairs (x,y) as double2 for 16-byte
// accesses; the Gauss points of a deformable body cut into tiles (mel_tiles.h) that the body kernel
// reads straight into registers, or, for bodies above MEL_MAX_BODY_NODES nodes, into chunks, each
// chunk one contiguous 16-byte-aligned image (header, dN/dx-dN/dy pairs, 16-bit body-local support
// indices, pull positions, per-point weights and offsets, touched-node records) that a single bulk
// copy moves into shared memory; contact elements in the reference's mel_contact record.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>
#include "melgpu.h"

#define MEL_BODY_THREADS 256      // threads per body CTA: warps 0-6 Gauss points and their sums, warp 7 contacts
#define MEL_TILE_GP 224           // Gauss points per tile (mel_tiles.h): one thread each
#define MEL_CHUNK_GP_FP64 224     // Gauss points per chunk of a wide body: one point thread each
#define MEL_PULL_WARPS 7          // warps 0-6 of the chunk loop: point pass, then pull
#define MEL_PIECE 8               // entries of one node a lane of the mixed pull sums before the warp combines
#define MEL_BAR_BYTES 128         // mbarriers, the flags of lost waits and the tail's ticket (at byte 64)
#define MEL_PLACES(mixed) ((mixed) ? 16 : 8)      // slots of one shared-memory wavefront (8 or 16 bytes each)
// head rows: derivative pairs of a point that its thread holds in registers (the rest are tail rows).
// Measured on B200, body kernel of 700 grains of 384 nodes: FP64 with 16 / 12 / 8 / 4 head rows 237 /
// 192 / 183 / 190 us (16 spill, few leave less shared memory for slots), mixed with 20 / 16 / 12 / 8
// 149 / 147 / 146 / 147 us
#define MEL_TILE_HEAD(mixed) ((mixed) ? 12 : 8)
#define MEL_TILE_SLOTS 3840       // slots of a tile: 224 points of 15 supports on average, groups padded
#define MEL_TILE_SLOTS_MAX 8192   // largest the tuning table may name
// support entries per chunk of a wide body, upper bound.  In the mixed form, whose images hold 12 bytes an
// entry instead of 20, 3,584 entries are the points of nearly all 224 threads.  Measured on B200, a step
// of 3 discs of 9,300 nodes (2 of 4,360) with at most 2,048 / 3,328 / 3,584 / 4,096 entries a chunk:
// 2,063 / 1,690 / 1,624 / 1,800 us (768 / 771 / 737 / 799)
#define MEL_CHUNK_E_MAX(mixed) ((mixed) ? 3584 : 2048)
#define MEL_WAIT_NS 1000000000u   // bound of every device-side wait (1 s)
#define MEL_WAIT_NOT 1u           // a wait with this bound gives up without a look (tests)
#define MEL_NBR_CAP_DEFAULT 64    // neighbour slots per body (grown on overflow)
// largest deformable body that keeps its node arrays in shared memory.  What a CTA has room for is less (176 or
// 184 bytes a node): 1,313 nodes in FP64, 1,256 in the mixed form; larger ones up to here are refused
#define MEL_MAX_BODY_NODES 4096
#define MEL_MAX_WIDE_NODES 65535  // larger bodies keep their node arrays in global memory (16-bit indices)
// bytes of a wide body's node arrays in global memory (mel_dev::gscr): s_f, s_fc, s_upf, then the
// post-loop arrays s_fn, s_fd, s_vp, s_ap, the six work terms and the temporary parameters
__host__ __device__ inline long long mel_wide_pre_bytes(int n) { return 32LL * n + 8LL * ((n + 1) & ~1); }
__host__ __device__ inline long long mel_wide_bytes(int n) { return mel_wide_pre_bytes(n) + (64LL + 48LL + 16LL) * n; }
#define MEL_SEGB 16               // segments per segment-block box (proximity pruning)
#define MEL_SEGB2 16              // blocks per superblock box (second pruning level)
#define MEL_MAX_SHIFT_SPAN 64     // periods one border box may span at a proximity update

// device error words (mel_dev::err)
enum { MEL_E_BOUNDS = 0, MEL_E_NBR_OVERFLOW = 1, MEL_E_STALE = 2, MEL_E_NAN = 3, MEL_E_CAPACITY = 4,
       MEL_E_NBR_NEED = 5, MEL_E_WAIT = 6, MEL_E_PRESSURE = 7, MEL_E_DEACT = 8, MEL_E_NWORDS = 9 };
#define MEL_PRESSURE_CAP 64       // contact contributions one border entry's pressure gathers

// Chunk image (all offsets in bytes from the image start, every section 16-byte aligned):
//   header   int4 {ngp, ne, ntn, nroff}
//   dN       ne x double2          dN/dx, dN/dy of every stored entry (float2 in the images of
//                                  the mixed-precision pass)
//   idx      ne x uint16           body-local support node of each entry
//   tpos     ne x uint16           entry positions in pull order, in pull rows (below)
//   c0       ngp2 x double         weight x jacobian of each point slot (ngp2 = ngp rounded to 2)
//   gpm      ngp4 x uint32         point slot: row table start | lane << 10 | support count << 15
//   tn       tn4 x uint32          pull slot: node | entry count << 12 | row table start << 20
//   tnode    ntn8 x uint16         (wide bodies only) each pull slot's node, 16 bits
//   roff     nroff8 x uint16       row tables: the point groups' rows, then the pull groups'
//                                  rows; each value is an offset (12 bits) | lane swizzle << 12
// Point slots: the chunk's points sorted by (support count descending, index), cut into groups of
// up to 32 slots, one warp each.  Row k of a group holds entry k of every slot whose point has
// more than k supports; these slots are a prefix of the group, so entry k of lane j sits at
// (r & 0xfff) + (j ^ (r >> 12)) with r = roff[r0 + k]: the lanes of a warp touch a permutation of
// consecutive entries.  The swizzle (k & 7 in rows whose width is a multiple of 8, else 0) spreads
// the entries of one point over the shared-memory bank groups.
// Pull slots: the touched nodes sorted by entry count (descending), cut into groups of 32 (slot t
// is lane t & 31 of group t >> 5).  Row j of a pull group holds, for every slot with more than j
// entries, the position of its node's entry j; a node's entries are in ascending point order.
// ne is the number of entries rounded up to a multiple of 8 (zero entries at the end).
// Images of the mixed pass's two-buffer loop replace the pull slots by pieces: tpos lists the
// positions of all entries in (node, point) order; the tn section holds MEL_PULL_WARPS + 1 uint16
// warp bounds (16 bytes), then one uint32 record per piece (first listed entry | (count - 1) << 13 |
// node << 16, 16 bits of node), a piece being at most MEL_PIECE consecutive entries of one node.  Pull warp w takes
// the pieces [bound w, bound w+1), which start and end at node boundaries; nroff counts the point
// rows only.
struct mel_chunk {        // one chunk of a body's Gauss points
    long long img;        // byte offset of the image in mel_dev::img
    int bytes;            // image size (multiple of 16)
    int ngp, ne, ntn;
    int gp0;              // first Gauss point (global index)
    int pad;
};

struct mel_chunk_layout {  // section offsets of an image
    int dN, idx, tpos, c0, gpm, tn, tnode, roff, bytes;
};
// dnb: bytes of one dN pair, 16 (FP64 images) or 8 (FP32 images of the mixed-precision pass).
// wide: the FP64 image of a body above MEL_MAX_BODY_NODES nodes, whose pull slots take their
// node from a uint16 section tnode (ntn8 entries) after tn instead of the record's 12 bits
__host__ __device__ inline mel_chunk_layout mel_chunk_sections(int ngp, int ne, int ntn, int nroff, int dnb, int wide = 0)
{
    mel_chunk_layout L;
    L.dN = 16;
    L.idx = L.dN + dnb * ne;
    L.tpos = L.idx + 2 * ne;
    L.c0 = L.tpos + 2 * ne;
    L.gpm = L.c0 + 8 * ((ngp + 1) & ~1);
    L.tn = L.gpm + 4 * ((ngp + 3) & ~3);
    L.tnode = L.tn + 4 * ((ntn + 3) & ~3);
    L.roff = L.tnode + (wide ? 2 * ((ntn + 7) & ~7) : 0);
    L.bytes = L.roff + 2 * ((nroff + 7) & ~7);
    return L;
}

// One tile of a body's Gauss points (sections: mel_tiles.h), a point's record and a pull slot's.
// base: offset / 128; rec_idx: bytes / 16 of the head pairs | of the tail pairs and index words << 16;
// counts: points | touched nodes << 16; pos: bytes / 16 of the position words | of the tail pairs << 16
struct mel_tile { unsigned base, rec_idx, counts, pos; };
struct mel_point { double c0; unsigned a, i; };     // weight x jacobian; a: first slot | supports << 16 | largest
                                                    // of the group << 24; i: first index word | (group
                                                    // width / 8 - 1) << 14 | slots of tail rows before << 16
struct mel_pull { unsigned node, p0; };             // node | entries << 16; first position word
__host__ __device__ inline size_t mel_tile_base(unsigned base) { return (size_t)base * 128; }
__host__ __device__ inline int mel_tile_o_rec(unsigned rec_idx) { return 16 * (int)(rec_idx & 0xffffu); }
__host__ __device__ inline int mel_tile_o_idx(unsigned rec_idx, unsigned counts) { return mel_tile_o_rec(rec_idx) + 16 * (int)(counts & 0xffffu); }
__host__ __device__ inline int mel_tile_idx_bytes(unsigned rec_idx) { return 16 * (int)(rec_idx >> 16); }
__host__ __device__ inline int mel_tile_o_slot(unsigned rec_idx, unsigned counts) { return mel_tile_o_idx(rec_idx, counts) + mel_tile_idx_bytes(rec_idx); }
// tail pairs and index words, brought by one copy; so are pull slots and position words
__host__ __device__ inline int mel_tile_pull_bytes(unsigned counts, unsigned pos) { return ((8 * (int)(counts >> 16) + 15) & ~15) + 16 * (int)(pos & 0xffffu); }
__host__ __device__ inline int mel_tile_tail_bytes(unsigned pos) { return 16 * (int)(pos >> 16); }

struct mel_dev {
    // sizes
    int nb, nn, nbd, ne, ng, nchunk, ncont, cont_cap;
    int nmat, self_contact, record_forces, precision;
    double xmin, period, gx, gy;
    // time: time2[parity] is the step's start time, time2[parity^1] its end (ping-pong)
    double* time2;
    double* dt;
    // materials and laws
    const int* mat_type; const double* mat_p;
    const int* law_type; const int* law_len; const double* law_p; const int* table;
    // bodies
    const int *b_type, *b_mat, *b_per, *b_node0, *b_bd0, *b_chunk0, *b_order;
    int* b_status;           // MEL_STATUS_*; Update_status turns bodies inactive during the run
    double* b_damage;        // Body::damage: the running value of Update_damage (starts at 0)
    const double* b_dist;
    const int* b_has_bc;     // body has a non-"none" border condition
    // bodies above MEL_MAX_BODY_NODES nodes: byte offset of the body's node arrays in gscr (-1 for
    // the others, whose node arrays live in shared memory); NULL when the model has none
    const long long* b_gscr;
    char* gscr;
    double *rg, *rf, *rtot, *drv, *works;
    // nodes
    const double2 *X0, *minv, *mass;
    double2 *x, *u, *v, *a, *up, *vp, *ap;
    const int* sup_ptr; const uint16_t* sup_idx; const double* sup_N;
    // the same supports of deformable bodies laid out for the kinematics: a body's nodes as slots
    // sorted by support count (slot ranges start at multiples of 32), groups of 32 slots; slot
    // record = node | support count << 16; entry k of lane l of group G at kg_base[G] + 32 k + l
    const int* b_ks0; const unsigned* ks_rec; const int* kg_base;
    const uint16_t* ks_idx; const double* ks_N;
    double2 *o_fint, *o_fcon, *o_fneu, *o_fdir, *o_ftot;
    // damping matrices (Body::Update_damping_forces): for each degree of freedom (2 node + direction)
    // the terms it receives, in matrix-entry order: source degree of freedom and coefficient; the
    // damping forces of the step (NULL without matrices)
    const int *dmp_ptr, *dmp_src;
    const double* dmp_c;
    double2* fdamp;
    // ALID layers (Body::Update_alid_forces): the bodies with a layer, each body's x and y history of
    // the layer's reference velocity, alid_beta per node, and per receiving degree of freedom its
    // stiffness terms (source degree of freedom, k / (1/alpha0 + 1/alpha1)) in entry order
    int n_alid;
    const int *alid_b, *alid_hptr;
    const double *alid_ht, *alid_hv, *alid_beta;
    const int *al_ptr, *al_src;
    const double* al_c;
    double2* falid;
    // borders and border entries
    const int *bd_body, *bd_per, *bd_bef, *bd_aft, *bd_e0, *bd_bc, *bd_h0;
    const double *bd_bcp, *ht, *hv;
    const int *e_node, *e_sn, *e_ss;         // e_sn/e_ss: 4 per entry (node0..3, shift0..3)
    const int* e_border;                      // border of each entry
    const double* e_len0;
    double* e_len;                            // lengths of the last Update_borders
    double2* e_bcp;                           // border-condition pressures of the last Update_bc_forces
                                              // (Border::x_bc_pressure, y_bc_pressure; zero on borders
                                              // whose conditions are both none)
    int nblk;                                 // segment blocks (MEL_SEGB segments of one border)
    const int* bd_blk0;                       // [nbd+1] first block of each border
    double4* seg_blk;                         // block boxes of the current proximity update
    int nsblk;                                // superblocks (MEL_SEGB2 consecutive blocks of one border)
    const int* bd_sblk0;                      // [nbd+1] first superblock of each border
    const int* sblk_border;                   // border of each superblock
    double4* seg_sblk;                        // superblock boxes (unions of their block boxes)
    // Gauss points: tile table and tiles; chunk table and chunk images of the wide bodies
    const mel_tile* tile;
    const int* b_tile0;
    const char* timg;
    int tile_cap, tile_q, tile_i;             // slots of a tile; shared-memory bytes of its contributions
                                              // and of its index words
    unsigned long long tile_pad;              // four positions that name the zero slot
    const mel_chunk* chunk;
    const char* img;
    int img_cap;                              // bytes of one shared-memory staging buffer
    // contacts
    mel_contact* cont;
    double* cont_w;                           // per-contact work increment of the last law evaluation
    double* cont_rt;                          // 6 per contact: rigid slave and rigid master force and
                                              // moment terms of the last contact pass (arms from the
                                              // positions before the body kernel moves any node)
    int any_damped;                           // a law with work terms is in use
    const int* b_cont0;                       // [nb+1] slave contact ranges (list is body-major)
    const int* b_inc0;                        // [nb+1] into inc_rng
    const int2* inc_rng;                      // incoming (master-side) contact ranges in send order
    // Solver_step (Code/Solver.h:98-486): phase of an adaptive launch (1: first half-step, 2: second
    // half-step), scheme and its parameters (mel_model_desc::solver_params), inverse distance
    // estimators of the nodes (Code/IO.h:1620,1819), temporary displacement parameters and
    // displacements, nodal errors, nodal mass-scaling factors; per body: total and largest error,
    // scaled mass, rigid mass-scaling factor and its last increment, rigid temporary kinematics
    // (x, y, r displacement then velocity)
    int phase, solver;
    double sp[8];
    const double* ide;
    double2 *upt, *ut, *errv, *fms;
    double *terr, *merr, *bmms, *bfms, *bdfms, *rg_tmp;
    // border contact pressures (Update_contact_pressures): per border entry, the contributions
    // gathered (contact << 2 | role, at most MEL_PRESSURE_CAP) and the pressures
    int* cp_cnt; int* cp_item;
    double *cpx, *cpy;
    // bounds of the body kernel's waits (MEL_WAIT_NS; the environment variables MELGPU_WAIT_NS, all of
    // them, and MELGPU_TILE_WAIT_NS read by mel_create shorten them so that tests can make a wait
    // give up): wait_tile_ns those for a tile's index words and for its pull sections
    unsigned wait_ns, wait_tile_ns[2];
    // error words
    unsigned int* err;
};

// kernel launch wrappers (mel_kernels.cu)
// Update_damping_forces of every deformable body with matrices, from the velocity parameters
void mel_launch_damping(const mel_dev& d, cudaStream_t s);
// Update_alid_forces at the step's start time time2[parity], or at T when use_T (Solver_step)
void mel_launch_alid(const mel_dev& d, int parity, double T, int use_T, cudaStream_t s);
void mel_launch_contact(const mel_dev& d, double law_dt_scale, cudaStream_t s);
// Initialize_CZM's pass over the contact list (contact geometry, then the initial bonds)
void mel_launch_czm_init(const mel_dev& d, cudaStream_t s);
// nblocks: bodies b_order[0, nblocks); nwide: the wide bodies after them
void mel_launch_body(const mel_dev& d, int parity, int nblocks, size_t smem, cudaStream_t s, int nwide = 0);
// one half-step of Solver_step (d.phase 1 or 2): T0 = Time, Tf = the time the forces see
void mel_launch_body_adaptive(const mel_dev& d, double T0, double Tf, int nblocks, size_t smem, cudaStream_t s, int nwide = 0);
// device-to-device copies of up to 16 arrays of 8-byte words by one launch
struct mel_copy_list { int n; const void* src[16]; void* dst[16]; size_t words[16]; };
void mel_launch_copy_many(const mel_copy_list& L, cudaStream_t s);
// Solver_step's error and mass sums over the bodies in order (Code/Solver.h:289-331): out =
// {mean_error, max_error, total_mass, max_mass}, then the MEL_E_NWORDS error words
void mel_launch_error_reduce(const mel_dev& d, double* out, cudaStream_t s);
// Update_bc(T) of every body's driven degrees of freedom (mel_dev::drv)
void mel_launch_drivendof(const mel_dev& d, double T, cudaStream_t s);
// Body::Restore of the rigid bodies' kinematics from a copy of the rigid records
void mel_launch_rigid_restore(const mel_dev& d, const double* rg_snap, cudaStream_t s);
// one step of a batch: the contact pass over thr0[nsamp] threads, the body pass over the ncta
// CTAs of cta (sample, CTA of the sample) and the per-sample time advance (devs, thr0, cta in device memory).  The body pass is two
// launches: CTAs [0, ncta_small) with smem_small bytes (members whose bodies fit two CTAs per SM,
// ordered first), then the rest with smem bytes
void mel_launch_batch_step(const mel_dev* devs, const int* thr0, int nthr, const int2* cta, int ncta_small, int ncta,
                           int nsamp, int mixed, size_t smem_small, size_t smem, cudaStream_t s);
// shared memory of a body CTA: node arrays of max_nodes nodes beside `stage` bytes of Gauss-point
// contributions or the post-loop arrays, whichever are larger
size_t mel_body_smem_bytes(int max_nodes, size_t stage, int mixed);
void mel_launch_update_borders(const mel_dev& d, cudaStream_t s);
void mel_launch_monitor(const mel_dev& d, double* part, const int* rigid_ids, int nrigid, double* out, cudaStream_t s);
// Update_contact_pressures (Code/Proximity.h:1014-1069) from the current contact list
void mel_launch_contact_pressures(const mel_dev& d, cudaStream_t s);

// one monitored entry of STATIC_CONTROL's MONITORING list (the vector Read_spy_line builds,
// Code/IO.h:11-590): type (0 position, 1 displacement, 2 velocity, 3 acceleration, 4 force,
// 7 contact, 9 energy, 10 work), kind (component or quantity), sub (force kind), body, node (-1:
// the whole body), border and border node (contact entries)
struct mel_mon_op { int type, kind, sub, body, node, border, bnode, pad; };
// the row's leading columns (Code/Monitoring.h:25)
struct mel_mon_head { double iteration, time, dt, neval, max_error, mean_error; };
// Monitoring after a step: per-body partial sums into part[3*nb], then the row into row[0..]
// (row[0] = number of values that follow)
// Update_status (Code/Proximity.h:550-1007): the DEACTIVATION entries (MEL_DEACT_NF doubles each)
// evaluated on the current state; bodies whose condition holds become inactive
void mel_launch_status(const mel_dev& d, const double* entries, int n, cudaStream_t s);
void mel_launch_monitor(const mel_dev& d, const mel_mon_op* ops, int nops, int energy, int boundaries,
                        double* part, double* row, const mel_mon_head& hd, cudaStream_t s);

int mel_body_kernel_configure(size_t smem);

#define MEL_CUDA_OK(call) do { cudaError_t e_ = (call); if (e_ != cudaSuccess) { mel_set_cuda_error(e_, #call, __FILE__, __LINE__); return MEL_ERR_CUDA; } } while (0)
void mel_set_cuda_error(cudaError_t e, const char* what, const char* file, int line);
void mel_set_error(const char* fmt, ...);
