// tb_tree.cuh -- hierarchical form of the ring field sums.
//
// The sum over 16 N rings at a point resolves every element with 16 rings,
// however far away it is; what the field at a distance d needs is a number of
// rings that grows with log(size / d).  The rings of a straight, axis-parallel
// stretch of electrode (r or z constant: tubes, caps, plates) are therefore
// gathered into a binary tree of element ranges, and every node carries
// TREE_P proxy rings at the Chebyshev nodes of its extent whose weights
// interpolate the node's rings (the kernel-independent treecode with
// barycentric Lagrange interpolation of Wang, Krasny and Tlupova, Commun.
// Comput. Phys. 28, 2020, in one dimension).
//
// Accuracy.  Along the stretch the ring kernels are analytic but for the
// points where rho2 or D vanish; the nearest of these to the interval
// [c - h, c + h] is the observation point itself seen as c + x + i y.  It
// lies on the Bernstein ellipse whose size rho obeys rho + 1/rho = (sum of
// its distances to the two ends) / h, and interpolation in P nodes leaves a
// relative error of at most 2 rho^-P.  A node is used when that sum is at
// least TREE_KAPPA h: rho = 10, 2 10^-16 at worst.  Against extended precision
// on the lens and pole-piece meshes the sums are off by 1e-16 of their terms,
// as much as the direct sums' rounding (rho = 8 took 20 % fewer rings but left
// 5e-16); the degree-7 forms of K and E leave 5e-13 in both.  Nearer nodes are
// split; leaves that are too near are summed ring by ring.
//
// A stretch counts as straight when its constant coordinate varies by
// rounding only (TREE_TOL); the proxies take the |w|-weighted mean of it, and
// a node is used only at distances at which that variation is invisible
// (TREE_JITTER).  Everything else (curved or sloped elements, non-finite
// rings, negative radii) is summed ring by ring.
#pragma once

#include <cstdint>
#include "tb_common.cuh"
#include "tb_internal.cuh"

namespace tb {

constexpr int TREE_P = 16;             // proxies per node = rings per element: one chunk is either
constexpr int TREE_LEAF = 4;           // elements of the smallest nodes
constexpr int TREE_MID = 32;           // elements of the largest nodes built from rings (larger ones from these)
constexpr float TREE_KAPPA = 10.2f;    // rho + 1/rho = 10.1 at rho = 10, and a margin for the FP32 test
constexpr double TREE_TOL = 4e-15;
constexpr float TREE_JITTER = 1e14f;
constexpr int64_t TREE_MAX_ELEMENTS = 1 << 18;
constexpr int TREE_CHUNK = 3 * TREE_P;  // doubles of a chunk: r[16], z[16], w[16]

enum TreeAxis : int { TREE_HORIZONTAL = 0, TREE_VERTICAL = 1, TREE_DIRECT = 2 };  // r constant, z constant, neither

// One node: its rings' range c +- h along the stretch and the constant
// coordinate v across it; reach: the smallest sum of distances to the ends at
// which the proxies may be used; tag = 8 ne + 4 (leaf) + axis with ne its
// elements (0: an empty slot); link: a leaf's first element, else the slot of
// the first of its two children.
struct alignas(16) TreeNode {
  double c, v;
  float h, reach;
  int tag, link;
};

struct TreeAux {  // of a node, for its ancestors
  double h, wabs, vmin, vmax;
};

// A tree in its workspace (device pointers).  Chunk e < n is element e's
// rings, chunk n + slot the proxies of node slot.
struct Tree {
  double* chunk = nullptr;
  TreeNode* node = nullptr;
  TreeAux* aux = nullptr;
  uint8_t* kind = nullptr;   // per element: axis, + 4 if a run starts there
  int* run_e0 = nullptr;     // [runs + 1] first element of each run
  int* run_slot = nullptr;   // [runs + 1] its root's slot
  int* group_run = nullptr;  // [groups + 1] first run of each group of rings
  int* count = nullptr;      // [3] runs, slots, 1: of no use, or a group does not start at an element
  int n = 0;                 // elements
  int groups = 0;
};

inline int64_t tree_round(int64_t b) { return (b + 255) / 256 * 256; }

// Lays a tree of n elements in `groups` groups out in `work`; returns its bytes.
inline int64_t tree_layout(int64_t n, int64_t groups, char* work, Tree* t) {
  int64_t o = 0;
  auto take = [&](int64_t bytes) {
    char* p = work ? work + o : nullptr;
    o += tree_round(bytes);
    return p;
  };
  Tree x;
  x.chunk = reinterpret_cast<double*>(take(2 * n * TREE_CHUNK * 8));
  x.node = reinterpret_cast<TreeNode*>(take(n * int64_t(sizeof(TreeNode))));
  x.aux = reinterpret_cast<TreeAux*>(take(n * int64_t(sizeof(TreeAux))));
  x.kind = reinterpret_cast<uint8_t*>(take(n));
  x.run_e0 = reinterpret_cast<int*>(take((n + 1) * 4));
  x.run_slot = reinterpret_cast<int*>(take((n + 1) * 4));
  x.group_run = reinterpret_cast<int*>(take((groups + 1) * 4));
  x.count = reinterpret_cast<int*>(take(3 * 4));
  x.n = int(n);
  x.groups = int(groups);
  if (t) *t = x;
  return o;
}

// Builds the tree of the rings src (3, 16 n) on the stream (tb_tree.cu).
// offsets (groups + 1, device memory): the first ring of each group, or null
// for one group.  Where one is not a multiple of 16 (count[2] is 1 then) the tree
// is not that of the groups.
int tree_build(const Tree& T, const double* src, const int64_t* offsets, cudaStream_t s);

// Scratch of one warp's walk.  A round of the walk takes at most 32 nodes off
// the stack and puts at most 64 children on it, the deepest first, so each
// level of the tree (at most 18) leaves at most 32 nodes behind.  It puts at
// most 32 TREE_LEAF chunks on the list, which is emptied above TREE_FLUSH.
constexpr int TREE_STACK = 32 * 18 + 64;
constexpr int TREE_FLUSH = 64;
constexpr int TREE_LIST = TREE_FLUSH + 32 * TREE_LEAF;
struct TreeScratch {
  int stack[TREE_STACK];
  int list[TREE_LIST];
};

// Adds this lane's share of the field sums of groups' runs run0 .. run1 - 1 at
// (r0, z0) to Sr, Sz (Sp); all lanes of the warp call it.  `part` of `parts`
// (a power of two) warps take the chunks in turn (each walks the tree for
// itself).
//
// Proxies and the elements of leaves that are too near for theirs go to one
// list of chunks, a half-warp per chunk, and each list starts with the
// half-warp after the one that took the last chunk of the one before: however
// short the runs are, all half-warps of all parts have the same number of
// rings to within one chunk (a half-warp per leaf, one leaf after another,
// left all but one idle on meshes whose neighbours are not on one line: 800
// elements in random order, one electron and eight warps 38 ms instead of the
// direct sums' 3.1).
template <bool POT>
__device__ __forceinline__ void tree_sums(const Tree& T, int run0, int run1, double r0, double z0, TreeScratch& sc,
                                          int part, int parts, double& Sr, double& Sz, double& Sp) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const double* mine = T.chunk + (lane & 15);
  const int step = 2 * parts;
  int turn = (lane >> 4) + 2 * part;  // this half-warp's first chunk of the next list
  int nst = 0, nl = 0;
  auto add = [&](int chunk) {
    const double* p = mine + int64_t(chunk) * TREE_CHUNK;
    ring_field_acc<POT>(r0, z0, p[0], p[TREE_P], p[2 * TREE_P], Sr, Sz, Sp);
  };
  auto flush = [&]() {
    __syncwarp();
#pragma unroll 2
    for (int i = turn; i < nl; i += step) add(sc.list[i]);
    turn = (turn - nl) & (step - 1);
    __syncwarp();
    nl = 0;
  };
  while (run0 < run1 || nst > 0) {
    int slot = -1;
    if (nst > 0) {
      const int take = nst < 32 ? nst : 32;
      nst -= take;
      if (lane < take) slot = sc.stack[nst + lane];
      __syncwarp();
    } else {
      if (run0 + lane < run1) slot = __ldg(T.run_slot + run0 + lane);
      run0 += 32;
    }
    bool use = false, split = false;
    int link = 0, ne = 0;
    if (slot >= 0) {
      const TreeNode nd = T.node[slot];
      ne = nd.tag >> 3;
      link = nd.link;
      const bool hor = (nd.tag & 3) == TREE_HORIZONTAL;
      const float du = float((hor ? z0 : r0) - nd.c), dv = float((hor ? r0 : z0) - nd.v);
      const float a = du + nd.h, b = du - nd.h, v2 = dv * dv;
      use = ne > 0 && sqrtf(fmaf(a, a, v2)) + sqrtf(fmaf(b, b, v2)) >= nd.reach;
      split = ne > 0 && !use && !(nd.tag & 4);
    }
    const bool near = ne > 0 && !use && !split;  // too near for the leaf's proxies: its elements' rings
    const unsigned mu = __ballot_sync(0xffffffffu, use), ms = __ballot_sync(0xffffffffu, split);
    const unsigned mn = __ballot_sync(0xffffffffu, near);
    if (use) sc.list[nl + __popc(mu & below)] = T.n + slot;
    nl += __popc(mu);
    if (split) {
      const int at = nst + 2 * __popc(ms & below);
      sc.stack[at] = link;
      sc.stack[at + 1] = link + 1;
    }
    nst += 2 * __popc(ms);
    if (mn) {
      // up to four chunks a leaf, at the sum of the lower lanes' counts
      const int c = near && ne <= TREE_LEAF ? ne : 0;
      const unsigned c1 = __ballot_sync(0xffffffffu, c & 1), c2 = __ballot_sync(0xffffffffu, c & 2),
                     c4 = __ballot_sync(0xffffffffu, c & 4);
      const int at = nl + __popc(c1 & below) + 2 * __popc(c2 & below) + 4 * __popc(c4 & below);
      for (int k = 0; k < c; k++) sc.list[at + k] = link + k;
      nl += __popc(c1) + 2 * __popc(c2) + 4 * __popc(c4);
      unsigned ml = __ballot_sync(0xffffffffu, near && ne > TREE_LEAF);
      while (ml) {  // a long run without proxies
        const int src = __ffs(ml) - 1;
        ml &= ml - 1;
        const int le0 = __shfl_sync(0xffffffffu, link, src), lne = __shfl_sync(0xffffffffu, ne, src);
#pragma unroll 2
        for (int i = turn; i < lne; i += step) add(le0 + i);
        turn = (turn - lne) & (step - 1);
      }
    }
    if (nl > TREE_FLUSH) flush();
    __syncwarp();
  }
  flush();
}

}  // namespace tb
