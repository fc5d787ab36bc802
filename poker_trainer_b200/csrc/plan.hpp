// Device plan of one traversal: POD task records shared by the host planner
// (engine.cu) and the kernels (kernels.cu).
//
// A traversal for traverser p over a subtree is level-synchronous:
//   down levels  — opponent nodes split the opponent reach by their
//                  strategy (regret matching + strategy-sum update in CFR
//                  mode), chance nodes fan the reach out per dealt card;
//   terminals    — fold and showdown values of every live terminal;
//   up levels    — deepest first: traverser nodes combine child values
//                  (and update regrets), opponent nodes and chance nodes sum.
// Reach rows live in "slots" (a traverser node's children share its slot);
// value rows are indexed by node id. Every row has HP floats (hands padded
// to a multiple of 8, padding kept at zero).
#pragma once

#include <cstdint>

namespace dcfr {

constexpr int VEC = 4;             // hands per thread in the row kernels (float4)
constexpr int ROW_MAX_THREADS = 352;  // row-kernel block: a thread per 4 hands, whole warps (1328 hands max)
constexpr int MAX_ACTIONS = 16;
constexpr uint32_t NONE32 = 0xFFFFFFFFu;

enum DownKind : uint32_t { D_OPP_SPLIT = 0, D_CHANCE_SPLIT = 1 };
enum UpKind : uint32_t { U_OWN = 0, U_OPP_SUM = 1, U_CHANCE_SUM = 2 };
enum TermKind : uint32_t { T_FOLD_SCALAR = 0, T_FOLD_BATCH = 1, T_SHOWDOWN_SCALAR = 2, T_SHOWDOWN_BATCH = 3 };
enum ModeId : int { M_CFR = 0, M_BR = 1, M_AVG = 2 };

struct DownTask {
  uint32_t kind;
  uint32_t in_slot;   // reach slot of the node
  uint32_t out_slot;  // slot of the first child (children's slots are consecutive)
  uint32_t nchild;
  uint64_t store;     // opponent split: float offset of the node's block
  uint32_t cards;     // chance split: offset of the children's cards in chance_cards;
                      // opponent split: the node's scale slot (compressed storage)
  float factor;       // chance split: reach multiplier
};

struct UpTask {
  uint32_t kind;
  uint32_t slot;        // reach slot of the node (liveness)
  uint32_t node;        // value row
  uint32_t child;       // first child's node id (value rows are consecutive)
  uint32_t nchild;
  uint32_t child_slot;  // first child's slot (opponent / chance nodes)
  uint64_t store;       // traverser node: float offset of its block
  uint32_t cards;       // chance: offset of the children's cards; decision node:
                        // its scale slot (compressed storage)
  uint32_t iso_first;   // chance: first isomorphic reference
  uint32_t iso_count;
  uint32_t pad;
};

// Fused segment: the down and up tasks of all its decision nodes, processed by
// one block (down: BFS order, LEVEL_BREAK on a level's first task, the node's
// slot counted in the segment above LOCAL_SHIFT: 0 for the root's, then the
// tasks' children in order; up: deepest level first).
struct FusedTree {
  uint32_t down_first, down_count;
  uint32_t up_first, up_count;
};
constexpr uint32_t LEVEL_BREAK = 0x100u;  // in DownTask::kind
constexpr uint32_t KIND_MASK = 0xFFu;
constexpr uint32_t LOCAL_SHIFT = 12;      // of DownTask::kind in a fused segment
constexpr int FUSED_MAX_NODES = 48;       // decision nodes of a fused segment

struct IsoRefD {
  uint16_t ci;    // canonical child index
  uint8_t pair;   // suit pair (0..5)
  uint8_t pad;
};

struct TermLane {
  uint32_t slot;  // reach slot
  uint32_t row;   // value row (node id)
  uint32_t frow;  // paired fold's value row, or NONE32
  uint32_t pad;
  double a;       // fold payoff / showdown win
  double b;       // showdown lose
  double c;       // showdown tie
  double d;       // paired fold payoff
};

// Strength-table entry (eval::Entry, crates/solver/src/eval.rs:11-18).
struct EntryD {
  uint32_t strength;
  uint16_t idx;
  uint8_t c1, c2;
};

struct DiscountD {
  float pos, neg, strat;
  int reach_weighted;
};

// One decision node's storage block for transfers to and from the
// reference's layout (HostStorage, crates/solver/src/storage.rs): its
// [rows][hp] block at element `dev` of the device storage, and its
// [rows][n] block at element `host` of the reference layout, counted from
// the start of the transfer chunk that holds it.
struct StorageBlockD {
  uint64_t dev, host;
  uint32_t rows, n, hp, pad;
};

// Fast-precision terminal evaluation (terminal_fast.cu): one task per live
// terminal; a showdown task also writes its paired fold's row.
struct FastTask {
  uint32_t kind;   // TermKind
  uint32_t board;  // layout index: showdown board, or the fold layout
  uint32_t slot;   // reach slot
  uint32_t row;    // value row (node id)
  uint32_t frow;   // paired fold's value row, or NONE32
  // A batch's task, whose spot has rows of its own length: its reach row, which
  // like row and frow counts ROW_UNITs there, and the row's entries (the
  // opponent's hands, padded).
  uint32_t reach, entries;
  uint32_t pad;
  double a, b, c, d;  // as TermLane
};

// A depth-limited solve's leaf in one traversal: the leaf's ordinal, the
// reach slot arriving at it and the value row (node id) it fills, and the
// state entering the network (pot and effective stack in chips).
struct LeafTask {
  uint32_t leaf;
  uint32_t slot;
  uint32_t row;
  uint32_t pad;
  float pot;
  float stack;
};

// Longest opponent hand list evaluated warp per terminal; longer lists use
// the block-wide scan of fast_terminal_kernel (measured: the block kernel is
// faster at 1128 hands, the warp kernel at 470).
constexpr int WARP_TERMINAL_MAX_HANDS = 768;
// A maximal run of fast terminal tasks on one layout. The warp terminal
// kernel (terminal_fast.cu) stages a run's layout in shared memory once per
// block whose task range meets the run.
struct TermUnit {
  uint32_t layout;  // FastTask::board of every task in the run
  uint32_t first;   // first task
  uint32_t count;   // tasks
  uint32_t pad;     // TileClass of its tasks, where the plan orders them by class
};
// Tasks that a tile of terminal_tile.cu evaluates alike: batched showdowns
// with neither tie payoff nor paired fold, other showdowns, folds.
constexpr int TILE_THREADS = 512;  // threads a block, and most tasks of a job
enum TileClass : uint32_t { TILE_PLAIN = 0, TILE_GENERAL = 1, TILE_FOLD = 2 };

// A panel of the panel terminal kernel (terminal_panel.cu): `count` (1..T)
// consecutive fast terminal tasks, all on one layout and all showdowns or
// all folds.
struct PanelD {
  uint32_t first;   // first task
  uint32_t count;   // tasks
  uint32_t layout;  // FastTask::board of every task in the panel
  uint32_t pad;
};

// Per (layout, traverser) scan layout of the opponent's hands: segment 0
// lists them in ascending strength, segment 1+c lists those holding card c
// (ascending strength). seg[j] is the first element of segment j
// (seg[53] = 3 * count). Per traverser hand h, rec[h] = {w | s << 16,
// aw | as << 16, bw | bs << 16, a | b << 8 | present << 16}: w (s) counts the
// opponent hands weaker than (not stronger than) h, aw/as (bw/bs) index the
// same boundaries inside card a's (b's) segment.
constexpr int ROW_UNIT = 8;  // rows are padded to this many hands
constexpr int FAST_SEGS = 54;
constexpr int FAST_THREADS = 256;

// Between two traversals that share a segment pass across the end of an
// iteration (Engine::enqueue_rolled), a terminal kernel clears the other
// traverser's liveness flags, whose last reader is done and whose next writer
// has not begun, and steps the discounts: TURN_NEXT writes the coming
// iteration's to cur[1], TURN_BEGIN counts that iteration and makes them
// cur[0].
enum TurnStep : uint32_t { TURN_KEEP = 0, TURN_NEXT = 1, TURN_BEGIN = 2 };
struct PassTurn {
  uint32_t* clear = nullptr;
  uint32_t nclear = 0;
  uint32_t step = TURN_KEEP;
  uint32_t* counter = nullptr;
  const DiscountD* table = nullptr;
  uint32_t table_len = 0;
  DiscountD* cur = nullptr;
};

// R is the row type: float for the solve, double for the FP64 best-response
// oracle (br64.cu).
template <typename R>
struct FastArgsT {
  const R* reach;
  R* vals;
  const uint32_t* alive;
  const uint16_t* cat;   // [(layout*2+p)][cstride] opponent hand per element
  const uint16_t* seg;   // [(layout*2+p)][FAST_SEGS]
  const uint4* rec;      // [(layout*2+p)][tstride]
  const uint32_t* same;  // traverser hand -> identical opponent hand (or NONE32)
  // A batch's spots (layout 2 * spot): {n0, n1, hp0, hp1} of each, and `same`
  // has rows of `stride` per (spot, traverser). Null: one game, n and hp.
  const int4* dims = nullptr;
  PassTurn turn;
  int cstride;
  int tstride;
  int emax;              // elements per thread (odd) for the largest layout
  int n[2];
  int hp[2];
  int stride;
  int p;
};
using FastArgs = FastArgsT<float>;
using FastArgs64 = FastArgsT<double>;

// Arguments of the row kernels (down/up levels) of one traversal.
struct RowArgs {
  float* regrets;
  float* sums;
  // 16-bit compressed storage (set instead of regrets / sums): i16 regrets,
  // u16 sums, one f32 scale of each per decision node (its ordinal).
  int16_t* rq;
  uint16_t* sq;
  float* rscale;
  float* sscale;
  int compressed;
  float* reach;
  float* vals;
  uint32_t* alive;
  const uint8_t* hc1[2];  // hand cards, padded to hp with 255
  const uint8_t* hc2[2];
  const uint16_t* perm;   // [(q*6+pair)*stride + h]
  const uint8_t* chance_cards;
  const IsoRefD* iso;
  const DiscountD* disc;
  int n[2];
  int hp[2];
  int stride;
  int p;
  int sms;                // the device's
};

// Segment passes (segment.cu). Tasks count slots, value rows and storage rows
// in the segment's own numbering; g* are the global ones.
constexpr int SEG_SLICE = 32;                  // hands per block
constexpr size_t SEG_SMEM_MAX = 200 << 10;     // shared memory of a pass
struct SegUp {
  uint32_t kind, nchild;
  uint32_t slot, node, child, child_slot;
  uint32_t store;   // traverser node: its first storage row
  uint32_t gnode;
  uint64_t gstore;  // traverser node: float offset of its block
  float uniform;    // 1 / nchild
  uint32_t pad;
};
struct SegDown {
  uint32_t in_slot, out_slot, nchild, store;
  uint64_t gstore;
  uint32_t gslot;   // first child's slot
  float uniform;
};
// A value row another kernel fills (a terminal's, a chance node's, a leaf's):
// its node and its row in the segment's numbering.
struct SegRow {
  uint32_t node, row;
};
// One traversal's root segment: its records in one array, the up tasks first,
// then at byte offsets the down tasks, the value rows to fetch, the global
// slot of each of its slots, and the level boundaries of the up (deepest
// first) and then the down tasks.
struct SegRes {
  const unsigned char* blob;
  uint32_t o_down, o_vals, o_slots, o_levs, bytes;
  const uint64_t* own[2];  // per player: float offsets of its storage rows
  uint32_t nup, ndown;     // levels
  uint32_t n_up, n_down;   // tasks
  uint32_t n_vals, n_rows, n_slots, n_own[2];  // fetched rows, value rows, slots, storage rows
  uint32_t root;           // the root's node
};

// One launch: the up pass of the traversal U (of traverser up.p) and then the
// down pass of D (of down.p); one that is not wanted has no blob.
struct SegPass {
  RowArgs up, down;
  SegRes U, D;
  const uint64_t* rows;        // storage rows of the player that both update
  uint32_t n_rows;
  int slices;
  const uint8_t* up_deferred;  // [slices][down task]
  uint8_t* down_deferred;
  float* root_out;             // the root's value row, or null
  const float* roots;          // the root's reach row
};

// Arguments of the FP64 best-response kernels (br64.cu): double reach and
// value rows, the f32 strategy sums.
struct Row64Args {
  const float* sums;
  const uint16_t* sq;     // compressed storage: u16 sums and per-node scales (sums is null)
  const float* sscale;
  double* reach;
  double* vals;
  uint32_t* alive;
  const uint8_t* hc1[2];
  const uint8_t* hc2[2];
  const uint16_t* perm;
  const uint8_t* chance_cards;
  const IsoRefD* iso;
  int n[2];
  int hp[2];
  int stride;
  int p;
};

}  // namespace dcfr
