// Device-side descriptors of one pipeline launch, filled by the host runtime
// (dq_runtime.cu) from the public IR (include/dogqc_b200.h) and passed to the
// pipeline kernel as one __grid_constant__ parameter.
#pragma once
#include <stdint.h>
#include "../../include/dogqc_b200.h"

namespace dq {

constexpr int kThreads = 256;          // pipeline kernel block size
constexpr int kMaxStages = 4;          // tile staging depth
constexpr int kMaxRes = 16;            // resources of a plan (every pipeline sees them all)
constexpr int kMaxStr = 8;             // string columns per pipeline
constexpr int kMaxStash = 24;          // values carried by one heavy work item
constexpr uint64_t kEmpty = ~0ull;     // empty tag of every hash table

// status bits written by device code
enum : int32_t {
  kErrHtFull = 1,
  kErrTimeout = 2,
  kErrOverflow = 4,
  kErrBadOp = 8,
  kErrKeyRange = 16,     // a key outside a key-domain bitmap's range: the host
                         // turns the table back into a hash table and re-runs
  kInfoHeavyFull = 32,   // informational: deferred expansion items exceeded their
                         // capacity; the rest ran in place (results stay exact)
  kErrMultiFull = 64,    // a multimap's build side has more rows than there is
                         // payload room for: nothing is scattered or probed, the
                         // host grows the multimap and re-runs
  kErrWideRange = 128,   // a long range in a run without room for deferred items:
                         // the host re-runs with room
};
constexpr int32_t kInfoMask = kInfoHeavyFull;
// A run that has one of these is repeated or fails, and its tables are not
// whole: the kernels that follow do nothing.
constexpr int32_t kErrStop = kErrHtFull | kErrTimeout | kErrMultiFull | kErrWideRange;

// A run without room for deferred items expands ranges in place, inside one warp,
// up to this many rows; a longer one ends the run, which is repeated with room.
// 32 ranges of 15,000 rows met by one warp took 4.4 ms in place, the run and its
// repetition 0.4.
constexpr uint32_t kWideRange = 1u << 11;

struct DevCol {           // staged fixed-width column
  const uint8_t* ptr;
  int32_t width;
  int32_t smem_off;       // offset inside one stage buffer
};

struct DevStr {           // string column, read in place
  const uint8_t* chars;
  const uint64_t* offsets;
  int32_t width;          // > 0: fixed-width strings
  int32_t sid;            // its index in the plan's string sources (string references)
};

// A string value carried as a 64-bit reference (group keys, join payloads and
// output columns hold these; the bytes stay in place): the plan's string source
// (bits 63..52), a substring flag (bit 51) with the substring's first and end
// byte offsets in the string (bits 50..43 and 42..35) and the row (bits 34..0).
constexpr int kStrRefShift = 52;
constexpr uint64_t kStrRefSub = 1ull << 51;
constexpr int kStrRefStartShift = 43;
constexpr int kStrRefEndShift = 35;
constexpr uint64_t kStrRefRow = (1ull << kStrRefEndShift) - 1;
constexpr int kStrRefMaxSources = 1 << 12;
constexpr int kStrRefMaxOffset = 255;

#ifdef __CUDACC__
// The bytes a reference names: its source's row, cut to the substring window
// when the flag is set (offsets past the string's end give the empty string).
__device__ __forceinline__ void str_ref_bytes(const DevStr* src, uint64_t ref, const uint8_t*& p, int& n) {
  const DevStr& d = src[ref >> kStrRefShift];
  const uint64_t row = ref & kStrRefRow;
  if (d.width > 0) {
    p = d.chars + row * (uint64_t)d.width;
    n = d.width;
  } else {
    p = d.chars + d.offsets[row];
    n = (int)(d.offsets[row + 1] - d.offsets[row]);
  }
  if (ref & kStrRefSub) {
    int st = (int)((ref >> kStrRefStartShift) & 0xff), en = (int)((ref >> kStrRefEndShift) & 0xff);
    st = st < n ? st : n;
    en = en < n ? en : n;
    if (en < st) en = st;
    p += st;
    n = en - st;
  }
}
#endif

struct DevSlot {
  int8_t kind, level, ctype, width;
  int16_t src, res;
  int32_t smem_off;       // REG: offset inside the level's register area
  int32_t stash;          // index in a heavy item's stash (-1: not carried)
};

struct DevRes {
  int32_t kind;           // dq_res_kind
  int32_t nkeys;
  int8_t key_ctype[DQ_MAX_KEYS];
  int32_t packed;         // keys packed into the 64-bit tag
  int32_t compact;        // UNIQUE, one key and one payload of at most 32 bits
                          // each: a slot is one word, key << 32 | payload
                          // (~0 empty); the all-ones key lives at slot cap
                          // (0 when present) with its payload at cap + 1
  int32_t words;          // 64-bit words per slot (tag + keys + payload/aggs)
  int32_t key_word;       // first key word (hashed keys only)
  int32_t val_word;       // first payload / accumulator word
  uint64_t cap;           // slots (UNIQUE/AGG), buckets (MULTI), rows (OUTPUT)
  uint64_t* slots;        // UNIQUE/AGG: cap+1 slots (last = tag ~0 key)
  uint32_t* counts;       // MULTI
  uint64_t* ranges;       // MULTI (cap+1): a bucket's rows << 32 | its first payload row
                          // (behind the last bucket: the rows of all)
  uint32_t* rank;         // MULTI, ranked: a source row's rank in its bucket, left by
                          // the count pass for the scatter pass (by source row)
  int32_t ranked;
  int32_t row_bytes;      // MULTI: > 0: a row's payload is one aligned item of that
                          // size (field j at pay_off[j]), else a column per field
  int8_t pay_off[DQ_MAX_PAY];
  int32_t npay;
  int32_t naggs;
  int8_t pay_ctype[DQ_MAX_PAY];
  int8_t pay_width[DQ_MAX_PAY];
  int8_t agg_red[DQ_MAX_AGGS];
  uint8_t* pay[DQ_MAX_PAY];   // MULTI payload columns / OUTPUT columns
  uint64_t* cursor;       // OUTPUT row cursor
  int32_t smem_slots;     // AGG: CTA-local table slots (0: global only)
  int32_t group_hint;     // AGG: groups the plan expects
  int32_t smem_off;       // AGG: offset of the CTA-local table
  int32_t bitmap;         // UNIQUE over a small key domain [bmin, bmin + brange):
                          // 1: no payload, slots hold one bit per key;
                          // 2: one 32-bit payload, slots hold a word per key,
                          //    (1 << 32) | payload, 0 when the key is absent
  int64_t bmin;
  uint64_t brange;
  uint32_t* bits;         // MULTI, filter: a bit per key of [bmin, bmin + brange) that
  int32_t filter;         // the build side holds (set by the count pass)
};

struct DevHeavy {         // deferred wide expansion ranges
  uint64_t* items;        // cap * words
  uint32_t* count;
  uint64_t* unit_prefix;  // work-unit prefix over items (heavy mode)
  uint32_t cap;
  int32_t words;          // 2 + number of stashed values
  int32_t nstash;
  int32_t op;             // index of the EXPAND op the items belong to
  uint64_t threshold;     // ranges longer than this are deferred
  // grouped mode (generated kernels): items whose probe rows matched the same
  // range form a group, and a warp gathers a chunk of the range once for all
  // of the group's items
  int32_t grouped;
  uint32_t gcap;          // group table slots
  uint64_t* gkey;         // (instance << 32) | range offset; kEmpty: free.  A
                          // range's offset identifies it within its instance
                          // (plain plans: instance 0; batches: shared buffers)
  uint32_t* glen;         // range length of a claimed group slot
  uint32_t* gcnt;         // items per group slot, then its scatter cursor
  uint32_t* glist;        // claimed group slots, in claim order
  uint32_t* ngroups;
  uint32_t* gstart;       // item prefix over glist (ngroups + 1 entries)
  uint64_t* sorted;       // the items' stashed values, grouped (cap * nstash)
};

constexpr int kGroupRows = 32;    // range rows per grouped work unit (a warp)
constexpr int kGroupItems = 64;   // items per grouped work unit
constexpr int kGroupThreshold = 128;   // grouped mode: ranges longer than this are deferred
constexpr int kGroupThresholdLow = 8;  // ... once a run showed several probe rows per range
constexpr int kBatchGroupThreshold = 128;  // the same in batches (their item buffers do not grow)

constexpr int kHotSlots = 512;         // CTA-local hot multimap buckets (generated kernels)
constexpr int kHotProbe = 4;           // probe window in that table
constexpr uint32_t kEmpty32 = 0xffffffffu;

struct DevPipe {
  int64_t nrows;
  const uint64_t* nrows_dev;   // row count produced on the device (temp tables)
  int32_t source_kind;         // dq_source_kind
  int32_t source_res;
  int32_t tile;                // rows per tile (multiple of 16)
  int32_t nstage;
  int32_t stage_bytes;
  int32_t exp_cap;             // rows per expansion chunk
  int32_t use_tma;
  int32_t mode;                // 0: tiles, 1: heavy work units
  int32_t clear_src;           // DQ_SRC_AGG: reset every slot read to its initial
                               // state (the table's only scan; the next run then
                               // needs no initialising kernel)
  int32_t ncols;
  DevCol cols[DQ_MAX_COLS];
  int32_t nstr;
  DevStr strs[kMaxStr];
  int32_t nslots;
  DevSlot slots[DQ_MAX_SLOTS];
  int32_t nops;
  dq_op ops[DQ_MAX_OPS];
  int16_t lists[DQ_MAX_LIST];
  int32_t nres;
  DevRes res[kMaxRes];
  const uint8_t* patterns;     // concatenated LIKE patterns / string constants
  int32_t pat_off[DQ_MAX_PATTERNS + 1];
  DevHeavy heavy;
  // shared-memory layout (bytes)
  int32_t off_stage;
  int32_t off_reg[DQ_MAX_LEVELS];
  int32_t off_sel[DQ_MAX_LEVELS];
  int32_t off_par[DQ_MAX_LEVELS];
  int32_t off_match[DQ_MAX_LEVELS];
  int32_t off_exp;             // expansion bookkeeping (off, cnt, pos) per parent level
  int32_t off_flags;           // per-row probe results
  int32_t off_stash;
  int32_t smem_bytes;
  const DevStr* strsrc;        // the plan's string sources (string references)
  int32_t nstrsrc;
  int32_t* status;
  uint32_t* tile_counter;      // dynamic tile scheduler; [1]: CTAs done (fused tail)
  uint64_t* scratch_ll;        // misc device counters
  uint64_t* profile;           // lane-activity histograms, 33 bins a profile point
};

// ---------------------------------------------------------------- batches --
// A batch runs many instances of one plan shape: these descriptors let one
// launch reset, scan or pack the per-instance buffers of all instances.

constexpr uint64_t kResetChunk = 8192;  // 64-bit words one CTA resets at a time

struct BatchReset {       // one buffer to reset before a run (8-byte aligned)
  void* ptr;
  uint64_t n;             // 64-bit words
  uint64_t value;         // kind 0
  uint64_t reds;          // kind 1: 4 bits of dq_red_kind per aggregate
  uint64_t chunk0;        // its first chunk of kResetChunk words among all buffers'
  int32_t kind;           // 0: fill u64, 1: aggregation table
  int32_t words;          // kind 1: words per slot
  int32_t val_word;       // kind 1: first accumulator word
  int32_t naggs;          // kind 1
};

// The buffers a plan's run starts by resetting, as a kernel parameter.
constexpr int kMaxResets = 48;
struct ResetList {
  int32_t n;
  int32_t pad;
  uint64_t chunks;
  BatchReset op[kMaxResets];
};

// A run's status word, row count and result columns in pinned host memory:
// the header, then a region per column.  A column that does not fit its region
// (more rows, longer strings) is copied by the host after the run.
constexpr uint64_t kPackBytes = 32768;  // bytes a column's region holds at most
constexpr uint32_t kPackRows = 2048;    // rows of a string column at most
constexpr int kPackHeader = 256;        // int32 status, uint64 rows at 8, uint64 heap
                                        // bytes of string column j at 16 + 8 j (~0: too large)

struct ResultPackCol {
  const uint8_t* src;
  uint64_t off;           // its region's offset (strings: the offsets, then kPackBytes of heap)
  uint64_t bytes;         // a fixed-width region's size
  int32_t width;          // 0: string references
  int32_t heap_off;       // strings: the heap's offset in the region
};

constexpr int kMaxPackStats = 8;
struct ResultPack {
  const int32_t* status;
  const uint64_t* cursor;
  uint64_t cap;
  const DevStr* strsrc;
  uint8_t* out;
  int32_t ncols;
  int32_t nstats;         // pairs of counters copied beside the result (deferred items)
  const uint32_t* stat_src[kMaxPackStats];
  uint32_t* stat_dst[kMaxPackStats];
  ResultPackCol c[DQ_MAX_PAY];
};

struct BatchScanSeg {     // one multimap's bucket counts -> offsets
  uint32_t* counts;
  uint64_t* ranges;
  uint64_t n;             // buckets
  uint64_t pay_rows;      // payload rows there is room for
  int32_t* status;
  uint64_t block0;        // first scan block of this segment
  uint64_t nblocks;
  int32_t ranked;         // the counts stay (a ranked multimap's scatter needs none)
  int32_t pad;
};

struct BatchPack {        // one output column of one instance
  const uint8_t* src;
  const uint64_t* cursor; // rows emitted (may exceed cap on overflow)
  uint64_t cap;
  uint64_t dst;           // byte offset in the packed buffer
  uint64_t* rows_out;     // where the kernel records min(cursor, cap)
  int32_t width;
  int32_t pad;
};

// ------------------------------------------------------------ text import --
constexpr int kImpTile = 16384;       // text bytes per CTA in the newline passes (64 a thread)
constexpr int kImpRows = 256;         // rows per CTA in the parse and string passes
constexpr int kImpMaxFields = 64;

// Field kinds (dq_text_kind) and the reasons a row is rejected.
enum : int32_t { kTxtInt = 1, kTxtDate = 2, kTxtChar = 3, kTxtDecimal = 4, kTxtString = 5, kTxtSkip = 6,
                 kTxtFloat = 7 };
enum : int32_t { kImpTooFew = 1, kImpTooMany = 2, kImpNoDigit = 3, kImpOverflow = 4, kImpNotChar = 5,
                 kImpShortDate = 6, kImpExponent = 7 };

struct ImpField {
  int32_t kind;
  int32_t scale;          // decimal digits kept after the point
  void* out;              // fixed-width column (nrows values)
  int32_t str;            // string ordinal (kTxtString)
  int32_t pad;
};

// The text as whole tiles: bytes [0, nmain) at `main`, the rest (one
// zero-padded tile at most) at `tail`.
struct ImpText {
  const uint8_t* main;
  const uint8_t* tail;
  uint64_t nmain;         // a multiple of kImpTile
};

struct ImpArgs {
  ImpText text;
  uint64_t nbytes;
  uint64_t nlines;        // newlines in the text
  uint64_t nrows;         // nlines, plus one for a last line without a newline
  const uint64_t* line_end;
  uint64_t* err;          // min over bad rows of row << 16 | field << 8 | reason
  uint64_t* spos;         // [nstr][nrows] first byte of each string
  uint32_t* slen;         // [nstr][nrows] its length
  uint64_t* bsum;         // [nstr][nblocks + 1] string bytes per parse block
  uint64_t* boff;         // the same, exclusive prefix sums (total last)
  uint64_t nblocks;
  int32_t nfields;
  int32_t nstr;
  uint32_t delim;
  int32_t pad;
  ImpField f[kImpMaxFields];
  uint64_t* soff[kImpMaxFields];  // string offsets (nrows + 1), by string ordinal
  uint8_t* sheap[kImpMaxFields];  // string heaps
};

}  // namespace dq
