// fm_merge.cu -- bulk insert of calls that are large beside their table, as
// one merge of the new records into the table, for tables without tombstones.
//
// On a table without tombstones (nothing removed since it was cleared) the
// Robin Hood order holds: the entries of a run of OCCUPIED slots are sorted
// by home, a key is stored at most once, and an insert of a key that is not
// stored (home g) appends it to g's entries and moves the first entry of
// every following group of equal homes to that group's end, up to the first
// EMPTY slot, which becomes OCCUPIED (the walk of src/rayon_cpu.rs:153-264:
// an eviction where depth > stored distance, so each group's first entry is
// evicted and passes the rest of its group).  So what a whole call does to
// the table has a closed form; nothing has to be moved op by op:
//
//  * An op whose key is stored before the call stays an update whatever the
//    call's other ops do, and an update moves nothing: the last op on each
//    key writes its value, first.
//  * Of several ops with one new key, the first inserts and the last gives
//    the value.
//  * The new keys as ops in index order: op j fills the first EMPTY slot F_j
//    at or after its home.  Left to right, an EMPTY slot takes the lowest op
//    index of those that came from the left or start there and have found no
//    slot yet (the ops carried to it), so the number of ops carried across a
//    slot boundary is c(s + 1) = max(0, c(s) + new(s) - empty(s)).
//  * The group of home h starts c(h) slots further right after the call, and
//    each op carried across h turns its entries by one (first to last) if it
//    has any at that time.  With a_1 < .. < a_k the new ops of home h, r_t of
//    the carried ones before a_t in index order: turn the m old entries r_1
//    times, append a_1, turn the m + 1 by r_2 - r_1, ... and at the end by
//    c(h) - r_k.
//
// Passes (all over memory once; n ops, C slots):
//   find     (a thread per op)   the stored slot or a place on its home's list
//   resolve  (a thread per op)   updates written; each home's list in index
//                                order without repeats
//   fn, carry, slots             c at every slot (a scan of the functions
//                                c -> max(a, c + b), MG_CHUNK slots a block)
//   rank     (a thread per op)   each new op's rank among the ops carried
//                                across its home (homes of several new ops)
//   new      (a thread per op)   where each new op goes:
//   old      (a thread per slot) where the stored entries go:
//                                seg_min[dest] = source
//   move     (a block per chunk) the records, once each, right to left between
//                                two slots with c = 0 (entries move only right)
// A call that outgrows a bound here (a home with too many ops or entries, a
// walk too long, no slot left EMPTY) is left to the other insert paths
// (Ctl::serial[0]) before any record moves; the updates already written are
// the ones those paths will write again.
//
// Bound by memory: the table's metadata is read about four times and each
// record that moves is read and written once.
#include <atomic>
#include <type_traits>

#include "fm_rounds.cuh"
#include "fm_probe.cuh"

namespace fm {
namespace {

constexpr uint32_t MG_LIST = 32;      // ops of one home a thread puts in order
constexpr uint32_t MG_GROUP = 64;     // stored entries of one home on either side of one of them
constexpr uint32_t MG_WALK = 1u << 14;  // slots a rank's walk looks back over
constexpr uint32_t MG_EMPTY = 0x80000000u, MG_FRESH = 0x40000000u, MG_COUNT = 0x3FFFFFFFu;  // carry words
constexpr uint32_t MG_SRC_OP = 0x80000000u;  // seg_min[dest]: the source is a new op,
constexpr uint32_t MG_SRC_VAL = 0x40000000u; //   with another op's value
constexpr uint32_t MG_MANY = 0x80000000u;    // seg_cnt[home]: the list has more than one op
constexpr uint64_t MG_UPDATE = 1ull << 63;   // op_slot: an update of that slot
constexpr int MG_THREADS = 256;

// Per new op (op_pt, four words): the op giving its value, its rank among the
// ops carried across its home, the number of ops on its home's list (first
// op of the list only), the next op of the list.  seg_cnt[home] heads a list
// (op + 1), with MG_MANY where it has several ops: the passes over the slots
// read the list only there.
struct __align__(16) MgOp {
    uint32_t val, rank, count, next;
};
__device__ __forceinline__ MgOp* mg_ops(const OpScratch& sc) { return reinterpret_cast<MgOp*>(sc.op_pt); }

__device__ __forceinline__ bool mg_left(const Ctl* ctl) { return *(volatile const uint32_t*)&ctl->serial[0] != 0; }

// For the kernels of a call: left, not for this path (tombstones; a call whose
// history the host does not know), or empty.
__device__ __forceinline__ uint32_t mg_n0(uint32_t n0, const Ctl* ctl) {
    return n0 != CMP_N0_CTL ? n0 : *(volatile const uint32_t*)&ctl->n0;
}
__device__ __forceinline__ bool mg_skip(uint32_t n0, const Ctl* ctl) {
    return mg_left(ctl) || *(volatile const uint32_t*)&ctl->tomb_claimed != 0 || mg_n0(n0, ctl) == 0;
}

// The passes are written for a crew of `step` threads of which this is number
// `me`: the grid, or the one block of k_mg_small.
template <int KB, bool RO>
__device__ __forceinline__ void mg_find(const TableView& t, const uint8_t* __restrict__ keys, uint32_t n0,
                                        const OpScratch& sc, uint32_t me, uint32_t step) {
    MgOp* ops = mg_ops(sc);
    for (uint32_t j = me; j < n0; j += step) {
        RegKey<KB> key;
        const uint64_t h = home_of<KB>(t, keys, j, key);
        const uint64_t x = get_probe_key<KB, RO>(t, key, h);
        if (x != NONE64) {
            sc.op_slot[j] = x | MG_UPDATE;
            sc.op_flag[j] = 0;
            atomicMin(&t.seg_min[x], upd_code(j));
        } else {
            sc.op_slot[j] = h;
            const uint32_t before = atomicExch(&t.seg_cnt[h], j + 1u);  // 0: an empty list
            ops[j].next = before ? before - 1u : IDLE;
            sc.op_flag[j] = before ? 0 : 1;  // the first op of a list puts it in order
            if (before) atomicOr(&sc.pend[0][(before - 1u) >> 5], 1u << ((before - 1u) & 31u));  // it is not alone
        }
    }
}

// Updates: the last op on each stored key writes its value.  Lists: the first
// op of each home's list sorts it, drops repeats of a key (the first op
// inserts, the last one's value counts), links the rest in index order.
// Returns the new keys this thread counted.
template <int KB, int VB>
__device__ __forceinline__ uint32_t mg_resolve(const TableView& t, const uint8_t* __restrict__ keys,
                                               const uint8_t* __restrict__ vals, uint32_t n0, const OpScratch& sc,
                                               Ctl* ctl, uint32_t me, uint32_t step) {
    MgOp* ops = mg_ops(sc);
    uint32_t fresh = 0;
    const uint32_t iters = (n0 + step - 1) / step;
    for (uint32_t it = 0; it < iters; it++) {  // warp-uniform trip count
        const uint32_t j = me + it * step;
        const uint8_t* src = nullptr;
        uint8_t* dst = nullptr;
        if (j < n0) {
            const uint64_t at = sc.op_slot[j];
            if (at & MG_UPDATE) {
                const uint64_t x = at & ~MG_UPDATE;
                if (t.seg_min[x] == upd_code(j)) {  // the others find another op's word, or idle
                    src = vals + (uint64_t)j * VB;
                    dst = t.vals + x * VB;
                    t.seg_min[x] = IDLE;
                }
            } else if (sc.op_flag[j]) {
                if (!(sc.pend[0][j >> 5] >> (j & 31u) & 1u)) {  // alone
                    ops[j] = MgOp{j, 0u, 1u, IDLE};
                    ++fresh;
                } else {
                    const uint32_t head = t.seg_cnt[at] - 1u;
                    uint32_t list[MG_LIST], val[MG_LIST];
                    uint32_t c = 0, x = head;
                    bool over = false;
                    while (x != IDLE) {
                        if (c == MG_LIST) {
                            over = true;
                            break;
                        }
                        uint32_t k = c++;
                        while (k > 0 && list[k - 1] > x) {
                            list[k] = list[k - 1];
                            --k;
                        }
                        list[k] = x;
                        x = ops[x].next;
                    }
                    if (over) {
                        ctl->serial[0] = 1u;
                    } else {
                        uint32_t u = 0;  // distinct keys so far, list[0..u)
                        for (uint32_t q = 0; q < c; q++) {
                            const uint32_t y = list[q];
                            RegKey<KB> key, other;
                            key.load(keys + (uint64_t)y * KB, KB);
                            uint32_t m = 0;
                            for (; m < u; m++) {
                                other.load(keys + (uint64_t)list[m] * KB, KB);
                                if (key.same(other)) break;
                            }
                            if (m < u) {
                                val[m] = y;  // a repeat
                                sc.op_slot[y] = NONE64 & ~MG_UPDATE;
                            } else {
                                list[u] = y;
                                val[u++] = y;
                            }
                        }
                        for (uint32_t q = 0; q < u; q++)
                            ops[list[q]] = MgOp{val[q], 0u, q == 0 ? u : 0u, q + 1 < u ? list[q + 1] : IDLE};
                        t.seg_cnt[at] = (list[0] + 1u) | (u > 1 ? MG_MANY : 0u);
                        fresh += u;
                    }
                }
            }
        }
        warp_copy_values<VB>(src, dst);
    }
    return fresh;
}

// c -> max(a, c + b) for c >= 0, a >= 0: what a stretch of slots makes of the
// ops carried to it.
struct MgFn {
    int a, b;
};
__device__ __forceinline__ MgFn then(const MgFn& f, const MgFn& g) {
    return MgFn{max(g.a, f.a + g.b), f.b + g.b};
}
__device__ __forceinline__ MgFn slot_fn(MgFn f, int fresh, bool empty) {
    const int d = fresh - (empty ? 1 : 0);
    f.b += d;
    f.a = max(0, f.a + d);
    return f;
}

__device__ __forceinline__ int fresh_of(const OpScratch& sc, uint32_t w) {
    return w & MG_MANY ? (int)mg_ops(sc)[(w & ~MG_MANY) - 1u].count : (w ? 1 : 0);
}
// The first op of a list.
__device__ __forceinline__ uint32_t first_of(uint32_t w) { return (w & ~MG_MANY) - 1u; }  // none: IDLE

__device__ __forceinline__ MgFn warp_scan_fn(MgFn f) {  // inclusive
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        MgFn o;
        o.a = __shfl_up_sync(0xFFFFFFFFu, f.a, d);
        o.b = __shfl_up_sync(0xFFFFFFFFu, f.b, d);
        if ((int)lane >= d) f = then(o, f);
    }
    return f;
}

// Four consecutive slots' metadata and new ops: their function and, per slot,
// the new ops and whether it is EMPTY.
struct MgQuad {
    uint32_t fresh[4];
    bool empty[4];
    MgFn f;
    __device__ __forceinline__ void load(const TableView& t, const OpScratch& sc, uint64_t s0) {
        const uint4 fl = *reinterpret_cast<const uint4*>(t.flags + s0);
        const uint4 nw = *reinterpret_cast<const uint4*>(t.seg_cnt + s0);
        const uint32_t f4[4] = {fl.x, fl.y, fl.z, fl.w}, n4[4] = {nw.x, nw.y, nw.z, nw.w};
        f = MgFn{0, 0};
#pragma unroll
        for (int l = 0; l < 4; l++) {
            fresh[l] = fresh_of(sc, n4[l]);
            empty[l] = is_free(f4[l]);
            f = slot_fn(f, (int)fresh[l], empty[l]);
        }
    }
    // The carry words, with c at the first of the slots.
    __device__ __forceinline__ void store(uint32_t* carry, uint64_t s0, int c) const {
        uint32_t w[4];
#pragma unroll
        for (int l = 0; l < 4; l++) {
            w[l] = (uint32_t)c | (empty[l] ? MG_EMPTY : 0u) | (fresh[l] ? MG_FRESH : 0u);
            c = max(0, c + (int)fresh[l] - (empty[l] ? 1 : 0));
        }
        *reinterpret_cast<uint4*>(carry + s0) = make_uint4(w[0], w[1], w[2], w[3]);
    }
};

// Exclusive composition over the block's threads (MG_THREADS), and the whole.
__device__ __forceinline__ MgFn block_scan_fn(MgFn f, MgFn* s_w, MgFn& total) {
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const MgFn inc = warp_scan_fn(f);
    if (lane == 31) s_w[w] = inc;
    __syncthreads();
    if (w == 0) {
        const MgFn v = warp_scan_fn(lane < nw ? s_w[lane] : MgFn{0, 0});
        s_w[lane] = v;
    }
    __syncthreads();
    MgFn ex;  // the threads before this one
    ex.a = __shfl_up_sync(0xFFFFFFFFu, inc.a, 1);
    ex.b = __shfl_up_sync(0xFFFFFFFFu, inc.b, 1);
    if (lane == 0) ex = MgFn{0, 0};
    if (w > 0) ex = then(s_w[w - 1], ex);
    total = s_w[31];
    __syncthreads();
    return ex;
}

// The function of every chunk: a block per chunk, four slots a thread.
__global__ void __launch_bounds__(MG_THREADS) k_mg_fn(TableView t, uint32_t n0, OpScratch sc, const Ctl* ctl,
                                                      int2* fn) {
    __shared__ MgFn s_w[32];
    if (mg_skip(n0, ctl)) return;
    MgQuad q;
    q.load(t, sc, (uint64_t)blockIdx.x * MG_CHUNK + threadIdx.x * 4);
    MgFn total;
    block_scan_fn(q.f, s_w, total);
    if (threadIdx.x == 0) fn[blockIdx.x] = make_int2(total.a, total.b);
}

// c at the start of every chunk (one block; the table is a ring: with fewer
// new records than EMPTY slots the ring's function has the fixed point a).
__global__ void __launch_bounds__(1024) k_mg_carry(uint64_t mask, uint32_t n0, Ctl* ctl, const int2* __restrict__ fn,
                                                   uint32_t* __restrict__ cin) {
    __shared__ MgFn s_w[32];
    if (mg_skip(n0, ctl)) return;  // block-uniform
    const uint64_t nch = (mask + 1) / MG_CHUNK;
    const uint64_t per = (nch + blockDim.x - 1) / blockDim.x;
    const uint64_t b0 = threadIdx.x * per, b1 = min(nch, b0 + per);
    MgFn f{0, 0}, total;
    for (uint64_t i = b0; i < b1; i++) {
        const int2 x = fn[i];
        f = then(f, MgFn{x.x, x.y});
    }
    const MgFn ex = block_scan_fn(f, s_w, total);
    if (total.b >= 0) {  // no slot stays EMPTY: not for this path
        if (threadIdx.x == 0) ctl->serial[0] = 1u;
        return;
    }
    int c = max(ex.a, total.a + ex.b);
    for (uint64_t i = b0; i < b1; i++) {
        cin[i] = (uint32_t)c;
        const int2 x = fn[i];
        c = max(x.x, c + x.y);
    }
}

// c at every slot (a block per chunk), with what a walk over the slots needs
// beside it: carry[s] = c(s) | MG_EMPTY | MG_FRESH (new ops start at s).
__global__ void __launch_bounds__(MG_THREADS) k_mg_slots(TableView t, uint32_t n0, OpScratch sc, const Ctl* ctl,
                                                         const uint32_t* __restrict__ cin,
                                                         uint32_t* carry) {
    __shared__ MgFn s_w[32];
    if (mg_skip(n0, ctl)) return;
    const uint64_t s0 = (uint64_t)blockIdx.x * MG_CHUNK + threadIdx.x * 4;
    MgQuad q;
    q.load(t, sc, s0);
    MgFn total;
    const MgFn ex = block_scan_fn(q.f, s_w, total);
    q.store(carry, s0, max(ex.a, (int)cin[blockIdx.x] + ex.b));
}

// The rank of op a among the ops carried across its home h: the ops before a
// in index order find their slots as if a and the ops after it were not
// there, so it is the c(h) of those ops alone, the largest sum over [s, h) of
// (their number starting at a slot - 1 if it is EMPTY) for any s, or 0.  The
// walk left ends where no op of the call is carried (c = 0), or once the sum
// has reached c(h).  A thread per op; no order between ops is needed.
__device__ __forceinline__ uint32_t mg_rank(const TableView& t, const MgOp* ops, const uint32_t* carry,
                                            uint32_t a, uint64_t h, uint32_t ch, bool& over) {
    const uint64_t mask = t.mask;
    int sum = 0, best = 0;
    uint64_t p = h + mask + 1;  // slots [p, h) are in the sum, unwrapped
    for (uint32_t step = 0; step < MG_WALK; step += 8) {
        // the eight slots that end at or behind p, with the lists that start there
        const uint64_t b = (p - 1) & ~7ull;
        const uint4* cp = reinterpret_cast<const uint4*>(carry + (b & mask));
        const uint4* lp = reinterpret_cast<const uint4*>(t.seg_cnt + (b & mask));
        const uint4 c0 = cp[0], c1 = cp[1], l0 = lp[0], l1 = lp[1];
        const uint32_t w8[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
        const uint32_t n8[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
#pragma unroll
        for (int l = 7; l >= 0; l--) {
            if (b + l >= p) continue;
            const uint32_t w = w8[l];
            if (w & MG_EMPTY) --sum;
            if (w & MG_FRESH) {
                uint32_t x = first_of(n8[l]);
                if (!(n8[l] & MG_MANY)) sum += x < a ? 1 : 0;
                else
                    for (; x < a; x = ops[x].next) ++sum;  // IDLE ends it
            }
            best = max(best, sum);
            if ((w & MG_COUNT) == 0 || best == (int)ch) return (uint32_t)best;
        }
        p = b;
    }
    over = true;
    return 0;
}

// An op that is the only one of its home's list.
__device__ __forceinline__ bool mg_one(const MgOp& op) { return op.count == 1u && op.next == IDLE; }

// The ranks of the ops that share a home with others of the call.
__device__ __forceinline__ void mg_ranks(const TableView& t, uint32_t n0, const OpScratch& sc, Ctl* ctl,
                                         const uint32_t* carry, uint32_t me, uint32_t step) {
    MgOp* ops = mg_ops(sc);
    bool over = false;
    for (uint32_t j = me; j < n0; j += step) {
        const uint64_t h = sc.op_slot[j];
        if (h > t.mask || mg_one(ops[j])) continue;  // an update, a repeat, or for mg_new
        const uint32_t c = carry[h] & MG_COUNT;
        if (c) ops[j].rank = mg_rank(t, ops, carry, j, h, c, over);
    }
    if (over) ctl->serial[0] = 1u;
}

// Where entry `pos` of a group of m stored entries, c ops carried across its
// home, ends up in the group; for a new op (mine != IDLE) its own place.
__device__ __forceinline__ uint32_t turned(const MgOp* ops, uint32_t head, uint32_t pos, uint32_t m, uint32_t c,
                                           uint32_t mine) {
    uint32_t size = m, seen = 0;
    bool in = mine == IDLE;
    for (uint32_t a = head; a != IDLE; a = ops[a].next) {
        const uint32_t r = ops[a].rank - seen;
        if (in && size) pos = (pos + size - r % size) % size;
        seen = ops[a].rank;
        if (a == mine) {
            in = true;
            pos = size;
        }
        ++size;
    }
    const uint32_t r = c - seen;
    return (pos + size - r % size) % size;
}

// Where every stored entry goes (seg_min[destination] = its slot); those that
// stay are left out.
__device__ __forceinline__ void mg_old(const TableView& t, const OpScratch& sc, Ctl* ctl,
                                       const uint32_t* carry, uint64_t x) {
    const uint64_t mask = t.mask;
    // what is carried across its home is carried on over every slot up to it
    if ((carry[x] & MG_COUNT) == 0) return;
    const uint32_t f = t.flags[x];
    if (st_of(f) != ST_OCC) return;
    const uint32_t d = (uint32_t)dist_of(f);
    const uint64_t h = (x - d) & mask;
    const uint32_t c = carry[h] & MG_COUNT;
    if (c == 0) return;
    uint32_t i = 0, m = 1;
    while (i < d && i < MG_GROUP) {  // entries of this home before it: distances count down
        const uint32_t g = t.flags[(x - i - 1) & mask];
        if (g != mk_flag(ST_OCC, d - i - 1)) break;
        ++i;
    }
    while (m < MG_GROUP && t.flags[(x + m) & mask] == mk_flag(ST_OCC, d + m)) ++m;
    if (i == MG_GROUP || m == MG_GROUP) {
        ctl->serial[0] = 1u;
        return;
    }
    const uint32_t w = t.seg_cnt[h];
    const uint32_t to = turned(mg_ops(sc), first_of(w), i, i + m, c, IDLE);
    const uint64_t dst = (x - i + c + to) & mask;
    if (dst != x) t.seg_min[dst] = (uint32_t)x;
}

// Where every new op goes, and the rank of an op that is alone on its home's
// list (which the entries stored there turn by; with none stored it does not
// matter).
__device__ __forceinline__ void mg_new(const TableView& t, uint32_t n0, const OpScratch& sc, Ctl* ctl,
                                       const uint32_t* carry, uint32_t me, uint32_t step) {
    const uint64_t mask = t.mask;
    MgOp* ops = mg_ops(sc);
    bool over = false;
    for (uint32_t j = me; j < n0; j += step) {
        const uint64_t h = sc.op_slot[j];
        if (h > mask) continue;  // an update or a repeat
        const uint32_t cw = carry[h];
        const uint32_t c = cw & MG_COUNT;
        MgOp op = ops[j];
        const uint32_t code = j | MG_SRC_OP | (op.val != j ? MG_SRC_VAL : 0u);
        const bool one = mg_one(op);
        if (one && c == 0 && (cw & MG_EMPTY)) {
            t.seg_min[h] = code;
            continue;
        }
        // the slots of this home's entries: behind those of lower homes, which
        // fill [h, s)
        uint32_t p = 0, m = 0;
        bool go = true;
        for (uint64_t wb = h & ~7ull; go; wb += 8) {
            const uint4* fp = reinterpret_cast<const uint4*>(t.flags + (wb & mask));
            const uint4 a = fp[0], b = fp[1];
            const uint32_t f8[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int l = 0; l < 8; l++) {
                if (!go || wb + l < h) continue;
                const uint32_t f = f8[l];
                if (st_of(f) != ST_OCC || dist_of(f) < p) {
                    go = false;
                } else {
                    m += dist_of(f) == p ? 1u : 0u;
                    ++p;
                }
            }
        }
        uint32_t to = 0;
        if (!one) {
            to = turned(ops, first_of(t.seg_cnt[h]), 0, m, c, j);
        } else if (m) {  // at the end of the m, then turned by those carried across after it
            if (c) {
                op.rank = mg_rank(t, ops, carry, j, h, c, over);
                ops[j].rank = op.rank;
            }
            to = m - (c - op.rank) % (m + 1);
        }
        t.seg_min[(h + p - m + c + to) & mask] = code;
    }
    if (over) ctl->serial[0] = 1u;
}

// The moves of the slots from the first one with c = 0 at or after lo to the
// first one at or after hi, by one block of NT threads: no entry crosses those
// two.  The
// destinations are listed highest first, MG_TILE slots at a time from the
// right; a batch loads all its records before it stores any, and a source
// lies at or left of its destination, so no record is overwritten before it
// is read.  Leaves seg_min and seg_cnt idle.
template <int NT>
struct MgMoveSmem {
    uint32_t dst[MG_MOVE_CHUNK], src[MG_MOVE_CHUNK];
    uint32_t woff[NT / 32];
    unsigned long long edge[2];
};
template <int KB, int VB, int NT>
__device__ __forceinline__ void mg_move(const TableView& t, const uint8_t* __restrict__ keys,
                                        const uint8_t* __restrict__ vals, const OpScratch& sc, Ctl* ctl,
                                        const uint32_t* carry, uint64_t lo, uint64_t hi,
                                        MgMoveSmem<NT>& sm) {
    constexpr int CK = (KB % 16 == 0 && VB % 16 == 0) ? 16 : 8;  // bytes of a piece
    using Ch = typename std::conditional<CK == 16, uint4, uint2>::type;
    constexpr int NK = KB / CK, NP = (KB + VB) / CK;  // pieces of a record
    constexpr int PER = 5;                            // pieces a thread holds
    constexpr int BATCH = PER * NT / NP < NT ? PER * NT / NP : NT;  // records at once
    constexpr uint32_t TILE = MG_MOVE_CHUNK;
    constexpr int SPT = TILE / NT;                    // slots of a tile per thread
    const uint64_t mask = t.mask;
    const MgOp* ops = mg_ops(sc);
    // the two edges: the first slot with c = 0 from lo and from hi on
    for (int side = 0; side < 2; side++) {
        if (threadIdx.x == 0) sm.edge[side] = NONE64;
        __syncthreads();
        for (uint64_t b = side ? hi : lo;; b += NT) {
            const uint64_t s = b + threadIdx.x;
            if ((carry[s & mask] & MG_COUNT) == 0) atomicMin(&sm.edge[side], (unsigned long long)s);
            __syncthreads();
            const bool got = sm.edge[side] != NONE64;
            __syncthreads();
            if (got || b - lo > 2 * mask) break;
        }
    }
    const uint64_t p0 = sm.edge[0], p1 = sm.edge[1];
    uint32_t md = 0;
    if (p0 < p1 && p1 != NONE64) {
        const uint64_t ntile = (p1 - p0 + TILE - 1) / TILE;
        for (uint64_t k = ntile; k-- > 0;) {
            const uint64_t a = p0 + k * TILE;
            const uint64_t z = min(a + TILE, p1);
            // this tile's destinations, highest first
            uint32_t src[SPT], cnt = 0;
#pragma unroll
            for (int q = 0; q < SPT; q++) {
                const uint64_t s = a + TILE - 1 - (threadIdx.x * SPT + q);
                src[q] = IDLE;
                if (s < z) {
                    const uint64_t sl = s & mask;
                    src[q] = t.seg_min[sl];
                    if (src[q] != IDLE) {
                        t.seg_min[sl] = IDLE;
                        ++cnt;
                    }
                    if (t.seg_cnt[sl]) t.seg_cnt[sl] = 0u;
                }
            }
            const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
            uint32_t inc = cnt;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, inc, d);
                if ((int)lane >= d) inc += o;
            }
            if (lane == 31) sm.woff[w] = inc;
            __syncthreads();
            uint32_t off = 0, total = 0;
            for (uint32_t i = 0; i < NT / 32; i++) {
                if (i < w) off += sm.woff[i];
                total += sm.woff[i];
            }
            off += inc - cnt;
#pragma unroll
            for (int q = 0; q < SPT; q++) {
                if (src[q] == IDLE) continue;
                sm.dst[off] = (uint32_t)((a + TILE - 1 - (threadIdx.x * SPT + q)) & mask);
                sm.src[off++] = src[q];
            }
            __syncthreads();
            for (uint32_t b = 0; b < total; b += BATCH) {
                const uint32_t nb = min((uint32_t)BATCH, total - b);
                Ch buf[PER];
                uint32_t flag = 0;
#pragma unroll
                for (int u = 0; u < PER; u++) {
                    const uint32_t g = threadIdx.x + u * NT;
                    if (g >= nb * NP) continue;
                    const uint32_t s = sm.src[b + g / NP], c = g % NP;
                    const uint8_t* from;
                    if (s & MG_SRC_OP) {
                        const uint32_t j = s & ~(MG_SRC_OP | MG_SRC_VAL);
                        from = c < (uint32_t)NK
                                   ? keys + (uint64_t)j * KB + c * CK
                                   : vals + (uint64_t)(s & MG_SRC_VAL ? ops[j].val : j) * VB + (c - NK) * CK;
                    } else {
                        from = c < (uint32_t)NK ? t.keys + (uint64_t)s * KB + c * CK
                                                : t.vals + (uint64_t)s * VB + (c - NK) * CK;
                    }
                    buf[u] = *reinterpret_cast<const Ch*>(from);
                }
                if (threadIdx.x < nb) {
                    const uint32_t s = sm.src[b + threadIdx.x];
                    const uint64_t dst = sm.dst[b + threadIdx.x];
                    uint64_t home;
                    if (s & MG_SRC_OP) {  // from the key, which the move reads anyway
                        RegKey<KB> key;
                        home = home_of<KB>(t, keys, s & ~(MG_SRC_OP | MG_SRC_VAL), key);
                    } else {
                        home = s - dist_of(t.flags[s]);
                    }
                    const uint32_t d = (uint32_t)((dst - home) & mask);
                    flag = mk_flag(ST_OCC, d);
                    md = max(md, d);
                }
                __syncthreads();
#pragma unroll
                for (int u = 0; u < PER; u++) {
                    const uint32_t g = threadIdx.x + u * NT;
                    if (g >= nb * NP) continue;
                    const uint64_t dst = sm.dst[b + g / NP];
                    const uint32_t c = g % NP;
                    uint8_t* to = c < (uint32_t)NK ? t.keys + dst * KB + c * CK : t.vals + dst * VB + (c - NK) * CK;
                    *reinterpret_cast<Ch*>(to) = buf[u];
                }
                if (threadIdx.x < nb) t.flags[sm.dst[b + threadIdx.x]] = flag;
                __syncthreads();
            }
        }
    }
    md = __reduce_max_sync(0xFFFFFFFFu, md);
    if ((threadIdx.x & 31u) == 0 && md > *(volatile uint32_t*)&ctl->dmax) atomicMax(&ctl->dmax, md);
}

template <int KB>
__global__ void __launch_bounds__(MG_THREADS) k_mg_find(TableView t, const uint8_t* __restrict__ keys, uint32_t n0,
                                                        OpScratch sc, Ctl* ctl) {
    if (mg_skip(n0, ctl)) {
        // a call that the host sent here for a table with tombstones: left
        if (n0 != CMP_N0_CTL && blockIdx.x == 0 && threadIdx.x == 0) ctl->serial[0] = 1u;
        return;
    }
    mg_find<KB, true>(t, keys, mg_n0(n0, ctl), sc, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

template <int KB, int VB>
__global__ void __launch_bounds__(MG_THREADS) k_mg_resolve(TableView t, const uint8_t* __restrict__ keys,
                                                           const uint8_t* __restrict__ vals, uint32_t n0,
                                                           OpScratch sc, Ctl* ctl) {
    __shared__ uint32_t s_tmp[MG_THREADS / 32];
    // (serial[0] is set in this kernel: not a reason to leave it)
    if (*(volatile const uint32_t*)&ctl->tomb_claimed != 0) return;
    const uint32_t fresh = mg_resolve<KB, VB>(t, keys, vals, mg_n0(n0, ctl), sc, ctl,
                                              blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
    block_add_count(ctl, fresh, s_tmp);
}

__global__ void __launch_bounds__(MG_THREADS) k_mg_rank(TableView t, uint32_t n0, OpScratch sc, Ctl* ctl,
                                                        const uint32_t* carry) {
    if (mg_skip(n0, ctl)) return;
    mg_ranks(t, mg_n0(n0, ctl), sc, ctl, carry, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

__global__ void __launch_bounds__(MG_THREADS) k_mg_old(TableView t, uint32_t n0, OpScratch sc, Ctl* ctl,
                                                       const uint32_t* carry) {
    if (mg_skip(n0, ctl)) return;
    mg_old(t, sc, ctl, carry, (uint64_t)blockIdx.x * blockDim.x + threadIdx.x);  // a thread per slot
}

// (eight blocks per SM: 4M u64 ops into 2^24 slots 250 -> 220 us)
__global__ void __launch_bounds__(MG_THREADS, 8) k_mg_new(TableView t, uint32_t n0, OpScratch sc, Ctl* ctl,
                                                       const uint32_t* carry) {
    if (mg_skip(n0, ctl)) return;
    mg_new(t, mg_n0(n0, ctl), sc, ctl, carry, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

template <int KB, int VB>
__global__ void __launch_bounds__(MG_THREADS) k_mg_move(TableView t, const uint8_t* __restrict__ keys,
                                                        const uint8_t* __restrict__ vals, uint32_t n0, OpScratch sc,
                                                        Ctl* ctl, const uint32_t* carry) {
    __shared__ MgMoveSmem<MG_THREADS> sm;
    if (mg_skip(n0, ctl)) return;
    const uint64_t lo = (uint64_t)blockIdx.x * MG_MOVE_CHUNK;
    mg_move<KB, VB, MG_THREADS>(t, keys, vals, sc, ctl, carry, lo, lo + MG_MOVE_CHUNK, sm);
}

// The call's end, on a block of its own: as the end of k_mg_move, the fence of
// each of its thousands of blocks cost 34 us (2^24 slots).
__global__ void __launch_bounds__(MG_THREADS) k_mg_publish(Ctl* ctl, Ctl* host) { publish_call(ctl, host); }

// After the passes of a call that has no host step: a call that was left has
// its slot words set idle (k_mg_undo), then its flags and count taken back,
// and one that is done has no ops for the passes that follow (k_mg_done).
__global__ void __launch_bounds__(MG_THREADS) k_mg_undo(TableView t, const Ctl* ctl) {
    if (*(volatile const uint32_t*)&ctl->tomb_claimed != 0 || !mg_left(ctl)) return;
    for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x <= t.mask; x += (uint64_t)gridDim.x * blockDim.x)
        t.seg_min[x] = IDLE, t.seg_cnt[x] = 0u;
}
__global__ void __launch_bounds__(32) k_mg_done(Ctl* ctl) {
    if (*(volatile const uint32_t*)&ctl->tomb_claimed != 0) return;
    const bool left = mg_left(ctl);
    __syncwarp();
    if (left) ctl->count_part[threadIdx.x][0] = 0;
    if (threadIdx.x == 0) {
        if (left) ctl->serial[0] = 0;
        else ctl->n0 = 0;
    }
}

// All the passes on one block, for tables of at most MG_SMALL_SLOTS.  Such a
// call is bound by launches and by the latency of each pass's few reads, so
// one launch does it all, with the table's metadata and everything else the
// passes share in shared memory (160 KB at 4096 slots): 1000 account pairs
// into 4096 slots took 37 us on one block over global memory.  The caller's
// pinned control block is written directly (what the host reads of it).
constexpr int MG_SMALL_THREADS = 1024;
struct MgSmall {
    uint64_t op_slot[MG_SMALL_SLOTS];
    MgOp ops[MG_SMALL_SLOTS];
    uint32_t flags[MG_SMALL_SLOTS], seg_min[MG_SMALL_SLOTS], seg_cnt[MG_SMALL_SLOTS], carry[MG_SMALL_SLOTS];
    uint32_t many[MG_SMALL_SLOTS / 32];
    uint8_t op_flag[MG_SMALL_SLOTS];
};
template <int KB, int VB>
__global__ void __launch_bounds__(MG_SMALL_THREADS) k_mg_small(TableView tg, const uint8_t* __restrict__ keys,
                                                               const uint8_t* __restrict__ vals, uint32_t n0,
                                                               Ctl* ctl, Ctl* host) {
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ MgMoveSmem<MG_SMALL_THREADS> sm;
    __shared__ MgFn s_w[32];
    __shared__ uint32_t s_n[MG_SMALL_THREADS / 32];
    __shared__ __align__(16) uint32_t s_ctl[sizeof(Ctl) / 4];
    MgSmall& m = *reinterpret_cast<MgSmall*>(s_dyn);
    Ctl* sctl = reinterpret_cast<Ctl*>(s_ctl);
    const uint32_t me = threadIdx.x, step = MG_SMALL_THREADS, lane = me & 31u;
    const uint32_t cap = (uint32_t)tg.mask + 1u;
    const uint32_t history = ctl->tomb_claimed;
    if (history != 0) {  // block-uniform: a table with tombstones is not for this path
        if (me == 0) host->serial[0] = 1u, host->err = 0, host->tomb_claimed = history;
        return;
    }
    TableView t = tg;
    t.flags = m.flags, t.seg_min = m.seg_min, t.seg_cnt = m.seg_cnt;
    OpScratch sc{};
    sc.op_slot = m.op_slot, sc.op_flag = m.op_flag, sc.op_pt = reinterpret_cast<uint32_t*>(m.ops), sc.pend[0] = m.many;
    if (me < MG_SMALL_SLOTS / 32) m.many[me] = 0;
    for (uint32_t x = me; x < cap / 4; x += step) {
        reinterpret_cast<uint4*>(m.flags)[x] = reinterpret_cast<const uint4*>(tg.flags)[x];
        reinterpret_cast<uint4*>(m.seg_min)[x] = make_uint4(IDLE, IDLE, IDLE, IDLE);
        reinterpret_cast<uint4*>(m.seg_cnt)[x] = make_uint4(0u, 0u, 0u, 0u);
    }
    if (me == 0) sctl->serial[0] = 0, sctl->dmax = ctl->dmax;
    __syncthreads();
    mg_find<KB, false>(t, keys, n0, sc, me, step);
    __syncthreads();
    uint32_t fresh = mg_resolve<KB, VB>(t, keys, vals, n0, sc, sctl, me, step);
    fresh = __reduce_add_sync(0xFFFFFFFFu, fresh);
    if (lane == 0) s_n[me >> 5] = fresh;
    __syncthreads();
    bool left = mg_left(sctl);  // block-uniform, as below: a barrier between the writes and this
    if (!left) {
        const bool mine = me * 4 < cap;  // four slots a thread
        MgQuad q;
        q.f = MgFn{0, 0};
        if (mine) q.load(t, sc, me * 4);
        MgFn total;
        const MgFn ex = block_scan_fn(q.f, s_w, total);
        left = total.b >= 0;  // no slot stays EMPTY
        if (!left) {
            if (mine) q.store(m.carry, me * 4, max(ex.a, total.a + ex.b));
            __syncthreads();
            mg_ranks(t, n0, sc, sctl, m.carry, me, step);
            __syncthreads();
            mg_new(t, n0, sc, sctl, m.carry, me, step);
            __syncthreads();
            for (uint64_t x = me; x < cap; x += step) mg_old(t, sc, sctl, m.carry, x);
            __syncthreads();
            left = mg_left(sctl);
        }
    }
    if (!left) {
        mg_move<KB, VB, MG_SMALL_THREADS>(t, keys, vals, sc, sctl, m.carry, 0, cap, sm);
        __syncthreads();
        for (uint32_t x = me; x < cap / 4; x += step)
            reinterpret_cast<uint4*>(tg.flags)[x] = reinterpret_cast<const uint4*>(m.flags)[x];
    }
    if (me < 32) {
        const uint32_t n = __reduce_add_sync(0xFFFFFFFFu, s_n[lane]);
        if (me == 0) {
            if (!left) ctl->dmax = sctl->dmax;
            host->serial[0] = left ? 1u : 0u;
            host->err = 0;
            host->rounds = 0;
            host->count = left ? 0u : n;
            host->tomb_claimed = history;
            __threadfence_system();
        }
        host->count_part[lane][0] = 0;
    }
}
static_assert(COUNT_PARTS == 32, "a lane per count part");

template <int KB, int VB>
void merge_shape(const TableView& t, const uint8_t* keys, const uint8_t* vals, uint32_t n0, uint32_t nmax,
                 const OpScratch& sc, Ctl* ctl, Ctl* host, cudaStream_t s) {
    const uint64_t cap = t.mask + 1;
    uint32_t* carry = sc.carry;
    int2* fn = reinterpret_cast<int2*>(carry + cap);  // before cin: one chunk's word would put it off 8 bytes
    uint32_t* cin = reinterpret_cast<uint32_t*>(fn + cap / MG_CHUNK);
    const unsigned g = grid_for(nmax, 8);
    const unsigned gc = (unsigned)(cap / MG_CHUNK);
    {
        KtScope kt(KC_INS_FIND, s);
        cudaMemsetAsync(sc.pend[0], 0, ((size_t)nmax + 31) / 32 * 4, s);
        k_mg_find<KB><<<g, MG_THREADS, 0, s>>>(t, keys, n0, sc, ctl);
        k_mg_resolve<KB, VB><<<g, MG_THREADS, 0, s>>>(t, keys, vals, n0, sc, ctl);
    }
    {
        KtScope kt(KC_INS_WALK, s);
        k_mg_fn<<<gc, MG_THREADS, 0, s>>>(t, n0, sc, ctl, fn);
        k_mg_carry<<<1, 1024, 0, s>>>(t.mask, n0, ctl, fn, cin);
        k_mg_slots<<<gc, MG_THREADS, 0, s>>>(t, n0, sc, ctl, cin, carry);
        k_mg_rank<<<g, MG_THREADS, 0, s>>>(t, n0, sc, ctl, carry);
    }
    {
        KtScope kt(KC_INS_EXEC, s);
        k_mg_new<<<g, MG_THREADS, 0, s>>>(t, n0, sc, ctl, carry);
        k_mg_old<<<(unsigned)((cap + MG_THREADS - 1) / MG_THREADS), MG_THREADS, 0, s>>>(t, n0, sc, ctl, carry);
    }
    {
        KtScope kt(KC_INS_LONG, s);
        k_mg_move<KB, VB><<<(unsigned)(cap / MG_MOVE_CHUNK), MG_THREADS, 0, s>>>(t, keys, vals, n0, sc, ctl, carry);
        if (host) k_mg_publish<<<1, MG_THREADS, 0, s>>>(ctl, host);
    }
    count_launches(host ? 10 : 9);
    if (n0 == CMP_N0_CTL) {
        k_mg_undo<<<grid_for(cap, 4), MG_THREADS, 0, s>>>(t, ctl);
        k_mg_done<<<1, 32, 0, s>>>(ctl);
        count_launches(2);
    }
}

template <int KB, int VB>
cudaError_t small_shape(const TableView& t, const uint8_t* keys, const uint8_t* vals, uint32_t n0, Ctl* ctl, Ctl* host,
                        cudaStream_t s) {
    static std::atomic<uint64_t> ready{0};  // devices on which the shared memory size is set, a bit each
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (!(ready.load() >> (dev & 63) & 1u)) {
        e = cudaFuncSetAttribute(k_mg_small<KB, VB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(MgSmall));
        if (e != cudaSuccess) return e;
        if (dev < 64) ready.fetch_or(1ull << dev);
    }
    KtScope kt(KC_INS_EXEC, s);
    k_mg_small<KB, VB><<<1, MG_SMALL_THREADS, sizeof(MgSmall), s>>>(t, keys, vals, n0, ctl, host);
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_ins_small(const TableView& t, Shape sh, const uint8_t* keys, const uint8_t* vals, uint32_t n0,
                             Ctl* ctl, Ctl* host, cudaStream_t s) {
    if (t.mask + 1 < MG_MIN_SLOTS || t.mask + 1 > MG_SMALL_SLOTS || n0 > MG_SMALL_SLOTS) return cudaErrorInvalidValue;
    switch (sh) {
        case SHAPE_8_8: return small_shape<8, 8>(t, keys, vals, n0, ctl, host, s);
        case SHAPE_32_128: return small_shape<32, 128>(t, keys, vals, n0, ctl, host, s);
        case SHAPE_32_64: return small_shape<32, 64>(t, keys, vals, n0, ctl, host, s);
        case SHAPE_32_32: return small_shape<32, 32>(t, keys, vals, n0, ctl, host, s);
        case SHAPE_8_32: return small_shape<8, 32>(t, keys, vals, n0, ctl, host, s);
        default: return cudaErrorInvalidValue;
    }
}

namespace {
cudaError_t merge_any(const TableView& t, Shape sh, const uint8_t* keys, const uint8_t* vals, uint32_t n0, uint32_t nmax,
                      const OpScratch& sc, Ctl* ctl, Ctl* host, cudaStream_t s) {
    if (!sc.carry || t.mask + 1 < MG_MIN_SLOTS || t.mask >= (uint64_t)DIST_MASK || nmax > MG_MAX_OPS)
        return cudaErrorInvalidValue;
    switch (sh) {
        case SHAPE_8_8: merge_shape<8, 8>(t, keys, vals, n0, nmax, sc, ctl, host, s); break;
        case SHAPE_32_128: merge_shape<32, 128>(t, keys, vals, n0, nmax, sc, ctl, host, s); break;
        case SHAPE_32_64: merge_shape<32, 64>(t, keys, vals, n0, nmax, sc, ctl, host, s); break;
        case SHAPE_32_32: merge_shape<32, 32>(t, keys, vals, n0, nmax, sc, ctl, host, s); break;
        case SHAPE_8_32: merge_shape<8, 32>(t, keys, vals, n0, nmax, sc, ctl, host, s); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}
}  // namespace

cudaError_t launch_ins_merge(const TableView& t, Shape sh, const uint8_t* keys, const uint8_t* vals, uint32_t n0,
                             const OpScratch& sc, Ctl* ctl, Ctl* host, cudaStream_t s) {
    return merge_any(t, sh, keys, vals, n0, n0, sc, ctl, host, s);
}

cudaError_t launch_ins_merge_ctl(const TableView& t, Shape sh, const uint8_t* keys, const uint8_t* vals,
                                 uint32_t nmax, const OpScratch& sc, Ctl* ctl, cudaStream_t s) {
    return merge_any(t, sh, keys, vals, CMP_N0_CTL, nmax, sc, ctl, nullptr, s);
}

}  // namespace fm
