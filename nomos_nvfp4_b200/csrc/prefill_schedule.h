// The order in which the prefill kernel's MMA lane takes ring units and issues its products (attn_prefill_kernel.cuh), and
// the order in which the dequant warps fill the ring.  Plain C++ over an `Ops` that does the waiting and issuing, so that
// the same walk runs on the CPU against a recorder that checks every hand-off.
//
// tcgen05.mma instructions of one thread are documented to run in order only among themselves on ONE accumulator and shape.
// A QK product (64 columns of S) overwrites the columns from which an earlier PV product (128 columns of O) reads its
// weights: neither accumulator nor shape is shared, so the walk waits for that PV's commit before it issues the QK.
// With one query tile there are four S buffers and the PV waited for is four tiles back, which costs nothing; with two (two
// buffers each) the other tile's product is issued in between, and what is left of the wait, and the issuing lane's time for
// it, is 3 to 6 % (2048 positions int8 65 -> 68 us).  QK of the second tile issued a step later, behind the first one's next
// PV, covers the wait altogether but holds a K slot meanwhile: 1 to 2 % slower at 2048 keys, 15 % with fp32 queries on
// block-32 caches (three units in the ring), 1 % faster behind 6144 keys.
#pragma once

#ifdef __CUDACC__
#define NOMOS_WALK __device__ __forceinline__
#else
#define NOMOS_WALK inline
#endif

namespace nomos {
namespace pf {

// Unit i of the ring (64 keys x 128 dims of K or of V): K0 K1 V0 K2 V1 ... with KU units per K tile and VU per V tile.
struct RingUnit { int tile, v, c; };
template <int KU, int VU>
NOMOS_WALK RingUnit ring_unit(int i, int n_tiles) {
    const int ahead = n_tiles < 2 ? n_tiles : 2, lead = KU * ahead;
    if (i < lead) return RingUnit{i / KU, 0, i % KU};
    i -= lead;
    const int body = (KU + VU) * (n_tiles - ahead);
    if (i < body) {
        const int q = i / (KU + VU), r = i % (KU + VU);
        return r < VU ? RingUnit{q, 1, r} : RingUnit{q + 2, 0, r - VU};
    }
    i -= body;
    return RingUnit{n_tiles - ahead + i / VU, 1, i % VU};
}

// Key tiles [first, last] of the CTA's n_tiles that a query tile attends (empty: first > last).
struct TileRange { int first, last; };

// S buffers of a query tile; buffer and barrier phase follow the query tile's own count of tiles.
template <int NQ> constexpr int s_buffers() { return 4 / NQ; }

// NQ query tiles.  Ops:
//   bool next_unit(int &slot)                  waits for the next ring unit
//   void release(int slot)                     hands a unit's slots back once all products issued so far are done
//   bool weights(int buf, int parity)          waits for the softmax warps' weights in S buffer buf
//   bool product(int buf, int parity)          waits for the PV product that reads S buffer buf
//   void qk(int g, int buf, int c, int slot), void s_done(int buf)      QK over 128 dims; commit of the tile's QK
//   void pv(int g, int buf, int c, int slot, bool first), void o_done(int buf)
template <int NQ, int KU, int VU, class Ops>
NOMOS_WALK bool walk_products(int n_tiles, const TileRange (&range)[NQ], Ops &op) {
    constexpr int NB = s_buffers<NQ>();
    auto active = [&](int g, int i) { return i >= range[g].first && i <= range[g].last; };
    auto use = [&](int g, int i) { return i - range[g].first; };
    auto buffer = [&](int g, int i) { return NB * g + use(g, i) % NB; };
    auto parity = [&](int g, int i) { return (use(g, i) / NB) & 1; };
    auto buffer_free = [&](int g, int j) { return use(g, j) < NB || op.product(buffer(g, j), parity(g, j) ^ 1); };
    if constexpr (NQ == 2) {
        static_assert(KU == 1 && VU == 1, "a unit per tile");
        auto qk = [&](int g, int j, int slot) {
            if (!active(g, j)) return true;
            if (!buffer_free(g, j)) return false;
            op.qk(g, buffer(g, j), 0, slot);
            op.s_done(buffer(g, j));
            return true;
        };
        auto pv = [&](int g, int i, int slot) {
            if (!active(g, i)) return true;
            if (!op.weights(buffer(g, i), parity(g, i))) return false;
            op.pv(g, buffer(g, i), 0, slot, use(g, i) == 0);
            op.o_done(buffer(g, i));
            return true;
        };
        auto qk_tile = [&](int j) {
            int n;
            if (!op.next_unit(n) || !qk(0, j, n) || !qk(1, j, n)) return false;
            op.release(n);
            return true;
        };
        if (!qk_tile(0) || (n_tiles > 1 && !qk_tile(1))) return false;
        for (int i = 0; i < n_tiles; ++i) {
            int n;
            if (!op.next_unit(n) || !pv(0, i, n) || !pv(1, i, n)) return false;
            op.release(n);
            if (i + 2 < n_tiles && !qk_tile(i + 2)) return false;
        }
    } else {
        static_assert(NQ == 1, "one or two query tiles");
        auto qk_tile = [&](int j) {
            if (!buffer_free(0, j)) return false;
#pragma unroll 1
            for (int c = 0; c < KU; ++c) {
                int n;
                if (!op.next_unit(n)) return false;
                op.qk(0, buffer(0, j), c, n);
                if (c == KU - 1) op.s_done(buffer(0, j));
                op.release(n);
            }
            return true;
        };
        if (!qk_tile(0) || (n_tiles > 1 && !qk_tile(1))) return false;
        for (int i = 0; i < n_tiles; ++i) {
            if (!op.weights(buffer(0, i), parity(0, i))) return false;
#pragma unroll 1
            for (int c = 0; c < VU; ++c) {
                int n;
                if (!op.next_unit(n)) return false;
                op.pv(0, buffer(0, i), c, n, i == 0);
                op.release(n);
            }
            op.o_done(buffer(0, i));
            if (i + 2 < n_tiles && !qk_tile(i + 2)) return false;
        }
    }
    return true;
}

}  // namespace pf
}  // namespace nomos
