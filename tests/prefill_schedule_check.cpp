// Walks the prefill kernel's product order (csrc/prefill_schedule.h) against a recorder that checks every hand-off: prints
// the first violation and returns 1, or the number of walks.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../nomos_nvfp4_b200/csrc/prefill_schedule.h"

using namespace nomos::pf;

#define CHECK(cond, ...) do { if (!(cond)) { std::printf(__VA_ARGS__); std::printf(" (%s)\n", #cond); std::exit(1); } } while (0)

template <int NQ, int KU, int VU>
struct Recorder {
    static constexpr int NB = s_buffers<NQ>();
    int n_tiles, units_in_ring;
    const TileRange (&range)[NQ];
    int next = 0, released = 0;
    int qks[4] = {}, weighed[4] = {}, pvs[4] = {};     // products and waits per S buffer
    bool read_by_pv[4] = {};                           // a PV that reads the buffer may still be running
    int qk_tiles[NQ] = {}, pv_tiles[NQ] = {};          // tiles finished per query tile
    Recorder(int n, int u, const TileRange (&r)[NQ]) : n_tiles(n), units_in_ring(u), range(r) {}
    bool next_unit(int &slot) {
        CHECK(next < units_in_ring || released > next - units_in_ring, "unit %d waits for a slot that is never released", next);
        slot = next++;
        return true;
    }
    void release(int slot) { CHECK(slot == released, "unit %d released behind %d", slot, released); ++released; }
    bool weights(int buf, int parity) {
        CHECK(qks[buf] == weighed[buf] + 1, "buffer %d: weights waited for without a QK", buf);
        CHECK(parity == (weighed[buf] & 1), "buffer %d: wrong phase of the weights", buf);
        ++weighed[buf];
        return true;
    }
    bool product(int buf, int parity) {
        CHECK(pvs[buf] > 0 && parity == ((pvs[buf] - 1) & 1), "buffer %d: wrong phase of the product", buf);
        read_by_pv[buf] = false;
        return true;
    }
    void held(int slot) { CHECK(slot < next && slot >= released, "a product reads unit %d, which is not held", slot); }
    void qk(int g, int buf, int c, int slot) {
        const int j = range[g].first + qk_tiles[g];
        const RingUnit u = ring_unit<KU, VU>(slot, n_tiles);
        held(slot);
        CHECK(u.tile == j && !u.v && u.c == c, "query tile %d: QK of tile %d takes unit %d", g, j, slot);
        CHECK(buf == NB * g + qk_tiles[g] % NB, "query tile %d, tile %d: buffer %d", g, j, buf);
        CHECK(!read_by_pv[buf], "QK of tile %d overwrites buffer %d under a PV that was not waited for", j, buf);
    }
    void s_done(int buf) { ++qks[buf]; ++qk_tiles[buf / NB]; }
    void pv(int g, int buf, int c, int slot, bool first) {
        const int j = range[g].first + pv_tiles[g];
        const RingUnit u = ring_unit<KU, VU>(slot, n_tiles);
        held(slot);
        CHECK(u.tile == j && u.v && u.c == c, "query tile %d: PV of tile %d takes unit %d", g, j, slot);
        CHECK(buf == NB * g + pv_tiles[g] % NB && weighed[buf] == pvs[buf] + 1, "query tile %d, tile %d: PV without weights", g, j);
        CHECK(first == (pv_tiles[g] == 0), "accumulation of query tile %d", g);
        read_by_pv[buf] = true;
    }
    void o_done(int buf) { ++pvs[buf]; ++pv_tiles[buf / NB]; }
    void finish() {
        CHECK(next == n_tiles * (KU + VU) && released == next, "%d of %d units taken, %d released", next, n_tiles * (KU + VU), released);
        for (int g = 0; g < NQ; ++g) {
            const int n = range[g].last >= range[g].first ? range[g].last - range[g].first + 1 : 0;
            CHECK(qk_tiles[g] == n && pv_tiles[g] == n, "query tile %d: %d and %d of %d tiles", g, qk_tiles[g], pv_tiles[g], n);
        }
    }
};

template <int NQ, int KU, int VU>
static int walk(int n_tiles, const TileRange (&range)[NQ]) {
    int walks = 0;
    for (int units : {2, 3, 5, 9, 14}) {               // units the ring holds
        Recorder<NQ, KU, VU> r(n_tiles, units, range);
        CHECK((walk_products<NQ, KU, VU>(n_tiles, range, r)), "the walk gave up");
        r.finish();
        ++walks;
    }
    return walks;
}

int main() {
    int walks = 0;
    for (int n = 1; n <= 23; ++n) {
        const TileRange all[1] = {{0, n - 1}};
        walks += walk<1, 1, 1>(n, all) + walk<1, 2, 2>(n, all) + walk<1, 4, 2>(n, all);
        // two query tiles: either may start later or end earlier, or have no keys at all
        for (int a = 0; a <= n; ++a)
            for (int b = 0; b <= n; ++b) {
                const TileRange causal[2] = {{0, n - 1 - a}, {b, n - 1}}, nested[2] = {{0, n - 1}, {a, n - 1 - b}};
                if (a + b <= n) walks += walk<2, 1, 1>(n, causal);
                walks += walk<2, 1, 1>(n, nested);
            }
        const TileRange one[2] = {{0, n - 1}, {0x3fffffff, -1}}, other[2] = {{0x3fffffff, -1}, {0, n - 1}};
        walks += walk<2, 1, 1>(n, one) + walk<2, 1, 1>(n, other);
    }
    std::printf("%d walks\n", walks);
    return 0;
}
