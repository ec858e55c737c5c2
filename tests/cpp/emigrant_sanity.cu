// The placement of a step's emigrants (launch_step_finish) on tables made by
// hand, where no grid can bring it: more leavers in the tiles' bits than the
// layout counted.  The status word must say so, and the slots that the layout
// gave the destination must hold its first immigrants; no slot past them is
// written and no record but a leaver's is read.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../dsdecompx_b200/csrc/dsx_kernels.cuh"

namespace {

int failures = 0;

void check(bool ok, const char* what, int leavers, int counted) {
    if (ok) return;
    std::printf("emigrant_sanity: %s (%d leavers, %d counted)\n", what, leavers, counted);
    ++failures;
}

template <class T>
T* device(const std::vector<T>& host) {
    T* p = nullptr;
    if (cudaMalloc(&p, host.size() * sizeof(T)) != cudaSuccess ||
        cudaMemcpy(p, host.data(), host.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess) {
        std::printf("emigrant_sanity: %s\n", cudaGetErrorString(cudaGetLastError()));
        std::exit(1);
    }
    return p;
}

template <class T>
std::vector<T> host(const T* p, std::size_t n) {
    std::vector<T> v(n);
    if (cudaMemcpy(v.data(), p, n * sizeof(T), cudaMemcpyDeviceToHost) != cudaSuccess) {
        std::printf("emigrant_sanity: %s\n", cudaGetErrorString(cudaGetLastError()));
        std::exit(1);
    }
    return v;
}

// Subdomain 0's first `leavers` of n0 particles leave for subdomain 1, whose
// layout counted `counted` of them.  No send lists, one axis split.
void run(int leavers, int counted) {
    constexpr int T = dsx::kTile, kEmigCounter = dsx::kHaloCounters + 1;
    const int n0 = leavers + 100, n1 = 500, N = n0 + n1;
    const int t0 = (n0 + T - 1) / T, t1 = (n1 + T - 1) / T, tiles = t0 + t1;
    const int ncap = N, max_tiles = (ncap + T - 1) / T + 2, stride = (max_tiles + 4) / 4 * 4;
    const int E = dsx::kMaxNeighbors;

    dsx::Grid G;
    G.P = 2;
    G.dims[0] = 2;
    for (int a = 0; a < 3; ++a) G.periodic[a] = 0;
    G.cut_offset[1] = 3;
    G.cut_offset[2] = 5;
    G.ncap = ncap;
    G.gcap = 1;
    G.tile = T;
    G.max_tiles = max_tiles;
    G.cuts = device(std::vector<double>{0.0, 0.5, 1.0, 0.0, 1.0, 0.0, 1.0});
    G.coord = device(std::vector<int>{0, 1 << 20});
    G.need = device(std::vector<unsigned char>(2 * 32, 0));
    G.lut = device(std::vector<unsigned>(2 * 64, 0u));
    G.shift = device(std::vector<double>(2 * E * 3, 0.0));
    G.n = device(std::vector<int>{n0, n1});
    G.obase = device(std::vector<int>{0, n0, N});
    G.tile_start = device(std::vector<int>{0, t0, tiles});
    std::vector<int4> rows(static_cast<std::size_t>(max_tiles), make_int4(0, 0, 0, 0));
    for (int g = 0; g < t0; ++g) rows[g] = make_int4(0, g * T, g * T + T < n0 ? g * T + T : n0, 0);
    for (int g = 0; g < t1; ++g)
        rows[t0 + g] = make_int4(1, n0 + g * T, n0 + (g * T + T < n1 ? g * T + T : n1), t0);
    G.tiles = device(rows);
    const int next0 = n0 - leavers, next1 = n1 + counted, base1 = next0 + n1;
    G.n_next = device(std::vector<int>{next0, next1});
    G.obase_next = device(std::vector<int>{0, next0, next0 + next1});
    const int nt0 = (next0 + T - 1) / T;
    G.tile_start_next = device(std::vector<int>{0, nt0, nt0 + (next1 + T - 1) / T});
    G.tiles_next = device(rows);
    G.status = device(std::vector<unsigned>{0u});

    // records: the owned half, then the half that the placement writes
    dsx::Arrays A;
    for (int a = 0; a < 11; ++a) {
        std::vector<double> v(2 * static_cast<std::size_t>(ncap), -1.0);
        for (int i = 0; i < N; ++i) v[i] = i < leavers && a == 0 ? 0.75 : 100.0 * a + i;
        A.d[a] = device(v);
    }
    std::vector<int> ids(2 * static_cast<std::size_t>(ncap), -1);
    for (int i = 0; i < N; ++i) ids[i] = i;
    A.type = device(ids);
    A.gid = device(ids);

    dsx::Scratch S;
    std::vector<unsigned> bits(static_cast<std::size_t>(max_tiles) * dsx::kTileBits, 0u);
    std::vector<int> pre(static_cast<std::size_t>(kEmigCounter + 1) * stride, 0);
    for (int i = 0; i < leavers; ++i)
        bits[static_cast<std::size_t>(i / T) * dsx::kTileBits + (i % T) / 32 * 8 + 7] |= 1u << (i % 32);
    for (int g = 0; g <= tiles; ++g)
        pre[static_cast<std::size_t>(kEmigCounter) * stride + g] = g * T < leavers ? g * T : leavers;
    S.bits = device(bits);
    S.pre = device(pre);
    S.stride = stride;
    S.dest16 = device(std::vector<unsigned short>(static_cast<std::size_t>(max_tiles) * T, 1));
    S.imm_total = device(std::vector<int>{0, counted});
    S.imm_base = device(std::vector<int>{next0, base1});
    S.imm_tile_start = device(std::vector<int>{0, 0, (counted + T - 1) / T});
    S.imm_tiles = device(rows);
    S.emig_src = device(std::vector<int>((static_cast<std::size_t>(ncap) + 3) / 4 * 4, 0));
    S.emig_dst = device(std::vector<int>((static_cast<std::size_t>(ncap) + 3) / 4 * 4, 0));
    S.emig_info = device(std::vector<int>{leavers, 0, 0, 0});
    S.cbase_imm = device(std::vector<int>(2 * dsx::kHaloCounters, 0));
    // what an unwritten entry of the order would name: a particle that stays
    S.mask = device(std::vector<unsigned>(static_cast<std::size_t>(ncap), static_cast<unsigned>(N - 1)));

    dsx::launch_step_finish(G, G, A, 0, ncap, 2ll * ncap, S, nullptr, false);
    check(cudaDeviceSynchronize() == cudaSuccess, "the launches failed", leavers, counted);
    const bool mismatch = host(G.status, 1)[0] & dsx::kStatusMigrationMismatch;
    check(mismatch == (leavers != counted), "status", leavers, counted);
    const std::vector<int> gid = host(A.gid, ids.size());
    const std::vector<double> x = host(A.d[0], ids.size());
    const int placed = leavers < counted ? leavers : counted;
    bool right = true, untouched = true;
    for (int k = 0; k < ncap; ++k) {
        const int got = gid[static_cast<std::size_t>(ncap) + k];
        const bool mine = k >= base1 && k < base1 + placed;
        if (mine) right = right && got == k - base1 && x[static_cast<std::size_t>(ncap) + k] == 0.75;
        else untouched = untouched && got == -1;
    }
    check(right, "an immigrant's record", leavers, counted);
    check(untouched, "a slot that is not the destination's was written", leavers, counted);
    for (void* p : {static_cast<void*>(G.cuts), (void*)G.coord, (void*)G.need, (void*)G.lut, (void*)G.shift,
                    (void*)G.n, (void*)G.obase, (void*)G.tile_start, (void*)G.tiles, (void*)G.n_next,
                    (void*)G.obase_next, (void*)G.tile_start_next, (void*)G.tiles_next, (void*)G.status,
                    (void*)A.type, (void*)A.gid, (void*)S.bits, (void*)S.pre, (void*)S.dest16,
                    (void*)S.imm_total, (void*)S.imm_base, (void*)S.imm_tile_start, (void*)S.imm_tiles,
                    (void*)S.emig_src, (void*)S.emig_dst, (void*)S.emig_info, (void*)S.cbase_imm,
                    (void*)S.mask})
        cudaFree(p);
    for (double* d : A.d) cudaFree(d);
}

}  // namespace

int main() {
    // the count right, short and over, inside a pass of the list, across its
    // passes, and across the CTAs of a cluster of either size
    for (int leavers : {5, 600, 2048, 5001, 20000, 150001})
        for (int off : {0, -1, 1, -4}) run(leavers, leavers + off);
    if (failures) return 1;
    std::printf("emigrant_sanity: ok\n");
    return 0;
}
