// The cross-tile carry fix-up kernels (gpupi_b200/csrc/carry_tile.cuh) run on
// the CPU, every row of the batch ending right before an unreadable page: an
// access past a row's own end, which in a ragged batch lies below the longest
// row's, ends this program.  The results are compared with a serial carry.
// Built and run by tests/test_carry_fixup_cpu.py.
#include <stdio.h>
#include <string.h>
#include <sys/mman.h>
#include <unistd.h>

#include <random>

#include "carry_tile.cuh"

using namespace gpupi;
namespace gpupi {
void count_launch() {}
}

static std::mt19937_64 rng(7);

// `len` limbs that end at a page without access
static uint32_t *guarded(size_t len) {
    const size_t page = (size_t)sysconf(_SC_PAGESIZE), bytes = (len * 4 + page - 1) / page * page;
    char *p = (char *)mmap(nullptr, bytes + page, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (p == MAP_FAILED || mprotect(p + bytes, page, PROT_NONE)) exit(2);
    return (uint32_t *)(p + bytes) - len;
}

struct Row {
    uint32_t *p;
    std::vector<uint32_t> want;
};

// Tile results with carry-in 0 for a row at p, flags and the row they give.
// Mostly carries, all-ones (for sub all-zeros) runs behind the first limbs, so
// that carries run far, also up to the last limb of the row.
template <bool SUB>
static Row make_row(uint32_t *p, uint32_t len, uint32_t span, uint32_t mis, uint32_t tiles, uint32_t *flags) {
    const uint32_t ones = SUB ? 0u : 0xffffffffu;
    uint32_t carry = 0;
    Row r{p, std::vector<uint32_t>(len)};
    for (uint32_t t = 0; t < tiles; ++t) {
        const uint64_t from = (uint64_t)t * span, a = from > mis ? from - mis : 0;
        const uint64_t b = std::min<uint64_t>(from + span - mis, len);
        flags[t] = 0;
        if (a >= b) continue;   // above the row: zeros, no carry
        const bool top = b == len;
        const bool all = !top && rng() % 3 == 0;
        // first limb that stops a carry: none, the last of the tile, or any
        const uint64_t stop = all ? b : (rng() % 2 ? b - 1 : a + rng() % (b - a));
        for (uint64_t i = a; i < b; ++i) p[i] = i < stop ? ones : (i == stop ? 5u : (uint32_t)rng());
        const uint32_t g = !top && !all && rng() % 4 != 0;
        flags[t] = g | (all ? 2u : 0u);
        uint32_t c = carry;
        for (uint64_t i = a; i < b; ++i) {
            r.want[i] = SUB ? p[i] - c : p[i] + c;
            c = c && p[i] == ones;
        }
        carry = g | (all ? carry : 0u);
    }
    return r;
}

static int compare(const std::vector<Row> &rows, const char *what) {
    for (size_t i = 0; i < rows.size(); ++i)
        if (memcmp(rows[i].p, rows[i].want.data(), rows[i].want.size() * 4)) {
            fprintf(stderr, "%s: row %zu differs\n", what, i);
            return 1;
        }
    return 0;
}

template <bool SUB>
static void fix(uint32_t *C, uint64_t sC, uint32_t N, uint32_t Lc, uint32_t tiles, uint32_t span, bool aligned,
                const std::vector<uint32_t> &flags, const RaggedRow *rows) {
    if (tiles > 32u) {   // as launch_carry_fixup
        const uint32_t bpr = (tiles + kFixTiles - 1u) / kFixTiles;
        for (unsigned b = 0; b < N * bpr; ++b)
            run_cta(b, N * bpr, kFixThreads, [&] {
                carry_fixup_rows_kernel<SUB>(C, sC, Lc, tiles, bpr, span, aligned, flags.data(), rows);
            });
    } else {
        run_cta(0, 1, 128, [&] { carry_fixup_kernel<SUB>(C, sC, N, Lc, tiles, span, aligned, flags.data(), rows); });
    }
}

// A ragged batch of one bucket: rows of the given lengths, the last the longest.
static int ragged(std::vector<uint32_t> len, uint32_t span) {
    const uint32_t N = (uint32_t)len.size(), most = len.back();
    const uint32_t tiles = (most + span - 1u) / span;
    std::vector<uint32_t> flags((size_t)N * tiles);
    std::vector<Row> rows;
    std::vector<RaggedRow> d;
    uint32_t *C = nullptr;
    for (uint32_t i = 0; i < N; ++i) {
        uint32_t *p = guarded(len[i]);
        if (!C) C = p;
        rows.push_back(make_row<false>(p, len[i], span, 0u, tiles, flags.data() + (size_t)i * tiles));
        // rows may lie below the first: the offset wraps, and the address with it
        d.push_back(RaggedRow{0, 0, (uint64_t)(((intptr_t)p - (intptr_t)C) / 4), len[i] - len[i] / 3, len[i] / 3});
    }
    fix<false>(C, 0, N, most, tiles, span, false, flags, d.data());
    return compare(rows, "ragged");
}

// Equal rows at every alignment, tiles counted from the 16-byte boundary.
template <bool SUB>
static int uniform(uint32_t N, uint32_t len, uint32_t span) {
    const uint32_t tiles = (len + 3u + span - 1u) / span;
    const uint64_t stride = len + 1u;
    uint32_t *C = guarded((N - 1) * stride + len);
    std::vector<uint32_t> flags((size_t)N * tiles);
    std::vector<Row> rows;
    for (uint32_t i = 0; i < N; ++i) {
        uint32_t *p = C + i * stride;
        rows.push_back(make_row<SUB>(p, len, span, ((uintptr_t)p >> 2) & 3u, tiles, flags.data() + (size_t)i * tiles));
    }
    fix<SUB>(C, stride, N, len, tiles, span, true, flags, nullptr);
    return compare(rows, SUB ? "sub" : "add");
}

int main() {
    for (int k = 0; k < 2; ++k) {
        if (ragged({2041, 2100, 2168, 4080, 4081, 4082, 4097, 4111, 8000}, 2040)) return 1;
        if (ragged({2100, 65280, 65281, 66000, 70000}, 2040)) return 1;   // 35 tiles: a CTA per row
    }
    if (ragged({300, 4 * 1024 + 1, 4 * 1500 + 3}, 4)) return 1;   // several CTAs per row
    for (uint32_t len : {4097u, 8190u, 8192u, 3u * 4096u})
        if (uniform<false>(5, len, 4096) || uniform<true>(5, len, 4096)) return 1;
    if (uniform<false>(4, 50 * 128 - 1, 128) || uniform<true>(4, 50 * 128 + 2, 128)) return 1;
    puts("carry fix-up ok");
    return 0;
}
