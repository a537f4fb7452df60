// Entries that name a base beyond the table, in the debug library's affine
// rounds: their pair must come out as an infinity with none of the record
// read.  The records lie within this program's allocation, so a missing check
// reads a known pattern, not foreign memory.
#include <cstdio>
#include <cstring>
#include <vector>
#include "msm.cuh"

using namespace lzk;

template <class F>
static int check(const char* name)
{
    constexpr uint32_t table = 4, all = 8, slots = 8;
    std::vector<Aff<F>> bases(all);
    for (uint32_t i = 0; i < all; i++) std::memset(&bases[i], i < table ? 0 : 0x11, sizeof(Aff<F>));
    const uint32_t ent[slots] = {5, 6, 0x80000005u, 7, kNoEntry, 6, 0, 5}, total = slots;
    Aff<F>*db, *fin;
    uint32_t *de, *dt;
    char* scratch;
    const AffineScratch<F> sz(slots, 1);
    if (cudaMalloc(&db, all * sizeof(Aff<F>)) || cudaMalloc(&fin, slots / 2 * sizeof(Aff<F>)) ||
        cudaMalloc(&de, sizeof(ent)) || cudaMalloc(&dt, sizeof(total)) || cudaMalloc(&scratch, sz.bytes()))
        return 1;
    cudaMemcpy(db, bases.data(), all * sizeof(Aff<F>), cudaMemcpyHostToDevice);
    cudaMemcpy(de, ent, sizeof(ent), cudaMemcpyHostToDevice);
    cudaMemcpy(dt, &total, sizeof(total), cudaMemcpyHostToDevice);
    lzk_debug_check_word(1);
    if (affine_sum<F>(db, de, dt, slots, slots, 1, table, scratch, fin, 0) != LZK_OK) return 1;
    std::vector<Aff<F>> got(slots / 2);
    if (cudaMemcpy(got.data(), fin, slots / 2 * sizeof(Aff<F>), cudaMemcpyDeviceToHost)) return 1;
    int bad = lzk_debug_check_word(1) != 4u;
    for (const Aff<F>& p : got) {
        const uint32_t* x = reinterpret_cast<const uint32_t*>(&p.x);
        const uint32_t* y = reinterpret_cast<const uint32_t*>(&p.y);
        bad += x[7] != 0xffffffffu;
        for (size_t i = 0; i < sizeof(F) / 4; i++) bad += y[i] != 0;
    }
    std::printf("%s: %d\n", name, bad);
    return bad;
}

int main()
{
    if (!lzk_debug_checks_enabled()) return 2;
    return check<Fq>("G1") + check<Fq2>("G2") ? 1 : 0;
}
