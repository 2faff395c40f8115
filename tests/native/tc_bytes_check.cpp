// The tensor-core scoring kernel's arithmetic restated in integers and floats
// (score_tc.cu), from the plan alone: random models over one or several regions
// to a row, with duplicate and cancelling terms and constants.  For random
// rows, every output and some columns:
//   - the sums D_s of digit products of coefficients (c0, c1) and raw bytes stay
//     below 2^23, so fp32 holds them exactly;
//   - D_s 2^-24 plus the output's m0 or m1 lands in [0.5, 1), and its bits, joined
//     by 256^s with `offset` and less the four magic numbers, plus the bias are the
//     output's word: sum of coefficient times word of the (rotated) row, mod 2^32;
//   - rotations are multiples of tc_rot_bytes / 4 words;
//   - tc_out_rows are the first and last row that an output reads.
// Prints one line per trial; exits non-zero on a mismatch.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <random>
#include <vector>

#include "plan.hpp"
using namespace idash;

static int32_t half_to_int(uint16_t h) {
    _Float16 f;
    std::memcpy(&f, &h, 2);
    return int32_t(float(f));
}
static uint32_t bits(float f) {
    uint32_t u;
    std::memcpy(&u, &f, 4);
    return u;
}

int main() {
    std::mt19937_64 rng(5);
    int failures = 0;
    constexpr uint32_t N = 256;  // short rows: rotations wrap often
    constexpr uint32_t kMagic = 0x3F400000u, kMagicSum = kMagic + (kMagic << 8) + (kMagic << 16) + (kMagic << 24);
    const uint32_t regions_of[] = {1, 2, 4, 7, 64, 256};
    for (int trial = 0; trial < 24; ++trial) {
        const uint32_t regions = regions_of[trial % 6], size = N / regions;
        const uint32_t n_rows = 60, n_feat = n_rows * regions;
        const uint64_t n_out = 100 + rng() % 200;
        const int32_t cmax = trial % 2 ? 32767 : 8192;
        std::vector<uint64_t> ptr{0};
        std::vector<uint32_t> feat;
        std::vector<int32_t> coef;
        for (uint64_t o = 0; o < n_out; ++o) {
            const uint32_t nb = uint32_t(std::vector<uint32_t>{0, 1, 6, 30}[rng() % 4]);
            const uint32_t base = uint32_t(o * (n_feat - 30) / n_out);
            for (uint32_t k = 0; k < nb; ++k) {
                feat.push_back(base + k);
                coef.push_back(trial % 4 < 2 ? int32_t(rng() % uint64_t(2 * cmax)) - cmax : (rng() % 2 ? cmax : -cmax));
            }
            if (nb && rng() % 3 == 0) { feat.push_back(base); coef.push_back(-coef[ptr.back()]); }  // cancels
            if (rng() % 2) { feat.push_back(0xFFFFFFFFu); coef.push_back(int32_t(rng() % 1000)); }
            ptr.push_back(feat.size());
        }
        PlanInput in;
        in.form = Form::kTrlwe;
        in.n_out = n_out;
        in.term_ptr = ptr.data();
        in.term_feat = feat.data();
        in.term_coef = coef.data();
        in.n_rows = n_rows;
        in.one_t32 = 1 << 18;
        in.N = N;
        in.num_regions = regions;
        in.region_size = size;
        Plan plan;
        bool index_error = false, ok = true;
        const std::string err = build_tc_plan(in, TcLimits{}, &plan, &index_error);
        if (!err.empty()) { std::printf("trial %d FAIL plan: %s\n", trial, err.c_str()); ++failures; continue; }
        ok = (plan.tc_rot_bytes != 0) == (regions > 1) && plan.tc_out_rows.size() == (regions > 1 ? n_out : 0);
        std::vector<std::vector<uint32_t>> rows(n_rows, std::vector<uint32_t>(N));
        for (auto &r : rows)
            for (auto &w : r) w = trial % 3 ? uint32_t(rng()) : (rng() % 2 ? 0xFFFFFFFFu : 0x80808080u);
        auto word = [&](uint32_t row, uint32_t rot, uint32_t j) {  // column j of X^(-rot) * row
            return j + rot < N ? rows[row][j + rot] : 0u - rows[row][j + rot - N];
        };
        int64_t worst = 0;
        for (const PlanBlock &b : plan.blocks) {
            const uint8_t *A = plan.tc_a.data() + uint64_t(b.group_begin) * 16;
            const uint64_t plane = tc_a_bytes(b.n_groups) / 2;
            for (uint32_t k = 0; k < b.n_slots; ++k) {
                const uint32_t rot = plan.slots[b.slot_begin + k].rot;
                if (regions == 1 ? rot != 0 : rot % (plan.tc_rot_bytes / 4) != 0) ok = false;
            }
            for (uint64_t o = b.out_lo; o < b.out_hi && ok; ++o) {
                const uint32_t m = uint32_t(o - b.out_lo), j = uint32_t(rng() % N);
                uint32_t want = 0, first = 0xFFFFFFFFu, end = 0;
                std::map<uint32_t, uint32_t> sum;
                for (uint64_t t = ptr[o]; t < ptr[o + 1]; ++t) {
                    if (feat[t] == 0xFFFFFFFFu) { want += uint32_t(coef[t]) << 18; continue; }
                    want += uint32_t(coef[t]) * word(feat[t] / regions, feat[t] % regions * size, j);
                    sum[feat[t]] += uint32_t(coef[t]);
                }
                for (auto &kv : sum)
                    if (kv.second) first = std::min(first, kv.first / regions), end = std::max(end, kv.first / regions + 1);
                if (regions > 1 && plan.tc_out_rows[o] != (end ? std::make_pair(first, end) : std::make_pair(0u, 0u))) ok = false;
                int64_t D[4] = {0, 0, 0, 0};
                for (uint32_t k = 0; k < b.n_slots; ++k) {
                    const uint64_t off = uint64_t(k / 8) * 2048 + (m / 8) * 128 + (m % 8) * 16 + (k % 8) * 2;
                    uint16_t h0, h1;
                    std::memcpy(&h0, A + off, 2);
                    std::memcpy(&h1, A + plane + off, 2);
                    const PlanSlot &s = plan.slots[b.slot_begin + k];
                    const uint32_t x = word(s.row, s.rot, j);
                    for (int i = 0; i < 4; ++i) {
                        const int64_t byte = (x >> (8 * i)) & 255u;
                        D[i] += half_to_int(h0) * byte;
                        if (i < 3) D[i + 1] += half_to_int(h1) * byte;
                        for (int64_t d : D) worst = std::max<int64_t>(worst, d < 0 ? -d : d);
                    }
                }
                const TcOut &oc = plan.tc_out[o];
                uint32_t v = oc.offset - kMagicSum + oc.bias;
                for (int s = 0; s < 4; ++s) {
                    const float sum_s = float(D[s]) * 0x1p-24f, r = sum_s + (s ? oc.m1 : oc.m0);
                    if (!(r >= 0.5f && r < 1.0f)) ok = false;
                    v += bits(r) << (8 * s);
                }
                if (v != want) ok = false;
            }
        }
        if (worst >= (1 << 23)) ok = false;
        std::printf("trial %d %s: regions=%u outputs=%llu blocks=%zu worst|D|=%lld\n", trial, ok ? "ok" : "FAIL", regions,
                    (unsigned long long)n_out, plan.blocks.size(), (long long)worst);
        failures += ok ? 0 : 1;
    }
    return failures != 0;
}
