// Checks plan_rows (lutgemm_kernels.h) over random sizes, with the kernel's own walk through a CTA's share: every (cell, k) is in
// one piece, no piece is empty or longer than the plan says, and every term block belongs to one group.
#include <stdio.h>

#include <algorithm>
#include <random>
#include <vector>

#include "lutgemm_kernels.h"

int main() {
    using namespace lutgemm;
    std::mt19937_64 gen(1);
    auto draw = [&](long lo, long hi) { return std::uniform_int_distribution<long>(lo, hi)(gen); };
    long grouped = 0, runs = 0;
    for (int i = 0; i < 20000; ++i) {
        const int sms = draw(0, 3) ? 148 : (int)draw(1, 200);
        const long rows = draw(1, draw(0, 1) ? 2000 : 300000), terms = draw(1, draw(0, 1) ? 700 : 60000);
        const int K = (int)draw(1, draw(0, 1) ? 70 : 5000);
        const RowsPlan p = plan_rows(rows, terms, K, sms);
        const long blocks = (terms + kRowsTerms - 1) / kRowsTerms, kunits = (K + kRowsUnit - 1) / kRowsUnit;
        bool ok = p.groups >= 1 && (long)p.groups * p.group_blocks >= blocks && (p.groups - 1L) * p.group_blocks < blocks &&
                  p.piece_k % kRowsUnit == 0 && p.piece_k > 0 && (p.group_blocks <= kRowsChain || p.piece_k <= kRowsMaxPer);
        const long total = rows_units(p, rows, K);
        const int grid = (int)std::min<long>(total, sms);
        long expect = 0;  // pieces have to follow each other without gaps
        for (int cta = 0; ok && cta < grid; ++cta) {
            long cur = total * cta / grid;
            const long end = total * (cta + 1) / grid;
            ok = cur == expect && end > cur;
            while (ok && cur < end) {
                const long k0 = cur % kunits, nk = std::min(std::min(end - cur, kunits - k0), (long)p.piece_k / kRowsUnit);
                ok = nk > 0 && k0 * kRowsUnit < K;
                cur += nk;
            }
            expect = end;
        }
        if (!ok || expect != total) {
            printf("rows %ld terms %ld K %d sms %d: groups %d x %d, pieces of %d\n", rows, terms, K, sms, p.groups, p.group_blocks, p.piece_k);
            return 1;
        }
        grouped += p.groups > 1;
        runs += p.group_blocks > kRowsChain;
    }
    return grouped > 1000 && runs > 1000 ? 0 : 2;
}
