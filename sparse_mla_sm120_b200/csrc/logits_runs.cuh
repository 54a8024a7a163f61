// Into how many runs the key tiles of a query group are cut (mqa_logits_tc_kernel).
#pragma once

namespace smla {

// `groups` query groups of `tiles` key tiles on `sms` CTAs.  About eight work items per SM, so that the CTAs finish together, of at least
// eight tiles, so that the q load and the pipeline fill stay a small share: that is the shortest run.  Longer ones, as many as
// fill one to eight rounds of the CTAs, are taken where they make the longest share of a CTA more than 1 % shorter; an item pays
// for its q and for filling and draining the pipeline what five tiles take.  us, shortest runs / these (64 heads): 16 tokens x 131072
// keys, one run of 28 tiles per CTA, 26.2 / 20.5; 700 x 9000 69.4 / 61.9; 1024 x 65536 607 / 593; 4096 x 4096 from the first token on
// 105.5 / 98.2.  Where only whole groups would fill the rounds (750 groups: six rounds of them, five and a bit of their halves) the
// shortest runs stay: 3000 x 65536 1791, whole 1983; with 32 heads 1257 and 1459.
inline int logits_runs(int groups, int tiles, int sms) {
    const int most = tiles > 8 ? (tiles + 7) / 8 : 1;
    auto share = [&](int c) { return ((long long)groups * c + sms - 1) / sms * ((tiles + c - 1) / c + 5); };
    if (groups >= 8 * sms) return 1;
    int best = (8 * sms + groups - 1) / groups;
    if (best > most) best = most;
    long long limit = share(best) * 99 / 100;
    for (int r = 1; r <= 8; ++r) {
        int c = r * sms / groups;
        c = c < 1 ? 1 : c > most ? most : c;
        if (share(c) < limit) { limit = share(c); best = c; }
    }
    return best;
}

}  // namespace smla
