// Stand-alone check, on the host, of how decode attention cuts the sequences of a merged step (attn_args.cuh): every position is in one part, the parts fit
// the list, and no part is much longer than its share.
//
//     parts_check        exit code 0 when every case passes
#include <algorithm>
#include <cstdio>
#include <random>
#include <vector>

#include "../attn_args.cuh"

int main() {
    std::mt19937 rng(1);
    long cases = 0, bad = 0;
    auto check = [&](const std::vector<int>& spans, int room, int each, int least) {
        const int B = (int)spans.size(), parts = room + B * each;
        long total = 0, used = 0, several = 0;
        for (int s : spans) total += s;
        const int length = attn_part_len(total, room, least);
        bool ok = length % 64 == 0 && length >= least;
        for (int s : spans) {
            int per = -1;
            const int n = attn_part_count(s, length, each, least, &per);
            ok = ok && n >= 1 && n <= 64 && per > 0 && (long)n * per >= s && (n == 1 || (long)(n - 1) * per < s);
            // a part is no longer than twice the length that all should have, but where a sequence would need more than 64 of those
            ok = ok && per <= std::max(std::max(2 * length, least), ((s + 63) / 64 + 63) & ~63);
            // and what is cut finer is no shorter than it need be
            ok = ok && (n <= each || per > length / 2);
            used += n;
            several += n > 1;
        }
        ok = ok && used <= parts && several <= attn_part_merges(parts, each, B);
        ++cases;
        if (!ok && bad++ < 10) std::printf("FAIL B=%d room=%d each=%d least=%d total=%ld length=%d used=%ld several=%ld\n", B, room, each, least, total, length, used, several);
    };
    for (int heads : {1, 2, 3, 8, 16, 64, 296, 500})
        for (int least : {1, 64, 100, 128, 512})
            for (int B : {2, 3, 16, 33, 64, 300}) {
                const int each = std::min(64, (296 + B * heads - 1) / (B * heads)), room = (296 + heads - 1) / heads;
                for (int s : {0, 1, 63, 64, 65, 127, 128, 129, 4096, 40960, 131072}) check(std::vector<int>(B, s), room, each, least);
                for (int i = 0; i < 40; ++i) {
                    std::vector<int> spans(B);
                    const double skew = i / 8.0;
                    for (int& s : spans) s = (int)std::min(262144.0, std::exp(std::normal_distribution<double>(4.0, skew)(rng)));
                    check(spans, room, each, least);
                }
                std::vector<int> one(B, 1);
                one[B / 2] = 131072;
                check(one, room, each, least);
            }
    std::printf("%s: %ld cases, %ld wrong\n", bad ? "FAILED" : "OK", cases, bad);
    return bad != 0;
}
