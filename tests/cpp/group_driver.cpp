// The adjoint's copies of aligned pixel groups over every window of small
// images, by the kernel's own index functions: no copied group reaches outside
// the image's storage, every image pixel that a window reads is copied unless
// the window is marked as cut, and it is marked only where one is not.
#include <algorithm>
#include <cstdio>
#include <vector>

#include "toed_groups.h"

template <int NU>
static long long windows(int H, int W, int pitch, int skew)
{
    constexpr int CH = (NU + 6) / 4, R = (NU - 5) / 2;
    const long long span = (long long)(H - 1) * pitch + W;
    const unsigned whole = toed::whole_groups(span);
    std::vector<char> copied(skew + span + 8);
    long long n = 0;
    for (int i = 0; i < H; ++i)
        for (int j = 0; j < W; ++j, ++n) {
            const int wy = i - R - 2, wx = j - R - 2, own = wy * pitch + wx + skew;
            bool missing = false;
            for (int u = 0; u < NU; ++u) {
                std::fill(copied.begin(), copied.end(), 0);
                for (int l = 0; l < 8; ++l) {
                    const int at = own + u * pitch + 4 * l;
                    if (!toed::group_copied<NU, CH>(at, l, skew, whole)) continue;
                    const int g = at & ~3;
                    if (g < skew || g + 4 > skew + span) {
                        std::printf("H %d W %d pitch %d skew %d NU %d window (%d, %d) row %d: pixels %d..%d of [%d, %lld)\n", H, W,
                                    pitch, skew, NU, wy, wx, u, g, g + 3, skew, skew + span);
                        return -1;
                    }
                    for (int e = 0; e < 4; ++e) copied[g + e] = 1;
                }
                if (wy + u < 0 || wy + u >= H) continue;
                for (int t = 0; t < NU; ++t)
                    if (wx + t >= 0 && wx + t < W) missing |= !copied[own + u * pitch + t];
            }
            if (missing != toed::window_cut(wy, wx, NU, H, W, skew, span)) {
                std::printf("H %d W %d pitch %d skew %d NU %d window (%d, %d): %s\n", H, W, pitch, skew, NU, wy, wx,
                            missing ? "a pixel is missing" : "marked without need");
                return -1;
            }
        }
    return n;
}

template <int NU>
static long long all_sizes()
{
    long long n = 0;
    for (int H : {1, 2, 3, 5, 9, NU - 1, NU, NU + 4})
        for (int W = 4; W <= NU + 6; ++W)
            for (int pitch = W; pitch < W + 5; ++pitch)
                for (int skew = 0; skew < 4; ++skew) {
                    const long long k = windows<NU>(H, W, pitch, skew);
                    if (k < 0) return -1;
                    n += k;
                }
    return n;
}

int main()
{
    // the window sides of radius 1, 2, 3, 6, 8, 12: NU = 2 r + 5
    const long long n[] = {all_sizes<7>(), all_sizes<9>(), all_sizes<11>(), all_sizes<17>(), all_sizes<21>(), all_sizes<29>()};
    long long sum = 0;
    for (long long k : n) {
        if (k < 0) return 1;
        sum += k;
    }
    std::printf("%lld windows\n", sum);
    return 0;
}
