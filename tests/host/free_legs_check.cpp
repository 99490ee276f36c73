// Host-side check of the rule that frees a field march of its wall limit (no
// GPU): for random reflections, volumes and boxes of non-vacuum labels, every
// leg the rule frees examines no position outside the volume before it meets
// vacuum, whichever increments it skips inside the box, in the reference's
// FP64 positions and in the march's fixed-point ones (with their margin, passed
// as MARGIN).  Prints "ok <free legs> <others that would have left>".
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>

#include "anacor_internal.h"

using namespace anacor;

int main()
{
    std::mt19937_64 gen(20240);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    auto pick = [&](int lo, int hi) { return lo + (int)(gen() % (unsigned long long)(hi - lo + 1)); };
    const double F[9] = {0.98, 0.1, -0.05, -0.08, 0.97, 0.12, 0.06, -0.11, 0.99};
    const double axis[3] = {1.0, 0.0, 0.0};
    long long freed = 0, left = 0;
    for (int it = 0; it < 60000; it++) {
        double v[2][3];
        for (auto &w : v) {
            double n = 0.0;
            for (double &x : w) {
                x = U(gen);
                n += x * x;
            }
            for (double &x : w)
                x /= std::sqrt(n);
        }
        ReflTable t;
        double rx[3], rs[3];
        if (setup_reflection(axis, 3.2 * (U(gen) + 1.0), F, v[0], v[1], &t, rx, rs) != kOk)
            continue;
        for (int leg = 0; leg < 2; leg++) {
            const uint32_t sb = t.head[leg].sign_bits;
            // face code -> (axis, max side): 1 x max, 6 x min, 5 y max, 4 y min, 3 z max, 2 z min
            const int faces[6][3] = {{1, 2, 1}, {6, 2, 0}, {5, 1, 1}, {4, 1, 0}, {3, 0, 1}, {2, 0, 0}};
            for (const auto &f : faces) {
                const int s = f[1], a = s == 0 ? 1 : 0, b = s == 2 ? 1 : 2;
                const FaceRule &R = t.rule[leg][f[0] - 1];
                if (!(f[2] ? ((sb >> s) & 1u) : ((sb >> (3 + s)) & 1u)) || R.status || !R.fast)
                    continue;
                const long long qm = std::max(std::llabs(R.Q[a]), std::llabs(R.Q[b]));
                if (qm > (30ll << 32))
                    continue;
                int dim[3], lo[3], hi[3], c[3], room[6];
                for (int x = 0; x < 3; x++) {
                    dim[x] = pick(1, 90);
                    lo[x] = pick(0, std::min(dim[x] - 1, 12));
                    hi[x] = pick(lo[x], dim[x] - 1);
                    if (gen() % 2)
                        hi[x] = std::max(lo[x], dim[x] - 1 - pick(0, 12));
                    room[x] = lo[x];
                    room[3 + x] = dim[x] - 1 - hi[x];
                    c[x] = pick(lo[x], hi[x]);
                }
                bool is_free = true;
                for (int x = 0; x < 3; x++)
                    is_free = is_free && room[wall_ahead(R.octant, x)] >= free_leg_room(qm);
                auto in = [&](const int *p, const int *l, const int *h) {
                    return p[0] >= l[0] && p[0] <= h[0] && p[1] >= l[1] && p[1] <= h[1] && p[2] >= l[2] && p[2] <= h[2];
                };
                const int zero[3] = {0, 0, 0}, last[3] = {dim[0] - 1, dim[1] - 1, dim[2] - 1};
                auto exact = [&](int i, int *p) {
                    for (int x = 0; x < 3; x++) {
                        const double y = (double)c[x] + (double)i * R.q[x];
                        p[x] = (int)(R.use_round ? std::round(y) : std::floor(y));
                    }
                };
                auto fixed = [&](int i, int *p) {
                    for (int x = 0; x < 3; x++) {
                        const bool half = R.use_round || ((R.exact_mask >> x) & 1) || (R.Q[x] == 0 && R.q[x] >= 0.0);
                        p[x] = c[x] + (int)(((half ? 1ll << 31 : 0ll) + MARGIN + (long long)i * R.Q[x]) >> 32);
                    }
                    p[s] = c[s] + i * (R.Q[s] > 0 ? 1 : -1);
                };
                int p[3], q[3], i = 0;
                for (;;) {
                    int k = 1;   // skipped increments lie in the box, then one is examined
                    for (; gen() % 5 < 2; k++) {
                        exact(i + k, p);
                        if (!in(p, lo, hi))
                            break;
                    }
                    i += k;
                    exact(i, p);
                    fixed(i, q);
                    if (!in(p, zero, last) || !in(q, zero, last)) {
                        if (is_free) {
                            std::printf("a free leg leaves: refl %d leg %d face %d increment %d\n", it, leg, f[0], i);
                            return 1;
                        }
                        left++;
                        break;
                    }
                    if (!in(p, lo, hi))
                        break;   // vacuum
                }
                freed += is_free;
            }
        }
    }
    std::printf("ok %lld %lld\n", freed, left);
    return freed > 10000 && left > 10000 ? 0 : 1;
}
