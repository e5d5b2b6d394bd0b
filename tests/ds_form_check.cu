// ds_form_check.cu -- host-only check of the DSSIM map pass's choice between
// tiles and strips (Engine::choose_ds_rows): submissions of n equal pairs whose
// DSSIM passes were timed in both forms on a B200 (us) go in the faster form,
// and none goes in strips that were slower.  Below two waves of strips, where
// the times of the two are close, only that direction is checked.  plan() makes
// no CUDA call (built and run by tests/test_cpu_ds_form.py).
#include <cstdio>
#include <vector>

#include "../turbo-metrics_b200/csrc/ssim2_engine_internal.h"

struct Timed {
    int n;
    uint32_t w, h;
    double tiles, strips;
};

int main() {
    const Timed timed[] = {
        {512, 32, 32, 240, 331},     {300, 8, 8, 162, 173},       {256, 64, 64, 187, 265},
        {128, 64, 64, 117, 203},     {256, 128, 128, 442, 530},   {64, 130, 600, 616, 684},
        {32, 240, 1080, 779, 569},   {64, 96, 2000, 1213, 1375},  {16, 96, 2000, 339, 437},
        {64, 121, 512, 407, 594},    {64, 200, 512, 616, 541},    {64, 300, 512, 779, 733},
        {100, 200, 200, 495, 370},   {64, 256, 256, 369, 399},    {128, 256, 256, 714, 735},
        {64, 360, 360, 757, 534},    {64, 512, 512, 1261, 1044},  {32, 512, 512, 627, 577},
        {16, 512, 512, 321, 352},    {64, 640, 480, 1373, 1100},  {16, 1280, 720, 979, 768},
        {8, 1280, 720, 499, 440},    {4, 1280, 720, 260, 278},    {64, 1920, 1080, 8230, 5377},
        {8, 1920, 1080, 1024, 782},  {4, 1920, 1080, 520, 452},   {2, 1920, 1080, 274, 284},
        {1, 1920, 1080, 161, 192},   {4, 2048, 2048, 1032, 817},  {1, 2560, 1440, 241, 272},
        {1, 3840, 2160, 497, 430},   {16, 3840, 2160, 7764, 5180}, {64, 2000, 96, 1090, 632},
        {4, 121, 6000, 307, 452},    {16, 481, 481, 366, 379},
    };
    int fails = 0;
    for (const Timed &t : timed) {
        Engine e;  // not initialised: planning is host-only
        e.metrics = S2_METRIC_DSSIM;
        std::vector<s2_pair_desc> d(t.n);
        for (auto &q : d) {
            memset(&q, 0, sizeof q);
            q.format = S2_FMT_SRGB8;
            q.width = t.w, q.height = t.h;
            q.ref = q.dis = (const void *)64;
            q.ref_pitch = q.dis_pitch = (size_t)t.w * 3;
        }
        Plan P;
        if (e.plan(d.data(), t.n, P) != S2_OK) return printf("FAILED plan\n"), 1;
        double waves = 0;
        for (const DsPair &D : P.ds)
            for (int s = 0; s < kDsLevels; s++)
                waves += ds_strips_x(D.w[s]) * ((D.h[s] + 63) / 64) / (double)(kDsStripBlocks * e.num_sms);
        const bool slower = P.ds_rows && t.strips > t.tiles;
        const bool missed = !P.ds_rows && t.strips < t.tiles && waves >= 2;
        if (slower || missed || (P.ds_rows != 0 && P.ds_rows != 64)) {
            fails++;
            printf("%d x %ux%u: rows %d, tiles %.0f strips %.0f us\n", t.n, t.w, t.h, P.ds_rows, t.tiles, t.strips);
        }
        // the strips cover every level: as many blocks as the launch starts
        int strips = 0;
        for (const DsSeg &g : P.dsegs) {
            if (P.ds_rows && g.first_strip != strips) fails++;
            const DsPair &D = P.ds[g.pair];
            if (P.ds_rows) strips += ds_strips_x(D.w[g.level]) * ((D.h[g.level] + P.ds_rows - 1) / P.ds_rows);
        }
        if (strips != P.ds_strips) fails++;
    }
    printf("%s fails=%d\n", fails ? "FAILED" : "OK", fails);
    return fails ? 1 : 0;
}
