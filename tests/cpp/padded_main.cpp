// Checks of the padded y pass: every line smoothed once, in runs of at least 32
// lines, and a padded copy no larger than a run needs; the copy itself.

static long check_runs(int yn, uint64_t nlines) {
    const int pitch = (yn + 7) & ~7;
    DevBuf ckpt, pad;
    std::vector<float> origin(1);
    g_work = origin.data();
    g_pad = &pad;
    g_runs.clear();
    g_accept = 1 << 30;
    g_fits = true;
    launch_smooth_y_padded(nullptr, g_work, yn, pitch, nlines, 3.0f, nullptr, ckpt, pad, nullptr);
    uint64_t next = 0, most = 0;
    long bad = 0;
    for (const Run &r : g_runs) {
        bad += r.first != next || r.lines < std::min<uint64_t>(32, nlines);
        next += r.lines;
        most = std::max(most, r.lines);
    }
    bad += next != nlines || !g_fits;
    bad += pad.cap > (most + 32) * (uint64_t)pitch * 2;  // no more than the longest run's lines
    bad += pad.cap > nlines * (uint64_t)pitch * 2;       // nor than the volume's
    if (bad) std::printf("runs of %d x %llu: %ld faults, copy of %zu bytes\n", yn, (unsigned long long)nlines, bad, pad.cap);
    return bad;
}

static long check_copy(int yn, uint64_t nlines) {
    const int pitch = (yn + 7) & ~7;
    std::vector<uint16_t> src(yn * nlines);
    for (size_t i = 0; i < src.size(); ++i) src[i] = (uint16_t)(i * 40503u >> 3);
    DevBuf ckpt, pad;
    std::vector<float> origin(1);
    g_work = origin.data();
    g_pad = &pad;
    g_runs.clear();
    g_accept = 1 << 30;
    g_copy = true;
    launch_smooth_y_padded(src.data(), g_work, yn, pitch, nlines, 3.0f, nullptr, ckpt, pad, nullptr);
    g_copy = false;
    const uint16_t *p = g_runs.at(0).buf;
    long bad = 0;
    for (uint64_t l = 0; l < nlines; ++l)
        for (int y = 0; y < pitch; ++y) bad += p[l * pitch + y] != (y < yn ? src[l * yn + y] : 0);
    if (bad) std::printf("copy of %d x %llu: %ld faults\n", yn, (unsigned long long)nlines, bad);
    return bad;
}

// launch_smooth: padded lines where every run is taken, else the passes of
// unpadded lines over the whole volume, and the pitch that the image then has
static long check_fallback() {
    DevBuf ckpt, pad;
    std::vector<float> origin(1);
    std::vector<uint16_t> img(1);
    g_work = origin.data();
    g_pad = &pad;
    long bad = 0;
    for (int accept : {0, 1, 2, 1 << 30}) {
        g_accept = accept;
        g_passes.clear();
        const int pitch = launch_smooth<float>(img.data(), g_work, 517, 400, 400, 520, 3.0f, nullptr, nullptr, ckpt,
                                               pad, nullptr);
        const bool padded = accept >= 2;  // two runs
        bad += pitch != (padded ? 520 : 517) || g_passes != (padded ? "x520 z520 " : "yx517 z517 ");
    }
    if (bad) std::printf("refused layouts: %ld faults\n", bad);
    return bad;
}

int main() {
    long bad = 0;
    bad += check_fallback();
    for (int yn : {65, 66, 67, 129, 517, 1013, 4095, 65534}) {
        const uint64_t step = std::max<uint64_t>(1024, (uint64_t(1) << 26) / ((yn + 7) & ~7));
        // the smallest volume that is padded, whole runs, and rests of 1 .. 33 lines
        for (uint64_t n : {(uint64_t(1) << 20) / yn + 1, step - 1, step, step + 1, step + 31, step + 32, step + 33,
                           2 * step, 2 * step + 31, 2 * step + 32, 3 * step + 1})
            if (n >= 32) bad += check_runs(yn, n);
    }
    for (int yn : {65, 66, 67, 70}) bad += check_copy(yn, 33);
    std::printf("faults %ld\n", bad);
    return bad != 0;
}
