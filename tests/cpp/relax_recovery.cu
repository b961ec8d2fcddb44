// relax_recovery.cu -- the 2D model's counting sort after a device error. Built with the model's own
// source, so that the error word and the counts, which nothing outside sets, can be set here: an
// error clears the handle's trust in its counts, whatever a refused step left in them, and the next
// step is a fresh handle's.
#include "../../libcl_gb300/csrc/fluid2d.cu"

#include <cstdio>

#define CHECK(x)                                                  \
    do {                                                          \
        if (!(x)) {                                               \
            std::printf("line %d: %s\n", __LINE__, #x);           \
            return 1;                                             \
        }                                                         \
    } while (0)

static const size_t N = 3000;

static int make(gbsph_fluid2d_t* f) {
    CHECK(gbsph_fluid2d_create(f) == GBSPH_OK);
    CHECK(gbsph_fluid2d_compile(*f) == GBSPH_OK);
    CHECK(gbsph_fluid2d_set_particle_count(*f, N) == GBSPH_OK);
    return 0;
}

static int fill(gbsph_fluid2d_t f) {
    std::vector<float> st(6 * N, 0.f);
    for (size_t i = 0; i < N; i++) {
        st[6 * i] = 2.f + 0.05f * (float)(i % 60) + 0.003f * (float)(i % 7);
        st[6 * i + 1] = 2.f + 0.05f * (float)(i / 60) + 0.002f * (float)(i % 11);
        st[6 * i + 4] = 0.7f;
    }
    CHECK(cudaMemcpy(gbsph_fluid2d_get_buffer(f, GBSPH2D_BUF_STATE, nullptr), st.data(), st.size() * 4, cudaMemcpyHostToDevice) == cudaSuccess);
    return 0;
}

static int zero_counts(gbsph_fluid2d_t f, bool* zero) {
    std::vector<uint32_t> c(count_words(f->table));
    CHECK(cudaMemcpy(c.data(), f->count, c.size() * 4, cudaMemcpyDeviceToHost) == cudaSuccess);
    *zero = std::all_of(c.begin(), c.end(), [](uint32_t v) { return v == 0; });
    return 0;
}

int main() {
    gbsph_fluid2d_t f = nullptr, g = nullptr;
    if (make(&f) || make(&g) || fill(f) || fill(g)) return 1;
    bool zero = false;
    if (zero_counts(f, &zero)) return 1;  // as allocated
    CHECK(zero);
    for (int i = 0; i < 2; i++) CHECK(gbsph_fluid2d_compute(f, nullptr) == GBSPH_OK);
    CHECK(gbsph_fluid2d_sync_status(f, nullptr) == GBSPH_OK);
    if (zero_counts(f, &zero)) return 1;  // as a step leaves them
    CHECK(zero && f->count_clean);

    const uint32_t bits = DEV_ERR_KEY_RANGE;
    CHECK(cudaMemcpy(f->err, &bits, 4, cudaMemcpyHostToDevice) == cudaSuccess);
    CHECK(gbsph_fluid2d_sync_status(f, nullptr) != GBSPH_OK);
    CHECK(!f->count_clean);
    const std::vector<uint32_t> left(count_words(f->table), 3u);
    CHECK(cudaMemcpy(f->count, left.data(), left.size() * 4, cudaMemcpyHostToDevice) == cudaSuccess);
    if (fill(f)) return 1;
    std::vector<float> a(6 * N), b(6 * N);
    for (gbsph_fluid2d_t h : {f, g}) {
        for (int i = 0; i < 2; i++) CHECK(gbsph_fluid2d_compute(h, nullptr) == GBSPH_OK);
        CHECK(gbsph_fluid2d_sync_status(h, nullptr) == GBSPH_OK);
        CHECK(cudaMemcpy(h == f ? a.data() : b.data(), gbsph_fluid2d_get_buffer(h, GBSPH2D_BUF_STATE, nullptr), a.size() * 4,
                         cudaMemcpyDeviceToHost) == cudaSuccess);
    }
    CHECK(std::memcmp(a.data(), b.data(), a.size() * 4) == 0);
    CHECK(gbsph_fluid2d_destroy(f) == GBSPH_OK && gbsph_fluid2d_destroy(g) == GBSPH_OK);
    std::printf("OK\n");
    return 0;
}
