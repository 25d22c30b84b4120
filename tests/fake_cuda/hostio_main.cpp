/* one scenario of the field transfers over the fake runtime; exit code 0 where
 * what the header promises holds */
#include "hostio.cu"

#include <stdio.h>

#include <string>

namespace {

struct Field {
    int nx, ny, pitch;
    std::vector<float> host;
    float *dev;
    Field(int nx, int ny, float v) : nx(nx), ny(ny), pitch((nx + 31) / 32 * 32), host((size_t)nx * ny) {
        for (size_t k = 0; k < host.size(); k++) host[k] = v + (float)k;
        dev = (float *)fake::make((size_t)pitch * ny * sizeof(float), cudaMemoryTypeDevice);
    }
    size_t row() const { return (size_t)pitch * sizeof(float); }
    bool there(const float *want) const {
        for (int j = 0; j < ny; j++)
            if (memcmp(dev + (size_t)j * pitch, want + (size_t)j * nx, (size_t)nx * sizeof(float))) return false;
        return true;
    }
};

#define CHECK(c)                                             \
    do {                                                     \
        if (!(c)) {                                          \
            printf("line %d: %s\n", __LINE__, #c);           \
            return 1;                                        \
        }                                                    \
    } while (0)

/* the caller's array may change as soon as an upload returned, whatever kind
 * of host memory it is */
int source(int nx, int ny, cudaMemoryType kind) {
    FakeStream s;
    Field f(nx, ny, 1.0f);
    float *h = kind == cudaMemoryTypeUnregistered ? f.host.data()
                                                  : (float *)fake::make(f.host.size() * sizeof(float), kind);
    const std::vector<float> want = f.host;
    memcpy(h, want.data(), want.size() * sizeof(float));
    CHECK(gc_field_upload(f.dev, f.row(), h, nx, ny, &s) == GC_OK);
    memset(h, 0xff, want.size() * sizeof(float));
    CHECK(cudaStreamSynchronize(&s) == cudaSuccess);
    CHECK(f.there(want.data()));
    return 0;
}

} // namespace

int main(int argc, char **argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    const int nx = argc > 2 ? atoi(argv[2]) : 200, ny = argc > 3 ? atoi(argv[3]) : 200;
    if (what == "pageable") return source(nx, ny, cudaMemoryTypeUnregistered);
    if (what == "locked") return source(nx, ny, cudaMemoryTypeHost);
    if (what == "managed") return source(nx, ny, cudaMemoryTypeManaged);
    printf("no scenario %s\n", what.c_str());
    return 2;
}
