/* one scenario of the field transfers over the fake runtime; exit code 0 where
 * what the header promises holds */
#include "hostio.cu"

#include <stdio.h>
#include <unistd.h>

#include <new>
#include <string>

static thread_local bool out_of_memory = false;
void *operator new(size_t n) {
    void *p = out_of_memory ? nullptr : malloc(n);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }

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

/* a field there and back on a stream of its own */
int round_trip(FakeStream &s, int nx, int ny) {
    Field f(nx, ny, 3.0f);
    std::vector<float> back(f.host.size());
    CHECK(gc_field_upload(f.dev, f.row(), f.host.data(), nx, ny, &s) == GC_OK);
    CHECK(gc_field_download(back.data(), f.dev, f.row(), nx, ny, &s) == GC_OK);
    CHECK(back == f.host && f.there(f.host.data()));
    return 0;
}

/* transfers on stream B end while those on stream A wait for A's earlier work:
 * `uploads` of them queued, then a blocking one (a download, or an upload that
 * needs its buffers again) in a thread */
int beside(int nx, int ny, int uploads, bool down) {
    FakeStream a, b;
    a.open = false;
    std::vector<Field> q;
    q.reserve(uploads + 1);
    for (int k = 0; k <= uploads; k++) q.emplace_back(nx, ny, 10.0f * k);
    std::vector<float> back(q[0].host.size());
    fake::push(&a, [] {}); /* the earlier work */
    for (int k = 0; k < uploads; k++)
        CHECK(gc_field_upload(q[k].dev, q[k].row(), q[k].host.data(), nx, ny, &a) == GC_OK);
    int rc = GC_OK;
    bool before_ok = true;
    std::thread t([&] {
        rc = down ? gc_field_download(back.data(), q[0].dev, q[0].row(), nx, ny, &a)
                  : gc_field_upload(q[uploads].dev, q[uploads].row(), q[uploads].host.data(), nx, ny, &a);
    });
    for (const cudaError_t before : {cudaSuccess, cudaErrorInvalidValue}) {
        /* an error that the caller has not fetched yet stays to be fetched, and none is left behind */
        fake::last = before;
        if (round_trip(b, nx, ny)) before_ok = false;
        before_ok = before_ok && cudaGetLastError() == before;
    }
    usleep(200000); /* the thread is waiting by now; were it not, the check would only be weaker */
    const int mine = round_trip(b, nx, ny) || round_trip(b, 300, 300);
    fake::set_open(&a, true);
    t.join();
    CHECK(before_ok && mine == 0 && rc == GC_OK && cudaStreamSynchronize(&a) == cudaSuccess);
    for (int k = 0; k < (down ? uploads : uploads + 1); k++) CHECK(q[k].there(q[k].host.data()));
    CHECK(!down || uploads == 0 || back == q[0].host);
    return 0;
}

/* a thread whose current device is not the stream's */
int foreign(int nx, int ny) {
    FakeStream s;
    s.device = 1;
    CHECK(round_trip(s, nx, ny) == 0);
    CHECK(fake::device == 0);
    return 0;
}

/* device memory on the caller's side: the runtime's own copies, no host access */
int device_caller(int nx, int ny) {
    CHECK(source(nx, ny, cudaMemoryTypeDevice) == 0 && fake::device_callers == 1);
    FakeStream s;
    Field f(nx, ny, 2.0f);
    float *to = (float *)fake::make(f.host.size() * sizeof(float), cudaMemoryTypeDevice);
    CHECK(gc_field_upload(f.dev, f.row(), f.host.data(), nx, ny, &s) == GC_OK);
    CHECK(gc_field_download(to, f.dev, f.row(), nx, ny, &s) == GC_OK && fake::device_callers == 2);
    CHECK(memcmp(to, f.host.data(), f.host.size() * sizeof(float)) == 0);
    return 0;
}

/* memory that work on the stream writes before an upload or reads after a
 * download: the transfer is in stream order, not ahead of it */
int ordered(int nx, int ny, cudaMemoryType kind) {
    FakeStream s;
    Field f(nx, ny, 5.0f);
    const size_t bytes = f.host.size() * sizeof(float);
    float *h = (float *)fake::make(bytes, kind);
    fake::push(&s, [&] { memcpy(h, f.host.data(), bytes); });
    CHECK(gc_field_upload(f.dev, f.row(), h, nx, ny, &s) == GC_OK);
    CHECK(cudaStreamSynchronize(&s) == cudaSuccess && f.there(f.host.data()));
    std::vector<float> seen(f.host.size());
    memset(h, 0xff, bytes);
    fake::push(&s, [&] { memcpy(seen.data(), h, bytes); });
    CHECK(gc_field_download(h, f.dev, f.row(), nx, ny, &s) == GC_OK && memcmp(h, f.host.data(), bytes) == 0);
    CHECK(memcmp(seen.data(), f.host.data(), 4) != 0); /* the reader that came first saw what was there */
    return 0;
}

/* a copy that can have no threads is made by its caller */
int no_memory(size_t bytes) {
    std::vector<char> a(bytes), b(bytes);
    for (size_t k = 0; k < bytes; k++) a[k] = (char)(k * 7 + k / 251);
    out_of_memory = true;
    const int rc = gc_host_copy(b.data(), a.data(), (long long)bytes);
    out_of_memory = false;
    CHECK(rc == GC_OK && a == b);
    return 0;
}

} // namespace

int main(int argc, char **argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    const int nx = argc > 2 ? atoi(argv[2]) : 200, ny = argc > 3 ? atoi(argv[3]) : 200;
    if (what == "pageable") return source(nx, ny, cudaMemoryTypeUnregistered);
    if (what == "locked") return source(nx, ny, cudaMemoryTypeHost);
    if (what == "managed") return source(nx, ny, cudaMemoryTypeManaged);
    alarm(20); /* a transfer that waits for another stream's work would wait for good */
    if (what == "beside-read") return beside(nx, ny, 0, true);
    if (what == "beside-queued-read") return beside(nx, ny, 1, true);
    if (what == "beside-upload") return beside(nx, ny, 2, false);
    if (what == "foreign-device") return foreign(nx, ny);
    if (what == "device-caller") return device_caller(nx, ny);
    if (what == "ordered-locked") return ordered(nx, ny, cudaMemoryTypeHost);
    if (what == "ordered-managed") return ordered(nx, ny, cudaMemoryTypeManaged);
    if (what == "ordered-device") return ordered(nx, ny, cudaMemoryTypeDevice);
    if (what == "no-memory") return no_memory((size_t)9 << 20);
    printf("no scenario %s\n", what.c_str());
    return 2;
}
