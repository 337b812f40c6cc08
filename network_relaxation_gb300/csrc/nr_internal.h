/* Internal declarations shared by the host C++ and CUDA translation units. */
#ifndef NR_INTERNAL_H
#define NR_INTERNAL_H

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <new>
#include <string>
#include <thread>
#include <vector>

#include "../../include/netrelax.h"

struct nr_host_network {
    int n_points = 0;
    double offset = 0, miny = 0, maxy = 0;
    std::vector<double> points;       // 2N
    std::vector<int> edge_ij;         // 2E
    std::vector<double> edge_l0;      // E
    std::vector<signed char> edge_wrap;
    std::vector<int> tri_hjk;         // 3T
    std::vector<signed char> tri_wrap;// 2T
    std::vector<double> bond_k;       // empty or E
    std::vector<double> tri_kb;       // empty or T
    std::vector<double> tri_phi0;     // empty or T
    // network-mesh composites (network_mesh_relax.cu): FEM triangles, their
    // areas, pairs of duplicate vertices on the left / right edges, x range
    std::vector<int> facets;          // 3F
    std::vector<double> areas;        // F
    std::vector<int> mesh_pairs;      // 2P
    double minx = 0, maxx = 0;
    int n_edges() const { return (int)edge_l0.size(); }
    int n_triples() const { return (int)(tri_hjk.size() / 3); }
    int n_facets() const { return (int)(facets.size() / 3); }
    int n_mesh_pairs() const { return (int)(mesh_pairs.size() / 2); }
};

namespace nr {

/* Thread-local error message + status helper. */
int fail(int status, const std::string &msg);
void clear_error();

/* f()'s status; NR_ERR_OOM when host memory runs out in it (an exception must
 * not leave a C function). */
template <class F>
int no_throw(F f) {
    try {
        return f();
    } catch (const std::bad_alloc &) {
        return fail(NR_ERR_OOM, "no host memory"); /* fits a string without memory of its own */
    }
}

/* work(k) for every k < n, on n host threads (the caller's is one).  A thread
 * that cannot be started leaves its part to the caller's; an exception in one is
 * thrown here once all have ended. */
template <class F>
void run_threads(int n, F work) {
    std::atomic<bool> thrown{false};
    std::exception_ptr error;
    auto guarded = [&](int k) {
        try {
            work(k);
        } catch (...) {
            if (!thrown.exchange(true)) error = std::current_exception();
        }
    };
    std::vector<std::thread> ts;
    int started = 1;
    try {
        ts.reserve(n);
        for (; started < n; ++started) ts.emplace_back(guarded, started);
    } catch (...) { /* std::system_error: no thread; bad_alloc: no room for its state */
    }
    guarded(0);
    for (int k = started; k < n; ++k) guarded(k);
    for (auto &t : ts) t.join();
    if (error) std::rethrow_exception(error);
}

/* An object's device memory: bytes that are uploaded, and behind them memory
 * that starts as zeros (zeros(): offsets from zeros_at()). */
class Image {
public:
    Image() = default;
    Image(const Image &) = delete;
    Image &operator=(const Image &) = delete;
    ~Image() { std::free(p_); }
    char *data() { return p_; }
    size_t size() const { return n_; }
    size_t add(size_t nbytes) { /* to be written by the caller */
        const size_t off = up(n_), end = off + nbytes;
        if (end > cap_) {
            cap_ = std::max(end, cap_ + cap_ / 2);
            char *const q = (char *)std::realloc(p_, cap_);
            if (!q) throw std::bad_alloc();
            p_ = q;
        }
        std::memset(p_ + n_, 0, off - n_);
        n_ = end;
        return off;
    }
    template <class T>
    size_t put(const T *src, size_t n) {
        const size_t off = add(n * sizeof(T));
        if (n) std::memcpy(p_ + off, src, n * sizeof(T));
        return off;
    }
    size_t zeros(size_t nbytes) {
        const size_t off = up(n_zeros_);
        n_zeros_ = off + nbytes;
        return off;
    }
    size_t zeros_at() const { return up(n_); }
    size_t zeros_size() const { return n_zeros_; }
    size_t total() const { return zeros_at() + n_zeros_; }

private:
    static size_t up(size_t n) { return (n + 255) / 256 * 256; }
    char *p_ = nullptr;
    size_t n_ = 0, cap_ = 0, n_zeros_ = 0;
};

/* A launch-policy knob: the environment variable `name`, else the tuning
 * table's entry of that name (tuning.cu), else null. */
const char *knob(const char *name);

/* Per-node incidence lists in canonical order: every bond (in index order,
 * first endpoint before second) and every triple (in index order, hinge, j,
 * k) touching the node.  Entry encodings: bond (b << 1) | role,
 * triple (t << 2) | role. */
struct Incidence {
    std::vector<int> bptr, bent, tptr, tent;
};
void build_incidence(int n_points, const int *edge_ij, int n_edges, const int *tri_hjk, int n_triples, bool use_bonds,
                     bool use_triples, Incidence &inc);

/* Per-node gel element entries 3 e + vertex, elements in index order
 * (eptr[N + 1], eent[3F]), and each node's duplicate partner (-1: none).
 * False when a vertex is in more than one pair (or paired with itself). */
bool element_incidence(const nr_host_network &h, std::vector<int> &eptr, std::vector<int> &eent,
                       std::vector<int> &partner);

/* Min/max y in the reader's convention (min starts at FLT_MAX, max at
 * FLT_MIN). */
void y_range(const std::vector<double> &points, double &miny, double &maxy);

/* n xy pairs written as "%2.10le\t%2.10le\n" lines (report_displaced,
 * large_strain_relax.cu:216-227), formatted in parallel. */
bool write_xy_file(const std::string &name, const double *xy, long n);

/* The duplicate-vertex search of read_network_mesh
 * (network_mesh_relax.cu:219-227): 2P indices. */
void find_mesh_pairs(const std::vector<double> &points, double offset, double minx, std::vector<int> &pairs);

}  // namespace nr

#endif
