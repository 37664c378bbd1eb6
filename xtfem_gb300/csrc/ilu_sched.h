// ilu_sched.h -- host form of a triangular factor's level schedule and small
// host helpers shared by the sweep builders (dev_ilu.cu, dev_ilu_rows.cu).
#pragma once

#include <algorithm>
#include <cstdlib>
#include <exception>
#include <string>
#include <thread>
#include <vector>

#include "xt_device.h"

namespace xt {

constexpr int kMaxG = 3;

struct TriHost {
    int ngroups = 0, nlevels = 0, g = 1, maxw = 0;
    std::vector<int> level_ptr, group_row0, ext_ptr, ext_col;
    std::vector<double> ext_v, int_v, dinv;
    std::vector<int> order;  // level order -> group id
    std::vector<int> pos;    // group id -> level-order position
    std::vector<int> slot;   // group id -> window slot
    int nslots = 0;
    std::vector<double> minv;  // level order, g*g: inverse of the group's diagonal block
};

// Both schedules, kept on the host to build staged sweeps on first use.
struct IluSched {
    TriHost L, U;
};

// The device error word that ilu_check reads (dev_ilu.cu).
int ilu_error_word(int** p);

inline int max_dyn_smem()
{
    static const int v = [] {
        int dev = 0, r = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&r, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
            r = 48 * 1024;
        return r;
    }();
    return v;
}

inline bool trace_on() { return std::getenv("XTFEM_TRACE") != nullptr; }

// Runs a() on a second host thread (on the caller's device) while b() runs
// on this one; returns the first failure, its message set on this thread
// (an exception in a() becomes XT_ERR_HOST; one in b() is rethrown after
// the join).
template <class A, class B>
int side_by_side(A&& a, B&& b)
{
    int dev = 0;
    XT_CUDA(cudaGetDevice(&dev));
    int ra = XT_OK;
    std::string ea;
    std::thread t([&] {
        try {
            if (cudaSetDevice(dev) != cudaSuccess) {
                ra = XT_ERR_CUDA;
                ea = "could not select the device on a helper thread";
                return;
            }
            ra = a();
            if (ra != XT_OK) ea = last_error();
        } catch (const std::exception& e) {
            ra = XT_ERR_HOST;
            ea = e.what();
        }
    });
    int rb = XT_OK;
    try {
        rb = b();
    } catch (...) {
        t.join();
        throw;
    }
    t.join();
    if (ra != XT_OK) {
        set_error(ea);
        return ra;
    }
    return rb;
}

// fn(begin, end) over [0, n), shared among as many host threads (eight at most)
// as get `least` items each; an exception is rethrown once all have ended.
template <class F>
void shared_out(size_t n, size_t least, F&& fn)
{
    const size_t hw = std::max(1u, std::thread::hardware_concurrency());
    const size_t T = std::max<size_t>(1, std::min({n / least, hw, (size_t)8}));
    std::vector<std::exception_ptr> err(T);
    auto part = [&](size_t k) {
        try {
            fn(n * k / T, n * (k + 1) / T);
        } catch (...) {
            err[k] = std::current_exception();
        }
    };
    std::vector<std::thread> th;
    th.reserve(T);
    size_t k = 1;
    try {
        for (; k < T; ++k) th.emplace_back(part, k);
    } catch (const std::exception&) {  // no more threads: the rest here
    }
    part(0);
    for (; k < T; ++k) part(k);
    for (std::thread& t : th) t.join();
    for (const std::exception_ptr& e : err)
        if (e) std::rethrow_exception(e);
}

inline int env_int(const char* name, int dflt)
{
    const char* e = std::getenv(name);
    return e ? std::atoi(e) : dflt;
}

// Polls of a ring wait for a level's data.  XTFEM_ILU_SPIN_LIMIT=N makes it
// N - 1, so that 1 gives up at once whatever has landed (tests make a wait run
// out with the GPU still answering).
inline int ring_polls()
{
    const int n = env_int("XTFEM_ILU_SPIN_LIMIT", 0);
    return n > 0 ? n - 1 : 1 << 20;
}

}  // namespace xt
