// Test harness (host only): the arithmetic of the parallel ordered float sums (film.cu, which it
// includes) on the CPU.  The increments are __host__ __device__, so what the kernels compose is
// checked here, addend by addend, without a GPU.
#include "../../mcrt_gb300/csrc/film.cu"

#include <cstring>

namespace mcrt {
// what film.cu takes from the rest of the library (its entry points are not called here)
int   set_error(int code, const std::string&) { return code; }
void* thread_scratch(int, size_t, bool& failed)
{
    failed = false;
    return nullptr;
}
}  // namespace mcrt

namespace {
unsigned bits_of(float f)
{
    unsigned u;
    std::memcpy(&u, &f, sizeof(u));
    return u;
}
float float_of(unsigned u)
{
    float f;
    std::memcpy(&f, &u, sizeof(f));
    return f;
}
}  // namespace

// what adding the float with these bits does to an even / odd multiple in binade e
extern "C" void film_sums_inc(unsigned bits, int e, int* out)
{
    const mcrt::Inc r = mcrt::inc_of(bits, e);
    out[0] = r.a[0];
    out[1] = r.a[1];
}

// The ordered sum of x[0 .. n) as the kernels make it: runs of `run` addends are composed as a tree
// of pairs, and a run in which the sum leaves its binade is redone addend by addend.  redone: runs
// redone; ties[0 / 1]: exact ties of a sum that stays in its binade, at an even / odd multiple.
extern "C" float film_sums_ordered(const float* x, long long n, int run, long long* redone, long long* ties)
{
    using namespace mcrt;
    float s = 0.f;
    *redone = 0;
    ties[0] = ties[1] = 0;
    Inc tree[1024];
    for (long long k = 0; k < n; k += run)
    {
        const int      count = static_cast<int>(n - k < run ? n - k : run);
        const unsigned b = bits_of(s);
        const int      e = binade(b), m = multiple(b);
        for (int j = 0; j < count; ++j) tree[j] = inc_of(bits_of(x[k + j]), e);
        int width = count;
        for (; width > 1; width = (width + 1) / 2)
            for (int j = 0; j < width; j += 2) tree[j / 2] = j + 1 < width ? inc_then(tree[j], tree[j + 1]) : tree[j];
        if (m + tree[0].a[m & 1] < kFull)
        {
            int at = m;
            for (int j = 0; j < count; ++j)
            {
                const Inc one = inc_of(bits_of(x[k + j]), e);
                if (one.a[0] != one.a[1]) ++ties[at & 1];
                at += one.a[at & 1];
            }
            s = float_of(float_from(m + tree[0].a[m & 1], e));
            continue;
        }
        ++*redone;
        for (int j = 0; j < count; ++j) s += x[k + j];
    }
    return s;
}
