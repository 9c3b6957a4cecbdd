// A bounded memo of planning results.  Finding the best way to deal out a
// convolution takes milliseconds of host time; a network has few distinct
// geometries and every layer asks for each of them several times (forward,
// backward data and backward filter plans; every replica).
#pragma once

#include "conv_simt.cuh"

#include <list>
#include <mutex>
#include <utility>
#include <vector>

namespace dcb
{

inline std::vector<long long> plan_key(const ConvGeom& g, long long what, long long mode)
{
    std::vector<long long> k = {what, mode, num_sms(), g.n, g.c, g.k, g.xs_n, g.xs_c, g.ys_n, g.ys_c};
    for (int i = 0; i < 3; ++i)
        for (long long v : {(long long) g.in[i], (long long) g.out[i], (long long) g.f[i], (long long) g.pad[i],
                            (long long) g.stride[i], (long long) g.dil[i], g.xs[i], g.ys[i]})
            k.push_back(v);
    return k;
}

template <class T>
class PlanCache
{
public:
    // *out = the value kept for `key`, or what `make` returns (kept from then on)
    template <class F>
    void get(const std::vector<long long>& key, T* out, F make)
    {
        {
            std::lock_guard<std::mutex> lock(m_mutex);
            for (auto it = m_list.begin(); it != m_list.end(); ++it)
                if (it->first == key)
                {
                    m_list.splice(m_list.begin(), m_list, it);
                    *out = it->second;
                    return;
                }
        }
        *out = make();
        std::lock_guard<std::mutex> lock(m_mutex);
        m_list.emplace_front(key, *out);
        if (m_list.size() > 48) // tens of kilobytes each at most
            m_list.pop_back();
    }

private:
    std::mutex m_mutex;
    std::list<std::pair<std::vector<long long>, T>> m_list;
};

} // namespace dcb
