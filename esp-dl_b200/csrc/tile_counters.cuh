// Which pair of tile counters (sched_counters in abi.cu) belongs to whom: a stream, or a stream during one capture.  Plain C++; the
// caller holds a lock.
#pragma once
#include <map>
#include <utility>
#include <vector>

namespace espdl {

class TileCounters {
public:
    explicit TileCounters(int pairs) : m_pairs(pairs) {}
    // The pair of (capture id, 0 for none; stream), -1 when all are taken.
    int get(unsigned long long capture, const void *stream)
    {
        const Key key(capture, stream);
        auto it = m_taken.find(key);
        if (it != m_taken.end())
            return it->second;
        int pair = m_fresh;
        if (!m_free.empty())
            pair = m_free.back(), m_free.pop_back();
        else if (m_fresh < m_pairs)
            m_fresh++;
        else
            return -1;
        m_taken.emplace(key, pair);
        return pair;
    }
    // Every pair of a capture, or that of a stream: no launch that uses them is in flight or will be made.
    void give_back_capture(unsigned long long capture)
    {
        auto it = m_taken.lower_bound(Key(capture, nullptr));
        while (it != m_taken.end() && it->first.first == capture) {
            m_free.push_back(it->second);
            it = m_taken.erase(it);
        }
    }
    void give_back_stream(const void *stream)
    {
        auto it = m_taken.find(Key(0ull, stream));
        if (it == m_taken.end())
            return;
        m_free.push_back(it->second);
        m_taken.erase(it);
    }
    int taken() const { return (int)m_taken.size(); }

private:
    typedef std::pair<unsigned long long, const void *> Key;
    std::map<Key, int> m_taken;
    std::vector<int> m_free;
    int m_pairs, m_fresh = 0;
};

} // namespace espdl
