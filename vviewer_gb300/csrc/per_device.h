// Values that belong to a device and are made once for it.
#pragma once
#include <map>
#include <mutex>

namespace vvpt {

// get() returns device `device`'s value, made by the first caller while others
// wait for it; values stay where they are.
template <class T>
class PerDevice {
public:
    template <class Make>
    const T &get(int device, Make make)
    {
        std::lock_guard<std::mutex> lk(m_mu);
        auto it = m_values.find(device);
        if (it == m_values.end())
            it = m_values.emplace(device, make()).first;
        return it->second;
    }

private:
    std::mutex m_mu;
    std::map<int, T> m_values;
};

}  // namespace vvpt
