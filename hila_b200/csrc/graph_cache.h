// Executable graphs of the engine by the launches they hold, the least recently used given up
// first (no CUDA types: a CPU test drives it).
#pragma once

#include <cstddef>

namespace hw {

template <class Exec, std::size_t N, void (*Destroy)(Exec)>
class GraphCache {
  public:
    ~GraphCache() { clear(); }
    // the graph of a key, or null
    Exec find(unsigned key) {
        for (Entry &e : e_)
            if (e.exec && e.key == key) {
                e.used = ++clock_;
                return e.exec;
            }
        return Exec();
    }
    // whether put() gives a graph up (which must not be running then)
    bool full() const {
        for (const Entry &e : e_)
            if (!e.exec) return false;
        return true;
    }
    void put(unsigned key, Exec exec) {
        Entry *at = &e_[0];
        for (Entry &e : e_) {
            if (!e.exec) {
                at = &e;
                break;
            }
            if (e.used < at->used) at = &e;
        }
        if (at->exec) Destroy(at->exec);
        *at = {key, ++clock_, exec};
    }
    void clear() {
        for (Entry &e : e_) {
            if (e.exec) Destroy(e.exec);
            e = Entry();
        }
    }

  private:
    struct Entry {
        unsigned key = 0;
        unsigned long long used = 0;
        Exec exec = Exec();
    };
    Entry e_[N];
    unsigned long long clock_ = 0;
};

}  // namespace hw
