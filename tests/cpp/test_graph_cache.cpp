// The engine's cache of executable graphs (hila_b200/csrc/graph_cache.h).  No GPU involved.
#include <cstdio>

#include "graph_cache.h"

static int alive = 0;
struct Graph {
    int id;
};
static void destroy(Graph *g) {
    alive--;
    delete g;
}

int main() {
    int failures = 0, builds = 0;
    {
        hw::GraphCache<Graph *, 4, destroy> C;
        auto get = [&](unsigned key) {
            Graph *g = C.find(key);
            if (!g) {
                builds++;
                alive++;
                C.put(key, g = new Graph{(int)key});
            }
            if (g->id != (int)key) failures++;
            return g;
        };
        for (int k = 0; k < 100; k++) get(k & 1);  // a stream that goes back and forth builds twice
        if (builds != 2) failures++;
        get(2), get(3);
        if (!C.full() || builds != 4) failures++;
        get(0);
        get(4);  // gives up the least recently used, 1
        if (alive != 4 || C.find(1) || !C.find(0) || !C.find(4)) failures++;
        for (unsigned k = 0; k < 1000; k++) get(k % 7);  // bounded
        if (alive != 4) failures++;
        C.clear();
        if (alive != 0 || C.find(0) || C.full()) failures++;
        get(5);
    }
    if (alive != 0) failures++;
    if (failures == 0) std::printf("graph cache passed\n");
    return failures;
}
