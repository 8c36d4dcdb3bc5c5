// Device colouring (exact sequential-greedy result, computed in parallel).
#pragma once
#include "world.cuh"

namespace cc {

constexpr uint32_t kMaxColors = 4096;

struct ColorView {
    uint32_t n;
    const uint32_t* lo_off;  // [n+1] lower-index neighbours of the material graph
    const uint32_t* lo;
    const uint4* head;       // [2n] .x, .y of each pair: first entry and length of the vertex's list in nb
    const uint32_t* nb;      // neighbours of the material graph
    ContactsView contacts;
    uint64_t n_incident;  // entries of contacts.inc
    int grab_active;
    uint32_t grab_v[3];
};

class Coloring {
   public:
    // lo_total: entries of the material graph's lower-neighbour lists
    void init(uint32_t n, uint64_t lo_total, cudaStream_t s);
    // Recompute the colouring for the current graph, starting from the last one.
    void compute(const ColorView& view, cudaStream_t s);
    uint32_t n_colors() const { return n_colors_; }
    const std::vector<uint32_t>& offsets() const { return offsets_h_; }
    const uint32_t* order() const { return order_.ptr; }
    const uint16_t* colors() const { return cur_; }
    // device word that receives DERR_SORT_WAIT if the colour sort's wait gives up
    void set_error_word(unsigned int* w) { error_word_ = w; }
    size_t last_iterations() const { return last_iterations_; }
    void download(std::vector<uint32_t>& colors);
    uint64_t launches() const { return launches_; }

   private:
    uint32_t n_ = 0;
    uint64_t lo_total_ = 0;
    DBuf<uint32_t> adj_;   // distinct lower neighbours of every vertex (k_color_rows)
    DBuf<uint4> row_head_;
    DBuf<uint16_t> a_, b_;
    uint16_t* cur_ = nullptr;
    DBuf<uint32_t> order_, iota_;
    // a colouring's words, cleared and read back as one: rounds, error, n - first failing vertex, (unused), vertices
    // per colour; behind them (not read back) the walk's dirty bits
    static constexpr size_t kWords = 4 + kMaxColors;
    DBuf<uint32_t> words_;
    Pinned<uint32_t> words_h_;
    RadixSorter sorter_;
    unsigned int* error_word_ = nullptr;  // receives DERR_SORT_WAIT (set_error_word)
    std::vector<uint32_t> offsets_h_;
    uint32_t n_colors_ = 0;
    size_t last_iterations_ = 0;
    uint64_t launches_ = 0;
};

}  // namespace cc
