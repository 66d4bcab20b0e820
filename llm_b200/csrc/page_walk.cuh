// Which cache pages and keys the queries of a differential attention see: a causal window beside which a sequence's
// first keep_first tokens stay visible.
#pragma once

#include "common.cuh"

namespace llmb {

// The pages a range of query positions [first_pos, last_pos] sees: `sink_pages` pages from page 0, then
// pages first_page .. last_page.
struct PageWalk {
    int sink_pages, first_page, count;
    __device__ __forceinline__ int logical(int i) const { return i < sink_pages ? i : first_page + (i - sink_pages); }
};
__device__ __forceinline__ PageWalk page_walk(int first_pos, int last_pos, int window, int keep_first) {
    PageWalk w;
    int last_page = last_pos / LLMB_PAGE;
    w.first_page = 0;
    w.sink_pages = 0;
    if (window > 0) {
        int first_key = first_pos - window + 1;
        w.first_page = first_key > 0 ? first_key / LLMB_PAGE : 0;
        int sinks = keep_first > 0 ? (keep_first - 1) / LLMB_PAGE + 1 : 0;
        w.sink_pages = sinks < w.first_page ? sinks : w.first_page;
    }
    w.count = w.sink_pages + last_page - w.first_page + 1;
    return w;
}
__device__ __forceinline__ bool key_visible(int key, int pos, int window, int keep_first) {
    return key <= pos && (window == 0 || pos - key < window || key < keep_first);
}

}  // namespace llmb
