// fednl_heap.cuh -- the 4-ary heap of the TopK / TopLEK selection in shared memory, step by step as the
// reference's (dopt/dopt/math_routines/include/MinHeap.h, D = 4); see k_select for how its parts are used.
#pragma once

namespace fednl {

struct HeapS {
    unsigned long long* key;   // bits of |value|
    unsigned* hid;             // packed upper position p
};

// minHeapify, MinHeap.h:255-290.  The entry (ck, ci) enters at node i with the carried comparison
// value lv.  The reference walks the children in order and moves to a child whose value is
// strictly below the running value, so it lands on the leftmost child holding the children's
// minimum whenever that minimum is strictly below lv; the carried value then becomes that
// minimum (the value that moved up, not the entry being sifted).  A two-level tree with strict
// '<' finds the same child.  The key array is placed so that the four children 4i+1..4i+4 of a
// node start on a 32-byte boundary (two 16-byte loads), the id array so that they start on a
// 16-byte boundary.  The path moves up one node and (ck, ci) is written where the walk stops,
// which equals the reference's chain of swaps.
//
// kWarp: a whole warp makes the same call, every lane with the same values and the same stores.  Lanes may run
// apart, and a level's stores replace what that level's loads read, so the lanes meet in between.
template <bool kWarp = false>
__device__ __forceinline__ void heap_descend(HeapS& h, int i, int n, unsigned long long lv,
                                             unsigned long long ck, unsigned ci)
{
    for (;;) {
        const int f = 4 * i + 1;
        int lo;
        unsigned long long m;
        if (f + 3 < n) {
            const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(h.key + f);
            const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(h.key + f + 2);
            const bool r12 = a.y < a.x, r34 = b.y < b.x;
            const unsigned long long m12 = r12 ? a.y : a.x, m34 = r34 ? b.y : b.x;
            const bool r = m34 < m12;
            m = r ? m34 : m12;
            lo = f + (r ? (r34 ? 3 : 2) : (r12 ? 1 : 0));
        } else {
            if (f >= n) break;
            lo = f;
            m = h.key[f];
            for (int c = f + 1; c < n; ++c) {
                const unsigned long long cv = h.key[c];
                if (cv < m) {
                    m = cv;
                    lo = c;
                }
            }
        }
        if (!(lv > m)) break;
        const unsigned hl = h.hid[lo];
        if (kWarp) __syncwarp();
        h.key[i] = m;
        h.hid[i] = hl;
        i = lo;
        lv = m;
    }
    h.key[i] = ck;
    h.hid[i] = ci;
}

__device__ __forceinline__ void heap_sift(HeapS& h, int i, int heap_size)
{
    const unsigned long long kv = h.key[i];
    heap_descend(h, i, heap_size, kv, kv, h.hid[i]);
}

// increaseMinimumInMinHeap (MinHeap.h:78-85): the root takes (cand, p) and sifts down; returns the
// new root value, which the scanning warp compares against next
__device__ __forceinline__ unsigned long long heap_replace_root(HeapS& h, int k, unsigned long long cand, unsigned p)
{
    if (k < 5) {
        heap_descend(h, 0, k, cand, cand, p);
        return h.key[0];
    }
    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(h.key + 1);
    const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(h.key + 3);
    const bool r12 = a.y < a.x, r34 = b.y < b.x;
    const unsigned long long m12 = r12 ? a.y : a.x, m34 = r34 ? b.y : b.x;
    const bool r = m34 < m12;
    const unsigned long long m = r ? m34 : m12;
    if (!(cand > m)) {
        h.key[0] = cand;
        h.hid[0] = p;
        return cand;
    }
    const int lo = 1 + (r ? (r34 ? 3 : 2) : (r12 ? 1 : 0));
    h.key[0] = m;
    h.hid[0] = h.hid[lo];
    heap_descend(h, lo, k, m, cand, p);
    return m;
}

// The heap's top in registers (at least 21 entries, so levels 0-2 are complete): the root's key and id
// (K0, I0) and the four level-1 keys sorted, s1 <= .. <= s4, equal keys by node (t: node 1..4, and bit 3
// set if the key is above the least of the node's children).  An entry that enters at the root is
// compared with all of them at once: against s1 it decides the new root, against s2..s4 the place of
// the value that replaces s1 (a tree over unsorted keys makes three dependent comparisons, and the
// chain of comparisons is what a step costs).  The level-1 ids and the least child keys (mn, by node)
// and positions stay in shared memory, those of the node of s1 loaded ahead (i1, m1, g1).
struct HeapMins {
    unsigned long long mn[5];   // least child's key, by node
    int gp[5];                  // its position
};

struct HeapTop {
    unsigned long long K0, s1, s2, s3, s4, m1;
    unsigned I0, i1, t1, t2, t3, t4;
    int g1;
    HeapMins* mins;             // shared

    // the least child of level-1 node s (the leftmost one): its key
    __device__ __forceinline__ unsigned long long children(const HeapS& h, unsigned s)
    {
        const int f = 4 * (int)s + 1;
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(h.key + f);
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(h.key + f + 2);
        const bool s01 = a.y < a.x, s23 = b.y < b.x;
        const unsigned long long n01 = s01 ? a.y : a.x, n23 = s23 ? b.y : b.x;
        const bool sr = n23 < n01;
        const unsigned long long m = sr ? n23 : n01;
        mins->gp[s] = f + (sr ? (s23 ? 3 : 2) : (s01 ? 1 : 0));
        mins->mn[s] = m;
        return m;
    }
    __device__ __forceinline__ void ahead(const HeapS& h)
    {
        i1 = h.hid[t1 & 7];
        m1 = mins->mn[t1 & 7];
        g1 = mins->gp[t1 & 7];
    }
    __device__ __forceinline__ void load(const HeapS& h, HeapMins* m)
    {
        mins = m;
        K0 = h.key[0];
        I0 = h.hid[0];
        s1 = h.key[1]; s2 = h.key[2]; s3 = h.key[3]; s4 = h.key[4];
        t1 = 1u | (s1 > children(h, 1u) ? 8u : 0u);
        t2 = 2u | (s2 > children(h, 2u) ? 8u : 0u);
        t3 = 3u | (s3 > children(h, 3u) ? 8u : 0u);
        t4 = 4u | (s4 > children(h, 4u) ? 8u : 0u);
        auto order = [](unsigned long long& a, unsigned& ta, unsigned long long& b, unsigned& tb) {
            if (b < a || (b == a && (tb & 7u) < (ta & 7u))) {
                const unsigned long long x = a;
                a = b;
                b = x;
                const unsigned y = ta;
                ta = tb;
                tb = y;
            }
        };
        order(s1, t1, s2, t2);
        order(s3, t3, s4, t4);
        order(s1, t1, s3, t3);
        order(s2, t2, s4, t4);
        order(s2, t2, s3, t3);
        ahead(h);
    }
    __device__ __forceinline__ void store(HeapS& h) const
    {
        h.key[0] = K0;
        h.hid[0] = I0;
        h.key[t1 & 7] = s1; h.key[t2 & 7] = s2; h.key[t3 & 7] = s3; h.key[t4 & 7] = s4;
    }
    // The entry (ck, ci) enters at the root of a heap of n >= 21 entries with its own key as the
    // comparison value (MinHeap.h:78-85 and :125-141: heap_descend(h, 0, n, ck, ck, ci)), in two steps:
    // the new root, true if the entry goes below it; then its place below.  below() returns true if
    // entries in shared memory moved.  kWarp as for heap_descend: the lanes meet once all have read what the
    // entry replaces (its node's id by the last ahead(), the entry that moves up).
    __device__ __forceinline__ bool root(unsigned long long ck, unsigned ci)
    {
        const bool gt = ck > s1;
        K0 = gt ? s1 : ck;
        I0 = gt ? i1 : ci;
        return gt;
    }
    template <bool kWarp = false>
    __device__ __forceinline__ bool below(HeapS& h, int n, unsigned long long ck, unsigned ci)
    {
        const unsigned nd = t1 & 7u;
        const bool deeper = (t1 & 8u) != 0u;
        unsigned long long x = ck, xm = m1;
        unsigned xi = ci;
        if (deeper) {       // level 2: the least child of the node is below the value that moved up
            x = m1;
            xi = h.hid[g1];
        }
        if (kWarp) __syncwarp();
        if (deeper) {
            heap_descend<kWarp>(h, g1, n, m1, ck, ci);
            xm = children(h, nd);
        }
        h.hid[nd] = xi;
        const unsigned tx = nd | (x > xm ? 8u : 0u);
        // x after s_k: above it, or equal with the later node
        const bool a2 = x >= s2 + ((t2 & 7u) > nd ? 1u : 0u);
        const bool a3 = x >= s3 + ((t3 & 7u) > nd ? 1u : 0u);
        const bool a4 = x >= s4 + ((t4 & 7u) > nd ? 1u : 0u);
        s1 = a2 ? s2 : x;
        t1 = a2 ? t2 : tx;
        s2 = a2 ? (a3 ? s3 : x) : s2;
        t2 = a2 ? (a3 ? t3 : tx) : t2;
        s3 = a3 ? (a4 ? s4 : x) : s3;
        t3 = a3 ? (a4 ? t4 : tx) : t3;
        s4 = a4 ? x : s4;
        t4 = a4 ? tx : t4;
        ahead(h);
        return deeper;
    }
};

// Extractions (extracFromMinHeap, MinHeap.h:125-141) that bring the heap from `size` to `target` entries,
// by one thread: the last entry leaves for the root and the root for the last place.  While the heap has
// more than 21 entries its top is in `top` (live), and the next last entry is loaded a step ahead; the
// answer is whether it still is.  100 cycles a step; 208 with a tree of comparisons over unsorted keys
// (and the windows between the chunks), 290 with a warp-wide minimum over lanes holding the nodes (its
// votes, and ties that need the keys' lower words), 165 on 32-bit ranks after 116 k cycles of sorting.
__device__ __forceinline__ bool extract_chunk(HeapS& h, HeapTop& top, bool live, int size, int target)
{
    if (live) {
        const int stop = max(target, 21);
        if (size > stop) {
            unsigned long long LK = h.key[size - 1];
            unsigned LI = h.hid[size - 1];
            for (; size > stop; --size) {
                const int n = size - 1;                  // heap size after the swap
                const unsigned long long nk = h.key[n - 1];
                const unsigned ni = h.hid[n - 1];
                h.key[n] = top.K0;
                h.hid[n] = top.I0;
                const bool moved = top.root(LK, LI) && top.below(h, n, LK, LI);
                LK = moved ? h.key[n - 1] : nk;
                LI = moved ? h.hid[n - 1] : ni;
            }
        }
        if (size > 21) return true;
        top.store(h);
    }
    for (; size > target; --size) {
        const int n = size - 1;
        const unsigned long long LK = h.key[n];
        const unsigned LI = h.hid[n];
        h.key[n] = h.key[0];
        h.hid[n] = h.hid[0];
        heap_descend(h, 0, n, LK, LK, LI);
    }
    return false;
}

// Two warps share TopLEK's extraction, step q = 1 .. nch: one extracts chunk q while the other tests the
// window of chunk q - 1, then they meet (a barrier of the two).  Step q's verdict stands in hit[q & 1], both
// zero before.  The word is written again in step q + 2, behind the meeting of step q + 1, which the
// extracting warp joins only after it has read it.  In a single word step q + 1's verdict could overtake a
// late read of step q's: the extracting warp would leave and the other wait for it for ever.
template <class Extract, class Meet>
__device__ __forceinline__ void extract_steps(int nch, const int* hit, Extract extract, Meet meet)
{
    for (int q = 1;; ++q) {
        if (q < nch) extract(q);
        meet();
        if (hit[q & 1] || q == nch) break;
    }
}

// window(q): whether chunk q holds a hit, the same in every lane; one lane writes
template <class Window, class Meet>
__device__ __forceinline__ void window_steps(int nch, int* hit, bool writer, Window window, Meet meet)
{
    for (int q = 1;; ++q) {
        const bool found = q > 1 && window(q - 1);
        if (writer) hit[q & 1] = found;
        meet();
        if (found || q == nch) break;
    }
}

}  // namespace fednl
