// Collapse of the binary BVH into 8-wide compressed nodes: the rules, and what
// both forms compute with. The library's form is collapseKernel (rt_build.cu),
// eight lanes per job; planCollapse, emitCollapse and collapseJob below are the
// same rules one job after another on the host, which the tests check against
// the reference's fixtures and hold the kernel's nodes against.
//
// One job per wide node. A job is either a binary node (interior or leaf) or
// a range of primitives (a leaf too large for one node). For a binary node,
// the children start as its two children; the interior child with the largest
// surface area is opened (replaced by its two children) while the result
// still fits in eight slots, where a leaf of k <= 8 * group triangles needs
// ceil(k / group) slots (groups of up to `group` triangles, 1..3, each with
// its own box) and anything else one slot. Leaves that still do not fit become wide children of their own.
// Slots are assigned by ray octant (slot s holds the child nearest along
// direction signs s), and child boxes are quantised outward against the
// node's grid, checked with the same fused multiply-add the traversal uses.
#pragma once
#include "rt_build.cuh"

namespace rt {

RT_HD int imin(int a, int b) { return a < b ? a : b; }
RT_HD int imax(int a, int b) { return a > b ? a : b; }
RT_HD float collapseHalfArea(const float lo[3], const float hi[3]) {
    float x = fmaxf(0.0f, hi[0] - lo[0]), y = fmaxf(0.0f, hi[1] - lo[1]), z = fmaxf(0.0f, hi[2] - lo[2]);
    return x * y + x * z + y * z;
}
RT_HD void collapseGrow(float lo[3], float hi[3], const float olo[3], const float ohi[3]) {
    for (int a = 0; a < 3; a++) { lo[a] = fminf(lo[a], olo[a]); hi[a] = fmaxf(hi[a], ohi[a]); }
}

struct Job { int kind; int node; int first; int count; int wide; };  // kind 0 binary node, 1 primitive range
struct Kid { int kind; int node; int first; int count; float lo[3], hi[3]; };  // kind 0/1 wide child, 2 triangle group

// Slots a binary child needs: one for an interior node, ceil(k / group) for a
// leaf of k <= width * group triangles held inline, one for a larger leaf.
RT_HD int slotsOf(const BinNode& n, int group, int width) {
    if (n.count == 0) return 1;
    return n.count <= width * group ? (n.count + group - 1) / group : 1;
}

// Cost of a child whose centre lies at c from the node's in slot s: how late
// rays whose direction signs are s meet it.
RT_HD float slotCost(const float c[3], int s) {
    return ((s & 4) ? -c[0] : c[0]) + ((s & 2) ? -c[1] : c[1]) + ((s & 1) ? -c[2] : c[2]);
}
// Exponent byte of a node's grid along an axis (steps of 2^(byte - 127), 255 of
// them at least the extent), and the step.
RT_HD unsigned char gridExponent(float extent) {
    int ex = -126;
    if (extent > 0.0f) { frexpf(extent / 255.0f, &ex); }
    return (unsigned char)(imax(-126, imin(127, ex)) + 127);
}
RT_HD float gridStep(unsigned char exponent) { return bitsToFloat((unsigned)exponent << 23); }
// A child's planes on the grid at p, rounded outward and checked with the
// traversal's arithmetic.
RT_HD void quantise(float lo, float hi, float p, float step, unsigned char& qlo, unsigned char& qhi) {
    int ql = (int)floorf((lo - p) / step);
    int qh = (int)ceilf((hi - p) / step);
    ql = imax(0, imin(255, ql));
    qh = imax(0, imin(255, qh));
    while (ql > 0 && fmaRn((float)ql, step, p) > lo) ql--;
    while (qh < 255 && fmaRn((float)qh, step, p) < hi) qh++;
    qlo = (unsigned char)ql;
    qhi = (unsigned char)qh;
}
// Meta bytes: a group of `count` triangles from `offset`, an interior child.
RT_HD unsigned char groupMeta(int count, int offset) { return (unsigned char)((((1u << count) - 1u) << 5) | (unsigned)offset); }
RT_HD unsigned char innerMeta(int slot) { return (unsigned char)(0x20u | (24u + (unsigned)slot)); }
// Triangle `index` as traversal reads it.
RT_HD void packTriangle(const SceneTri& t, int index, float4* dst) {
    dst[0] = make_float4(t.origin.x, t.origin.y, t.origin.z, t.edge1.x);
    dst[1] = make_float4(t.edge1.y, t.edge1.z, t.edge2.x, t.edge2.y);
    dst[2] = make_float4(t.edge2.z, bitsToFloat(t.oneSided != 0 ? 1u : 0u), bitsToFloat((unsigned)index), 0.0f);
}

// A job's wide node before its storage is allocated: the children, their
// slots and boxes, and the triangles of each triangle group.
struct CollapsePlan {
    Kid kids[8];
    int nk, wide;
    int slotKid[8];
    int groupTris[8][3], groupCount[8];
    int nInterior, nTris;  // wide children (= next-level jobs) and packed triangles
    float nlo[3], nhi[3];
};

// Chooses up to eight children of job J's wide node, their boxes and slots,
// and the triangles of its triangle groups. width (4 or 8): most children
// per node; the node format keeps eight slots either way. primTri: the
// triangle of each primitive when primitives are triangle pieces (null:
// primitive p is triangle p).
inline void planCollapse(Job J, const BinNode* bn, const int* order, const float4* plo, const float4* phi, int group,
                        int width, const int* primTri, CollapsePlan& P) {
    if (J.kind == 0 && bn[J.node].count > 0) { J.kind = 1; J.first = bn[J.node].first; J.count = bn[J.node].count; }
    P.wide = J.wide;
    Kid* kids = P.kids;
    int nk = 0;
    if (J.kind == 0) {
        // Candidates with what opening one needs, read once each: its slots,
        // and for an interior one its area and the slots after opening it.
        int cand[8], slots[8], opened[8], nc = 0, total = 0;
        float area[8];
        bool asNode[8] = {false, false, false, false, false, false, false, false};
        auto place = [&](int i, int node) {
            const BinNode& c = bn[node];
            cand[i] = node;
            slots[i] = slotsOf(c, group, width);
            area[i] = -1.0f;
            if (c.count == 0) {
                float lo[3] = {c.low.x, c.low.y, c.low.z}, hi[3] = {c.high.x, c.high.y, c.high.z};
                area[i] = collapseHalfArea(lo, hi);
                opened[i] = slotsOf(bn[c.first], group, width) + slotsOf(bn[c.first + 1], group, width);
            }
            total += slots[i];
        };
        const int children = bn[J.node].first;
        place(nc++, children);
        place(nc++, children + 1);
        for (;;) {
            int best = -1; float bestArea = -1.0f;
            for (int i = 0; i < nc; i++)
                if (area[i] > bestArea && nc < width && total - 1 + opened[i] <= width) { bestArea = area[i]; best = i; }
            if (best < 0) break;
            const int first = bn[cand[best]].first;
            total -= slots[best];
            place(best, first);
            place(nc++, first + 1);
        }
        // Leaves that do not fit inline become wide children of their own.
        for (;;) {
            int total = 0;
            for (int i = 0; i < nc; i++) total += asNode[i] ? 1 : slotsOf(bn[cand[i]], group, width);
            if (total <= width) break;
            int pick = -1, most = 0;
            for (int i = 0; i < nc; i++) {
                const BinNode& c = bn[cand[i]];
                if (!asNode[i] && c.count > group && c.count > most) { most = c.count; pick = i; }
            }
            if (pick < 0) break;
            asNode[pick] = true;
        }
        for (int i = 0; i < nc && nk < width; i++) {
            const BinNode& c = bn[cand[i]];
            if (c.count == 0) {
                kids[nk++] = Kid{0, cand[i], 0, 0, {c.low.x, c.low.y, c.low.z}, {c.high.x, c.high.y, c.high.z}};
            } else if (asNode[i] || c.count > width * group) {
                kids[nk++] = Kid{1, -1, c.first, c.count, {c.low.x, c.low.y, c.low.z}, {c.high.x, c.high.y, c.high.z}};
            } else {
                for (int g = 0; g < c.count && nk < width; g += group)
                    kids[nk++] = Kid{2, -1, c.first + g, imin(group, c.count - g), {0, 0, 0}, {0, 0, 0}};
            }
        }
    } else if (J.count <= width * group) {
        for (int g = 0; g < J.count && nk < width; g += group)
            kids[nk++] = Kid{2, -1, J.first + g, imin(group, J.count - g), {0, 0, 0}, {0, 0, 0}};
    } else {
        int chunk = (J.count + width - 1) / width;
        for (int g = 0; g < J.count && nk < width; g += chunk) {
            int c = imin(chunk, J.count - g);
            kids[nk++] = Kid{c <= group ? 2 : 1, -1, J.first + g, c, {0, 0, 0}, {0, 0, 0}};
        }
    }
    // Boxes of primitive-range kids: union of padded primitive boxes.
    float nlo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, nhi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    for (int k = 0; k < nk; k++) {
        Kid& K = kids[k];
        if (K.kind != 0) {
            float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
            for (int i = 0; i < K.count; i++) {
                int p = order[K.first + i];
                float4 a = plo[p], b = phi[p];
                lo[0] = fminf(lo[0], a.x); lo[1] = fminf(lo[1], a.y); lo[2] = fminf(lo[2], a.z);
                hi[0] = fmaxf(hi[0], b.x); hi[1] = fmaxf(hi[1], b.y); hi[2] = fmaxf(hi[2], b.z);
            }
            for (int a = 0; a < 3; a++) { K.lo[a] = lo[a]; K.hi[a] = hi[a]; }
        }
        collapseGrow(nlo, nhi, K.lo, K.hi);
    }
    // Slot assignment: slot s holds the kid met first by rays whose direction
    // signs are s (bit 2 = x negative, bit 1 = y, bit 0 = z).
    int* slotKid = P.slotKid;
    for (int s = 0; s < 8; s++) slotKid[s] = -1;
    {
        float cn[3], ck[8][3];
        for (int a = 0; a < 3; a++) cn[a] = 0.5f * (nlo[a] + nhi[a]);
        for (int k = 0; k < nk; k++)
            for (int a = 0; a < 3; a++) ck[k][a] = 0.5f * (kids[k].lo[a] + kids[k].hi[a]) - cn[a];
        // Greedy: the cheapest (kid, slot) pair first, the lower kid and slot
        // of equals. Each kid keeps its cheapest free slot, looked up again only
        // when that slot is taken.
        float cost[8];
        int at[8];
        unsigned freeSlots = 0xFFu, left = (1u << nk) - 1u;
        auto cheapest = [&](int k) {
            cost[k] = FLT_MAX;
            at[k] = -1;
            for (int s = 0; s < 8; s++) {
                if (!((freeSlots >> s) & 1u)) continue;
                float c = slotCost(ck[k], s);
                if (c < cost[k]) { cost[k] = c; at[k] = s; }
            }
        };
        for (int k = 0; k < nk; k++) cheapest(k);
        for (int round = 0; round < nk; round++) {
            float best = FLT_MAX; int bk = -1, bs = -1;
            for (int k = 0; k < nk; k++)
                if (((left >> k) & 1u) && cost[k] < best) { best = cost[k]; bk = k; bs = at[k]; }
            if (bk < 0) {  // non-finite costs: first free kid into the first free slot
                for (int k = 0; k < nk && bk < 0; k++) if ((left >> k) & 1u) bk = k;
                for (int s = 0; s < 8 && bs < 0; s++) if ((freeSlots >> s) & 1u) bs = s;
            }
            left &= ~(1u << bk);
            freeSlots &= ~(1u << bs);
            slotKid[bs] = bk;
            for (int k = 0; k < nk; k++)
                if (((left >> k) & 1u) && at[k] == bs) cheapest(k);
        }
    }
    // Triangles of each triangle group, once each: pieces of one triangle in
    // the same group would only repeat its test (the group's box covers them).
    int (*groupTris)[3] = P.groupTris;
    int* groupCount = P.groupCount;
    int nInterior = 0, nTris = 0;
    for (int k = 0; k < nk; k++) {
        groupCount[k] = 0;
        if (kids[k].kind != 2) { nInterior++; continue; }
        for (int i = 0; i < kids[k].count; i++) {
            const int prim = order[kids[k].first + i];
            const int tri = primTri ? primTri[prim] : prim;
            bool seen = false;
            for (int j = 0; j < groupCount[k]; j++) seen = seen || groupTris[k][j] == tri;
            if (!seen) groupTris[k][groupCount[k]++] = tri;
        }
        nTris += groupCount[k];
    }
    P.nk = nk;
    P.nInterior = nInterior;
    P.nTris = nTris;
    for (int a = 0; a < 3; a++) { P.nlo[a] = nlo[a]; P.nhi[a] = nhi[a]; }
}

// Writes a planned wide node whose storage has been allocated: wide children
// from childBase, packed triangles from triBase, next-level jobs from
// jobBase (nInterior of each). counters[3] receives an error code when an
// allocation passes its capacity.
inline void emitCollapse(const CollapsePlan& P, int childBase, int triBase, int jobBase, const SceneTri* tris,
                        Job* nextJobs, WideNode* wide, float4* packed, int* counters, int wideCapacity,
                        int jobCapacity, int triCapacity) {
    const Kid* kids = P.kids;
    const int* slotKid = P.slotKid;
    const int (*groupTris)[3] = P.groupTris;
    const int* groupCount = P.groupCount;
    const float* nlo = P.nlo;
    const float* nhi = P.nhi;
    if (childBase + P.nInterior > wideCapacity || triBase + P.nTris > triCapacity) { counters[3] = 3; return; }
    WideNode W;
    W.px = nlo[0]; W.py = nlo[1]; W.pz = nlo[2];
    unsigned char ebits[3];
    for (int a = 0; a < 3; a++) ebits[a] = gridExponent(nhi[a] - nlo[a]);
    W.ex = ebits[0]; W.ey = ebits[1]; W.ez = ebits[2];
    W.imask = 0;
    W.childBase = (unsigned)childBase;
    W.triBase = (unsigned)triBase;
    int interiorSeen = 0, triOffset = 0;
    for (int s = 0; s < 8; s++) {
        int k = slotKid[s];
        if (k < 0) {
            W.meta[s] = 0;
            for (int a = 0; a < 3; a++) { W.qlo[a][s] = 0; W.qhi[a][s] = 0; }
            continue;
        }
        const Kid& K = kids[k];
        for (int a = 0; a < 3; a++) quantise(K.lo[a], K.hi[a], nlo[a], gridStep(ebits[a]), W.qlo[a][s], W.qhi[a][s]);
        if (K.kind == 2) {
            const int count = groupCount[k];
            W.meta[s] = groupMeta(count, triOffset);
            for (int i = 0; i < count; i++)
                packTriangle(tris[groupTris[k][i]], groupTris[k][i], packed + (size_t)(triBase + triOffset + i) * 3);
            triOffset += count;
        } else {
            W.meta[s] = innerMeta(s);
            W.imask |= (unsigned char)(1u << s);
            const int q = jobBase + interiorSeen;
            if (q >= jobCapacity) { counters[3] = 4; interiorSeen++; continue; }
            nextJobs[q] = Job{K.kind == 0 ? 0 : 1, K.node, K.first, K.count, childBase + interiorSeen};
            interiorSeen++;
        }
    }
    wide[P.wide] = W;
}

// Builds wide node J.wide for one job: planCollapse, then allocation of its
// wide children, packed triangles and next-level jobs, then emitCollapse.
// counters: [0] wide nodes, [1] packed triangles, [2] next-level jobs,
// [3] error code.
inline void collapseJob(Job J, const BinNode* bn, const int* order, const float4* plo, const float4* phi,
                       const SceneTri* tris, Job* nextJobs, WideNode* wide, float4* packed, int* counters,
                       int wideCapacity, int jobCapacity, int triCapacity, int group, int width = 8,
                       const int* primTri = nullptr) {
    CollapsePlan P;
    planCollapse(J, bn, order, plo, phi, group, width, primTri, P);
    const int childBase = counters[0], triBase = counters[1], jobBase = counters[2];
    counters[0] += P.nInterior;
    counters[1] += P.nTris;
    counters[2] += P.nInterior;
    emitCollapse(P, childBase, triBase, jobBase, tris, nextJobs, wide, packed, counters, wideCapacity, jobCapacity,
                 triCapacity);
}

}  // namespace rt
