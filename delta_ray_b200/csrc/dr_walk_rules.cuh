// The warp walk's stacks (dr_edge_walk.cuh): which class a pending node goes to
// and how many nodes of each class a step takes.  Host and device, so that the
// bound they keep can be tested on the CPU: no stack outgrows its entries
// (the pushes are not checked).
//
// Classes of pending nodes, each with its own stack in the warp's shared
// memory: 2 the all walk's nodes that split (bound above 1, or around the
// point), whose children's bounds only meet thresholds and whose cone tests
// decide nothing (k_edge_walk's fast step; three in four nodes of a glossy
// heightfield); of the others, 1 the all walk's off the cone walk's path, 0 the
// rest, which take the cone tests.
//
// Off the path a node's cone-walk share cp is 0, and its children's are 0 too
// unless their own share is undefined (0 times NaN, below a node with an
// infinite bound).  The all walk's weight of an edge, ap / (cp^2 + ap^2), is NaN
// where either share is, and nothing else reads them there, so such a child
// takes its undefined share as ap and 0 as cp (walk_undefined): class 1 never
// adds to class 0.
//
// While all stacks have room for a step's children (walk_room) the classes are
// stepped as they fill.  Without that room (or room to hand the nodes on) no
// node goes to class 2 any more (`two`): a child then stays in its parent's
// class or goes to class 1, and a step takes only as many nodes as leave
// DR_WALK_RESERVE slots of its class free, and at least one.  Taking one at a
// time needs one slot per tree level (trees are split at the median, node ids
// have 27 bits: at most DR_WALK_LEVELS), so the reserve always suffices; steps
// of classes 0 and 2 also add up to 32 nodes to the classes below, which are
// drained first.
#pragma once

#define DR_WALK_N0 128
#define DR_WALK_N1 128
#define DR_WALK_N2 224
#define DR_WALK_RESERVE 32
#define DR_WALK_LEVELS 28
static_assert(DR_WALK_RESERVE >= DR_WALK_LEVELS, "one node at a time needs a slot per tree level");
static_assert(DR_WALK_N0 >= 2 * (DR_WALK_RESERVE + 32) && DR_WALK_N1 >= 2 * (DR_WALK_RESERVE + 32) && DR_WALK_N2 >= 64,
              "room for a step's children above the reserve");

// An all-walk child whose cone-walk share is undefined (see above).
DEV void walk_undefined(bool all_walk, float &cp, float &ap) {
    if (all_walk && cp != cp) {
        ap = cp;
        cp = 0.f;
    }
}

// The class of a node with code `code` (mode << 30, all-split << 31) and
// cone-walk share cp.
DEV int walk_class(unsigned code, float cp, bool two) {
    const bool all_walk = (code >> 30) & 1;
    if (two && all_walk && (code >> 31)) return 2;
    return all_walk && cp == 0.f ? 1 : 0;
}

// Whether every stack has room for a step's children with the reserve left.
DEV bool walk_room(int n0, int n1, int n2) {
    return n0 <= DR_WALK_N0 - DR_WALK_RESERVE - 32 && n1 <= DR_WALK_N1 - DR_WALK_RESERVE - 32 && n2 <= DR_WALK_N2 - 32;
}

// The nodes a step takes off each stack, up to 16: of one class where a class
// fills the step, else of all (which only the general step takes).  fast: the
// step of 16 class-2 nodes.
struct WalkTake {
    int k0, k1, k2;
    bool fast;
};
DEV WalkTake walk_take(int n0, int n1, int n2, bool two) {
    WalkTake t;
    t.k0 = t.k1 = t.k2 = 0;
    t.fast = two && n2 >= 16;
    if (t.fast) {
        t.k2 = 16;
    } else if (!two) {  // short of room: class 1 first, then 0, which add to none but themselves and 1
        const int r0 = DR_WALK_N0 - n0 - DR_WALK_RESERVE, r1 = DR_WALK_N1 - n1 - DR_WALK_RESERVE;
        if (n1 >= 16) t.k1 = r1 > 16 ? 16 : (r1 > 1 ? r1 : 1);
        else if (n0 >= 16) t.k0 = r0 > 16 ? 16 : (r0 > 1 ? r0 : 1);
        else if (n2 > 0) t.k2 = n2 < 16 ? n2 : 16;
        else if (n0 > 0) t.k0 = n0;
        else t.k1 = n1;
    } else if (n1 >= 16) {
        t.k1 = 16;
    } else if (n0 >= 16) {
        t.k0 = 16;
    } else {
        t.k2 = n2;
        t.k1 = n1 < 16 - t.k2 ? n1 : 16 - t.k2;
        t.k0 = n0 < 16 - t.k2 - t.k1 ? n0 : 16 - t.k2 - t.k1;
    }
    return t;
}
