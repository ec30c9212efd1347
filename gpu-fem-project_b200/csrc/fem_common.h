// Shared internals of libfemb200: error reporting and small helpers.
#pragma once

#include <cstdint>
#include <cstdio>
#include <vector>

#include "fem_b200.h"

namespace fem {

namespace dev {
// A strip of a plan's strip layout (HostPlan::strips): listed elements [begin, begin +
// count), each the right neighbour of the one before; lead: id of the first element
// that is not the halo.
struct alignas(16) Strip {
  int begin, count, flags, lead;
};
// Flags of a strip (kHalo, kRight) and of one of its steps: its first element is a halo,
// assembled for its right edge only; its first element continues the strip and takes
// the sums of its left edge from the element before it; its last element has a right
// neighbour, which owns the edge between them.
enum : int { kHalo = 1, kCarry = 2, kRight = 4 };
}  // namespace dev

// Records a message for fem_last_error() on this host thread and returns `status`.
int fail(int status, const char *fmt, ...);
void clear_error();
const char *last_error_cstr();

inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Host builders (fem_host.cpp).
int build_pattern(int numNodes, const int *connPtr, const int *conn, int numElements, int *rowp, int *cols,
                  int64_t *nnzb);
int colour_greedy(int numNodes, const int *connPtr, const int *conn, int numElements, int *colour,
                  int *numColours);

// Plan topology built on the host before upload (fem_host.cpp).
struct HostPlan {
  int order = 0, nn = 0, numNodes = 0, numElements = 0, numColours = 0;
  int64_t nnzb = 0;
  std::vector<int> rowp, cols;                // pattern
  std::vector<int> elemList;            // elements in colour order
  std::vector<int> colourPtr;           // numColours+1 offsets into elemList
  std::vector<int> connList;            // conn in elemList order, nn per element
  // Per listed element k a record of codeStride bytes: [a*nn + b] = rank of the
  // block (a, b) in row conn[a] | 0x80 when this element stores it first, then
  // [nn*nn + a] = 1 when this element writes node a's residual first; zero padding
  // to a multiple of 16 bytes (records are copied to shared memory in 16-byte chunks).
  int codeStride = 0;
  std::vector<uint8_t> blockCode;
  // Order 1, row assembly (each block row written once by the warp that owns it):
  // rowElemPtr[numNodes+1] indexes rowElem, two ints per (node r, element k listing
  // r): {k << 2 | a (local index of r), ranks of the element's four nodes in row r,
  // one byte each, | 0x80 in the row's first entry with that block}; rowChunk[numChunks+1]
  // cuts the rows into chunks of at most kRowChunkRows rows and kRowChunkBlocks blocks.
  // Empty when not applicable.
  std::vector<int> rowElemPtr, rowElem, rowChunk;
  // Orders 2-4, pair layout of the fragment kernel's single-mesh assembly: elements
  // paired with the neighbour across their right edge (its left edge, node for
  // node), pairs coloured so that the pairs of one colour share no node, each
  // colour listing its pairs (two consecutive positions, the pair's first element
  // first) and then its unpaired elements.  Codes as above, in list order, so the
  // second element of a pair adds to the blocks and residual rows of the shared
  // edge that the first one stored.
  int numPairColours = 0;
  int64_t numPairs = 0;
  std::vector<int> pairColourPtr, pairList, pairConnList;
  std::vector<int> pairRegionEnd;  // per colour: the end of its pairs (its unpaired elements follow)
  std::vector<uint8_t> pairCode;
  // Order kStripOrder: strip layout (LINEAR Jacobians, in the pair layout's place; up to
  // kStripColours colours the pair tables are then left out).  Chains of right neighbours are coloured so that the
  // chains of one colour share no node and cut into strips.  The blocks of an edge's nodes among
  // themselves and their residual rows belong to the element right of the edge; a strip
  // that does not begin its chain lists the element before it first, as a halo whose
  // share of the strip's left edge is assembled again, so the strips of a chain share no
  // output and one launch takes all of a colour.  strips: by colour, ascending lead.
  // Codes in list order (a halo's are unused); a block left to the right neighbour has
  // the store flag, so that nothing is added there.
  int numStripColours = 0;
  std::vector<dev::Strip> strips;
  std::vector<int> stripColourPtr, stripConn, stripLo, stripHi;  // Lo, Hi: node span per strip, halo included
  std::vector<uint8_t> stripCode;
};
constexpr int kPairMinElements = 4 * 148 * 12;  // four colours of one element per resident warp
constexpr int kStripOrder = 3;
constexpr int kStripWarps = 148 * 12;  // resident warps of the strip kernel
// Strips against pairs, by the colours of the chains (order 3, us, strips / pairs).  Up to
// three (the rows of a grid, in any numbering, or of a ring) strips win at every size: 64^2
// 27 / 29, 128^2 49 / 67, 256^2 160 / 183, 512^2 537 / 704, eight wide 59 / 67, MIXED 512^2
// 633 / 669.  Chains that cross (blocks with turned axes, turned elements) need four to
// seven, and their launches are smaller: strips lose up to about 440^2 (four blocks with
// crossed axes 128^2 95 / 76, 400^2 456 / 422; blocks of 8 256^2 255 / 194, 430^2 511 / 480) and win
// beyond in FP64 (470^2: crossed 577 / 627, blocks of 8, 20, 64 575 / 604, 598 / 603, 581 / 604, with 2
// and 10 % of the elements turned 569 / 593, 600 / 620; 700^2: 1172 / 1318, 1196 / 1314, 1193 / 1312,
// 1174 / 1311, 1129 / 1276, 1232 / 1330), not in MIXED (512^2 833 / 760, 758 / 735), which runs the pairs.
// Strips longer than kStripCrossedLength lose there (blocks of 20: 470^2 707 us with 19).
constexpr int kStripColours = 3, kStripColoursLarge = 7, kStripLargeElements = 210000, kStripCrossedLength = 7;
constexpr int kRowChunkRows = 32, kRowChunkBlocks = 320;
int build_host_plan(int order, int numNodes, const int *connPtr, const int *conn, int numElements, HostPlan &hp,
                    bool strips = true);

}  // namespace fem
