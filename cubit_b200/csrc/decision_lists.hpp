// Decision lists: what variant selection does inside a leaf of the match tree, unrolled into tests in a fixed order.
//
// select_variant (codec_core.cuh) finds every class of a leaf that matches the word, ranks the matches and applies the
// disambiguation rules.  Each question it asks of a word is whether some bits have some values, so its whole decision inside
// one leaf can be written down beforehand as an ordered list of (mask, value, outcome): the first entry that agrees with the
// word holds the answer.  DecisionLists::compile follows select_variant over every leaf with the word's bits unknown and
// records one entry per way its questions can be answered.
//
// Two lists are made per leaf.  The decode list answers with the variant (and its extraction record and tie bit).  The
// roundtrip list asks one question more, whether the word is what the variant encodes to, and answers with the status; which
// variant it was does not matter to it, so that many entries of the decode list fall into one.
#pragma once
#include <cstdint>
#include <vector>

#include "flat_table.hpp"

namespace cubit {

struct DecisionLists {
    std::vector<uint32_t> decode, roundtrip;   // table images for the kernels; offsets in `at` (ListLayout)
    ListLayout decode_at{}, roundtrip_at{};
    uint32_t decode_entries = 0, roundtrip_entries = 0, longest = 0;

    // Both images are empty when a table does not fit the form: leaves of more than 16 classes, more variants or field layouts
    // than an entry has bits for, a leaf whose decision takes hundreds of entries, ones among the constant bits of the upper limb.
    // Such tables keep the kernels that scan classes.
    static DecisionLists compile(const FlatTable& ft);
};

}  // namespace cubit
