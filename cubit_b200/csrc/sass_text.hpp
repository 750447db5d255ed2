// Host text layer: SASS text -> typed instruction -> (record, patch) for the batch encoder.
//
// Mirrors the behaviour of the reference's parser (src/parser.rs) and of the text-semantic
// half of its encoder (src/encoder.rs:42-258 lookup chain and operand checks, :615-1060
// operand -> field value conversions, :395-443 register placement fixups, :1069-1146 branch
// targets, :468-516 raw-address LDG/STG, :1181-1215 PLOP3 / FADD fixups, :560-608 control
// word).  Text never goes to the GPU: an instruction is lowered to
//   * a record (variant id, one value per table field, guard nibble, reuse bits, scheduling)
//     that the batch encode kernel turns into and_base | fields | guard | reuse | control, and
//   * a patch (clear mask, set value) holding every bit the reference derives from the text
//     rather than from table fields; the final word is (kernel word & ~clear) | set.
#pragma once
#include <cstdint>
#include <deque>
#include <stdexcept>
#include <string>
#include <string_view>
#include <unordered_map>
#include <utility>
#include <vector>

#include "isa_table.hpp"

namespace cubit {

// Message texts follow the reference's ("unrecognized SASS: ...", "no operand-compatible
// table entry; attempted keys: [...]", "invalid control code string: ...").
//
// A line costs a few hundred nanoseconds: nothing here allocates for it.  Parsed text is views into the caller's text
// (or into a TextArena, for the few statements that are rewritten before they are read), failures are return values whose
// message is put together only when the caller asks for it, and names are looked up by view.
struct TextError : std::runtime_error {
    using std::runtime_error::runtime_error;
};

enum class OperandKind : uint8_t {
    Reg, UReg, Pred, UPred, Imm32, Imm64, FloatImm, Addr, ConstMem, Desc, BranchTarget, Barrier, SysReg, Label,
};

// One typed operand (reference src/ir.rs:38-84).  Only the members of its kind are meaningful.
struct TextOperand {
    OperandKind kind = OperandKind::Label;
    uint8_t num = 0;                       // register / predicate / barrier number (RZ = 255, URZ = 63, PT = 7)
    bool neg = false, abs = false, inv = false, reuse = false, is_zero = false;
    bool has_base = false, has_suffix = false, has_ur = false;
    uint8_t base = 0;                      // Addr / ConstMem / Desc base register
    uint8_t ur = 0;                        // Addr / ConstMem uniform register
    uint8_t ur_idx = 0;                    // Desc
    uint16_t bank = 0;                     // ConstMem
    uint32_t target = 0;                   // BranchTarget (absolute byte offset)
    int64_t imm = 0;                       // Imm32
    uint64_t bits = 0;                     // Imm64 value, FloatImm as f64 bits
    int64_t offset = 0;
    std::string_view suffix;               // ".64"-style suffix of the base register, without the dot
    std::string_view text;                 // SysReg name, Label text
};

// The operands of one instruction: the first few in place, all of them in `more` when there are more than that.
class OperandList {
public:
    size_t size() const { return n_; }
    bool empty() const { return n_ == 0; }
    TextOperand& operator[](size_t i) { return data()[i]; }
    const TextOperand& operator[](size_t i) const { return data()[i]; }
    TextOperand* begin() { return data(); }
    TextOperand* end() { return data() + n_; }
    const TextOperand* begin() const { return data(); }
    const TextOperand* end() const { return data() + n_; }
    void clear() { n_ = 0; more_.clear(); }
    TextOperand& add() {
        if (n_ < kInPlace) { fixed_[n_] = TextOperand(); return fixed_[n_++]; }
        if (n_ == kInPlace) more_.assign(fixed_, fixed_ + kInPlace);
        more_.emplace_back();
        ++n_;
        return more_.back();
    }

private:
    enum { kInPlace = 8 };
    TextOperand* data() { return n_ > kInPlace ? more_.data() : fixed_; }
    const TextOperand* data() const { return n_ > kInPlace ? more_.data() : fixed_; }
    TextOperand fixed_[kInPlace];
    std::vector<TextOperand> more_;
    size_t n_ = 0;
};

struct TextControl {                       // reference src/ir.rs:17-36 and its defaults
    uint8_t stall = 1;
    bool yield_flag = false;
    uint8_t write_bar = 7, read_bar = 7, wait_mask = 0;
};

// Text that a statement was rewritten to; views into its strings stay valid as long as it lives.
typedef std::deque<std::string> TextArena;

struct TextInstruction {                   // reference src/ir.rs:87-113
    uint32_t addr = 0;
    bool raw = false;                      // "__raw__0x<hex>": raw_hex is all there is
    std::string_view opcode, opcode_full, raw_hex;
    uint32_t op_class = 0;                 // what the opcode's name says about it (OC_*, sass_text.cpp)
    bool has_guard = false;
    uint8_t guard_pred = 7; bool guard_neg = false, guard_uniform = false;
    OperandList operands;
    TextControl ctrl;
    bool hand_sched = false;
    std::string_view raw_text;
    bool needs_addr() const;               // the word it lowers to depends on where it stands
    std::string key() const;               // opcode and operand types, "IADD3_R_P_P_R_R_R"
};

// "B------:R-:W-:-:S01" <-> TextControl (reference src/scheduling.rs:31-100).
bool parse_control_code(std::string_view s, TextControl* out);
std::string format_control_code(const TextControl& c);
uint32_t pack_control_code(const TextControl& c);   // the 17-bit scheduling value, not shifted
TextControl unpack_control_code(uint32_t sched17);

const char* operand_type_label(const TextOperand& op);

// One instruction, bare (parse_sass) or with a "[B..:R.:W.:.:S..]" prefix (parse_cuasm_line).  False when the text is not
// an instruction; `error`, when given, gets the reference's message.
bool parse_sass(std::string_view text, uint32_t addr, TextArena* arena, TextInstruction* out, std::string* error);
bool parse_cuasm_line(std::string_view line, uint32_t addr, TextArena* arena, TextInstruction* out, std::string* error);

// Branch operands that name a label become its address (find(name, &target) says whether it is known).
template <typename Find>
void resolve_labels(TextInstruction* insn, Find find) {
    for (TextOperand& op : insn->operands)
        if (op.kind == OperandKind::Label) {
            uint32_t target;
            if (!find(op.text, &target)) continue;
            op = TextOperand();
            op.kind = OperandKind::BranchTarget;
            op.target = target;
        }
}
bool resolves_labels(const TextInstruction& insn);   // the opcode is one of those whose labels are resolved

// Sorted, comma-joined dot-modifiers of the mnemonic (reference src/table.rs:477-502).
std::string extract_mod_group(std::string_view sass);

struct LoweredInstruction {
    bool raw = false;                // "__raw__0x..." statement: `set` is the whole word, nothing to encode
    uint32_t variant = 0;
    std::vector<uint64_t> values;    // one per table field of the variant, already masked
    uint32_t ctrl = 0;               // record control word: [16:0] scheduling, [19:17] reuse, [23:20] guard
    u128 clear = 0, set = 0;
};

class TextEncoder {
public:
    explicit TextEncoder(const IsaTable& table);
    // False when no table entry fits the operands (`error`, when given, gets the reference's message).  `out` can be used
    // for one instruction after another.
    bool lower(const TextInstruction& insn, LoweredInstruction* out, std::string* error) const;
    // Variant id of (key, mod_group), -1 when the table has no such pair.
    int find(std::string_view key, std::string_view mod_group) const;

private:
    // What the register and reuse fixups ask of a variant's fields.
    struct VariantShape {
        bool has_rd = false, has_ra = false, has_opaque = false;
        bool have_slot[3] = {false, false, false}, explicit_reuse[3] = {false, false, false};
        int32_t slot_tok[3] = {0, 0, 0};
    };
    const IsaTable& table_;
    std::unordered_map<std::string_view, uint32_t> key_index_;
    std::vector<VariantShape> shape_;
    const IsaKey* key(std::string_view name) const;
    const IsaVariant* get(std::string_view key, std::string_view mod_group, uint32_t* id) const;
};

// ---- printing ------------------------------------------------------------------------------

// Text that grows at the end.
class TextOut {
public:
    TextOut() = default;
    TextOut(const TextOut&) = delete;
    TextOut& operator=(const TextOut&) = delete;
    TextOut(TextOut&& o) noexcept : data_(o.data_), size_(o.size_), room_(o.room_) { o.data_ = nullptr; o.size_ = o.room_ = 0; }
    TextOut& operator=(TextOut&& o) noexcept {
        std::swap(data_, o.data_); std::swap(size_, o.size_); std::swap(room_, o.room_);
        return *this;
    }
    ~TextOut();
    void need(size_t n) { if (room_ - size_ < n) grow(n); }
    void put(char c) { need(1); data_[size_++] = c; }
    void put(std::string_view s) {
        need(s.size());
        if (!s.empty()) __builtin_memcpy(data_ + size_, s.data(), s.size());
        size_ += s.size();
    }
    void hex(uint64_t v, int digits = 1);        // at least that many digits, no prefix
    void dec(uint64_t v);
    void cut(size_t size) { size_ = size; }
    size_t size() const { return size_; }
    std::string_view view(size_t from = 0) const { return std::string_view(data_ + from, size_ - from); }

private:
    void grow(size_t n);
    char* data_ = nullptr;
    size_t size_ = 0, room_ = 0;
};
void put_control_code(const TextControl& c, TextOut* out);

struct VariantMeta;

// One field as the printer reads it: which spellings its extraction name (reference src/decoder.rs:679-705) equals or
// starts with, as PK_* bits, and where a record holds its value.
struct PrintField {
    uint32_t shift = 0, bits = 0, dst_pos = 0, stored_bits = 0;
    int32_t token_idx = 0;
    uint32_t shr = 0;        // the number behind the last "shr" of the name
    uint64_t kinds = 0;
    uint64_t value = 0;
};

// What printing derives from a variant alone: made once per variant, read for every word.
struct PrintPlan {
    std::vector<PrintField> fields;          // in token order, table order within a token
    std::vector<uint8_t> op_types;           // operand-type segments of the key (reference src/printer.rs:345-370), OT_*
    std::vector<std::string> op_names;       // their spelling, for the ones the printer does not know
    std::string mnemonic;                    // opcode + ordered modifiers (reference src/printer.rs:430-445)
    int32_t ra_tok = 0, rb_tok = 0;          // operands that the synthesized abs / neg modifiers belong to
    int32_t reuse_tok[3] = {0, 0, 0};        // operand whose register sits in the slot of reuse bit 122 + i; 0: none
    uint32_t traits = 0;                     // PT_*, sass_print.cpp
    uint8_t branch = 0;                      // BK_*, sass_print.cpp
};
PrintPlan make_print_plan(const VariantMeta& meta);

// Appends the SASS text of one decoded word, without the trailing " ;" (reference src/printer.rs:12-212).
void print_record(const PrintPlan& plan, const uint32_t slots[8], uint32_t ctrl, u128 raw, uint32_t addr, TextOut* out);

// ---- statements of a program ------------------------------------------------------------------

namespace text_detail {
inline bool is_space(char c) { return c == ' ' || c == '\t' || c == '\n' || c == '\r' || c == '\v' || c == '\f'; }
inline std::string_view trim(std::string_view s) {
    size_t b = 0, e = s.size();
    while (b < e && is_space(s[b])) ++b;
    while (e > b && is_space(s[e - 1])) --e;
    return s.substr(b, e - b);
}
// Length of the leading "/*<hex>*/" of s, 0 when there is none.
inline size_t address_comment(std::string_view s) {
    if (s.size() < 5 || s[0] != '/' || s[1] != '*') return 0;
    size_t k = 2;
    while (k < s.size() && ((s[k] >= '0' && s[k] <= '9') || (s[k] >= 'a' && s[k] <= 'f'))) ++k;
    return k > 2 && s.compare(k, 2, "*/") == 0 ? k + 2 : 0;
}
// Position of the colon of a leading "name:", 0 when there is none.
inline size_t label_colon(std::string_view s) {
    for (size_t k = 0; k < s.size(); ++k) {
        const char c = s[k];
        if (c == ':') return k;
        if (!((c >= '0' && c <= '9') || (c >= 'a' && c <= 'z') || (c >= 'A' && c <= 'Z') || c == '_')) return 0;
    }
    return 0;
}
}  // namespace text_detail

// Cuts whole lines of a program into labels and candidate statements, in order (reference src/parser.rs:485-588):
// ';' and newlines separate, // and # start comments, a leading /*addr*/ is dropped.  fn(text, is_label) for each.
template <typename Fn>
void for_each_statement(std::string_view text, Fn fn) {
    using namespace text_detail;
    for (size_t pos = 0; pos < text.size();) {
        size_t nl = text.find('\n', pos);
        if (nl == std::string_view::npos) nl = text.size();
        std::string_view line = text.substr(pos, nl - pos);
        pos = nl + 1;
        if (!line.empty() && line.back() == '\r') line.remove_suffix(1);
        size_t cut = line.find("//");
        if (cut == std::string_view::npos) cut = line.find('#');
        if (cut != std::string_view::npos) line = line.substr(0, cut);
        for (size_t at = 0; at <= line.size();) {
            size_t semi = line.find(';', at);
            if (semi == std::string_view::npos) semi = line.size();
            std::string_view seg = trim(line.substr(at, semi - at));
            at = semi + 1;
            if (const size_t skip = address_comment(seg)) seg = trim(seg.substr(skip));
            if (seg.empty()) continue;
            if (const size_t colon = label_colon(seg)) {
                fn(seg.substr(0, colon), true);
                seg = trim(seg.substr(colon + 1));
                if (seg.empty()) continue;
            }
            fn(seg, false);
        }
    }
}

}  // namespace cubit
