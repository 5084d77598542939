// Queries as find_value runs them: the bytecode (jsonpath.h) decoded once on
// the host into 16-byte steps, one aligned load each, with what a key search
// needs worked out and the keys' bytes on four-byte boundaries.  Decoding the
// bytecode in the kernel was half of its loads: every opcode, length and key
// byte of a query, read again for every line.
#pragma once

#include <cstdint>
#include <vector>

#include "interp.cuh"

namespace gpj {

// Appends the program of validated bytecode `ir` to `out` (on a 16-byte
// boundary of it); returns where it begins.
inline int32_t append_program(const uint8_t* ir, std::vector<uint8_t>* out) {
    out->resize((out->size() + 15) / 16 * 16, 0);
    const size_t begin = out->size();
    std::vector<ProgramStep> steps;
    std::vector<uint8_t> strings;
    ByteCode code{ir};
    for (;;) {
        ProgramStep s{static_cast<uint32_t>(code.next()), code.value, 0, 0};
        if (s.op == 4 || s.op == 6) {
            if (s.op == 4) {
                const auto key = code.key();
                s.op |= static_cast<uint32_t>(key.span) << 8;
                s.op |= (key.mask == 0 ? 0u : (key.mask == ~0u ? 2u : 1u)) << 16;
                s.tail = key.tail;
            }
            s.at = static_cast<uint32_t>(strings.size());
            strings.insert(strings.end(), code.bytes, code.bytes + code.value);
            strings.resize((strings.size() + 3) / 4 * 4, 0);
        }
        steps.push_back(s);
        if (s.op == 0 || s.op > 0xFFFFFFu) break;
        if ((s.op & 0xFF) > 6) break;
    }
    for (auto& s : steps)
        if ((s.op & 0xFF) == 4 || (s.op & 0xFF) == 6) s.at += static_cast<uint32_t>(steps.size() * sizeof(ProgramStep));
    const uint8_t* p = reinterpret_cast<const uint8_t*>(steps.data());
    out->insert(out->end(), p, p + steps.size() * sizeof(ProgramStep));
    out->insert(out->end(), strings.begin(), strings.end());
    return static_cast<int32_t>(begin);
}

}  // namespace gpj
