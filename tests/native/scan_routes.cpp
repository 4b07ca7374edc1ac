// Prints what a step does for each line of "kind channels states sms chunk length count [length count ...]" on standard input: apart, or the form of
// its call (csrc/scan_routes.h).
#include <cstdio>
#include <iostream>
#include <sstream>
#include <string>

#include "scan_routes.h"

int main() {
    using namespace ingot_scan;
    std::string line;
    while (std::getline(std::cin, line)) {
        std::istringstream in(line);
        std::string name;
        int channels, states, sms, chunk, len, count;
        in >> name >> channels >> states >> sms >> chunk;
        const Kind kind = name == "scan" ? Kind::selective : Kind::gated;
        Load all = {}, small = {}, large = {};
        while (in >> len >> count)
            for (Load* l : {&all, len <= kShort ? &small : &large}) {
                l->tokens += static_cast<long long>(len) * count;
                l->longest = std::max(l->longest, len);
                l->sequences += count;
                l->most_chunks = (l->longest + chunk - 1) / chunk;
            }
        const Form form = choose(kind, all, channels, states, sms).form;
        std::printf("%s\n", apart(kind, all, small, large, channels, states, sms) ? "apart" : form == Form::stream ? "stream" : form == Form::tile ? "tile" : "chunks");
    }
}
