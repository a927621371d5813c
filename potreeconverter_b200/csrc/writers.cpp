// hierarchy.bin and metadata.json writers. Both files are byte contracts
// with the reference's readers (Potree), so their layout follows the
// reference writers step for step, including its quirks:
//  * every node starts as LEAF and only turns NORMAL when one of its children
//    is met later in the same batch (HierarchyBuilder.h:149-163); since
//    children complete before parents, inner nodes keep type LEAF with a
//    non-zero child mask;
//  * batch roots are PROXY in the root batch and NORMAL inside their own
//    batch (HierarchyBuilder.h:257-264, 316-327);
//  * byte sizes pass through a 32-bit field (indexer.h:221, HierarchyBuilder.h:104).

#include "writers.h"

#include <algorithm>
#include <iomanip>
#include <cstring>
#include <limits>
#include <sstream>
#include <type_traits>
#include <utility>

namespace pcg {

namespace {

constexpr int kStep = 4;           // hierarchyStepSize, indexer.cpp:19
constexpr int kRecordBytes = 22;   // type, childMask, numPoints, offset, size

enum NodeType : uint8_t { T_NORMAL = 0, T_LEAF = 1, T_PROXY = 2 };

// A node's name as a number: a 1, then three bits per digit after the "r". The
// parent is code >> 3, and the order by length, then text, is the order of
// the codes. 64 bits hold 21 levels, 128 bits 42. A cube of 2^32 units of the
// smallest scale has at most 33 and one round of five more, but every axis has
// a scale of its own: a header box that is long in one axis only has as many
// levels as its doubles resolve. Names past 42 levels stay text.
class TextCode {
public:
	TextCode() = default;
	explicit TextCode(uint64_t code) {
		for (int b = 63 - __builtin_clzll(code) - 3; b >= 0; b -= 3) digits_ += (char)('0' + (code >> b & 7));
	}
	TextCode(const char* name, size_t len) : digits_(name + 1, len - 1) {}
	friend TextCode operator>>(const TextCode& c, int bits) {  // the root has no parent
		TextCode up;
		if ((size_t)bits / 3 > c.digits_.size()) up.none_ = true;
		else up.digits_ = c.digits_.substr(0, c.digits_.size() - (size_t)bits / 3);
		return up;
	}
	friend int operator&(const TextCode& c, int) { return c.digits_.empty() ? 1 : c.digits_.back() - '0'; }
	friend bool operator==(const TextCode& a, const TextCode& b) { return a.none_ == b.none_ && a.digits_ == b.digits_; }
	friend bool operator!=(const TextCode& a, const TextCode& b) { return !(a == b); }
	friend bool operator<(const TextCode& a, const TextCode& b) {
		if (a.none_ != b.none_) return a.none_;
		return a.digits_.size() != b.digits_.size() ? a.digits_.size() < b.digits_.size() : a.digits_ < b.digits_;
	}

private:
	std::string digits_;
	bool none_ = false;  // above the root
};

template <class Code>
Code code_of(const char* name, size_t len) {
	if constexpr (std::is_same_v<Code, TextCode>) {
		return TextCode(name, len);
	} else {
		Code c = 1;
		for (size_t i = 1; i < len; i++) c = c << 3 | (Code)(name[i] - '0');
		return c;
	}
}

template <class Code>
struct BNode {
	Code code{};
	int32_t num_points = 0;
	uint32_t order = 0;  // in the file
	uint8_t child_mask = 0;
	uint8_t type = T_LEAF;
	uint64_t byte_offset = 0, byte_size = 0;
	uint64_t proxy_offset = 0, proxy_size = 0;
};

template <class Code>
struct BChunk {
	Code code{};
	size_t first = 0, count = 0;  // its entries
};

// The chunks of a batch in order, and their nodes in order.
template <class Code>
struct Batch {
	Code code{};
	std::vector<BNode<Code>> nodes;                  // by code
	std::vector<BChunk<Code>> chunks;                // by code
	std::vector<std::pair<Code, uint32_t>> entries;  // (chunk, node), chunk by chunk
	std::vector<std::pair<Code, uint32_t>> by_code;  // (node, record)
	int64_t byte_size = 0;

	BNode<Code>* find(Code c) {
		auto it = std::lower_bound(nodes.begin(), nodes.end(), c, [](const BNode<Code>& n, Code v) { return n.code < v; });
		return it != nodes.end() && it->code == c ? &*it : nullptr;
	}
	bool has_chunk(Code c) const {
		auto it = std::lower_bound(chunks.begin(), chunks.end(), c, [](const BChunk<Code>& n, Code v) { return n.code < v; });
		return it != chunks.end() && it->code == c;
	}
};

// HierarchyBuilder::loadBatch (HierarchyBuilder.h:82-197) over the records a
// flusher file holds.
template <class Code>
void load_batch(Batch<Code>& b, Code code, const std::vector<const HierRecord*>& recs) {
	b.code = code;
	b.nodes.clear();
	b.chunks.clear();
	b.entries.clear();
	b.by_code.clear();
	for (uint32_t i = 0; i < recs.size(); i++) b.by_code.push_back({code_of<Code>(recs[i]->name.data(), recs[i]->name.size()), i});
	std::sort(b.by_code.begin(), b.by_code.end());
	size_t up = 0;  // the first node not before the parent
	for (uint32_t i = 0; i < b.by_code.size(); i++) {
		const HierRecord& r = *recs[b.by_code[i].second];
		BNode<Code> n;
		n.code = b.by_code[i].first;
		n.order = b.by_code[i].second;
		n.num_points = (int32_t)(uint32_t)r.num_points;
		n.byte_offset = (uint64_t)r.byte_offset;
		n.byte_size = (uint64_t)(int64_t)(int32_t)(uint32_t)r.byte_size;
		// chunk: "r" for names up to 5 chars, then the first 4k+1 chars
		const int len = (int)r.name.size(), key = len <= 5 ? 1 : kStep * ((len - 2) / 4) + 1;
		b.entries.push_back({n.code == code ? code : n.code >> (3 * (len - key)), i});
		if ((len - 1) % kStep == 0 && len > kStep + 1 && n.code != code) b.entries.push_back({n.code, i});
		while (up < i && b.nodes[up].code < n.code >> 3) up++;
		if (up < i && b.nodes[up].code == n.code >> 3) {
			if (n.order > b.nodes[up].order) b.nodes[up].type = T_NORMAL;
			b.nodes[up].child_mask |= (uint8_t)(1 << (int)(n.code & 7));
		}
		b.nodes.push_back(n);
	}
	std::sort(b.entries.begin(), b.entries.end());
	for (size_t i = 0; i < b.entries.size(); i++) {
		if (i == 0 || b.entries[i].first != b.entries[i - 1].first) b.chunks.push_back({b.entries[i].first, i, 0});
		b.chunks.back().count++;
	}
	for (const auto& c : b.chunks)
		if (auto* n = b.find(c.code)) n->type = T_PROXY;
}

template <class Code>
bool process_batch(Batch<Code>& b, std::string& err) {  // HierarchyBuilder.h:199-238
	for (const auto& c : b.chunks) {
		if (c.code == b.code) continue;
		if (!b.has_chunk(c.code >> (3 * kStep))) { err = "hierarchy: missing parent chunk"; return false; }
		auto* n = b.find(c.code);
		if (!n) { err = "hierarchy: missing proxy node"; return false; }
		n->proxy_offset = (uint64_t)kRecordBytes * c.first;
		n->proxy_size = (uint64_t)kRecordBytes * c.count;
	}
	return true;
}

template <class Code>
void serialize_batch(Batch<Code>& b, int64_t bytes_written, std::vector<uint8_t>& out, size_t at) {  // :240-282
	b.byte_size = (int64_t)(kRecordBytes * b.entries.size());
	if (out.size() < at + (size_t)b.byte_size) out.resize(at + (size_t)b.byte_size);
	uint8_t* p = out.data() + at;
	for (const auto& [chunk, i] : b.entries) {
		const auto& n = b.nodes[i];
		const bool is_proxy = n.type == T_PROXY && n.code != chunk;
		const uint8_t type = (n.type == T_PROXY && !is_proxy) ? (uint8_t)T_NORMAL : n.type;
		const uint64_t size = is_proxy ? n.proxy_size : n.byte_size;
		const uint64_t offset = is_proxy ? (uint64_t)bytes_written + n.proxy_offset : n.byte_offset;
		const uint32_t np = (uint32_t)n.num_points;
		p[0] = type;
		p[1] = n.child_mask;
		std::memcpy(p + 2, &np, 4);
		std::memcpy(p + 6, &offset, 8);
		std::memcpy(p + 14, &size, 8);
		p += kRecordBytes;
	}
}

template <class Code>
bool build(const std::vector<HierRecord>& completed, std::vector<uint8_t>& out, int64_t& first_chunk_size, std::string& err) {
	// flusher files: the root's nodes, and per node of depth 4 its subtree
	// (indexer.h:171-193); the builder visits files in file-name order, which
	// equals key order.
	std::vector<const HierRecord*> top, recs;
	std::vector<uint64_t> filed;  // file, record
	for (size_t i = 0; i < completed.size(); i++) {
		const std::string& name = completed[i].name;
		if (name.size() <= (size_t)kStep + 1) top.push_back(&completed[i]);
		if (name.size() > (size_t)kStep) filed.push_back(code_of<uint64_t>(name.data(), kStep + 1) << 32 | i);
	}
	std::sort(filed.begin(), filed.end());
	if (top.empty()) { err = "hierarchy: no root batch"; return false; }
	Batch<Code> root, b;
	load_batch(root, Code(1), top);
	out.assign(kRecordBytes * root.nodes.size(), 0);
	int64_t written = (int64_t)out.size();
	for (size_t i = 0; i < filed.size();) {
		const uint64_t file = filed[i] >> 32;
		recs.clear();
		for (; i < filed.size() && filed[i] >> 32 == file; i++) recs.push_back(&completed[filed[i] & 0xffffffffu]);
		load_batch(b, Code(file), recs);
		if (!process_batch(b, err)) return false;
		serialize_batch(b, written, out, out.size());
		auto* n = root.find(b.code);
		if (!n) { err = "hierarchy: batch root missing from root batch"; return false; }
		if (b.nodes.size() > 1) {
			n->type = T_PROXY;
			n->proxy_offset = (uint64_t)written;
			size_t own = 0;
			for (const auto& c : b.chunks)
				if (c.code == b.code) own = c.count;
			n->proxy_size = (uint64_t)kRecordBytes * own;
		} else {
			n->type = T_LEAF;
		}
		written += b.byte_size;
	}
	std::vector<uint8_t> head;
	serialize_batch(root, 0, head, 0);
	std::memcpy(out.data(), head.data(), head.size());
	first_chunk_size = root.byte_size;
	return true;
}

}  // namespace

bool build_hierarchy(const std::vector<HierRecord>& completed, std::vector<uint8_t>& out,
                     int64_t& first_chunk_size, std::string& err) {
	size_t longest = 0;
	for (const auto& r : completed) longest = std::max(longest, r.name.size());
	if (longest <= 22) return build<uint64_t>(completed, out, first_chunk_size, err);
	if (longest <= 43) return build<unsigned __int128>(completed, out, first_chunk_size, err);
	return build<TextCode>(completed, out, first_chunk_size, err);
}

std::string build_metadata(const std::string& name, const std::string& projection, int64_t points_total,
                           int64_t first_chunk_size, int64_t depth, const Setup& s,
                           const std::vector<AttrStats>& stats, double spacing) {
	auto num = [](double v) {
		std::ostringstream o;
		o << std::setprecision(std::numeric_limits<double>::max_digits10) << v;
		return o.str();
	};
	auto q = [](const std::string& v) { return "\"" + v + "\""; };
	auto tabs = [](int n) { return std::string(n, '\t'); };
	auto vec3 = [&](const Vec3d& v) { return "[" + num(v.x) + ", " + num(v.y) + ", " + num(v.z) + "]"; };
	auto list = [&](std::initializer_list<double> vs) {
		std::string o = "[";
		size_t i = 0;
		for (double v : vs) { o += num(v); if (++i < vs.size()) o += ", "; }
		return o + "]";
	};
	std::ostringstream m;
	const char* nl = "\n";
	m << "{" << nl;
	m << tabs(1) << q("version") << ": " << q("2.0") << "," << nl;
	m << tabs(1) << q("name") << ": " << q(name) << "," << nl;
	m << tabs(1) << q("description") << ": " << q("") << "," << nl;
	m << tabs(1) << q("points") << ": " << points_total << "," << nl;
	m << tabs(1) << q("projection") << ": " << q(projection) << "," << nl;
	m << tabs(1) << q("hierarchy") << ": {" << nl;
	m << tabs(2) << q("firstChunkSize") << ": " << first_chunk_size << ", " << nl;
	m << tabs(2) << q("stepSize") << ": " << kStep << ", " << nl;
	m << tabs(2) << q("depth") << ": " << depth << nl;
	m << tabs(1) << "}," << nl;
	m << tabs(1) << q("offset") << ": " << vec3(s.pos_offset) << "," << nl;
	m << tabs(1) << q("scale") << ": " << vec3(s.pos_scale) << "," << nl;
	m << tabs(1) << q("spacing") << ": " << num(spacing) << "," << nl;
	m << tabs(1) << q("boundingBox") << ": {" << nl;
	m << tabs(2) << q("min") << ": " << vec3(s.cube_min) << ", " << nl;
	m << tabs(2) << q("max") << ": " << vec3(s.root_max) << nl;
	m << tabs(1) << "}," << nl;
	m << tabs(1) << q("encoding") << ": " << q("DEFAULT") << "," << nl;
	m << tabs(1) << q("attributes") << ": [" << nl;
	for (size_t i = 0; i < s.attrs.size(); i++) {
		const AttrDesc& a = s.attrs[i];
		const AttrStats& st = stats[i];
		if (i == 0) m << tabs(2) << "{" << nl;
		m << tabs(3) << q("name") << ": " << q(a.name) << "," << nl;
		m << tabs(3) << q("description") << ": " << q(a.description) << "," << nl;
		m << tabs(3) << q("size") << ": " << a.size << "," << nl;
		m << tabs(3) << q("numElements") << ": " << a.numElements << "," << nl;
		m << tabs(3) << q("elementSize") << ": " << a.elementSize << "," << nl;
		m << tabs(3) << q("type") << ": " << q(attr_type_name(a.type)) << "," << nl;
		bool any = false;
		for (int64_t h : st.histogram) any = any || h != 0;
		if (a.size == 1 && any) {
			m << tabs(3) << q("histogram") << ": [";
			for (size_t k = 0; k < st.histogram.size(); k++) { m << st.histogram[k]; if (k + 1 < st.histogram.size()) m << ", "; }
			m << "], " << nl;
		}
		if (a.numElements == 1) {
			m << tabs(3) << q("min") << ": " << list({st.min.x}) << "," << nl;
			m << tabs(3) << q("max") << ": " << list({st.max.x}) << "," << nl;
			m << tabs(3) << q("scale") << ": " << list({a.scale.x}) << "," << nl;
			m << tabs(3) << q("offset") << ": " << list({a.offset.x}) << nl;
		} else if (a.numElements == 2) {
			m << tabs(3) << q("min") << ": " << list({st.min.x, st.min.y}) << "," << nl;
			m << tabs(3) << q("max") << ": " << list({st.max.x, st.max.y}) << "," << nl;
			m << tabs(3) << q("scale") << ": " << list({a.scale.x, a.scale.y}) << "," << nl;
			m << tabs(3) << q("offset") << ": " << list({a.offset.x, a.offset.y}) << nl;
		} else if (a.numElements == 3) {
			m << tabs(3) << q("min") << ": " << list({st.min.x, st.min.y, st.min.z}) << "," << nl;
			m << tabs(3) << q("max") << ": " << list({st.max.x, st.max.y, st.max.z}) << "," << nl;
			m << tabs(3) << q("scale") << ": " << list({a.scale.x, a.scale.y, a.scale.z}) << "," << nl;
			m << tabs(3) << q("offset") << ": " << list({a.offset.x, a.offset.y, a.offset.z}) << nl;
		}
		m << tabs(2) << (i + 1 < s.attrs.size() ? "},{" : "}") << nl;
	}
	m << tabs(1) << "]" << nl;
	m << "}" << nl;
	return m.str();
}

}  // namespace pcg
